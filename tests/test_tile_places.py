"""The places in a plane that the grid engine's tile walks hand out, on the
host: the walk of the device code, compiled as plain C++. The free operator
takes any grid whose planes the device holds (32 bytes a cell: some 73000
cells a side), so its places pass 2^31 at 46341 cells a side and 2^32 at
65536; a sheet has at most 32768."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dirty-gen_b200", "csrc")
PROGRAM = r"""
#include "tile_geom.cuh"
#include <cstdio>
#include <cstdlib>

struct One {
    static constexpr int NT = 1;
    int tid = 0;
};
static long long wrong = 0, seen = 0;

template <class G, bool EDGE>
void walk(int tx0, int ty0, int res) {
    silt::region<One, G, EDGE, G::H, G::H>(One(), tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
        const __int128 place = (__int128)gy * res + gx;
        wrong += gx < 0 || gy < 0 || gx >= res || gy >= res || (__int128)g != place ||
                 (__int128)silt::plane_index<size_t>(gx, gy, res) != place || s < 0 || s >= G::PLANE;
        ++seen;
    });
}

template <class G>
void walk_all(int res) {
    const int last = (res - 1) / silt::FT * silt::FT;
    const int tiles[] = {0, last / 2 / silt::FT * silt::FT, last - silt::FT, last};
    for (int ty0 : tiles)
        for (int tx0 : tiles) walk<G, true>(tx0, ty0, res);
    walk<G, false>(tiles[1], tiles[1], res);
    walk<G, false>(tiles[1], last - 2 * silt::FT, res);
}

int main(int, char** argv) {
    const int res = atoi(argv[1]);
    // As launch_force picks: 32-bit places up to MAX_NEAR_RES.
    if (res > silt::MAX_NEAR_RES)
        walk_all<silt::FarSnap>(res);
    else
        walk_all<silt::Snap>(res);
    if (res <= silt::MAX_SHEET_RES) walk_all<silt::Sweep>(res);
    printf("%lld %lld\n", seen, wrong);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("places")
    (d / "places.cpp").write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fwrapv", "-I", CSRC, str(d / "places.cpp"), "-o",
                           str(d / "places")])
    return str(d / "places")


@pytest.mark.parametrize("res", [513, 32767, 32768, 46340, 46341, 65535, 65536, 73000])
def test_places_of_a_tile_walk(program, res):
    seen, wrong = map(int, subprocess.check_output([program, str(res)]).split())
    assert seen > 0 and wrong == 0
