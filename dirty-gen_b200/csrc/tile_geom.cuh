// The tiles of the grid engine's passes: their halos, how a team of threads
// walks a tile's cells, and the cells' places in the planes. Plain C++ apart
// from the function qualifier, so a host compiler takes it too.
#pragma once
#include <cstddef>

#ifdef __CUDACC__
#define SILT_TILE_FN __device__ __forceinline__
#else
#define SILT_TILE_FN inline
#endif

namespace silt {

constexpr int FT = 32;  // force tile edge

// A cell's place in a plane, in the type that the pass's planes need.
template <class Index>
SILT_TILE_FN Index plane_index(int gx, int gy, int res) {
    return (Index)gy * (Index)res + (Index)gx;
}

// Shared-memory layout of a force tile (the halo its widest stage reads, the
// planes' width and size, their number) and the type of its cells' places.
template <int HALO, int PLANES, class INDEX>
struct TileGeom {
    using Index = INDEX;
    static constexpr int H = HALO;
    static constexpr int W = FT + 2 * H;
    static constexpr int PLANE = W * W;
    static constexpr size_t BYTES = sizeof(float) * PLANES * PLANE;
};

// Every cell of the tile's region of radius (RX, RY): f(gx, gy, s, g) with s
// the shared-memory index and g the global one. The rectangle is walked as one
// flat range (a compile-time width), which keeps every lane busy; on edge
// tiles cells outside the grid are left out.
template <class TM, class G, bool EDGE, int RX, int RY, class F>
SILT_TILE_FN void region(const TM& T, int tx0, int ty0, int res, F f) {
    const int ox = tx0 - G::H, oy = ty0 - G::H;
    constexpr int RW = FT + 2 * RX, RH = FT + 2 * RY;
    for (int k = T.tid; k < RW * RH; k += TM::NT) {
        const int r = k / RW;
        const int gy = ty0 - RY + r, gx = tx0 - RX + (k - r * RW);
        if (EDGE && ((unsigned)gx >= (unsigned)res || (unsigned)gy >= (unsigned)res)) continue;
        f(gx, gy, (gy - oy) * G::W + (gx - ox), plane_index<typename G::Index>(gx, gy, res));
    }
}

// The snapshot form carries every stage of a cell through one tile:
// p (2) + gravity (1) + vorticity (2) + projection (4). Seven planes (70 KB):
// three CTAs share an SM. Their time is block barriers between ten short
// stages, so a third tile on the SM fills the other two's waits: k_force on a
// flooded 1000^2 grid 90 us with eight planes and two CTAs, 83 so.
// 32-bit places reach MAX_NEAR_RES cells a side: every sheet (MAX_SHEET_RES at
// most) and the free operator's grids up to there. The free operator takes any
// grid whose planes the device holds (70 000 cells a side and more), and above
// that size 64-bit places (FarSnap), which cost register pairs: on a flooded
// 1000^2 grid k_force takes 67.7 us with 32-bit places and 69.0 with 64-bit
// ones, and the batch's kernel 73 registers a thread for 64, one CTA per SM for
// two.
constexpr int MAX_NEAR_RES = 46340;
constexpr int MAX_SHEET_RES = 32768;
static_assert((long long)MAX_NEAR_RES * MAX_NEAR_RES <= 0x7fffffffLL && MAX_SHEET_RES <= MAX_NEAR_RES,
              "a near grid's places fit an int");
using Snap = TileGeom<9, 7, int>;
using FarSnap = TileGeom<9, 7, size_t>;
// The sweep form's stages meet in global memory, so no stage reaches further
// than the projection's 4 cells: 51 KB a tile instead of 80. Only sheets take it.
using Sweep = TileGeom<4, 8, int>;

}  // namespace silt
