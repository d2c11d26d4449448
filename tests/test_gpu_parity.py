"""Parity of the CUDA sheet step with the CPU oracle (the restated reference).

Tolerance (from the build's pass criteria): max |dh| <= 1e-4 m per layer after
100 steps. The window engine (windows up to 512 cells) steps box by box with
the reference's Gauss-Seidel confinement, and the grid engine (any size)
solves the same sweep as a fixed point. The water layer's damping factor
is computed on the host with the reference's libm; the slurry's powf and expf
are the double-precision functions rounded once, which agree with the C
library's on all but a few inputs in 10^4, so on these scenes both layers
match bit for bit. The grid engine's snapshot form (the reference's
free-operator confinement) stays selectable.
"""
import numpy as np
import pytest

import oracle as O
import silt_b200 as G
import silt_scenes as S

pytestmark = pytest.mark.gpu
DT = 1.0 / 120.0
TOL_H = 1.0e-4


def run_pair(steps, scene, check_every=0, engine=G.ENGINE_AUTO):
    ref = O.Core()
    dev = G.Sheet(engine=engine)
    S.seed_core(ref, scene)
    S.seed_core(dev, scene)
    worst = []
    for k in range(steps):
        ref.step(DT)
        dev.step(DT, want_spray=False)
        if check_every and (k + 1) % check_every == 0:
            worst.append(max(np.abs(ref.get("water") - dev.get("water")).max(),
                             np.abs(ref.get("slurry") - dev.get("slurry")).max()))
    return ref, dev, worst


def test_window200_100_steps_depth_parity():
    scene = S.window200()
    ref, dev, worst = run_pair(100, scene, check_every=10)
    dw = np.abs(ref.get("water") - dev.get("water")).max()
    ds = np.abs(ref.get("slurry") - dev.get("slurry")).max()
    print(f"max |dh| water {dw:.3e} slurry {ds:.3e} trace {worst}")
    assert dw <= TOL_H and ds <= TOL_H
    # Velocities follow the same physics; they are not the pass criterion.
    for name in ("uw", "vw", "us", "vs"):
        assert np.abs(ref.get(name) - dev.get(name)).max() < 5e-3, name
    assert dev.non_finite_count() == 0


def test_window200_water_is_bit_exact_after_100_steps():
    scene = S.window200()
    ref, dev, _ = run_pair(100, scene)
    a, b = ref.get("water"), dev.get("water")
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), float(np.abs(a - b).max())
    for name in ("uw", "vw"):
        a, b = ref.get(name), dev.get(name)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (name, float(np.abs(a - b).max()))


def test_window200_slurry_is_bit_exact_after_100_steps():
    scene = S.window200()
    ref, dev, _ = run_pair(100, scene)
    for name in ("slurry", "us", "vs"):
        a, b = ref.get(name), dev.get(name)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (name, float(np.abs(a - b).max()))


def test_grid_engine_window200_within_tolerance():
    scene = S.window200()
    ref, dev, _ = run_pair(100, scene, engine=G.ENGINE_GRID)
    for name in ("water", "slurry"):
        assert np.abs(ref.get(name) - dev.get(name)).max() <= TOL_H, name


def test_window200_ledger_matches_oracle_in_fp64():
    scene = S.window200()
    ref, dev, _ = run_pair(20, scene)
    lr = ref.ledger()
    ld = dev.ledger()
    assert abs(ld["water_m3"] - lr["water64"]) <= 1e-6 * lr["water64"]
    assert abs(ld["slurry_m3"] - lr["slurry64"]) <= 1e-6 * lr["slurry64"]


def test_grid_engine_water_is_bit_exact_on_a_jacobi_sized_box():
    """The grid engine's snapshot form (SILT_CONFINE_SNAPSHOT) on a pond wider
    than 48 x 32 cells, against the oracle's pair with the free operator's
    threading: the reference then confines from a snapshot too (force_gravity_par, src/fluid_core.rs:2229-2231) and the
    water damping factor is computed on the host with the reference's libm, so
    every operation is the reference's own IEEE sequence and the depths must
    match bit for bit."""
    scene = S.window200()
    ref = O.Core(inner_par=True)
    dev = G.Sheet(engine=G.ENGINE_GRID)
    dev.set_confinement(G.CONFINE_SNAPSHOT)
    for core in (ref, dev):
        core.map_water_bed(scene["bed"], np.zeros_like(scene["water"]))
        core.pour_water(-7.0, 7.0, -7.0, 7.0, 0.06)
        core.read_substrate(scene["bed"], scene["moisture"], scene["grain"])
    for k in range(5):
        ref.step(DT)
        dev.step(DT, want_spray=False)
        a, b = ref.get("water"), dev.get("water")
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (k, float(np.abs(a - b).max()))


def test_grid_engine_device_substep_count_is_exact():
    """A fast start (15 m/s water) needs two substeps, which the grid engine
    decides on the device without waiting: the host launches three from its
    speed bound and the water layer copies itself through the third. The slurry
    pool, slow, takes one substep and copies itself through two. With two
    substeps the cells the first one wets sit two cells inside the reference's
    work box, where the box edge reaches their pressure solve, so the grid
    engine (which has no box edge) differs there by float rounding (~3e-8 m);
    a wrong substep count would move the pond's rim by ~1e-3 m."""
    scene = S.window200()
    ref = O.Core()
    dev = G.Sheet(engine=G.ENGINE_GRID)
    dev.set_step_timing(True)
    n = scene["water"].size
    fast_u = np.full(n, 15.0, np.float32)
    fast_v = np.full(n, -2.0, np.float32)
    for core in (ref, dev):
        core.map_water_bed(scene["bed"], np.zeros_like(scene["water"]))
        core.pour_water(-7.0, 7.0, -7.0, 7.0, 0.06)
        core.pour_slurry(10.0, 13.0, 10.0, 13.0, 0.03, 0, 0.55)
        core.read_substrate(scene["bed"], scene["moisture"], scene["grain"])
        core.map_water_velocity(fast_u, fast_v)
    for k in range(4):
        ref.step(DT)
        dev.step(DT, want_spray=False)
        assert np.abs(ref.get("water") - dev.get("water")).max() <= 1.0e-6, k
        assert np.abs(ref.get("slurry") - dev.get("slurry")).max() <= TOL_H, k
    assert dev.step_parts()["device_counts"] >= 1
    ld, lr = dev.ledger(), ref.ledger()
    assert abs(ld["water_m3"] - lr["water64"]) <= 1e-6 * lr["water64"]
    assert abs(ld["slurry_m3"] - lr["slurry64"]) <= 1e-6 * lr["slurry64"]


@pytest.mark.parametrize("res,cell,dt,vort", [(48, 0.06, 0.05, 0.0), (96, 0.2, 0.05, 0.02), (160, 0.1, 0.02, 0.08)])
def test_free_step_sheet_matches_oracle(res, cell, dt, vort):
    import torch
    rng = np.random.default_rng(res)
    n = res * res
    jj, ii = np.mgrid[0:res, 0:res]
    bed = (-0.03 * jj + 0.02 * np.sin(ii * 0.3)).astype(np.float32).ravel()
    h = np.where(((ii - res / 2) ** 2 + (jj - res / 3) ** 2) < (res / 5) ** 2, 0.05, 0.0).astype(np.float32).ravel()
    h += np.where(rng.random(n) < 0.05, 0.01, 0.0).astype(np.float32)
    nu = np.full(n, O.dynamic_viscosity(0, 0.55), np.float32)
    nu[: n // 2] = 0.9
    gate = np.ones(n, np.uint8)
    u = np.zeros(n, np.float32)
    v = np.zeros(n, np.float32)
    ref = [h.copy(), u.copy(), v.copy()]
    sc = O.Scratch()
    dev = [torch.tensor(x, device="cuda") for x in (h, u, v, bed, nu)]
    dgate = torch.tensor(gate, device="cuda")
    scratch = torch.zeros(G.lib().silt_step_sheet_scratch_bytes(res) // 4 + 16, dtype=torch.float32, device="cuda")
    for _ in range(20):
        O.step_sheet(ref[0], ref[1], ref[2], bed, nu, gate, res, cell, dt, vort, scratch=sc)
        G.step_sheet_device(dev[0].data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), dev[3].data_ptr(),
                            dev[4].data_ptr(), dgate.data_ptr(), res, cell, dt, vort, scratch.data_ptr())
    torch.cuda.synchronize()
    dh = np.abs(dev[0].cpu().numpy() - ref[0]).max()
    assert dh <= TOL_H, dh


def free_operator(res, speed, depth):
    """A disc of water on a wavy slope for the operator on tiles: step(dt) on
    the device, its planes, and the host's copies."""
    import torch
    n = res * res
    jj, ii = np.mgrid[0:res, 0:res]
    bed = (-0.01 * jj + 0.02 * np.sin(ii * 0.3)).astype(np.float32).ravel()
    wet = (((ii - res / 2) ** 2 + (jj - res / 3) ** 2) < (res / 5) ** 2).ravel()
    h = np.where(wet, depth, 0.0).astype(np.float32)
    u = np.where(wet, speed, 0.0).astype(np.float32)
    v = np.where(wet, -0.25 * speed, 0.0).astype(np.float32)
    nu = np.full(n, 0.05, np.float32)
    dev = [torch.tensor(x, device="cuda") for x in (h, u, v, bed, nu)]
    gate = torch.ones(n, dtype=torch.uint8, device="cuda")
    scratch = torch.zeros(G.lib().silt_step_sheet_scratch_bytes(res) // 4 + 16, dtype=torch.float32, device="cuda")

    def step(dt):
        rc = G.step_sheet_device(*[x.data_ptr() for x in dev], gate.data_ptr(), res, 0.1, dt, 0.02, scratch.data_ptr())
        torch.cuda.synchronize()
        return rc

    return step, dev, (h, u, v, bed, nu)


@pytest.mark.parametrize("res,speed,depth", [(513, 0.0, 0.05), (520, 0.4, 3.0e-6)])
def test_free_step_sheet_above_512_matches_oracle(res, speed, depth):
    """Still water, and a film whose cells cross the dry cut."""
    step, dev, (h, u, v, bed, nu) = free_operator(res, speed, depth)
    gate, sc = np.ones(res * res, np.uint8), O.Scratch()
    for _ in range(3):
        O.step_sheet(h, u, v, bed, nu, gate, res, 0.1, 0.05, 0.02, scratch=sc)
        assert step(0.05) == 0
    dh = np.abs(dev[0].cpu().numpy() - h).max()
    assert dh <= TOL_H, dh


@pytest.mark.parametrize("pattern", ["cells", "rows", "halves"])
def test_free_step_sheet_above_512_with_mixed_viscosity_matches_oracle(pattern):
    """A thread keeps the damping factor of the viscosity it met last: planes
    that change it at every cell, every row, and once."""
    import torch
    res = 513
    step, dev, (h, u, v, bed, nu) = free_operator(res, 0.5, 0.05)
    jj, ii = np.mgrid[0:res, 0:res]
    key = {"cells": ii + jj, "rows": jj, "halves": (ii >= res // 2).astype(int)}[pattern]
    nu = np.array([0.05, 0.9, 30.0, 240.0], np.float32)[key % 4].ravel()
    dev[4].copy_(torch.tensor(nu))
    gate, sc = np.ones(res * res, np.uint8), O.Scratch()
    for _ in range(3):
        O.step_sheet(h, u, v, bed, nu, gate, res, 0.1, 0.05, 0.02, scratch=sc)
        assert step(0.05) == 0
    dh = np.abs(dev[0].cpu().numpy() - h).max()
    assert dh <= TOL_H, dh


@pytest.mark.parametrize("res,speed,count", [(513, 0.5, 1), (600, 2.6, 4), (515, 5.0, 7)])
def test_free_step_sheet_above_512_counts_its_substeps(res, speed, count):
    """The first substep's dt is the device's own count of the speed, the
    others' is the host's: one call gives the same bits as `count` calls with
    a `count`-th of its dt, each of which takes one substep."""
    import torch
    dt = np.float32(0.05)
    assert int(np.ceil(dt * np.float32(np.hypot(speed, 0.25 * speed)) / np.float32(0.042))) == count
    whole, a, _ = free_operator(res, speed, 0.05)
    parts, b, _ = free_operator(res, speed, 0.05)
    assert whole(float(dt)) == 0
    for _ in range(count):
        assert parts(float(dt / np.float32(count))) == 0
    assert all(torch.equal(x, y) for x, y in zip(a[:3], b[:3]))


def test_free_step_sheet_above_512_leaves_a_dry_sheet_alone():
    """At or below 1e-6 of summed depth the operator is a no-op: its return
    value says so and no plane changes, on a fresh sheet and after a wet one."""
    import torch
    res = 520
    scratch = torch.zeros(G.lib().silt_step_sheet_scratch_bytes(res) // 4 + 16, dtype=torch.float32, device="cuda")
    z = torch.zeros(res * res, device="cuda")
    gate = torch.ones(res * res, dtype=torch.uint8, device="cuda")
    nu = torch.full_like(z, 0.05)

    def step(h, u, v):
        return G.lib().silt_step_sheet(h.data_ptr(), u.data_ptr(), v.data_ptr(), z.data_ptr(), nu.data_ptr(),
                                       gate.data_ptr(), res, 0.1, 0.05, 0.0, scratch.data_ptr(), None)

    for k in range(3):
        dry = [z.clone(), torch.full_like(z, 0.3), torch.full_like(z, -0.2)]
        dry[0][:5] = 1.0e-7
        was = [x.clone() for x in dry]
        torch.cuda.synchronize()
        assert step(*dry) == 1  # SILT_OK_NOOP
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(dry, was)), k
        wet = [torch.full_like(z, 0.05), z.clone(), z.clone()]
        torch.cuda.synchronize()
        assert step(*wet) == 0


@pytest.mark.parametrize("engine", [G.ENGINE_WINDOW, G.ENGINE_GRID])
def test_open_water_and_surface_diffusion_match_oracle(engine):
    """Open-water mode (mobility 1, Manning 0.035, eddy 0.06 m^2/s, the ford
    reach's settings, src/ford.rs:338-343) and surface diffusion 0.024 m^2/s on
    a basin with a 0.75 m/s current: depth within the 1e-4 m criterion after
    60 steps, velocity within 1e-3 m/s (Manning's powf and hypotf may differ
    from glibc's by an ulp), and the FP64 books closed. The grid engine runs
    against the oracle's snapshot-confinement form."""
    sc = S.basin()
    dev = G.Sheet(res=sc["res"], cell=sc["cell"], engine=engine)
    # The grid engine confines from a snapshot: the oracle's pair with the
    # free operator's form does too on boxes of at least 48 x 32 (the basin's).
    ref = O.Core(threads=1)
    for c in (dev, ref):
        S.seed_basin(c, sc)
        c.set_open_water(True, 1.0, 0.035, 0.06)
        c.set_surface_diffusion(0.024)
    v0 = dev.ledger()
    for _ in range(60):
        dev.step(DT, want_spray=False)
        ref.step(DT)
    for name in ("water", "slurry"):
        d = float(np.abs(dev.get(name) - ref.get(name)).max())
        assert d <= 1e-4, (name, d)
    du = float(np.abs(dev.get("uw") - ref.get("uw")).max())
    assert du <= 1e-3, du
    led = dev.ledger()
    gap = abs(led["total_m3"] + led["cut_m3"] - v0["total_m3"] - v0["cut_m3"]) / v0["total_m3"]
    assert gap < 1e-6, gap
    # The current slowed under the bed friction, as on the oracle.
    assert float(np.abs(dev.get("uw")).max()) < 0.9


def test_sample_reads_the_coarse_cell():
    sc = S.basin()
    dev = G.Sheet(res=sc["res"], cell=sc["cell"])
    ref = O.Core(threads=1)
    for c in (dev, ref):
        S.seed_basin(c, sc)
    for _ in range(5):
        dev.step(DT, want_spray=False)
        ref.step(DT)
    for x, z in ((0.3, -1.1), (2.0, 2.5), (-5.9, 0.1)):
        g = dev.sample(x, z)
        r = ref.sample(x, z)
        assert abs(g["water_m"] - r["water_m"]) <= 1e-4 and abs(g["bed_m"] - r["bed_m"]) == 0.0
        assert abs(g["moisture"] - r["moisture"]) == 0.0
    assert dev.sample(1000.0, 0.0) is None


def _pair_planes(ref, dev, names=("water", "slurry", "uw", "vw", "us", "vs", "moisture")):
    return {k: float(np.abs(ref.get(k) - dev.get(k)).max()) for k in names}


def test_recenter_scroll_and_jump_match_oracle():
    """Window moves between steps: a whole-cell scroll, a jump with no overlap
    (every cell parked), the way back; depths within the 1e-4 m criterion of
    the oracle throughout and the FP64 books (frozen included) equal."""
    scene = S.window200()
    ref, dev = O.Core(threads=1), G.Sheet()
    for c in (ref, dev):
        S.seed_core(c, scene)
    v0 = dev.ledger()["total_m3"]
    plan = [(3, None), (10, (3.1, -2.2)), (2, (100.0, 37.0)), (10, (0.0, 0.0)), (5, (-1.4, 0.8))]
    for steps, move in plan:
        if move is not None:
            ref.recenter(*move)
            dev.recenter(*move)
            assert dev.origin() == ref.origin()
            d = _pair_planes(ref, dev)
            assert d["water"] <= 1e-4 and d["slurry"] <= 1e-4 and d["moisture"] == 0.0, d
        for _ in range(steps):
            ref.step(DT)
            dev.step(DT, want_spray=False)
        d = _pair_planes(ref, dev)
        assert d["water"] <= 1e-4 and d["slurry"] <= 1e-4, (move, d)
        lr, ld = ref.ledger(), dev.ledger()
        assert abs(ld["frozen_water_m3"] - lr["frozen_water_m3"]) <= 1e-6 + 1e-5 * lr["frozen_water_m3"]
        assert abs(ld["frozen_slurry_m3"] - lr["frozen_slurry_m3"]) <= 1e-6 + 1e-5 * lr["frozen_slurry_m3"]
    led = dev.ledger()
    assert abs(led["total_m3"] + led["cut_m3"] - v0) <= 1e-6 * v0


@pytest.mark.parametrize("engine", [G.ENGINE_WINDOW, G.ENGINE_GRID])
def test_patch_water_outside_the_window_is_parked_and_restored(engine):
    """Tires at the window's west edge: the per-tire patches reach past it, so
    their off-window water is parked under its coarse world cell
    (src/fluid_core.rs:8484-8487); moving the window west restores it. The
    near field is off on both sides (the device releases tiles that leave the
    window; the reference keeps them by world cell)."""
    scene = S.grid(res=128, seed=0xABC, puddles=6)
    ox = S.snap_origin(0.0, 0.0, 128 * 0.2, 0.2)[0]
    ref = O.Core(res=128, fine_res=64, layout=1, threads=1)
    dev = G.Sheet(res=128, fine_res=64, layout=G.FINE_PER_TIRE, engine=engine)
    for c in (ref, dev):
        S.seed_core(c, scene)
        c.set_near_field(False)
        c.pour_water(ox - 1.0, ox + 2.0, -3.0, 3.0, 0.05)
    v0 = dev.ledger()["total_m3"]
    for k in range(20):
        # The west tires 0.2 m inside the window's edge: their patches reach 0.44 m past it.
        for t in S.tires_at(k * DT, speed=3.0, center=(ox + 0.95, 0.0), z0=-1.2):
            ref.push_tire(**t)
            dev.push_tire(**t)
        ref.step(DT)
        dev.step(DT, want_spray=False)
    lr, ld = ref.ledger(), dev.ledger()
    assert lr["frozen_water_m3"] > 0.0
    assert abs(ld["frozen_water_m3"] - lr["frozen_water_m3"]) <= 1e-3 * lr["frozen_water_m3"]
    for c in (ref, dev):
        c.recenter(-3.0, 0.0)
    lr, ld = ref.ledger(), dev.ledger()
    assert abs(ld["frozen_water_m3"] - lr["frozen_water_m3"]) <= 1e-6 + 1e-3 * lr["frozen_water_m3"]
    d = _pair_planes(ref, dev, ("water", "slurry"))
    assert d["water"] <= 1e-4 and d["slurry"] <= 1e-4, d
    led = dev.ledger()
    assert abs(led["total_m3"] + led["cut_m3"] - led["opened_m3"] - v0) <= 1e-5 * v0


@pytest.mark.parametrize("engine", [G.ENGINE_WINDOW, G.ENGINE_GRID])
def test_river_reach_and_wave_maker_match_oracle(engine):
    """A river channel through the window with the reach's inlet and outlet
    (src/fluid_core.rs:7638-7745), a paddle strip (:7420-7480) and open water:
    depth within 1e-4 m of the oracle after 60 steps, the reach bank within
    f32 rounding of the oracle's, and the FP64 books closed (the bank is on
    the ledger)."""
    sc = S.channel()
    reach = dict(along_z=False, positive=True, cross0=-4.0, cross1=4.0, rows=4, inlet_eta=0.3, outlet_eta=0.28,
                 inlet_speed_m_s=0.75)
    wave = dict(x0=5.0, x1=7.0, z0=-3.0, z1=3.0, dir_x=1.0, dir_z=0.0, amplitude_m_s=0.3, period_s=0.5, ramp_s=0.2)
    dev = G.Sheet(res=sc["res"], cell=sc["cell"], engine=engine)
    ref = O.Core(threads=1)
    for c in (dev, ref):
        S.seed_basin(c, sc)
        c.set_open_water(True, 1.0, 0.035, 0.06)
        c.set_river_reach(reach)
        c.set_wave_maker(wave)
    v0 = dev.ledger()
    for _ in range(60):
        dev.step(DT, want_spray=False)
        ref.step(DT)
    d = _pair_planes(ref, dev, ("water", "uw", "vw"))
    assert d["water"] <= 1e-4 and d["uw"] <= 1e-3, d
    led = dev.ledger()
    assert led["reach_m3"] > 0.0
    assert abs(led["reach_m3"] - ref.reach_bank_m3()) <= 1e-4 * led["reach_m3"] + 1e-6
    gap = abs(led["total_m3"] + led["cut_m3"] - v0["total_m3"] - v0["cut_m3"]) / v0["total_m3"]
    assert gap < 1e-6, gap


@pytest.mark.parametrize("pattern", ["comb", "spiral", "checker", "bars", "dots", "one", "edges"])
@pytest.mark.parametrize("res", [33, 64, 200, 257])
def test_work_boxes_of_awkward_wet_shapes_match_oracle(pattern, res):
    """Wet shapes that stress the work boxes: a comb and a spiral (one body of
    many runs, joined late), a checkerboard (more runs than the labelling
    tables hold on the larger windows, more bodies than boxes), bars and dots
    (two to many bodies, merged or not), one cell, and the window's edges.
    Depths and velocities bit for bit with the oracle after 3 steps: a wrong
    box, or one in another order, steps other cells."""
    j, i = np.mgrid[0:res, 0:res]
    m = np.zeros((res, res), bool)
    if pattern == "comb":
        m = (i % 4 == 1) | (j == res - 2)
    elif pattern == "spiral":
        d = np.minimum(np.minimum(i, j), np.minimum(res - 1 - i, res - 1 - j))
        m = (d % 4 == 0) & ~((i == d + 1) & (j == d + 2))
        m |= (d % 4 != 0) & (i == d) & (j == d + 2) & (d < res // 2 - 3)
    elif pattern == "checker":
        m = (i + j) % 2 == 0
    elif pattern == "bars":
        m = (j == 5) | (j == res - 7)
    elif pattern == "dots":
        m = (i % 17 == 3) & (j % 19 == 5)
    elif pattern == "one":
        m[res // 2, res // 3] = True
    else:
        m = (i == 0) | (j == 0) | (i == res - 1) | (j == res - 1)
    rng = np.random.default_rng(res)
    bed = rng.uniform(-0.05, 0.05, (res, res)).astype(np.float32)
    water = np.where(m, rng.uniform(0.01, 0.1, (res, res)), 0.0).astype(np.float32)
    ref, dev = O.Core(res=res), G.Sheet(res=res, engine=G.ENGINE_WINDOW)
    for c in (ref, dev):
        c.map_water_bed(bed.ravel(), water.ravel())
    for _ in range(3):
        ref.step(1.0 / 120.0)
        dev.step(1.0 / 120.0, want_spray=False)
    for name in ("water", "uw", "vw"):
        a, b = ref.get(name), dev.get(name)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (name, float(np.abs(a - b).max()))


@pytest.mark.parametrize("res,level", [(513, 0.0), (700, 1.0e-12)])
def test_a_dry_call_above_512_steps_no_tile(res, level):
    """A call that finds nothing wet leaves the caller's planes and the
    scratch planes, which only a substep writes, as they are; water on the
    same arrays afterwards steps as on fresh ones."""
    import torch

    def arrays():
        h = torch.full((res, res), level, device="cuda")
        u = torch.full((res, res), 0.3, device="cuda")
        v = torch.full((res, res), -0.2, device="cuda")
        bed = torch.zeros((res, res), device="cuda")
        nu = torch.full((res, res), 0.9, device="cuda")
        scratch = torch.zeros(G.lib().silt_step_sheet_scratch_bytes(res) // 4 + 16, device="cuda")
        return h, u, v, bed, nu, scratch

    def step(a):
        rc = G.lib().silt_step_sheet(*(x.data_ptr() for x in a[:5]), None, res, 0.2, 1.0 / 120.0, 0.08,
                                     a[5].data_ptr(), None)
        torch.cuda.synchronize()
        return rc

    a, b = arrays(), arrays()
    planes = a[5][64:64 + 3 * res * res]  # u, v and h of a substep, behind 256 bytes
    planes.fill_(7.0)
    for _ in range(3):
        assert step(a) == G.SILT_OK_NOOP
    for x, y in zip(a[:5], b[:5]):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32))
    assert bool((planes == 7.0).all())
    for q in (a, b):
        q[0][40:300, 100:333] = 0.05
        assert step(q) == 0
    for x, y in zip(a[:3], b[:3]):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32))
