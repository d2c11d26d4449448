"""Performance cases of the sheet step: the work its users have it do.

A case is a dict of plain values. `prepare` makes what a program holds before
the call (sheets, batches, networks, torch tensors), `run` makes one pass
through the public entry points and returns the outputs, `work` states what a
pass cannot do without, and `exact` gives a training step's values in 64 bits.

The kinds of case:

* operator -- the free one-sheet operator on the caller's device arrays;
* window   -- one sheet handle, stepped frame by frame: tire pushes, step,
              publish of the film and flow maps into device memory;
* batch    -- many windows stepped together (scenes or vehicles), their maps
              and FP64 ledgers read every few steps;
* train    -- one optimiser step's gradients of the flux closure network.

Handles share one CUDA stream, as one program's frame loop does. A window is
an episode of one second: after 120 steps it is put back to its first state
(silt_sheet_copy_state) and its vehicle to its start.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "dirty-gen_b200"))

import silt_b200 as G  # noqa: E402
import silt_closure as C  # noqa: E402

DT = 1.0 / 120.0
CELL = 0.2
EPISODE = 120
WEIGHTS = os.path.join(ROOT, "dirty-gen_b200", "closure_weights.npz")
TRACK, WHEELBASE = 1.5, 2.4
CORNERS = ((-0.5, -0.5), (0.5, -0.5), (-0.5, 0.5), (0.5, 0.5))


def listed():
    return [
        # A small film on arrays the caller owns, one step: launch and wait latency.
        dict(name="operator_64", kind="operator", res=64, level=0.05),
        # A large flooded grid through the same operator, an odd number of tiles.
        dict(name="operator_1000", kind="operator", res=1000, level=0.15),
        # The library's default window (200 cells of 20 cm): a puddle and a slurry film in two ruts, nothing driving.
        dict(name="window_200", kind="window", res=200, tires=0, speed=0.0, fine=160, per_tire=False, puddles=1,
             level=-1.0, walls=False, river=False, spray=False, steps=1),
        # The same window with a vehicle: the default 160-cell patch under four tires, spray read every frame.
        dict(name="drive_200", kind="window", res=200, tires=4, speed=5.0, fine=160, per_tire=False, puddles=3,
             level=-1.0, walls=False, river=False, spray=True, steps=1),
        # A vehicle standing in a flooded window: its belly and wheels are walls, the load on them is read every frame.
        dict(name="walls_200", kind="window", res=200, tires=0, speed=0.0, fine=160, per_tire=False, puddles=2,
             level=0.02, walls=True, river=False, spray=False, steps=1),
        # Open water: a river through the window with inlet, outlet, paddle, bed friction, eddy viscosity and diffusion.
        dict(name="river_301", kind="window", res=301, tires=0, speed=0.0, fine=160, per_tire=False, puddles=0,
             level=0.3, walls=False, river=True, spray=False, steps=1),
        # A large terrain, mostly dry, with an inflow strip and a vehicle with one patch per tire.
        dict(name="grid_2048_drive", kind="window", res=2048, tires=4, speed=5.0, fine=64, per_tire=True, puddles=8,
             level=-1.0, walls=False, river=False, spray=False, steps=2),
        # A large terrain under a flood: half of its cells wet, odd side.
        dict(name="grid_1501_flood", kind="window", res=1501, tires=0, speed=0.0, fine=64, per_tire=True, puddles=20,
             level=0.0, walls=False, river=False, spray=False, steps=2),
        # A few small scenes stepped together, no vehicles.
        dict(name="batch_24", kind="batch", windows=24, lo=64, hi=160, tires=0, closure=False, steps=4),
        # Many scenes of uneven size, 0 to 4 tires each on nested 2 cm sheets.
        dict(name="batch_256_drive", kind="batch", windows=256, lo=64, hi=512, tires=4, closure=False, steps=4),
        # One vehicle per window with the learned closure in place of the nested sheets.
        dict(name="batch_128_closure", kind="batch", windows=128, lo=200, hi=200, tires=4, closure=True, steps=4),
        # Training of the closure: forward, loss and parameter gradients of one batch of crops.
        dict(name="train_256", kind="train", crops=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    kind = rng.choice(["operator", "operator", "window", "window", "window", "grid", "batch", "batch", "train"])
    if kind == "operator":
        return dict(kind="operator", res=_log(rng, 48, 1100), level=round(rng.uniform(0.0, 0.2), 3))
    if kind == "train":
        return dict(kind="train", crops=_log(rng, 16, 512))
    if kind == "batch":
        closure = rng.random() < 0.3
        n = _log(rng, 4, 96)
        if closure:
            return dict(kind="batch", windows=n, lo=200, hi=200, tires=4, closure=True, steps=4)
        lo = rng.randint(40, 120)
        return dict(kind="batch", windows=n, lo=lo, hi=lo + rng.randint(20, 300), tires=rng.choice([0, 4]),
                    closure=False, steps=rng.randint(2, 4))
    if kind == "grid":
        return dict(kind="window", res=_log(rng, 520, 2000), tires=rng.choice([0, 4]),
                    speed=round(rng.uniform(2.0, 10.0), 2), fine=64, per_tire=True, puddles=rng.randint(1, 30),
                    level=rng.choice([-1.0, -0.05, 0.0]), walls=False, river=False, spray=False,
                    steps=rng.randint(1, 3))
    sort = rng.choice(["still", "drive", "drive", "walls", "river"])
    return dict(kind="window", res=rng.randint(120, 360), tires=4 if sort == "drive" else 0,
                speed=round(rng.uniform(2.0, 10.0), 2), fine=rng.choice([160, 64]), per_tire=rng.random() < 0.5,
                puddles=0 if sort == "river" else rng.randint(1, 6),
                level={"walls": 0.02, "river": 0.3}.get(sort, -1.0), walls=sort == "walls", river=sort == "river",
                spray=sort == "drive", steps=1)


# ------------------------------------------------------------------ scenes

_shared = {}


def _stream():
    if "stream" not in _shared:
        _shared["stream"] = torch.cuda.Stream()
    return _shared["stream"]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _bed(res, gen):
    """Four octaves of value noise, 0.3 m."""
    x = (torch.arange(res, device="cuda", dtype=torch.float32) + 0.5) * CELL
    bed = torch.zeros((res, res), device="cuda")
    for o in range(4):
        p = x * (0.25 * 2.0 ** o)
        i = p.floor().long()
        f = p - i
        s = f * f * (3.0 - 2.0 * f)
        n = int(0.25 * 2.0 ** o * CELL * res) + 3
        lattice = torch.rand((n, n), device="cuda", generator=gen) * 2.0 - 1.0
        rows = lattice[:, i] + (lattice[:, i + 1] - lattice[:, i]) * s
        bed += 0.5 ** o * (rows[i] + (rows[i + 1] - rows[i]) * s[:, None])
    return bed * (0.3 / 1.875)


def _scene(res, puddles, level, gen, rng):
    """Noise bed with two ruts, slurry in the ruts, puddles of 0.05 to 0.2 m and 2 to 8 m radius, and water up to
    `level` everywhere when it is above -1."""
    bed = _bed(res, gen)
    half = 0.5 * res * CELL
    x = (torch.arange(res, device="cuda", dtype=torch.float32) + 0.5) * CELL - half
    ruts = torch.zeros(res, dtype=torch.bool, device="cuda")
    for c in (-0.75, 0.75):
        d = (x - c).abs()
        bed = bed - torch.where(d < 0.125, 0.075 * (1.0 + torch.cos(math.pi * d / 0.125)), 0.0)
        ruts |= d < 0.125
    water = torch.zeros_like(bed)
    for _ in range(puddles):
        depth, rad = rng.uniform(0.05, 0.2), rng.uniform(2.0, min(8.0, 0.4 * half))
        px, pz = (rng.uniform(-1.0, 1.0, 2) * (half - rad)).tolist()
        r2 = (x[None, :] - px) ** 2 + (x[:, None] - pz) ** 2
        water = torch.maximum(water, torch.where(r2 < rad * rad, depth * (1.0 - r2 / (rad * rad)), 0.0))
    if level > -1.0:
        water = torch.maximum(water, level - bed)
    slurry = torch.where(ruts[None, :] & (x.abs() < 20.0)[:, None], rng.uniform(0.02, 0.05), 0.0)
    return bed, water, slurry


def _host(t):
    return t.contiguous().cpu().numpy().ravel()


def _seed(sheet, bed, water, slurry):
    n = bed.numel()
    b = _host(bed)
    sheet.map_water_bed(b, _host(water))
    sheet.lay_slurry_mask(_host(slurry), G.CLAY, 0.55)
    sheet.read_substrate(b, np.full(n, 0.55, np.float32), np.full(n, G.CLAY, np.uint8))


def _channel(sheet, res, level, gen):
    """A river along x: a sand floor 8 m wide between banks, a current of 0.5 m/s."""
    z = ((torch.arange(res, device="cuda", dtype=torch.float32) + 0.5) - 0.5 * res) * CELL
    bed = ((z.abs() - 4.0).clamp_min(0.0) * 0.6)[:, None] + _bed(res, gen) * (0.05 / 0.3)
    water = (level - bed).clamp_min(0.0)
    n = res * res
    sand = np.full(n, G.SAND, np.uint8)
    sheet.read_substrate(_host(bed), np.full(n, 0.9, np.float32), sand)
    sheet.map_grain(sand)
    sheet.map_water_bed(_host(bed), _host(water))
    sheet.map_water_velocity(_host((water > 0.0).float() * 0.5), np.zeros(n, np.float32))


def _vehicle_bodies():
    belly = dict(x=0.1, z=0.4, yaw=0.35, half_length=1.15, half_width=0.70, bottom_y=-1.0, top_y=2.0, contact=0)
    return [belly] + [dict(x=0.1 + dx, z=0.4 + dz, yaw=0.35, half_length=0.25, half_width=0.15, bottom_y=-1.0,
                           top_y=2.0, contact=1, radius=0.38, width=0.2) for dx in (-0.75, 0.75) for dz in (-1.2, 1.2)]


# ------------------------------------------------------------------ prepare

def _prepare_operator(case, seed):
    res, gen = case["res"], _generator(seed)
    bed = _bed(res, gen)
    depth = torch.maximum(case["level"] - bed, torch.zeros((), device="cuda"))
    wet = (depth > 0.0).float()
    return dict(kind="operator", res=res, bed=bed, h=depth,
                u=wet * (torch.rand((res, res), device="cuda", generator=gen) - 0.5),
                v=wet * (torch.rand((res, res), device="cuda", generator=gen) - 0.5),
                nu=torch.full((res, res), 0.9, device="cuda"),
                gate=torch.ones((res, res), dtype=torch.uint8, device="cuda"),
                scratch=torch.zeros(G.lib().silt_step_sheet_scratch_bytes(res), dtype=torch.uint8, device="cuda"))


def _prepare_window(case, seed):
    res, gen, rng = case["res"], _generator(seed), np.random.default_rng(seed)

    def sheet():
        return G.Sheet(res=res, cell=CELL, fine_res=case["fine"], fine_cell=0.02,
                       layout=G.FINE_PER_TIRE if case["per_tire"] else G.FINE_MEAN_PATCH,
                       stream=_stream().cuda_stream)

    first, live = sheet(), sheet()
    if case["river"]:
        _channel(first, res, case["level"], gen)
        live.set_open_water(True, 0.35, 0.03, 0.05)
        live.set_surface_diffusion(0.024)
        live.set_river_reach(dict(along_z=False, positive=True, cross0=-4.0, cross1=4.0, rows=4, inlet_eta=0.3,
                                  outlet_eta=0.28, inlet_speed_m_s=0.5, inlet_turbidity=0.1))
        live.set_wave_maker(dict(x0=5.0, x1=7.0, z0=-3.0, z1=3.0, dir_x=1.0, dir_z=0.0, amplitude_m_s=0.3,
                                 period_s=0.5, ramp_s=0.2))
    else:
        _seed(first, *_scene(res, case["puddles"], case["level"], gen, rng))
    if case["walls"]:
        n = res * res
        first.map_water_velocity(np.full(n, 0.15, np.float32), np.full(n, 0.45, np.float32))
        live.set_hydro_solids(_vehicle_bodies())
    if res > 512:
        live.set_inflow(2, -10.0, 10.0, 0.5)
    live.copy_state_from(first)
    live.sync()
    n = res * res
    return dict(kind="window", sheet=live, first=first, t=0, yaw=float(rng.uniform(0.0, 2.0 * math.pi)),
                tires=case["tires"], speed=case["speed"], spray=case["spray"], walls=case["walls"],
                steps=case["steps"], particles=np.zeros((2048, 8)), film=torch.zeros(2 * n, device="cuda"),
                flow=torch.zeros(4 * n, device="cuda"))


def _prepare_batch(case, seed):
    gen, rng = _generator(seed), np.random.default_rng(seed)
    sheets, idx, recs, way = [], [], [], []
    net = None
    if case["closure"]:
        w = np.load(WEIGHTS)
        net = C.Closure(w["params"], w["norm"])
    sides = np.random.default_rng(case["windows"])  # the fleet's window sizes: the case's, not the seed's
    for k in range(case["windows"]):
        res = int(round(math.exp(sides.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        sh = G.Sheet(res=res, cell=CELL, fine_res=64, fine_cell=0.02, layout=G.FINE_PER_TIRE,
                     stream=_stream().cuda_stream, engine=G.ENGINE_GRID)
        _seed(sh, *_scene(res, int(rng.integers(1, 5)), -1.0, gen, rng))
        if net is not None:
            C.set_coupling(sh, C.COUPLING_CLOSURE, net, 1e30)
        tires = case["tires"] if case["closure"] else int(rng.integers(0, case["tires"] + 1))
        yaw, speed, start = rng.uniform(0.0, 2.0 * math.pi), rng.uniform(2.0, 10.0), rng.uniform(0.0, 1.0)
        for dx, dz in CORNERS[:tires]:
            idx.append(k)
            recs.append((math.sin(yaw), math.cos(yaw), 0.38, 0.2, speed, 0.3))
            way.append((dx * TRACK, dz * WHEELBASE, start, 0.5 * res * CELL))
        sheets.append(sh)
    rec = np.zeros(len(recs), G.TIRE_DTYPE)
    for q, name in enumerate(("forward_x", "forward_z", "radius", "width", "speed", "slip")):
        rec[name] = [r[q] for r in recs]
    cells = [s.res * s.res for s in sheets]
    torch.cuda.synchronize()
    return dict(kind="batch", batch=G.Batch(sheets), net=net, idx=np.asarray(idx, np.int32), rec=rec,
                way=np.asarray(way, np.float64).reshape(-1, 4), t=0, steps=case["steps"],
                at=np.concatenate([[0], np.cumsum(cells)]), film=torch.zeros(2 * sum(cells), device="cuda"),
                flow=torch.zeros(4 * sum(cells), device="cuda"))


def _train_inputs(crops, seed):
    """Crops as the training's normalised inputs and targets: standard normal features, depth and velocity changes in
    the scale of their deviations, about half of the cells wet."""
    norm = np.load(WEIGHTS)["norm"]
    gen = _generator(seed)
    n = C.CROP
    x = torch.zeros((crops, n, n, C.CIN), device="cuda")
    x[..., :C.IN_USED] = torch.randn((crops, n, n, C.IN_USED), device="cuda", generator=gen)
    scale = torch.tensor(norm[12:20], device="cuda")
    spread = torch.stack([scale[0], scale[2], scale[4], scale[5], scale[6], scale[7]])
    t = torch.randn((crops, n, n, 8), device="cuda", generator=gen)
    t[..., :6] *= spread
    t[..., 6:] = (t[..., 6:] > 0.0).float()
    return dict(x=x.to(torch.bfloat16), t=t, scale=scale, inv_var=1.0 / spread ** 2, lam=1e-3,
                params=C.init_params(seed))


def prepare(case, seed):
    torch.cuda.set_device(0)
    if case["kind"] == "operator":
        return _prepare_operator(case, seed)
    if case["kind"] == "window":
        return _prepare_window(case, seed)
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    s = _train_inputs(case["crops"], seed)
    s.update(kind="train", net=C.Net(s["params"]))
    return s


# ---------------------------------------------------------------------- run

def _run_operator(s):
    G.step_sheet_device(*(s[k].data_ptr() for k in ("h", "u", "v", "bed", "nu", "gate")), s["res"], CELL, DT, 0.08,
                        s["scratch"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return dict(h=s["h"], u=s["u"], v=s["v"])


def _run_window(s):
    sheet, out = s["sheet"], {}
    for _ in range(s["steps"]):
        if s["t"] == EPISODE:
            sheet.copy_state_from(s["first"])
            s["t"] = 0
        s["t"] += 1
        if s["tires"]:
            fx, fz = math.sin(s["yaw"]), math.cos(s["yaw"])
            d = s["speed"] * (s["t"] * DT - 0.5)
            for dx, dz in CORNERS[:s["tires"]]:
                a, b = dx * TRACK, d + dz * WHEELBASE
                sheet.push_tire(x=a * fz + b * fx, z=b * fz - a * fx, forward_x=fx, forward_z=fz, radius=0.38,
                                width=0.2, speed=s["speed"], slip=0.3)
        events = sheet.step(DT, want_spray=s["spray"])
    if s["spray"]:
        s["particles"][:] = 0.0  # a particle buffer of fixed size, as a renderer keeps
        if events:
            s["particles"][:len(events)] = events[:len(s["particles"])]
        out["spray"] = s["particles"]
    if s["walls"]:
        out["load"] = sheet.hydro_load()
    G.check(G.lib().silt_publish_film_flow_device(sheet.h, s["film"].data_ptr(), s["flow"].data_ptr()), "publish")
    out.update(film=s["film"], flow=s["flow"])
    return out


def _run_batch(s):
    b, rec = s["batch"], s["rec"]
    ahead, up, start, half = s["way"].T
    for _ in range(s["steps"]):
        s["t"] += 1
        if len(rec):
            d = ((start * half + rec["speed"] * (s["t"] * DT)) % half) - 0.5 * half + up
            rec["x"] = ahead * rec["forward_z"] + d * rec["forward_x"]
            rec["z"] = d * rec["forward_z"] - ahead * rec["forward_x"]
            b.push_tires(s["idx"], rec)
        b.step(DT)
    publish, film, flow = G.lib().silt_publish_film_flow_device, s["film"].data_ptr(), s["flow"].data_ptr()
    for sheet, at in zip(b.sheets, s["at"]):
        G.check(publish(sheet.h, film + 8 * int(at), flow + 16 * int(at)), "publish")
    return dict(ledgers=b.ledger_rows(), film=s["film"], flow=s["flow"])


def _run_train(s):
    a1, a2, y = s["net"].forward(s["x"])
    dy, loss = C.step_loss_grad(y, s["t"], s["scale"], s["inv_var"], s["lam"])
    return dict(loss=loss, y=y, grads=s["net"].grads(s["x"], a1, a2, dy))


def run(state):
    return {"operator": _run_operator, "window": _run_window, "batch": _run_batch,
            "train": _run_train}[state["kind"]](state)


# ----------------------------------------------------------- work and exact

def work(case):
    """Bytes and operations of one pass. A wet cell of a layer reads its depth, velocity and bed (the slurry its
    material too) and writes its depth and velocity every step: 28 and 33 bytes, about 250 operations. The maps of a
    publish read 8 planes and write 6 values per cell. Wet cells are counted from the scene's own sizes."""
    if case["kind"] == "operator":
        n = case["res"] ** 2
        return dict(bytes=33.0 * n, flops=250.0 * n)
    if case["kind"] == "train":
        pixels = case["crops"] * C.CROP * C.CROP
        macs = 9 * (C.CIN * C.HID + C.HID * C.HID + C.HID * C.COUT)
        # forward, input gradients of the two upper layers, weight gradients of all three
        flops = 2.0 * pixels * (2 * macs + 9 * (C.HID * C.HID + C.HID * C.COUT))
        return dict(bytes=pixels * (2.0 * C.CIN + 4.0 * 8 + 4.0 * C.COUT), flops=flops)

    def wet_cells(res, puddles, level):
        if level > 0.0:
            return 0.5 * res * res
        area = puddles * math.pi * 28.0 / CELL ** 2
        return min(res * res, area + (0.5 * res * res if level > -0.01 else 0.2 * res * res if level > -1.0 else 0.0))

    fine_cell = 28.0 + 33.0
    if case["kind"] == "window":
        res, steps = case["res"], case["steps"]
        fine = (case["tires"] if case["per_tire"] else min(case["tires"], 1)) * case["fine"] ** 2
        ruts = 3 * min(res, 200)
        step = wet_cells(res, case["puddles"], case["level"]) * 28.0 + ruts * 33.0 + fine * fine_cell
        return dict(bytes=steps * step + 56.0 * res * res, flops=250.0 * steps * step / 30.0)
    n = case["windows"]
    mean = (case["hi"] ** 2 - case["lo"] ** 2) / (2.0 * math.log(case["hi"] / case["lo"])) \
        if case["hi"] > case["lo"] else float(case["lo"] ** 2)
    step = n * (min(mean, 2.5 * math.pi * 28.0 / CELL ** 2) * 28.0 + 600 * 33.0)
    if case["tires"] and not case["closure"]:
        step += n * 0.5 * case["tires"] * 64 * 64 * fine_cell
    flops = 250.0 * step / 30.0
    if case["closure"]:
        flops += n * 2.0 * C.CROP ** 2 * 9 * (C.CIN * C.HID + C.HID * C.HID + C.HID * C.COUT)
    return dict(bytes=case["steps"] * step + 56.0 * n * mean, flops=case["steps"] * flops)


def _exact_train(case, seed):
    s = _train_inputs(case["crops"], seed)
    f64 = torch.float64
    p = torch.tensor(s["params"], dtype=f64, device="cuda").requires_grad_()
    P = C.split_params(p)

    def conv(x, name):
        w = P["W" + name]
        return torch.nn.functional.conv2d(x, w.view(3, 3, *w.shape[1:]).permute(3, 2, 0, 1), P["b" + name], padding=1)

    x = s["x"].to(f64).permute(0, 3, 1, 2)
    y = conv(conv(conv(x, "1").relu(), "2").relu(), "3").permute(0, 2, 3, 1)
    scale, inv_var, t = s["scale"].to(f64), s["inv_var"].to(f64), s["t"].to(f64)
    g = y[..., :8] * scale
    total = s["lam"] * (y[..., :8] ** 2).sum()
    for layer in range(2):
        gx = torch.nn.functional.pad(g[:, :, :-1, 2 * layer], (0, 1))
        gz = torch.nn.functional.pad(g[:, :-1, :, 2 * layer + 1], (0, 0, 0, 1))
        inflow = torch.nn.functional.pad(gx[:, :, :-1], (1, 0)) + torch.nn.functional.pad(gz[:, :-1, :], (0, 0, 1, 0))
        total = total + (inv_var[layer] * (inflow - gx - gz - t[..., layer]) ** 2).sum()
    for k in range(4):
        total = total + (inv_var[2 + k] * t[..., 6 + k // 2] * (g[..., 4 + k] - t[..., 2 + k]) ** 2).sum()
    loss = total / (case["crops"] * C.CROP ** 2)
    grads = torch.autograd.grad(loss, p)[0]
    G_ = C.split_params(grads)
    G_["W1"][:, C.IN_USED:, :] = 0.0
    G_["W3"][:, :, C.OUT_USED:] = 0.0
    G_["b3"][C.OUT_USED:] = 0.0
    return dict(loss=loss.detach().reshape(1), y=y.detach().contiguous(), grads=grads)


def exact(case, seed):
    """A training step in 64 bits from the FP32 parameters (the sheet step has no such value: its outputs are the
    32-bit arithmetic of the step itself, wet-dry decisions included)."""
    return _exact_train(case, seed) if case["kind"] == "train" else None
