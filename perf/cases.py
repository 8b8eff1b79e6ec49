"""Performance cases: the calls that programs built on this library make,
over the sizes they make them at.

Five kinds of pass, each through public entry points:

flow      a window of timesteps of one solver (a closed box, or a stream past
          a sphere or a blunt capsule), then the readback that ends such a
          window: the sampled per-cell fields and totals, or the particles
ensemble  a window of timesteps of independent sphere flows advanced together
          (DSMCBatch), then every member's sampled fields
stages    one timestep stage by stage on the caller's device tensors
          (cudadsmc_b200.stages)
fill      a particle population seeded from per-cell fields (the warm start)
          and its first few timesteps, then their sampled fields
mlp       the warm-start network: a prediction, or a training step (loss,
          gradients, Adam)

Argon throughout, as in bench.py.  A case is a dict of plain values;
`prepare` holds what a program has before the call.
"""
import math

import numpy as np
import torch

import cudadsmc_b200 as cb
from cudadsmc_b200 import stages
from cudadsmc_b200.surrogate import WarmStartMLP

KB = 1.380649e-23
ARGON = dict(gas_mass=6.63e-26, gas_diam=4.17e-10, gas_tref=273.0)
T_INF = 200.0
SOUND = math.sqrt(5.0 / 3.0 * KB * T_INF / ARGON["gas_mass"])
OUTFLOW = {"-x": "inflow", "+x": "outflow", "-y": "outflow", "+y": "outflow", "-z": "outflow",
           "+z": "outflow"}


def listed():
    return [
        # A small box stepped by direct launches, the particles read after
        # every few steps: an interactive run, in the reference's own mode
        # (HybridTaus streams, hard spheres).  Launch latency decides.
        dict(name="box_8cube_direct", kind="flow", body="none", nx=8, ny=8, nz=8, ppc=16, rng="taus",
             omega=0.5, periodic="n", api="direct", steps=10, sample_every=0, settle=20, back="state"),
        # The relaxation of a two-temperature gas in a closed box of 16^3
        # cells, 98,304 particles (bench.py's box100k), from the step graph.
        dict(name="box_16cube", kind="flow", body="none", nx=16, ny=16, nz=16, ppc=24, rng="philox",
             omega=0.81, periodic="n", api="graph", steps=100, sample_every=100, settle=20,
             back="state"),
        # The largest grid of the reference's own random streams, 524,288
        # particles, in its mode (the second case of the speed test against
        # the reference's kernels).
        dict(name="box_64x32x32_taus", kind="flow", body="none", nx=64, ny=32, nz=32, ppc=8,
             rng="taus", omega=0.5, periodic="n", api="graph", steps=100, sample_every=100,
             settle=20, back="fields"),
        # Stream past a diffuse sphere, 500k particles, sampled every other
        # step as the warm-start study does.
        dict(name="sphere_500k", kind="flow", body="sphere", tris=3, nx=64, ny=32, nz=32, ppc=7.63,
             mach=5.7, wall=300.0, rng="philox", omega=0.81, api="graph", steps=100, sample_every=2,
             settle=200, back="fields"),
        # bench.py's default workload: Mach 7 past a capsule of 20k
        # triangles, 4.26M particles at the fill.
        dict(name="capsule_4m", kind="flow", body="capsule", tris=20000, nx=128, ny=64, nz=64,
             ppc=8.4, mach=7.0, wall=500.0, rng="philox", omega=0.81, api="graph", steps=100,
             sample_every=100, settle=300, back="fields"),
        # The ensemble that generates training fields: uneven sphere flows in
        # one launch sequence per step.
        dict(name="ensemble_32", kind="ensemble", members=32, particles_lo=50000,
             particles_hi=2000000, steps=50, sample_every=2, settle=50),
        # Stage by stage on caller's tensors, at the box's size with the
        # allocation-free sort, and at the capsule's size with a workspace.
        dict(name="stages_98k", kind="stages", nx=16, ny=16, nz=16, n=98304, sort="static",
             rng="taus", omega=0.5),
        dict(name="stages_4m", kind="stages", nx=128, ny=64, nz=64, n=4194304, sort="workspace",
             rng="philox", omega=0.81),
        # The warm start of the 64x32x32 sphere flow: the fill from a
        # prediction and the first timesteps after it.
        dict(name="fill_64x32x32", kind="fill", nx=64, ny=32, nz=32, ppc=7.6, weight=0.7, radius=0.1,
             steps=10),
        # Fields predicted for one condition, and for the 100 held-out ones.
        dict(name="predict_1", kind="mlp", call="predict", batch=1, cells=65536, hidden=512, depth=4,
             modes=256),
        dict(name="predict_100", kind="mlp", call="predict", batch=100, cells=65536, hidden=512,
             depth=4, modes=256),
        # One late training step (the schedule's final rate) on a batch of
        # half of the study's 2000 conditions.
        dict(name="train_1024", kind="mlp", call="train", batch=1024, cells=65536, hidden=512, depth=4,
             modes=256),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["flow", "flow", "flow", "flow", "ensemble", "stages", "stages", "fill", "mlp",
                       "mlp"])
    if kind == "flow":
        body = rng.choice(["none", "sphere", "capsule"])
        if body == "none":
            # boxes of 4k to 1.5M particles
            nx, ny, nz = (int(_log(rng, 7, 61)) for _ in range(3))
            ppc = rng.randint(6, 30)
            while nx * ny * nz * ppc > 1500000:
                nx, ny, nz = nx * 3 // 4, ny * 3 // 4, nz * 3 // 4
            mode = rng.choice(["taus", "philox"])
            api = rng.choice(["graph", "graph", "direct"])
            steps = rng.choice([10, 20, 50])
            return dict(kind=kind, body=body, nx=nx, ny=ny, nz=nz, ppc=ppc, rng=mode,
                        omega=0.5 if mode == "taus" else rng.choice([0.5, 0.74, 0.81]),
                        periodic=rng.choice(["n", "x", "y", "z"]), api=api, steps=steps,
                        sample_every=rng.choice([0, 1, 10]) if api == "direct" else rng.choice([2, 10]),
                        settle=20, back="state" if nx * ny * nz * ppc < 200000 else "fields")
        # streams past a body, 60k to 4.2M particles
        f = _log(rng, 0.45, 1.9)
        nx, ny, nz = int(64 * f), int(32 * f * rng.uniform(0.9, 1.1)), int(32 * f * rng.uniform(0.9, 1.1))
        every = rng.choice([1, 2, 10, 50])
        return dict(kind=kind, body=body, tris=rng.randint(2, 4) if body == "sphere" else
                    int(_log(rng, 1500, 20000)), nx=nx, ny=ny, nz=nz, ppc=round(rng.uniform(5, 9), 2),
                    mach=round(rng.uniform(2, 10), 2), wall=round(rng.uniform(200, 600), 1), rng="philox",
                    omega=0.81, api=rng.choice(["graph", "graph", "direct"]), steps=50,
                    sample_every=every, settle=100, back="fields")
    if kind == "ensemble":
        return dict(kind=kind, members=int(_log(rng, 3, 24)), particles_lo=50000,
                    particles_hi=int(_log(rng, 2e5, 1.5e6)), steps=20,
                    sample_every=rng.choice([2, 10, 20]), settle=20)
    if kind == "stages":
        n = int(_log(rng, 20000, 4000000))
        small = n <= stages.SORT_STATIC_MAX_N
        cells = max(64, n // rng.randint(6, 24))
        nx = max(4, int((2 * cells) ** (1 / 3)))
        ny = max(4, int(nx * rng.uniform(0.4, 1.0)))
        nz = max(4, min(cells // (nx * ny), 120000 // (nx * ny) if small else 1 << 30))
        mode = rng.choice(["taus", "philox"])
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, n=n,
                    sort=rng.choice(["static", "workspace"]) if small else "workspace", rng=mode,
                    omega=0.5 if mode == "taus" else 0.81)
    if kind == "fill":
        f = _log(rng, 0.4, 1.3)
        return dict(kind=kind, nx=int(64 * f), ny=int(32 * f), nz=int(32 * f * rng.uniform(0.8, 1.0)),
                    ppc=round(rng.uniform(4, 10), 2), weight=rng.choice([0.0, round(rng.uniform(0.1, 1), 2)]),
                    radius=round(rng.uniform(0.05, 0.15), 3), steps=10)
    net = dict(hidden=16 * rng.randint(4, 32), depth=rng.randint(2, 4))
    if rng.random() < 0.6:
        return dict(kind=kind, call="predict", batch=int(_log(rng, 1, 140)), cells=8 * int(_log(rng, 500, 8000)),
                    modes=16 * rng.randint(2, 16), **net)
    # training on a coarse grid's fields
    return dict(kind=kind, call="train", batch=8 * int(_log(rng, 1, 128)), cells=8 * int(_log(rng, 40, 300)),
                modes=16 * rng.randint(2, 16), **net)


# ------------------------------------------------------------------ solvers --

def _flow_solver(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["body"] == "none":
        dom = (1.0, 1.0, 1.0) if case["rng"] == "philox" else (1.2, 0.6, 0.6)
        s = dict(init_kind="bimodal", init_temp2=600.0, part_per_cell=case["ppc"],
                 periodic=case["periodic"], dt=1e-5)
    else:
        dom = (1.2, 0.6, 0.6)
        u = case["mach"] * SOUND
        cmp = math.sqrt(2 * KB * T_INF / ARGON["gas_mass"])
        s = dict(init_kind="maxwell", ntc_local=1, stream_vel=(u, 0.0, 0.0), wall_diffuse=1,
                 wall_temp=case["wall"], geom_nearest=1, face_kind=OUTFLOW, capacity_factor=1.6,
                 dt=min(dom[0] / nx, dom[1] / ny, dom[2] / nz) / (u + 3 * cmp))
    cell_v = dom[0] * dom[1] * dom[2] / (nx * ny * nz)
    s.update(grid_min=(0, 0, 0), grid_max=dom, grid_dim=(nx, ny, nz), density=1e20, temp=T_INF,
             fnum=1e20 * cell_v / case["ppc"], rng=case["rng"], gas_omega=case["omega"],
             sample_every=case["sample_every"], seed=seed + 1, **ARGON)
    sol = cb.DSMCSolver().Init(cb.settings_t().set(**s))
    if case["body"] == "sphere":
        sol.SetModel(*cb.mesh_icosphere(case["tris"], 0.1, (0.4, 0.3, 0.3)), (16, 16, 16))
    elif case["body"] == "capsule":
        sol.SetModel(*cb.mesh_capsule(0.15, 20.0, 0.26, (0.5, 0.3, 0.3), case["tris"], 7), (48, 64, 64))
    return sol, s["dt"]


def _pinned_fields(*shape):
    return torch.zeros(shape, dtype=torch.float64).pin_memory().numpy()


def _prepare_flow(case, seed):
    sol, dt = _flow_solver(case, seed)
    sol.InitSystemState()
    sol.StepGraph(dt, case["settle"])
    sol.Sync()
    out = None if case["back"] == "state" else _pinned_fields(case["nx"] * case["ny"] * case["nz"], 5)
    return dict(sol=sol, dt=dt, out=out)


def _run_flow(case, s):
    sol = s["sol"]
    step = sol.StepGraph if case["api"] == "graph" else sol.RunSimulationStep
    if case["back"] == "state":
        step(s["dt"], case["steps"])
        return sol.DownloadState(soa=True), sol.Totals()
    sol.ResetSamples()
    step(s["dt"], case["steps"])
    return sol.Fields(s["out"]), sol.Totals()


def _prepare_ensemble(case, seed):
    # bench.py's batch64 conditions: particles log-uniform, Mach 2-10, Knudsen
    # number (on the sphere's diameter) log-uniform in 0.01-1, T_wall/T_inf 1-3
    r = np.random.default_rng(seed)
    dom, dim, radius = (1.2, 0.6, 0.6), (64, 32, 32), 0.1
    cells = dim[0] * dim[1] * dim[2]
    cell = [dom[k] / dim[k] for k in range(3)]
    m, d = ARGON["gas_mass"], ARGON["gas_diam"]
    cmp = math.sqrt(2 * KB * T_INF / m)
    cbar = math.sqrt(8 * KB * T_INF / (math.pi * m))
    mesh = cb.mesh_icosphere(3, radius, (0.4, 0.3, 0.3))
    # the same spread of member sizes for every seed, in another order
    q = (np.arange(case["members"]) + 0.5) / case["members"]
    parts = case["particles_lo"] * (case["particles_hi"] / case["particles_lo"]) ** r.permutation(q)
    sols = []
    for i in range(case["members"]):
        u = r.uniform(2, 10) * SOUND
        kn = math.exp(r.uniform(math.log(0.01), 0.0))
        nd = 1.0 / (math.sqrt(2.0) * math.pi * d * d * kn * 2 * radius)
        st = cb.settings_t().set(
            grid_min=(0, 0, 0), grid_max=dom, grid_dim=dim, density=nd, temp=T_INF,
            fnum=nd * cell[0] * cell[1] * cell[2] * cells / parts[i], stream_vel=(u, 0.0, 0.0),
            dt=min(0.2 * min(cell) / (u + 3 * cmp), 0.2 * kn * 2 * radius / cbar), rng="philox",
            ntc_local=1, sample_every=case["sample_every"], init_kind="maxwell", wall_diffuse=1,
            wall_temp=r.uniform(1, 3) * T_INF, capacity_factor=1.6, seed=seed + i + 1, geom_nearest=1,
            face_kind=OUTFLOW, gas_omega=0.81, **ARGON)
        sol = cb.DSMCSolver().Init(st)
        sol.SetModel(*mesh, (16, 16, 16))
        sol.InitSystemState()
        sols.append(sol)
    batch = cb.DSMCBatch(sols)
    batch.Step(case["settle"])
    batch.Sync()
    return dict(batch=batch, sols=sols, out=_pinned_fields(case["members"], cells, 5))


def _run_ensemble(case, s):
    for sol in s["sols"]:
        sol.ResetSamples()
    s["batch"].Step(case["steps"])
    s["batch"].Sync()
    for i, sol in enumerate(s["sols"]):
        sol.Fields(s["out"][i])
    return s["out"]


# ------------------------------------------------------------------- stages --

def _prepare_stages(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    nx, ny, nz, n = case["nx"], case["ny"], case["nz"], case["n"]
    cells = nx * ny * nz
    dom = (0.01 * nx, 0.01 * ny, 0.01 * nz)
    f32 = dict(dtype=torch.float32, device="cuda")
    # the order a run leaves: sorted by the cells of the step before, most
    # particles moved by less than a cell since
    home = (torch.arange(n, device="cuda") * cells) // n
    at = [home % nx, (home // nx) % ny, home // (nx * ny)]
    pos = []
    for k in range(3):
        x = 0.01 * (at[k].to(torch.float32) + torch.rand(n, generator=g, **f32))
        x = x + 0.004 * torch.randn(n, generator=g, **f32)
        pos.append(x.clamp_(1e-5, dom[k] - 1e-5))
    vstd = math.sqrt(KB * 300.0 / ARGON["gas_mass"])
    vel = [vstd * torch.randn(n, generator=g, **f32) for _ in range(3)]
    vel[0] += 300.0
    i32 = dict(dtype=torch.int32, device="cuda")
    maxrem = torch.stack([torch.full((cells,), 6.0 * vstd * math.pi * ARGON["gas_diam"] ** 2, **f32),
                          torch.rand(cells, generator=g, **f32)], dim=1).contiguous()
    seeds = torch.randint(129, 1 << 31, (cells, 4), generator=g, device="cuda").to(torch.int32)
    fnum = 1e20 * 1e-6 * cells / n
    gref = 0.0
    w = case["omega"]
    if w != 0.5:
        gref = math.sqrt(4 * KB * ARGON["gas_tref"] / ARGON["gas_mass"]) * math.gamma(2.5 - w) ** (-1 / (2 * w - 1))
    grid = stages.make_grid((0, 0, 0), dom, (nx, ny, nz))
    dt = 3e-6
    ws = None
    if case["sort"] == "workspace":
        ws = torch.empty(stages.sort_workspace_bytes(n, cells), dtype=torch.uint8, device="cuda")
    return dict(
        grid=grid, src=pos + vel, dst=[torch.empty(n, **f32) for _ in range(6)],
        keys=torch.empty(n, **i32), idx=torch.empty(n, **i32), start=torch.empty(cells + 1, **i32),
        cse=torch.empty(2 * cells, **i32), maxrem=maxrem, seeds=seeds, ws=ws,
        sums=torch.zeros((cells, 5), dtype=torch.float64, device="cuda"), cells=cells,
        cp=stages.collide_params(cells, 1e-6, math.pi * ARGON["gas_diam"] ** 2, fnum, n / cells, dt,
                                 omega=w, vhs_gref=gref, ntc_local=int(case["rng"] == "philox"),
                                 rng=case["rng"], seed=seed + 1),
        mp=stages.move_params(grid, dt, seed=seed + 1))


def _run_stages(case, s):
    src, dst = s["src"], s["dst"]
    stages.cell_index(s["grid"], src[0], src[1], src[2], s["keys"], s["idx"])
    if case["sort"] == "static":
        stages.sort_static(s["keys"], s["idx"], s["cells"], cell_start=s["start"])
    else:
        stages.sort(s["keys"], s["idx"], s["cells"], cell_start=s["start"], workspace=s["ws"])
    stages.bounds_reorder(s["keys"], s["idx"], s["cells"], s["cse"], src, dst)
    stages.collide(s["cp"], dst[3], dst[4], dst[5], s["start"], s["maxrem"],
                   s["seeds"] if case["rng"] == "taus" else None)
    stages.move(s["mp"], *dst)
    s["sums"].zero_()
    stages.sample(dst[3], dst[4], dst[5], s["start"], s["cells"], s["sums"])
    return s["keys"], s["idx"], s["start"], s["cse"], dst, s["maxrem"], s["seeds"], s["sums"]


# --------------------------------------------------------------------- fill --

def _prepare_fill(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    u = 6.0 * SOUND
    dom = (1.2, 0.6, 0.6)
    cell_v = dom[0] * dom[1] * dom[2] / (nx * ny * nz)
    st = dict(grid_min=(0, 0, 0), grid_max=dom, grid_dim=(nx, ny, nz), density=1e20, temp=T_INF,
              fnum=1e20 * cell_v / case["ppc"], stream_vel=(u, 0.0, 0.0), dt=2e-6, rng="philox", ntc_local=1,
              sample_every=2, init_kind="maxwell", wall_diffuse=1, wall_temp=2 * T_INF, gas_omega=0.81,
              capacity_factor=2.0, seed=seed + 1, geom_nearest=1, face_kind=OUTFLOW, **ARGON)
    sol = cb.DSMCSolver().Init(cb.settings_t().set(**st))
    sol.SetModel(*cb.mesh_icosphere(3, case["radius"], (0.4, 0.3, 0.3)), (16, 16, 16))
    # a predicted flow: compressed, slowed and heated ahead of the body, thin
    # behind it, with the roughness of a prediction
    r = np.random.default_rng(seed)
    z, y, x = np.meshgrid((np.arange(nz) + 0.5) / nz * 0.6, (np.arange(ny) + 0.5) / ny * 0.6,
                          (np.arange(nx) + 0.5) / nx * 1.2, indexing="ij")
    dx, rad = x - 0.4, np.hypot(y - 0.3, z - 0.3)
    bow = np.exp(-((np.sqrt(dx * dx + rad * rad) / case["radius"] - 1.5) ** 2) - 4 * np.maximum(dx, 0))
    wake = np.exp(-(rad / case["radius"]) ** 2) * (dx > 0)
    f = np.stack([1e20 * (1 + 2.5 * bow - 0.9 * wake), u * (1 - 0.8 * bow - 0.6 * wake),
                  300 * bow * (y - 0.3) / 0.3, 300 * bow * (z - 0.3) / 0.3,
                  T_INF * (1 + 6 * bow + 2 * wake)], axis=-1).reshape(-1, 5)
    f *= 1 + 0.02 * r.standard_normal(f.shape)
    return dict(sol=sol, fields=f.astype(np.float32), weight=case["weight"], dt=st["dt"],
                out=_pinned_fields(nx * ny * nz, 5))


def _run_fill(case, s):
    if s["weight"] > 0:
        n = s["sol"].InitFromFieldsTwoStream(s["fields"], s["weight"])
    else:
        n = s["sol"].InitFromFields(s["fields"])
    s["sol"].StepGraph(s["dt"], case["steps"])
    return n, s["sol"].Fields(s["out"])


# ---------------------------------------------------------------------- mlp --

def _conditions(case, seed):
    return np.random.default_rng(seed + 1).uniform(-1, 1, (case["batch"], 4)).astype(np.float32)


def _biases(case, seed):
    r = np.random.default_rng(seed + 2)
    sizes = {f"b{l}": case["hidden"] for l in range(case["depth"])}
    sizes["bout"] = case["modes"]
    return {k: torch.from_numpy(r.normal(0, 0.1, n).astype(np.float32)).cuda() for k, n in sizes.items()}


def _targets(case, seed):
    """Normalized fields of a batch, [batch, cells * 5], BF16; cells without a
    particle are NaN."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["batch"], case["cells"], 5)
    t = 1 + 0.3 * torch.randn(shape, generator=g, device="cuda")
    t[torch.rand(shape[:2], generator=g, device="cuda") < 0.02] = float("nan")
    return t.reshape(case["batch"], -1).to(torch.bfloat16).contiguous()


def _prepare_mlp(case, seed):
    net = WarmStartMLP(case["cells"] * 5, hidden=case["hidden"], depth=case["depth"],
                       modes=case["modes"], seed=seed)
    net.set_mean(np.ones(case["cells"] * 5, np.float32))
    for k, b in _biases(case, seed).items():  # as after some training
        net.params[k].copy_(b)
    s = dict(net=net, x=_conditions(case, seed))
    if case["call"] == "train":
        s["t"] = _targets(case, seed)
    return s


def _run_mlp(case, s):
    net = s["net"]
    if case["call"] == "predict":
        return net.predict(s["x"])
    loss, count, grads, y = net.loss_and_grads(s["x"], s["t"])
    net.adam_step(grads, lr=1e-5)
    return dict(loss=loss, count=count, grads=grads, y=y, params=net.params)


def _exact_mlp(case, seed):
    """The same network in 64 bits: the weights drawn as the network draws
    them, nothing rounded to 16 bits but the targets."""
    F, hidden, modes, depth = case["cells"] * 5, case["hidden"], case["modes"], case["depth"]
    r = np.random.default_rng(seed)
    f64 = dict(dtype=torch.float64, device="cuda")

    def normal(std, shape):
        return torch.from_numpy(r.normal(0, std, shape).astype(np.float32)).to(**f64)

    P = {}
    for l in range(depth):
        fan = 4 if l == 0 else hidden
        w = normal(math.sqrt(2.0 / fan), (fan, hidden))
        P[f"W{l}"] = torch.cat([w, torch.zeros((12, hidden), **f64)]) if l == 0 else w
    P["Wout"] = normal(math.sqrt(1.0 / hidden), (hidden, modes))
    P["B"] = normal(0.02, (modes, F))
    P["mean"] = torch.ones(F, **f64)
    P.update({k: b.to(**f64) for k, b in _biases(case, seed).items()})
    x = torch.from_numpy(_conditions(case, seed)).to(**f64)
    h, zs, hs = torch.cat([x, torch.zeros((len(x), 12), **f64)], dim=1), [], []
    for l in range(depth):
        hs.append(h)
        zs.append(h @ P[f"W{l}"] + P[f"b{l}"])
        h = torch.nn.functional.gelu(zs[-1])
    c = h @ P["Wout"] + P["bout"]
    y = c @ P["B"] + P["mean"]
    if case["call"] == "predict":
        return y
    t = _targets(case, seed).to(torch.float64)
    ok = ~torch.isnan(t)
    e = torch.where(ok, y - t, torch.zeros((), **f64))
    dy = 2 * e / y.numel()
    g = {"B": c.T @ dy, "mean": dy.sum(0)}
    dc = dy @ P["B"].T
    g["Wout"], g["bout"] = h.T @ dc, dc.sum(0)
    dh = dc @ P["Wout"].T
    for l in range(depth - 1, -1, -1):
        z = zs[l]
        dz = dh * (0.5 * (1 + torch.erf(z / math.sqrt(2))) +
                   z * torch.exp(-z * z / 2) / math.sqrt(2 * math.pi))
        g[f"W{l}"], g[f"b{l}"] = hs[l].T @ dz, dz.sum(0)
        dh = dz @ P[f"W{l}"].T
    # Adam's first step: the corrected moments are g and g^2
    new = {k: w - 1e-5 * g[k] / (g[k].abs() + 1e-8) for k, w in P.items()}
    return dict(loss=(e * e).sum().reshape(1), count=None, grads=g, y=y, params=new)


# ---------------------------------------------------------------- interface --

_PREPARE = dict(flow=_prepare_flow, ensemble=_prepare_ensemble, stages=_prepare_stages,
                fill=_prepare_fill, mlp=_prepare_mlp)
_RUN = dict(flow=_run_flow, ensemble=_run_ensemble, stages=_run_stages, fill=_run_fill, mlp=_run_mlp)


def prepare(case, seed):
    s = _PREPARE[case["kind"]](case, seed)
    s["case"] = case
    return s


def run(state):
    return _RUN[state["case"]["kind"]](state["case"], state)


def work(case):
    kind = case["kind"]
    if kind == "flow":
        # per step the six state arrays read once and written once
        cells = case["nx"] * case["ny"] * case["nz"]
        n = cells * case["ppc"]
        back = 24 * n if case["back"] == "state" else 40 * cells
        return dict(bytes=48 * n * case["steps"] + back, flops=60 * n * case["steps"])
    if kind == "ensemble":
        lo, hi = case["particles_lo"], case["particles_hi"]
        n = case["members"] * (hi - lo) / math.log(hi / lo)
        return dict(bytes=48 * n * case["steps"] + 40 * 65536 * case["members"],
                    flops=60 * n * case["steps"])
    if kind == "stages":
        # state read and written, keys and indices written, per-cell state
        cells = case["nx"] * case["ny"] * case["nz"]
        per_cell = 4 + 8 + 16 + 40 + (32 if case["rng"] == "taus" else 0)
        return dict(bytes=(48 + 8) * case["n"] + per_cell * cells, flops=80 * case["n"])
    if kind == "fill":
        cells = case["nx"] * case["ny"] * case["nz"]
        n = cells * case["ppc"]
        return dict(bytes=60 * cells + 24 * n + 48 * n * case["steps"], flops=(100 + 60 * case["steps"]) * n)
    b, F, h, k, d = case["batch"], case["cells"] * 5, case["hidden"], case["modes"], case["depth"]
    small = 16 * h + (d - 1) * h * h + h * k
    if case["call"] == "predict":
        return dict(bytes=2 * (small + k * F) + 4 * F + 4 * b * F, flops=2.0 * b * (small + k * F))
    w = small + k * F + F
    # weights and both moments read and written, gradients and the BF16 copies
    # written, the BF16 weights read; targets read, fields written
    return dict(bytes=w * (24 + 4 + 2 + 2) + b * F * (2 + 4), flops=6.0 * b * (small + k * F))


def exact(case, seed):
    """The network's passes have an exact result.  The others follow random
    draws (collisions, walls, fills): theirs has no closed form, and the whole
    numbers among them (cells, order, counts) are fixed by their definition."""
    return _exact_mlp(case, seed) if case["kind"] == "mlp" else None
