"""Performance cases of the fluid engine: what a user's program has it do.

Kinds of case:
  step       one solver step of one scene (DFSPH, IISPH or implicit SPH) from a
             state the program loads: the frame loop of a simulation, or one
             evaluation of a parameter study
  batch      one DFSPH step of several independent scenes in one call
  neighbors  the standalone neighbor update with the reference-layout list
  sample     density, velocity and vorticity at sample points (statistics)
  volume     a body's volume map, built once per body when a scene is set up

`exact` restates each of them in 64-bit torch without the engine.
"""
import math

import numpy as np
import torch

from alluvion_b200 import _capi, scenes

DT = 2e-4
DENSITY0 = 1000.0
VISCOSITY = 0.01
EPS = 1e-6  # dfsph_factor_epsilon
GAP = 2.9     # particle radii between the block and the walls it leans on
SPACING = 2.0  # of the lattice, in particle radii
JITTER = 0.05  # of its points, in particle radii
_engine = []


def _lib():
    """The process's engine (a program keeps one) and the library."""
    if not _engine:
        _engine.append(_capi.Engine(0))
    return _engine[0], _capi.lib()


# ------------------------------------------------------------------- cases
def _step(name, method, nx, ny, nz, radius, dtype="f32", bodies=0, periodic=False, map_res=24):
    return {"name": name, "kind": "step", "method": method, "nx": nx, "ny": ny, "nz": nz,
            "radius": radius, "dtype": dtype, "bodies": bodies, "periodic": periodic,
            "map_res": map_res}


def listed():
    return [
        # an interactive scene: launches and latency are all there is
        _step("df-4k", "df", 16, 16, 16, 0.01, map_res=16),
        # the small benchmark scene (32^3 lattice)
        _step("df-32k", "df", 32, 32, 32, 0.01, map_res=24),
        # the ordinary production scene with coupled bodies (128 x 64 x 128 lattice)
        _step("df-1m", "df", 128, 64, 128, 0.005, bodies=2, map_res=32),
        # the largest single-GPU scene (256 x 128 x 256 lattice)
        _step("df-8m", "df", 256, 128, 256, 0.0025, bodies=2, map_res=48),
        # periodic flow: no walls, the y seam wraps
        _step("df-periodic-209k", "df", 67, 48, 65, 0.01, periodic=True),
        # double precision, the reference's other solver type, ragged size
        _step("df-f64-128k", "df", 53, 47, 51, 0.01, dtype="f64", map_res=16),
        # the other two pressure solvers, ragged sizes
        _step("ii-491k", "ii", 97, 61, 83, 0.005, bodies=2, map_res=32),
        _step("i-147k", "i", 63, 41, 57, 0.01, bodies=1, map_res=24),
        # many small scenes at once (parameter sweeps, training data)
        {"name": "batch-24", "kind": "batch", "scenes": 24, "min_n": 8192, "max_n": 65536,
         "radius": 0.01, "map_res": 16},
        # a program that reads the neighbor list itself
        {"name": "neighbors-300k", "kind": "neighbors", "nx": 75, "ny": 61, "nz": 67,
         "radius": 0.01, "dtype": "f32"},
        # statistics on a cloud of probes
        {"name": "sample-1m", "kind": "sample", "nx": 100, "ny": 100, "nz": 100, "radius": 0.01,
         "samples": 1 << 20, "dtype": "f32"},
        # scene set-up: the container's map
        {"name": "volume-box-32", "kind": "volume", "shape": "box", "grid": False, "res": 32,
         "radius": 0.01, "size": 64.0, "dtype": "f32"},
    ]


def _lattice(rng, lo, hi):
    """A lattice of lo..hi particles (log-uniform), sides within a factor of about two."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    side = n ** (1 / 3)
    nx = max(8, int(side * rng.uniform(0.75, 1.35)))
    nz = max(8, int(side * rng.uniform(0.75, 1.35)))
    return nx, max(8, min(int(hi / (nx * nz)), round(n / (nx * nz)))), nz


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["batch", "neighbors", "sample", "volume"])
    radius = rng.choice([0.005, 0.01])
    dtype = rng.choice(["f32", "f32", "f32", "f64"])
    if kind == "step":
        method = rng.choice(["df", "df", "df", "ii", "i"])
        nx, ny, nz = _lattice(rng, 2000, 400000 if dtype == "f64" else 3000000)
        periodic = rng.random() < 0.2
        if periodic:
            ny = max(8, 4 * round(ny / 4))  # four layers are two cells
        bodies = 0 if periodic or min(nx, nz) < 16 else rng.choice([0, 1, 2])
        c = _step("", method, nx, ny, nz, radius, dtype, bodies, periodic,
                  rng.choice([12, 16, 24, 32]))
        del c["name"]
        return c
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(2, 32), "min_n": rng.randint(2000, 9000),
                "max_n": rng.randint(20000, 90000), "radius": radius,
                "map_res": rng.choice([12, 16])}
    if kind == "neighbors":
        nx, ny, nz = _lattice(rng, 2000, 600000)
        return {"kind": "neighbors", "nx": nx, "ny": ny, "nz": nz, "radius": radius,
                "dtype": dtype}
    if kind == "sample":
        nx, ny, nz = _lattice(rng, 2000, 1500000)
        return {"kind": "sample", "nx": nx, "ny": ny, "nz": nz, "radius": radius,
                "samples": int(math.exp(rng.uniform(math.log(1000), math.log(1500000)))),
                "dtype": dtype}
    grid = rng.random() < 0.4
    return {"kind": "volume", "shape": rng.choice(["box", "sphere"]), "grid": grid,
            "res": rng.randint(8, 20 if grid else 36), "radius": radius,
            "size": float(rng.randint(16, 80)), "dtype": "f32"}


# ------------------------------------------------------------------- inputs
def _np_dtype(case):
    return np.float64 if case.get("dtype") == "f64" else np.float32


def _generator(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + salt)


def _block(nx, ny, nz, radius, gen):
    """A jittered lattice block (spacing SPACING r: near rest density), z fastest, f64."""
    s = SPACING * radius
    ax = [s * torch.arange(k, device="cuda", dtype=torch.float64) for k in (nx, ny, nz)]
    x = torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    return x + JITTER * radius * (2 * torch.rand(x.shape, device="cuda", dtype=torch.float64,
                                               generator=gen) - 1)


def _flow(x, extent, gen):
    """A smooth velocity field with a little noise."""
    v = 0.005 * torch.randn(x.shape, device="cuda", dtype=torch.float64, generator=gen)
    for _ in range(3):
        k = torch.randn(3, device="cuda", dtype=torch.float64, generator=gen) * 3 / extent
        a = 0.1 * torch.randn(3, device="cuda", dtype=torch.float64, generator=gen)
        v += torch.sin(x @ k + 6.28 * torch.rand(1, device="cuda", dtype=torch.float64,
                                                 generator=gen))[:, None] * a
    return v


def _scene_inputs(case, seed):
    """Host description of a step case and its particle state (f64 on the device):
    block in the low corner of a tank, free in x, open above, bodies floating on it."""
    r, nx, ny, nz = case["radius"], case["nx"], case["ny"], case["nz"]
    gen = _generator(seed)
    x = _block(nx, ny, nz, r, gen)
    ext = SPACING * r * np.array([nx, ny, nz], float)
    dt = np.float32(DT).item() if case["dtype"] == "f32" else DT
    h = 4 * r
    specs, lo, hi, period = [], None, None, 0.0
    if case["periodic"]:  # a free slab, y wraps at a whole number of cells
        period = max(2, round(ext[1] / (2 * h))) * 2 * h  # an even number of cells
        x[:, 1] *= period / ext[1]
        x[:, 1] += -period / 2 + r
        x[:, 1] = torch.where(x[:, 1] < -period / 2, x[:, 1] + period, x[:, 1])
        x[:, 0] += h
        x[:, 2] += h
        lo, hi = (0.0, -period / 2, 0.0), (ext[0] + 3 * h, period / 2, ext[2] + 3 * h)
        depth = torch.zeros_like(x[:, 1])
    else:
        x += GAP * r
        top = GAP * r + ext[1]
        size = np.array([1.3 * ext[0] + 4 * h, 1.4 * ext[1] + 12 * h,
                         ext[2] - SPACING * r + 2 * GAP * r])
        specs.append(dict(shape=_capi.SHAPE_BOX, params=scenes.box_params(size), sign=-1.0,
                          resolution=case["map_res"], use_distance_grid=False, mass=0.0,
                          x=tuple(size / 2)))
        rr, w = 8 * r, 12 * r
        if case["bodies"] > 0:
            m = 800 * 4 / 3 * math.pi * rr ** 3
            specs.append(dict(shape=_capi.SHAPE_SPHERE, params=[rr], sign=1.0, resolution=16,
                              use_distance_grid=True, mass=m,
                              inertia=scenes.sphere_inertia(m, rr),
                              x=(0.3 * ext[0], top + rr + 0.5 * r, 0.35 * ext[2]),
                              v=(0.05, -0.2, 0.0), omega=(0.3, 0.0, 0.5)))
        if case["bodies"] > 1:
            m = 600 * w ** 3
            specs.append(dict(shape=_capi.SHAPE_BOX, params=scenes.box_params((w,) * 3),
                              sign=1.0, resolution=16, use_distance_grid=True, mass=m,
                              inertia=scenes.box_inertia(m, (w,) * 3),
                              x=(0.7 * ext[0], top + w / 2 + 0.5 * r, 0.65 * ext[2]),
                              q=(0.0, math.sin(0.2), 0.0, math.cos(0.2)), v=(0.0, -0.1, 0.1)))
        lo, hi = -0.5 * h * np.ones(3), size + 0.5 * h
        depth = top - x[:, 1]
    v = _flow(x, float(ext.max()), gen)
    noise = 1 + 0.1 * torch.rand(x.shape[0], device="cuda", dtype=torch.float64, generator=gen)
    td = torch.float32 if case["dtype"] == "f32" else torch.float64
    depth = depth * noise
    state = {"x": x.to(td), "v": v.to(td)}
    if case["method"] == "df":  # the previous step's kappa (hydrostatic) and kappa_v
        state["kappa"] = (-9.81 * depth * dt * dt).to(td)
        state["kappa_v"] = (-0.01 * depth).to(td)
    else:
        state["pressure"] = (9.81 * depth).to(td)
    return {"specs": specs, "lo": lo, "hi": hi, "period": period, "state": state, "dt": dt}


def _step_state(case, seed):
    engine, _ = _lib()
    dtype = _np_dtype(case)
    inp = _scene_inputs(case, seed)
    n = inp["state"]["x"].shape[0]
    cn = scenes.make_const(dtype, case["radius"], viscosity=VISCOSITY,
                           boundary_viscosity=VISCOSITY, dfsph_factor_epsilon=EPS)
    cni = scenes.make_consti(inp["lo"], inp["hi"], float(cn.kernel_radius), len(inp["specs"]))
    sp = scenes.solver_params(max_dt=DT)
    if inp["period"]:
        cells = round(inp["period"] / float(cn.kernel_radius))
        cni.grid_offset[1], cni.grid_res[1] = -(cells // 2), cells
        sp.wrap_y, sp.wrap_length = 1, cells * float(cn.kernel_radius)
    scene = scenes.DeviceScene(engine, dtype, cn, cni, np.zeros((n, 3), dtype), inp["specs"])
    start = scene.snapshot()[1]
    return {"scene": scene, "sp": sp, "inputs": inp["state"], "rigid": start, "dt": inp["dt"],
            "method": case["method"]}


def _load(st):
    """The program's new state into the scene's buffers."""
    for k, t in st["inputs"].items():
        getattr(st["scene"], k).copy_(t)
    st["scene"].restore(({}, st["rigid"]))


def _outputs(st):
    sc = st["scene"]
    out = {k: getattr(sc, k) for k in ("x", "v", "density", *list(st["inputs"])[2:])}
    if sc.num_boundaries > 1:
        rig = scenes.rigid_array(sc.dtype, [sc.rigid[b] for b in range(1, sc.num_boundaries)])
        out["rigid_pose"] = rig[:, [0, 1, 2, 6, 7, 8, 9]]
        out["rigid_velocity"] = rig[:, [3, 4, 5, 10, 11, 12]]
    return out


def _batch_cases(case, seed):
    """The scenes of a batch: cubic lattices, sizes log-uniform, up to two bodies."""
    rng = np.random.default_rng(1234)  # the sizes belong to the case, the states to the seed
    out = []
    for k in range(case["scenes"]):
        n = math.exp(rng.uniform(math.log(case["min_n"]), math.log(case["max_n"])))
        side = max(10, round(n ** (1 / 3)))
        out.append(dict(_step("", "df", side, side, side, case["radius"],
                              bodies=k % 3 if side >= 16 else 0, map_res=case["map_res"]),
                        seed=seed * 64 + k))
    return out


def _sample_inputs(case, seed):
    td = torch.float32 if case["dtype"] == "f32" else torch.float64
    gen = _generator(seed, 7)
    r = case["radius"]
    x = _block(case["nx"], case["ny"], case["nz"], r, gen) + 4 * r
    ext = SPACING * r * torch.tensor([case["nx"], case["ny"], case["nz"]], device="cuda",
                                   dtype=torch.float64)
    v = _flow(x, float(ext.max()), gen)
    rho = DENSITY0 * (0.97 + 0.06 * torch.rand(x.shape[0], device="cuda", dtype=torch.float64,
                                               generator=gen))
    out = {"x": x.to(td), "v": v.to(td), "rho": rho.to(td), "hi": (ext + 8 * r).cpu().numpy()}
    if case["kind"] == "sample":
        out["s"] = (torch.rand((case["samples"], 3), device="cuda", dtype=torch.float64,
                               generator=gen) * ext + 4 * r).to(td)
    return out


def _volume_body(case, seed):
    """The body of a volume map: extents vary a little with the seed."""
    r = case["radius"]
    f = 1 + 0.02 * np.random.default_rng(seed).random(3)
    w = case["size"] * r * f
    if case["shape"] == "box":
        shape, params = _capi.SHAPE_BOX, scenes.box_params(w)
    else:
        shape, params = _capi.SHAPE_SPHERE, [0.5 * w[0]]
    sign = 1.0 if case["grid"] else -1.0
    return dict(shape=shape, params=params, sign=sign, resolution=case["res"],
                use_distance_grid=case["grid"], mass=0.0)


def prepare(case, seed):
    engine, _ = _lib()
    dtype = _np_dtype(case)
    td = torch.float32 if dtype == np.float32 else torch.float64
    kind = case["kind"]
    if kind == "step":
        return dict(_step_state(case, seed), kind=kind)
    if kind == "batch":
        return {"kind": kind, "sp": scenes.solver_params(max_dt=DT),
                "scenes": [_step_state(c, c["seed"]) for c in _batch_cases(case, seed)]}
    cn = scenes.make_const(dtype, case["radius"])
    h = float(cn.kernel_radius)
    if kind in ("neighbors", "sample"):
        inp = _sample_inputs(case, seed)
        st = dict(inp, kind=kind, cn=cn, sfx=case["dtype"],
                  cni=scenes.make_consti(np.zeros(3), inp["hi"], h, 0))
        n = inp["x"].shape[0]
        zeros = lambda *s, t=td: torch.zeros(*s, dtype=t, device="cuda")
        if kind == "neighbors":
            st.update(density=zeros(n), count=zeros(n, t=torch.int32), list=zeros(n, 64, 4))
            return st
        ns = inp["s"].shape[0]
        st.update(density=zeros(ns), vel=zeros(ns, 3), vort=zeros(ns, 3))
        return st
    spec = _volume_body(case, seed)
    body = scenes.body_from_spec(dtype, cn, spec)
    st = {"kind": kind, "cn": cn, "body": body,
          "nodes": torch.zeros(body.num_nodes, dtype=td, device="cuda"), "sfx": case["dtype"]}
    if case["grid"]:
        st["dist"] = _body_distance(spec, _node_positions(*_body_grid(spec, h, dtype))).to(td)
        body.distance_nodes = st["dist"].data_ptr()
    return st


# ---------------------------------------------------------------------- run
def run(state):
    engine, lib = _lib()
    p, kind = _capi.ptr, state["kind"]
    if kind == "step":
        _load(state)
        state["scene"].step(state["method"], state["sp"], state["dt"])
        return _outputs(state)
    if kind == "batch":
        for s in state["scenes"]:
            _load(s)
        scenes.batch_step(engine, [s["scene"] for s in state["scenes"]], state["sp"],
                          [s["dt"] for s in state["scenes"]])
        # every scene's particles in one tensor each: x, v, density
        return {k: torch.cat([getattr(s["scene"], k) for s in state["scenes"]])
                for k in ("x", "v", "density", "kappa", "kappa_v")}
    if kind == "neighbors":
        fn = getattr(lib, "al_update_particle_neighbors_" + state["sfx"])
        _capi.check(fn(engine.handle, p(state["cn"]), p(state["cni"]), p(state["x"]),
                       state["x"].shape[0], None, p(state["density"]), p(state["count"]),
                       p(state["list"]), None, None), "al_update_particle_neighbors")
        ints = state["list"].view(torch.int32 if state["sfx"] == "f32" else torch.int64)
        return {"density": state["density"], "count": state["count"],
                "displacement": state["list"][..., :3], "index": ints[..., 3]}
    if kind == "sample":
        req = (_capi.SampleF32 if state["sfx"] == "f32" else _capi.SampleF64)()
        req.sample_x, req.num_samples = p(state["s"]).value, state["s"].shape[0]
        req.particle_density, req.particle_v = p(state["rho"]).value, p(state["v"]).value
        req.sample_density, req.sample_v = p(state["density"]).value, p(state["vel"]).value
        req.sample_vorticity = p(state["vort"]).value
        fn = getattr(lib, "al_sample_fluid_" + state["sfx"])
        _capi.check(fn(engine.handle, p(state["cn"]), p(state["cni"]), p(state["x"]),
                       state["x"].shape[0], None, p(req), None), "al_sample_fluid")
        return {"density": state["density"], "v": state["vel"], "vorticity": state["vort"]}
    fn = getattr(lib, "al_build_volume_field_" + state["sfx"])
    _capi.check(fn(engine.handle, p(state["cn"]), p(state["body"]), p(state["nodes"]), None),
                "al_build_volume_field")
    return state["nodes"]


# --------------------------------------------------------------------- work
PAIRS = 30  # neighbors per particle near rest density (h = 4 r)


def _step_work(case):
    """One step at its minimum iteration counts.  Bytes: the caller's state in and
    out once.  Flops: the pair sums (about 30 per neighbor and pass)."""
    n = case["nx"] * case["ny"] * case["nz"]
    w = 4 if case["dtype"] == "f32" else 8
    io = {"df": 6 + 2 + 9 + 5, "ii": 6 + 1 + 9 + 3, "i": 6 + 1 + 9 + 3}[case["method"]]
    passes = {"df": 14, "ii": 9, "i": 6}[case["method"]]
    return n * w * io, n * PAIRS * 30 * passes


def work(case):
    kind = case["kind"]
    if kind == "step":
        b, f = _step_work(case)
    elif kind == "batch":
        parts = [_step_work(c) for c in _batch_cases(case, 0)]
        b, f = sum(q[0] for q in parts), sum(q[1] for q in parts)
    else:
        w = 8 if case["dtype"] == "f64" else 4
        if kind == "neighbors":
            n = case["nx"] * case["ny"] * case["nz"]
            b, f = n * (3 * w + w + 4 + PAIRS * 4 * w), n * PAIRS * 30
        elif kind == "sample":
            n = case["nx"] * case["ny"] * case["nz"]
            b, f = w * (7 * n + 10 * case["samples"]), case["samples"] * PAIRS * 60
        else:
            # the quadrature is defined on 27,000 points of each node's ball; only nodes
            # whose ball meets the surface need them
            m = scenes.num_grid_nodes([case["res"]] * 3)
            ext = case["size"] + (8 if not case["grid"] else 16)
            inner = max(0.0, (case["size"] - 8) / ext) ** 3 if not case["grid"] else 0.0
            b, f = m * w, (1 - inner) * m * 27000 * (12 if not case["grid"] else 200)
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times the distance from `exact` that was seen, which is what sums in
    another order show too.  Steps amplify rounding through kappa (rho_adv - 1 is a small
    difference); the finest scene most, and single particles at a clamp more than the rest."""
    f32 = case.get("dtype", "f32") == "f32"
    if case["kind"] in ("step", "batch"):
        if not f32:
            return {"rel": 2e-13, "max": 1e-9}
        return {"rel": 5e-4 if case["radius"] < 0.005 else 6e-5, "max": 1e-2}
    return {"rel": 1e-6 if f32 else 2e-15, "max": 1e-4 if f32 else 1e-12}


# ------------------------------------------------------- 64-bit restatement
def _real(case):
    return torch.float32 if case["dtype"] == "f32" else torch.float64


class _Kernel:
    """The cubic spline and the constants derived from the particle radius."""

    def __init__(self, radius, f32):
        self.r = np.float32(radius).item() if f32 else radius
        self.h = 4 * self.r
        self.k = 8 / self.h ** 3 / math.pi
        self.l = 48 / self.h ** 4 / math.pi
        self.vol = (2 * self.r) ** 3
        self.mass = DENSITY0 * self.vol

    def W(self, dist):
        q = dist.abs() / self.h
        s = torch.where(q <= 0.5, (6 * q - 6) * q * q + 1, 2 * (1 - q).clamp(min=0) ** 3)
        return s * self.k

    def grad(self, d):
        rl = d.square().sum(-1).sqrt()
        q = rl / self.h
        s = torch.where(q <= 0.5, (3 * q - 2) / self.h,
                        torch.where(q <= 1, -(1 - q) ** 2 / rl.clamp(min=1e-300),
                                    torch.zeros_like(q)))
        return (self.l * s)[..., None] * d


def _pairs(pts, x, h, period=0.0, skip=True):
    """(i, j, d): points pts[i] and particles x[j] closer than h (the test in the
    inputs' own precision), i ascending, without j == i when skip."""
    dt = x.dtype
    hh = torch.tensor(h, dtype=dt, device=x.device)
    h2 = hh * hh
    lo = torch.minimum(pts.amin(0), x.amin(0)).double() - 0.5 * h
    if period:
        lo[1] = -period / 2
    cell = lambda p: ((p.double() - lo) / h).floor().long()
    cx, cp = cell(x), cell(pts)
    top = torch.maximum(cx.amax(0), cp.amax(0)) + 2
    ny = round(period / h) if period else None
    if period:
        cx[:, 1] %= ny
        cp[:, 1] %= ny
    key = lambda c: ((c[:, 0] + 1) * (top[1] + 2) + c[:, 1] + 1) * (top[2] + 2) + c[:, 2] + 1
    order = torch.argsort(key(cx), stable=True)
    sorted_key = key(cx)[order]
    out_i, out_j = [], []
    chunk = 1 << 21
    half = torch.tensor(period / 2, dtype=dt, device=x.device)
    full = torch.tensor(period, dtype=dt, device=x.device)

    def diff(i, j):
        d = pts[i] - x[j]
        if period:
            y = d[:, 1]
            d[:, 1] = torch.where(y >= half, y - full, torch.where(y < -half, y + full, y))
        return d
    for c0 in range(0, pts.shape[0], chunk):
        ii = torch.arange(c0, min(c0 + chunk, pts.shape[0]), device=x.device)
        gi, gj = [], []
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dz in (-1, 0, 1):
                    c = cp[ii] + torch.tensor([dx, dy, dz], device=x.device)
                    if period:
                        c[:, 1] %= ny
                    kk = key(c)
                    b = torch.searchsorted(sorted_key, kk)
                    m = torch.searchsorted(sorted_key, kk, right=True) - b
                    i = torch.repeat_interleave(ii, m)
                    off = torch.arange(i.shape[0], device=x.device) - torch.repeat_interleave(
                        torch.cumsum(m, 0) - m, m)
                    j = order[torch.repeat_interleave(b, m) + off]
                    d = diff(i, j)
                    s = d * d
                    near = (s[:, 0] + s[:, 1]) + s[:, 2] < h2
                    if skip:
                        near &= i != j
                    gi.append(i[near])
                    gj.append(j[near])
        i, j = torch.cat(gi), torch.cat(gj)
        o = torch.argsort(i, stable=True)
        out_i.append(i[o])
        out_j.append(j[o])
    i, j = torch.cat(out_i), torch.cat(out_j)
    d = pts[i].double() - x[j].double()
    if period:
        d[:, 1] -= period * torch.round(d[:, 1] / period)
    return i, j, d


def _sum(n, i, v):
    return torch.zeros((n, *v.shape[1:]), dtype=torch.float64, device=v.device).index_add_(0, i, v)


# ---- bodies
def _body_grid(spec, h, dtype):
    """(domain_min, cell_size, res) of a body's grid in the solver's type, as f64."""
    T = np.dtype(dtype).type
    if spec["shape"] == _capi.SHAPE_BOX:
        lo = -np.asarray(spec["params"][:3])
    else:
        lo = -np.full(3, spec["params"][0])
    margin = T(h) if spec["sign"] < 0 else T(h) * T(2)
    dmin = lo.astype(T) - margin
    dmax = (-lo).astype(T) + margin
    res = spec["resolution"]
    return (torch.tensor(dmin.astype(np.float64), device="cuda"),
            torch.tensor(((dmax - dmin) / T(res)).astype(np.float64), device="cuda"), res)


def _node_positions(dmin, cs, res):
    """The 32-node element's nodes: vertices (x fastest), then two third-points on
    every x-edge (y fastest after x), y-edge and z-edge."""
    r = lambda k: torch.arange(k, device="cuda", dtype=torch.float64)
    third = torch.tensor([1 / 3, 2 / 3], device="cuda", dtype=torch.float64)

    def grid(slow, mid, fast, axes):
        g = torch.stack(torch.meshgrid(slow, mid, fast, indexing="ij"), -1).reshape(-1, 3)
        out = torch.empty_like(g)
        for k, a in enumerate(axes):
            out[:, a] = g[:, k]
        return out

    def edge(axis, slow, mid, axes):
        g = grid(slow, mid, r(res), axes).repeat_interleave(2, 0)
        g[:, axis] += third.repeat(g.shape[0] // 2)
        return g
    v = r(res + 1)
    p = torch.cat([grid(v, v, v, (2, 1, 0)), edge(0, v, v, (2, 1, 0)),
                   edge(1, v, v, (0, 2, 1)), edge(2, v, v, (1, 0, 2))])
    return dmin + cs * p


def _body_distance(spec, x):
    if spec["shape"] == _capi.SHAPE_SPHERE:
        return x.square().sum(-1).sqrt() - spec["params"][0]
    d = x.abs() - torch.tensor(spec["params"][:3], device=x.device, dtype=torch.float64)
    return d.clamp(min=0).square().sum(-1).sqrt() + d.amax(-1).clamp(max=0)


def _locate(dmin, cs, res, x):
    t = (x - dmin) / cs
    inside = ((t >= 0) & (t <= res)).all(-1)
    ip = t.floor().clamp(0, res - 1)
    return inside, ip.long(), 2 * (t - ip) - 1


_EDGES = ((0, 2, 1), (1, 0, 2), (2, 1, 0))  # axis, axis of bit 1, axis of bit 2


def _interpolate(nodes, res, ip, xi, grad=False):
    """Value (and reference-space gradient) of the cubic element at xi of cells ip, for
    each node array of `nodes`."""
    n1 = res + 1
    x, y, z = ip.unbind(-1)
    val = [torch.zeros_like(xi[:, 0]) for _ in nodes]
    der = [torch.zeros_like(xi) for _ in nodes] if grad else None
    r2 = xi.square().sum(-1)

    def add(index, N, dN):
        for k, a in enumerate(nodes):
            w = a[index]
            val[k] += w * N
            if grad:
                der[k] += w[:, None] * dN
    for j in range(8):
        s = [1.0 if j >> k & 1 else -1.0 for k in range(3)]
        a = [1 + s[k] * xi[:, k] for k in range(3)]
        f = 9 * r2 - 19
        dN = None
        if grad:
            dN = torch.stack([a[(k + 1) % 3] * a[(k + 2) % 3] * (s[k] * f + 18 * xi[:, k] * a[k])
                              for k in range(3)], -1) / 64
        add(n1 * n1 * (z + (j >> 2 & 1)) + n1 * (y + (j >> 1 & 1)) + x + (j & 1),
            a[0] * a[1] * a[2] * f / 64, dN)
    base = n1 ** 3
    for fam, (ax, a1, a2) in enumerate(_EDGES):
        for e in range(8):
            s, b1, b2 = (1.0 if e & 1 else -1.0), e >> 1 & 1, e >> 2 & 1
            s1, s2 = 2.0 * b1 - 1, 2.0 * b2 - 1
            t, A, B = xi[:, ax], 1 + s1 * xi[:, a1], 1 + s2 * xi[:, a2]
            g = (1 - t * t) * (1 + 3 * s * t)
            if fam == 0:
                idx = res * n1 * (z + b1) + res * (y + b2) + x
            elif fam == 1:
                idx = res * n1 * (x + b1) + res * (z + b2) + y
            else:
                idx = res * n1 * (y + b1) + res * (x + b2) + z
            dN = None
            if grad:
                dN = torch.zeros_like(xi)
                dN[:, ax] = (3 * s * (1 - t * t) - 2 * t * (1 + 3 * s * t)) * A * B
                dN[:, a1] = g * s1 * B
                dN[:, a2] = g * A * s2
                dN = dN * (9 / 64)
            add(base + 2 * idx + (e & 1), 9 / 64 * g * A * B, dN)
        base += 2 * res * n1 * n1
    return val, der


def _quadrature():
    """Peirce's m = 14 rule on the unit ball: points [27000, 3] and weights."""
    cphi, b = np.polynomial.legendre.leggauss(30)
    # Gauss rule for the weight sqrt(s) on [0, 1] (radius = sqrt(s)) from odd Legendre nodes:
    # the 15 positive nodes of the 31-point Legendre rule, weight r^2
    t, wt = np.polynomial.legendre.leggauss(31)
    r, c = t[16:], wt[16:] * t[16:] ** 2
    th = 2 * np.pi * (np.arange(60) + 1) / 60
    sphi = np.sqrt(1 - cphi ** 2)
    u = np.stack([sphi[None] * np.cos(th)[:, None], sphi[None] * np.sin(th)[:, None],
                  np.broadcast_to(cphi, (60, 30))], -1)
    p = u[:, :, None, :] * r[None, None, :, None]
    w = np.broadcast_to(2 * np.pi / 60 * b[None, :, None] * c[None, None, :], (60, 30, 15))
    return (torch.tensor(p.reshape(-1, 3), device="cuda"),
            torch.tensor(np.ascontiguousarray(w).reshape(-1), device="cuda"))


def _volume_map(spec, K, dtype, dist=None):
    """Volume nodes of a body: quadrature of 1 inside and W / W(0) outside over each
    node's ball (constant where the ball misses the surface's neighborhood)."""
    dmin, cs, res = _body_grid(spec, K.h, dtype)
    x = _node_positions(dmin, cs, res)
    pts, w = _quadrature()
    phi = _body_distance(spec, x) * spec["sign"]
    full = w.sum()
    out = torch.where(phi <= 0, full, torch.zeros_like(phi))
    # a grid's interpolated distance follows the exact one closely: one h of slack
    slack = K.h if dist is not None else 1e-6 * K.h
    near = ((phi < 2 * K.h + slack) & (phi > -K.h - slack)).nonzero()[:, 0]
    if dist is not None:
        near = torch.arange(x.shape[0], device="cuda")
    step = max(1, (1 << 23) // pts.shape[0] if dist is None else (1 << 22) // pts.shape[0])
    for k in range(0, near.shape[0], step):
        idx = near[k:k + step]
        p = (x[idx][:, None, :] + K.h * pts[None]).reshape(-1, 3)
        if dist is None:
            d = _body_distance(spec, p)
        else:
            inside, ip, xi = _locate(dmin, cs, res, p)
            d = _interpolate([dist], res, ip, xi)[0][0]
            d = torch.where(inside, d, torch.full_like(d, 1e30))
        d = d * spec["sign"]
        e = torch.where(d <= 0, torch.ones_like(d), K.W(d) / K.k)
        out[idx] = e.reshape(idx.shape[0], -1) @ w
    return out * K.h ** 3


def _rotate(q, v, inverse=False):
    u = torch.tensor(q[:3], device=v.device, dtype=torch.float64) * (-1.0 if inverse else 1.0)
    c = torch.linalg.cross(u.expand_as(v), v)
    return v + 2 * (q[3] * c + torch.linalg.cross(u.expand_as(v), c))


class _Boundary:
    """One body's boundary terms for the particles within its kernel range."""

    def __init__(self, spec, K, dtype, x):
        T = np.dtype(dtype).type
        f = lambda key, default: [float(T(t)) for t in spec.get(key, default)]
        td = torch.float32 if T == np.float32 else torch.float64
        self.spec = dict(spec, params=[float(T(t)) for t in spec["params"]])
        spec = self.spec
        self.x, self.v = (torch.tensor(f(k, (0, 0, 0)), device="cuda", dtype=torch.float64)
                          for k in ("x", "v"))
        self.omega = torch.tensor(f("omega", (0, 0, 0)), device="cuda", dtype=torch.float64)
        self.q = f("q", (0, 0, 0, 1))
        self.mass = float(T(spec["mass"]))
        self.inertia = torch.tensor(f("inertia", (1, 1, 1)), device="cuda", dtype=torch.float64)
        dmin, cs, res = _body_grid(spec, K.h, dtype)
        dist = None
        if spec["use_distance_grid"]:
            dist = _body_distance(spec, _node_positions(dmin, cs, res)).to(td).double()
        vol = _volume_map(spec, K, dtype, dist).to(td).double()
        local = _rotate(self.q, x - self.x, inverse=True)
        near = (_body_distance(spec, local) * spec["sign"] < 1.5 * K.h)
        self.i = near.nonzero()[:, 0]
        local = local[self.i]
        inside, ip, xi = _locate(dmin, cs, res, local)
        if dist is not None:
            (phi, V), (g, _) = _interpolate([dist, vol], res, ip, xi, grad=True)
            g = g * 2 / cs
        else:
            V = _interpolate([vol], res, ip, xi)[0][0]
            phi = _body_distance(spec, local)
            s = K.h / 256
            e = torch.eye(3, device="cuda", dtype=torch.float64) * s
            g = torch.stack([_body_distance(spec, local + e[k]) -
                             _body_distance(spec, local - e[k]) for k in range(3)], -1)
        d = phi * spec["sign"]
        nrm = _rotate(self.q, g * spec["sign"])
        nrm = nrm / nrm.square().sum(-1, keepdim=True).sqrt().clamp(min=1e-300)
        sep = d[:, None] * nrm
        ok = inside & (V != 0)
        self.i, V, sep, d = self.i[ok], V[ok], sep[ok], d[ok]
        self.at = x[self.i] - sep
        self.V = V
        self.gw = V[:, None] * K.grad(sep)
        self.w = V * K.W(d)
        self.force = torch.zeros(3, device="cuda", dtype=torch.float64)
        self.torque = torch.zeros(3, device="cuda", dtype=torch.float64)

    def velocity(self, at):
        return torch.linalg.cross(self.omega.expand_as(at), at - self.x) + self.v

    def push(self, f, at):
        self.force += f.sum(0)
        self.torque += torch.linalg.cross(at - self.x, f).sum(0)

    def advance(self, dt):
        """Pile::integrate_kinematics: (pose [x, q], velocity [v, omega])."""
        v, omega = self.v + dt / self.mass * self.force, self.omega
        m = _rotate(self.q, torch.eye(3, device="cuda", dtype=torch.float64)).T
        omega = omega + dt * (m @ torch.diag(1 / self.inertia) @ m.T @ self.torque)
        q = torch.tensor(self.q, device="cuda", dtype=torch.float64)
        u, s = q[:3], q[3]
        dq = torch.cat([0.5 * (omega * s + torch.linalg.cross(omega, u)),
                        -0.5 * (omega @ u)[None]])
        q = q + dt * dq
        q = q / q.norm()
        g = torch.tensor([0.0, -9.81, 0.0], device="cuda", dtype=torch.float64)
        v = v + g * dt
        return torch.cat([self.x + v * dt, q]), torch.cat([v, omega])


def _viscosity(K, n, i, j, d, gw, x, v, rho, bodies):
    """Acceleration: gravity, viscosity, boundary viscosity at four points per pair."""
    eps = 0.01 * K.h ** 2
    s = VISCOSITY * K.mass / rho[j] * (d * gw).sum(-1) / (d.square().sum(-1) + eps)
    a = _sum(n, i, s[:, None] * (v[i] - v[j]))
    for b in bodies:
        nrm = b.at - x[b.i]
        ln = nrm.square().sum(-1, keepdim=True).sqrt()
        nrm = nrm / ln.clamp(min=1e-300)
        ref = torch.zeros_like(nrm)
        steep = nrm[:, 0].abs() > 0.999
        ref[:, 0] = (~steep).double()
        ref[:, 1] = steep.double()
        t1 = torch.linalg.cross(nrm, ref)
        t2 = torch.linalg.cross(nrm, t1)
        t1, t2 = t1 / t1.norm(dim=-1, keepdim=True), t2 / t2.norm(dim=-1, keepdim=True)
        off = K.h - ln
        for at in (b.at - t1 * off, b.at + t1 * off, b.at - t2 * off, b.at + t2 * off):
            sep = x[b.i] - at
            c = (VISCOSITY * 0.25 * b.V * (sep * K.grad(sep)).sum(-1) /
                 (sep.square().sum(-1) + eps))[:, None] * (v[b.i] - b.velocity(at))
            a.index_add_(0, b.i, c)
            b.push(-K.mass * c, at)
    a[:, 1] -= 9.81
    return a


def _exact_step(case, seed):
    f32 = case["dtype"] == "f32"
    dtype = _np_dtype(case)
    inp = _scene_inputs(case, seed)
    K = _Kernel(case["radius"], f32)
    st = inp["state"]
    dt = float(np.float32(DT)) if f32 else DT
    xr = st["x"]
    period = 0.0
    if inp["period"]:
        period = round(inp["period"] / K.h) * K.h
    n = xr.shape[0]
    i, j, d = _pairs(xr, xr, K.h, period)
    x, v = xr.double(), st["v"].double()
    gw = K.grad(d) * K.vol
    cnt = torch.bincount(i, minlength=n)
    bodies = [_Boundary(s, K, dtype, x) for s in inp["specs"]]
    den = K.vol * K.k + K.vol * _sum(n, i, K.W(d.square().sum(-1).sqrt()))
    grad = _sum(n, i, gw)
    for b in bodies:
        den.index_add_(0, b.i, b.w)
        grad.index_add_(0, b.i, b.gw)
    rho = den * DENSITY0

    def divergence(v):
        out = _sum(n, i, ((v[i] - v[j]) * gw).sum(-1))
        for b in bodies:
            out.index_add_(0, b.i, ((v[b.i] - b.velocity(b.at)) * b.gw).sum(-1))
        return out

    def push(v, k):
        """Velocities after the updates of k."""
        ks = k[i] + k[j]
        ks = torch.where(ks.abs() > EPS, ks, torch.zeros_like(ks))
        dv = dt * _sum(n, i, ks[:, None] * gw)
        for b in bodies:
            kb = torch.where(k[b.i].abs() > EPS, k[b.i], torch.zeros_like(k[b.i]))
            a = -kb[:, None] * b.gw
            b.push(K.mass * a, b.at)
            dv.index_add_(0, b.i, -dt * a)
        return v + dv

    if case["method"] == "df":
        s2 = _sum(n, i, gw.square().sum(-1)) + grad.square().sum(-1)
        alpha = torch.where(s2 > EPS, -1 / s2, torch.zeros_like(s2))

        def change(v):
            return torch.where(cnt < 20, torch.zeros_like(den), divergence(v).clamp(min=0))
        adv = change(v)
        kv = torch.where(adv > 0, 0.5 * st["kappa_v"].double().clamp(min=-0.5) / dt, 0 * adv)
        v = push(v, kv)
        k, it = change(v) * alpha / dt, 0
        while True:
            v = push(v, k)
            kv = kv + k
            adv = change(v)
            k, it = adv * alpha / dt, it + 1
            if not ((adv.mean() > 1e-3 / dt or it < 1) and it < 100):
                break
        kv = kv * dt
        v = v + dt * _viscosity(K, n, i, j, d, gw / K.vol, x, v, rho, bodies)

        def advected(v):
            return (den + dt * divergence(v)).clamp(min=1)
        kp = torch.where(advected(v) > 1, 0.5 * st["kappa"].double().clamp(min=-0.00025) / dt ** 2,
                         0 * den)
        v = push(v, kp)
        k, it = (advected(v) - 1) * alpha / dt ** 2, 0
        while True:
            v = push(v, k)
            kp = kp + k
            adv = advected(v)
            k, it = (adv - 1) * alpha / dt ** 2, it + 1
            if not (((adv - 1).mean() > 1e-3 or it < 2) and it < 100):
                break
        extra = {"kappa": kp * dt ** 2, "kappa_v": kv}
        xn = x + dt * v
    else:
        v = v + dt * _viscosity(K, n, i, j, d, gw / K.vol, x, v, rho, bodies)
        last = 0.5 * st["pressure"].double()
        it = 0
        if case["method"] == "ii":
            dii = -grad * (DENSITY0 / rho ** 2)[:, None]
            dji = (DENSITY0 * K.vol / rho[i] ** 2)[:, None] * gw / K.vol
            adv = den + dt * divergence(v)
            aii = _sum(n, i, ((dii[i] - dji) * gw).sum(-1))
            for b in bodies:
                t = DENSITY0 / rho[b.i] ** 2
                aii.index_add_(0, b.i, ((dii[b.i] - t[:, None] * b.gw) * b.gw).sum(-1))
            aii = aii * DENSITY0
            while True:
                dp = -DENSITY0 * _sum(n, i, (last / rho ** 2)[j][:, None] * gw)
                s = _sum(n, i, ((dp[i] - dii[j] * last[j][:, None] -
                                 (dp[j] - dji * last[i][:, None])) * gw).sum(-1))
                for b in bodies:
                    s.index_add_(0, b.i, (dp[b.i] * b.gw).sum(-1))
                s, term, denom = s * DENSITY0, 1 - adv, aii * dt ** 2
                p = torch.where(denom.abs() > 1e-9,
                                (last / 3 + 2 / 3 / denom * (term - dt ** 2 * s)).clamp(min=0),
                                0 * last)
                err = torch.where(p == 0, 0 * p, denom * p + s * dt ** 2 - term)
                last, it = p, it + 1
                if not ((err.mean() > 1e-3 or it < 2) and it < 100):
                    break
        else:
            eps = 0.01 * K.h ** 2
            c = ((rho[i] + rho[j]) / (rho[i] * rho[j]) / (d.square().sum(-1) + eps) *
                 (d * gw).sum(-1))
            adv = den + dt * divergence(v)
            diag = _sum(n, i, c)
            for b in bodies:
                sep = x[b.i] - b.at
                diag.index_add_(0, b.i, (rho[b.i] + DENSITY0) / (rho[b.i] * DENSITY0) /
                                (sep.square().sum(-1) + eps) * (sep * b.gw).sum(-1))
            diag = diag * DENSITY0
            while True:
                off = -DENSITY0 * _sum(n, i, c * last[j])
                term, denom = 1 - adv, diag * dt ** 2
                p = torch.where(denom.abs() > 1e-9,
                                (last / 3 + 2 / 3 * (term / denom - off / diag)).clamp(min=0),
                                0 * last)
                err = torch.where(p == 0, 0 * p, denom * p + off * dt ** 2 - term)
                last, it = p, it + 1
                if not ((err.mean() > 1e-3 or it < 2) and it < 100):
                    break
        dp = last / rho ** 2
        a = -K.mass / K.vol * _sum(n, i, (dp[i] + dp[j])[:, None] * gw)
        for b in bodies:
            t = (DENSITY0 * dp[b.i])[:, None] * b.gw
            b.push(K.mass * t, b.at)
            a.index_add_(0, b.i, -t)
        v = v + dt * DENSITY0 * a
        xn = x + dt * v
        extra = {"pressure": last}
    if period:
        y = xn[:, 1]
        xn[:, 1] = torch.where(y >= period / 2, y - period,
                               torch.where(y < -period / 2, y + period, y))
    out = {"x": xn, "v": v, "density": rho, **extra}
    if len(bodies) > 1:
        moved = [b.advance(dt) for b in bodies[1:]]
        out["rigid_pose"] = torch.stack([m[0] for m in moved]).cpu().numpy()
        out["rigid_velocity"] = torch.stack([m[1] for m in moved]).cpu().numpy()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        return _exact_step(case, seed)
    if kind == "batch":
        parts = [_exact_step(c, c["seed"]) for c in _batch_cases(case, seed)]
        return {k: torch.cat([p[k] for p in parts])
                for k in ("x", "v", "density", "kappa", "kappa_v")}
    f32 = case["dtype"] == "f32"
    K = _Kernel(case["radius"], f32)
    if kind == "volume":
        spec = _volume_body(case, seed)
        dtype = _np_dtype(case)
        spec = dict(spec, params=[float(dtype(t)) for t in spec["params"]])
        dist = None
        if case["grid"]:
            dist = _body_distance(_volume_body(case, seed), _node_positions(
                *_body_grid(spec, K.h, dtype))).to(_real(case)).double()
        return _volume_map(spec, K, dtype, dist)
    inp = _sample_inputs(case, seed)
    x, v, rho = inp["x"], inp["v"].double(), inp["rho"].double()
    n = x.shape[0]
    if kind == "neighbors":
        i, j, d = _pairs(x, x, K.h)
        den = K.vol * K.k + K.vol * _sum(n, i, K.W(d.square().sum(-1).sqrt()))
        # the list's order: ascending cell of j, then j
        cell = (x / torch.tensor(K.h, dtype=x.dtype, device=x.device)).floor().long()
        key = ((cell[:, 0] << 20) + cell[:, 1] << 20) + cell[:, 2]
        o = torch.argsort(j, stable=True)
        o = o[torch.argsort(key[j[o]], stable=True)]
        o = o[torch.argsort(i[o], stable=True)]
        count = torch.bincount(i, minlength=n)
        slot = torch.arange(i.shape[0], device="cuda") - (count.cumsum(0) - count)[i]
        disp = torch.zeros((n, 64, 3), dtype=torch.float64, device="cuda")
        disp[i, slot] = d[o]
        index = torch.zeros((n, 64), dtype=torch.int64, device="cuda")
        index[i, slot] = j[o]
        return {"density": den * DENSITY0, "count": count, "displacement": disp, "index": index}
    s = inp["s"]
    ns = s.shape[0]
    # particle k is left out of sample k's sums, as the sampling defines it
    i, j, d = _pairs(s, x, K.h)
    w = K.W(d.square().sum(-1).sqrt())
    den = DENSITY0 * K.vol * _sum(ns, i, w)
    mw = (K.mass / rho)[j]
    vel = _sum(ns, i, (mw * w)[:, None] * v[j])
    vort = _sum(ns, i, mw[:, None] * torch.linalg.cross(v[j] - vel[i], K.grad(d)))
    return {"density": den, "v": vel, "vorticity": vort}
