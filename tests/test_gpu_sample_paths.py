"""The two sampling kernels: the list kernel and the list-free one (which also
serves pellets) give the same bits, for bodies, quantities, both types and
periodic grids."""
import numpy as np
import pytest
import torch

from alluvion_b200 import _capi, scenes

pytestmark = pytest.mark.gpu

LIST_FREE = 1 << 26  # a neighbor capacity that the list kernel does not serve
OUTPUTS = dict(density=1, position_density=1, quantity=3, v=3, vorticity=3)


def _dev(a, dtype):
    return torch.from_numpy(np.ascontiguousarray(a, dtype)).cuda()


def _sample(engine, cn, cni, x, rho, v, sx, q=None, rigid=None, bnd=None, wrap=0.0,
            outputs=("density", "v", "vorticity")):
    """Status and host outputs of one call; arrays are device tensors."""
    f64 = x.dtype == torch.float64
    req = (_capi.SampleF64 if f64 else _capi.SampleF32)()
    p = lambda t: _capi.ptr(t).value
    out = {k: torch.zeros((len(sx), OUTPUTS[k]), dtype=x.dtype, device="cuda") for k in outputs}
    req.sample_x, req.num_samples = p(sx), len(sx)
    req.particle_density, req.particle_v = p(rho), p(v)
    if q is not None:
        req.particle_quantity, req.quantity_dim = p(q), q.shape[1]
    if bnd is not None:
        req.sample_boundary, req.sample_boundary_kernel = p(bnd[0]), p(bnd[1])
    if wrap:
        req.wrap_y, req.wrap_length = 1, wrap
    for k, t in out.items():
        setattr(req, "sample_" + k, p(t))
    fn = getattr(_capi.lib(), "al_sample_fluid_f64" if f64 else "al_sample_fluid_f32")
    status = fn(engine.handle, _capi.ptr(cn), _capi.ptr(cni), _capi.ptr(x), len(x),
                _capi.ptr(rigid) if rigid is not None else None, _capi.ptr(req), None)
    return status, {k: t.cpu().numpy() for k, t in out.items()}


def _cloud(dtype, n, extent, seed):
    rng = np.random.default_rng(seed)
    x = rng.random((n, 3)) * extent
    return (_dev(x, dtype), _dev(1000 + 50 * rng.random(n), dtype),
            _dev(rng.normal(0, 1, (n, 3)), dtype), _dev(rng.normal(0, 1, (n, 3)), dtype))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("periodic", [False, True])
def test_list_and_list_free_sums_agree(engine, dtype, periodic):
    cn = scenes.make_const(dtype, 0.01)
    h = float(cn.kernel_radius)
    extent = np.array([5.3, 6.0, 4.7]) * h
    x, rho, v, q = _cloud(dtype, 2500, extent, 5)
    sx = _dev(np.random.default_rng(6).random((3001, 3)) * extent, dtype)
    got = []
    for cap in (128, LIST_FREE):
        cni = scenes.make_consti((0, 0, 0), extent, h, 0, max_num_neighbors_per_particle=cap)
        if periodic:
            cni.grid_offset[1], cni.grid_res[1] = 0, 6
        got.append(_sample(engine, cn, cni, x, rho, v, sx, q, wrap=6 * h if periodic else 0.0,
                           outputs=OUTPUTS))
    assert got[0][0] == got[1][0] == 0
    for k in OUTPUTS:
        assert np.array_equal(got[0][1][k], got[1][1][k]), k
    assert np.abs(got[0][1]["vorticity"]).max() > 0


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_list_and_list_free_sums_agree_with_bodies(engine, dtype):
    """A moving, spinning sphere above the block: the body terms of both."""
    sphere = dict(shape=_capi.SHAPE_SPHERE, params=[0.04], sign=1.0, resolution=16,
                  use_distance_grid=True, mass=0.0, x=(0.12, 0.255, 0.11), v=(0.3, -0.1, 0.2),
                  omega=(1.0, 2.0, -0.5))
    sc = scenes.dam_break(engine, dtype, (10, 10, 10), 0.01, (0.3, 0.3, 0.3), [sphere], seed=3,
                          volume_resolution=16)
    sc.step("df", scenes.solver_params(integrate_rigids=0), 2e-4)
    rng = np.random.default_rng(8)
    sx = _dev(rng.random((2000, 3)) * 0.3, dtype)
    q = _dev(rng.normal(0, 1, (sc.n, 3)), dtype)
    bnd = [torch.zeros(sc.num_boundaries, len(sx), 4, dtype=sx.dtype, device="cuda")
           for _ in range(2)]
    fn = getattr(_capi.lib(), "al_compute_particle_boundary_" +
                 ("f64" if dtype == np.float64 else "f32"))
    _capi.check(fn(engine.handle, _capi.ptr(sc.cn), sc.num_boundaries, _capi.ptr(sc.bodies),
                   _capi.ptr(sc.rigid), _capi.ptr(sx), len(sx), _capi.ptr(bnd[0]),
                   _capi.ptr(bnd[1]), None), "boundary")
    assert float(bnd[1].abs().max()) > 0
    got = []
    for cap in (64, LIST_FREE):
        sc.cni.max_num_neighbors_per_particle = cap
        got.append(_sample(engine, sc.cn, sc.cni, sc.x, sc.density, sc.v, sx, q, sc.rigid, bnd,
                           outputs=OUTPUTS))
    assert got[0][0] == got[1][0] == 0
    for k in OUTPUTS:
        assert np.array_equal(got[0][1][k], got[1][1][k]), k


@pytest.mark.parametrize("cap", [1024, 1767, 1771, 1 << 18, 1 << 20])
@pytest.mark.parametrize("samples", [1, 5000, 65281, 65282])
def test_list_scratch_stays_within_256_mib(engine, cap, samples):
    """A call whose lists do not fit 2^26 entries runs in launches of at least one
    block per SM, or list-free; results equal the list-free kernel's and the
    device memory a call takes stays below 256 MiB and the sorted copies."""
    dtype = np.float32
    cn = scenes.make_const(dtype, 0.01)
    h = float(cn.kernel_radius)
    extent = np.array([4.3, 5.0, 4.7]) * h
    x, rho, v, _ = _cloud(dtype, 1200, extent, 9)
    sx = _dev(np.random.default_rng(10).random((samples, 3)) * extent, dtype)
    per = (cap + 1 + 3) // 4 * 4
    most = (1 << 26) // per
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if samples <= most:
        launches = 2  # gather, sums
    elif most >= sms * 256:
        launches = 1 + -(-samples // (most // 256 * 256))
    else:
        launches = 2  # densities and velocities, vorticity
    cni = scenes.make_consti((0, 0, 0), extent, h, 0, max_num_particles_per_cell=512,
                             max_num_neighbors_per_particle=LIST_FREE)
    _, want = _sample(engine, cn, cni, x, rho, v, sx)
    cni.max_num_neighbors_per_particle = cap
    own = _capi.Engine(0)
    try:
        tiny = _sample(own, cn, scenes.make_consti((0, 0, 0), extent, h, 0, 512, 64), x, rho, v,
                       sx[:1])  # the context's own allocations come first
        assert tiny[0] == 0
        sorts = own.launch_count()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        status, got = _sample(own, cn, cni, x, rho, v, sx)
        torch.cuda.synchronize()
        taken = free - torch.cuda.mem_get_info()[0]
        count = own.launch_count() - sorts
    finally:
        own.close()
    assert status == 0
    for k in want:
        assert np.array_equal(got[k], want[k]), k
    assert taken <= (256 + 32) << 20
    assert count == sorts - 2 + launches  # the two sorts and the sums


def _reference(x, s, cn, cni, wrap):
    """Density sums of every sample in canonical order over its first cap
    neighbors (float32 tests, float64 sums), and the accepted counts."""
    f = np.float32
    h, cap = f(cn.kernel_radius), cni.max_num_neighbors_per_particle
    off, res = list(cni.grid_offset), list(cni.grid_res)
    cell = np.floor(x / h).astype(np.int64) - off
    at = np.floor(s / h).astype(np.int64) - off
    order = np.lexsort((np.arange(len(x)), cell[:, 2], cell[:, 1], cell[:, 0]))
    hd = float(h)
    dens, count = np.zeros(len(s)), np.zeros(len(s), int)
    for i in range(len(s)):
        near = []
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                cy = at[i, 1] + dy
                if wrap:
                    cy = cy - res[1] if cy >= res[1] else cy + res[1] if cy < 0 else cy
                m = ((cell[order, 0] == at[i, 0] + dx) & (cell[order, 1] == cy) &
                     (np.abs(cell[order, 2] - at[i, 2]) <= 1))
                j = order[m]
                d = (s[i] - x[j]).astype(f)
                if wrap:
                    y = d[:, 1]
                    half, full = f(wrap) * f(0.5), f(wrap)
                    d[:, 1] = np.where(y >= half, y - full, np.where(y < -half, y + full, y))
                d2 = (d * d)[:, 0] + (d * d)[:, 1] + (d * d)[:, 2]
                ok = (d2 < h * h) & (j != i)
                near += list(np.sqrt((d[ok].astype(float) ** 2).sum(1)) / hd)
        count[i] = len(near)
        q = np.array(near[:cap])
        w = np.where(q <= 0.5, (6 * q - 6) * q * q + 1, 2 * (1 - q) ** 3)
        dens[i] = w.sum() * 8 / np.pi / hd ** 3 * float(cn.particle_vol) * float(cn.density0)
    return dens, count


# float32 sums of up to 200 positive terms with a few rounded operations each:
# (200 + 20) * 2^-24
SUM_BOUND = 1.4e-5


@pytest.mark.parametrize("cells", [1, 2, 3, 4])
def test_capacity_of_narrow_periodic_grids(engine, cells):
    """Periodic grids of one or two cells along y walk a row more than once, and
    meet the sample's own particle as often: capacities of the accepted count,
    and one less, with samples on the particles."""
    cn = scenes.make_const(np.float32, 0.01)
    h = float(np.float32(cn.kernel_radius))
    extent = np.array([2.0, cells, 2.0]) * h
    x, rho, v, _ = _cloud(np.float32, 60, extent, cells)
    xs = x.cpu().numpy()
    for spare in (0, -1):
        cni = scenes.make_consti((0, 0, 0), extent, h, 0, max_num_particles_per_cell=512)
        cni.grid_offset[1], cni.grid_res[1] = 0, cells
        cni.max_num_neighbors_per_particle = 10000
        _, count = _reference(xs, xs, cn, cni, cells * h)
        cni.max_num_neighbors_per_particle = cap = int(count.max()) + spare
        want, _ = _reference(xs, xs, cn, cni, cells * h)
        status, got = _sample(engine, cn, cni, x, rho, v, x, wrap=cells * h)
        assert status == (_capi.AL_ERR_NEIGHBOR_OVERFLOW if spare else 0)
        np.testing.assert_allclose(got["density"][:, 0], want, rtol=SUM_BOUND)


@pytest.mark.parametrize("own", [False, True])
@pytest.mark.parametrize("spare", [-2, -1, 0, 1])
def test_capacity_edges(engine, own, spare):
    """Forty particles within h of every sample: capacities from two below the
    accepted count to one above it, for samples that share an index with one of
    the forty (own; it is anywhere in the list, the first and the last entry
    among them) and for samples that do not."""
    cn = scenes.make_const(np.float32, 0.01)
    h = float(np.float32(cn.kernel_radius))
    rng = np.random.default_rng(12)
    xs = (1.5 * h + 0.25 * h * (2 * rng.random((40, 3)) - 1)).astype(np.float32)
    ss = (1.5 * h + 0.1 * h * (2 * rng.random((40, 3)) - 1)).astype(np.float32)
    if not own:  # samples 0..39 elsewhere, the next ones among the particles
        ss = np.concatenate([np.full((40, 3), 5.5 * h, np.float32), ss])
    x, sx = _dev(xs, np.float32), _dev(ss, np.float32)
    rho = torch.full((40,), 1000.0, device="cuda")
    cni = scenes.make_consti((0, 0, 0), (6 * h,) * 3, h, 0)
    accepted = 39 if own else 40
    cni.max_num_neighbors_per_particle = accepted + spare
    want, count = _reference(xs, ss, cn, cni, 0.0)
    assert set(count) == ({39} if own else {0, 40})
    status, got = _sample(engine, cn, cni, x, rho, torch.zeros_like(x), sx,
                          outputs=("density", "v"))
    assert status == (_capi.AL_ERR_NEIGHBOR_OVERFLOW if spare < 0 else 0)
    np.testing.assert_allclose(got["density"][:, 0], want, rtol=SUM_BOUND)


@pytest.mark.parametrize("frame", [0.0, 100.0])
def test_velocity_and_vorticity_in_a_moving_frame(engine, frame):
    """Float sums against 64-bit ones, at rest and with a large common velocity;
    the vorticity against the sample's velocity that the call returned.  Bound:
    one rounding per term and sum and about 20 in the kernel's factors, on the
    sum of the terms' magnitudes (the gradient's by its maximum over q)."""
    cn = scenes.make_const(np.float32, 0.01)
    h = float(np.float32(cn.kernel_radius))
    extent = np.array([4.3, 5.0, 4.7]) * h
    x, rho, v, _ = _cloud(np.float32, 1200, extent, 13)
    v += frame
    sx = _dev(np.random.default_rng(14).random((400, 3)) * extent, np.float32)
    cni = scenes.make_consti((0, 0, 0), extent, h, 0, max_num_neighbors_per_particle=128)
    status, got = _sample(engine, cn, cni, x, rho, v, sx)
    assert status == 0
    xs, vs, rs, ps = (t.cpu().numpy().astype(float) for t in (x, v, rho, sx))
    mass = float(cn.particle_mass)
    k, l = 8 / np.pi / h ** 3, 48 / np.pi / h ** 4
    eps = 2.0 ** -23
    for i in range(len(ps)):
        d = ps[i] - xs
        r = np.sqrt((d ** 2).sum(1))
        near = (r < h) & (np.arange(len(xs)) != i)
        d, r, mr, vj = d[near], r[near], (mass / rs)[near], vs[near]
        q = r / h
        w = k * np.where(q <= 0.5, (6 * q - 6) * q * q + 1, 2 * (1 - q) ** 3)
        s = l * np.where(q <= 0.5, (3 * q - 2) / h, -(1 - q) ** 2 / r)
        n = near.sum() + 20
        want = ((mr * w)[:, None] * vj).sum(0)
        assert np.abs(got["v"][i] - want).max() <= n * eps * (mr * w @ np.abs(vj)).max()
        rel = vj - got["v"][i].astype(float)
        want = (mr[:, None] * np.cross(rel, s[:, None] * d)).sum(0)
        scale = (mr * np.sqrt((rel ** 2).sum(1))).sum() * l / 3  # |grad W| <= l / 3
        assert np.abs(got["vorticity"][i] - want).max() <= n * eps * scale


@pytest.mark.parametrize("radius", [0.01, 0.0037, 0.07, 0.1])
def test_double_kernel_is_as_exact_as_ieee_operations(engine, radius):
    """Densities of samples with one neighbor each, against 80-bit values: no
    further off (root mean square) than numpy's square root and divisions in
    double.  (The device contracts products and sums, which leaves it 3 % below;
    1 / h rounded once and |d| by a reciprocal square root put it 1-5 % above.)"""
    cn = scenes.make_const(np.float64, radius)
    h = float(cn.kernel_radius)
    rng = np.random.default_rng(2)
    g, lag = 24, 7
    n = g ** 3
    cells = np.stack(np.meshgrid(*[np.arange(g)] * 3, indexing="ij"), -1).reshape(-1, 3)
    xs = 4 * h * cells + 2 * h + 0.1 * h * rng.random((n, 3))
    away = rng.normal(size=(n, 3))
    away *= 0.98 * h * rng.random((n, 1)) / np.linalg.norm(away, axis=1)[:, None]
    ss = np.roll(xs + away, lag, 0)  # sample k beside particle k - lag, not its own
    x, sx = _dev(xs, np.float64), _dev(ss, np.float64)
    cni = scenes.make_consti((0, 0, 0), xs.max(0) + h, h, 0)
    rho = torch.full((n,), 1000.0, dtype=torch.float64, device="cuda")
    status, got = _sample(engine, cn, cni, x, rho, torch.zeros_like(x), sx,
                          outputs=("density", "v"))
    assert status == 0

    def density(t):
        d = ss.astype(t) - np.roll(xs, lag, 0).astype(t)
        r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
        q, q2 = np.sqrt(r2) / t(h), r2 / t(cn.kernel_radius_sqr)
        w = np.where(q <= 0.5, (6 * q - 6) * q2 + 1, 2 * (1 - q) * (1 - q) * (1 - q))
        return t(cn.density0) * (t(cn.particle_vol) * (w * t(cn.cubic_kernel_k)))

    exact = density(np.longdouble)
    rms = lambda a: float(np.sqrt(((a - exact) ** 2).mean()))
    assert rms(got["density"][:, 0]) <= rms(density(np.float64))
