"""Edges of the step's and the sampling's kernels: list groups and packed
distance tests at ragged sizes, the two forms of the cell scan, large sample
capacities, solver loops of no iteration or several, unaligned list rows, the
boundary stop."""
import ctypes

import numpy as np
import pytest
import torch

from alluvion_b200 import _capi, scenes
from test_gpu_step import TOL, _close, _oracle_run, _scene

pytestmark = pytest.mark.gpu


def _cloud(n, h, cells, seed):
    """n float32 points in a few cells of side h (rows of many candidates)."""
    rng = np.random.default_rng(seed)
    return (rng.random((n, 3)) * np.asarray(cells) * h).astype(np.float32)


def _neighbors_numpy(x, h, cap):
    """Lists in canonical order: ascending cell, then index; float32 tests."""
    h = np.float32(h)
    cell = np.floor(x / h).astype(np.int64)
    key = (cell[:, 0] << 40) + (cell[:, 1] << 20) + cell[:, 2]
    order = np.lexsort((np.arange(len(x)), key))
    out = []
    for i in range(len(x)):
        d = x[i] - x[order]
        s = d * d
        near = (s[:, 0] + s[:, 1]) + s[:, 2] < h * h
        out.append([j for j in order[near] if j != i][:cap])
    return out


def _update(engine, cn, cni, x, cap, offset=0):
    n = len(x)
    xd = torch.from_numpy(x).cuda()
    density = torch.zeros(n, device="cuda")
    count = torch.zeros(n, dtype=torch.int32, device="cuda")
    store = torch.zeros(n * cap * 4 + 4, device="cuda")
    rows = store[offset:offset + n * cap * 4]
    status = _capi.lib().al_update_particle_neighbors_f32(
        engine.handle, _capi.ptr(cn), _capi.ptr(cni), _capi.ptr(xd), n, None, _capi.ptr(density),
        _capi.ptr(count), _capi.ptr(rows), None, None)
    _capi.check(status, "al_update_particle_neighbors_f32", allow=_capi.ANOMALY_STATUSES)
    rows = rows.cpu().numpy().reshape(n, cap, 4)
    return count.cpu().numpy(), rows, density.cpu().numpy()


@pytest.mark.parametrize("n", [1, 2, 5, 31, 32, 33, 63, 130, 257])
@pytest.mark.parametrize("cap", [1, 3, 4, 5, 64, 131])
@pytest.mark.parametrize("offset", [0, 1])
def test_lists_at_group_and_round_edges(engine, n, cap, offset):
    """Lists, counts and displacements exactly as a direct search finds them,
    whatever the row lengths, the list capacity and the alignment of the
    caller's rows (offset in floats)."""
    cn = scenes.make_const(np.float32, 0.01)
    h = float(cn.kernel_radius)
    x = _cloud(n, h, (2.3, 2.1, 3.7), seed=n)
    cni = scenes.make_consti((0, 0, 0), x.max(0), h, 0, max_num_particles_per_cell=512,
                             max_num_neighbors_per_particle=cap)
    count, rows, _ = _update(engine, cn, cni, x, cap, offset)
    want = _neighbors_numpy(x, h, cap)
    for i, w in enumerate(want):
        assert count[i] == len(w)
        assert rows[i, :len(w), 3].view(np.uint32).tolist() == [int(j) for j in w]
        assert np.array_equal(rows[i, :len(w), :3], x[i] - x[w].reshape(-1, 3))


@pytest.mark.parametrize("res", [(3, 5, 7), (64, 32, 64), (128, 128, 128), (256, 256, 160)])
def test_sort_over_few_and_many_scan_tiles(engine, res):
    """The cell scan's two-launch form serves up to 4,096 tiles of 2,048 cells,
    the three-launch form beyond (10.5 M cells): both give the canonical order."""
    cn = scenes.make_const(np.float32, 0.01)
    h = float(cn.kernel_radius)
    rng = np.random.default_rng(res[0])
    n = 5000
    x = ((0.01 + 0.98 * rng.random((n, 3))) * np.asarray(res) * h).astype(np.float32)
    cni = scenes.make_consti((0, 0, 0), (h, h, h), h, 0, max_num_particles_per_cell=n)
    for k in range(3):
        cni.grid_offset[k], cni.grid_res[k] = 0, res[k]
    xd = torch.from_numpy(x).cuda()
    cell = torch.zeros(n, dtype=torch.int32, device="cuda")
    perm = torch.zeros(n, dtype=torch.int32, device="cuda")
    start = torch.zeros(int(np.prod(res)) + 1, dtype=torch.int32, device="cuda")
    _capi.check(_capi.lib().al_grid_sort_f32(
        engine.handle, _capi.ptr(cn), _capi.ptr(cni), _capi.ptr(xd), n, _capi.ptr(cell),
        _capi.ptr(perm), _capi.ptr(start), None, None), "al_grid_sort_f32")
    c = np.floor(x / np.float32(h)).astype(np.int64)
    key = (c[:, 0] * res[1] + c[:, 1]) * res[2] + c[:, 2]
    assert np.array_equal(cell.cpu().numpy(), key)
    assert np.array_equal(perm.cpu().numpy(), np.lexsort((np.arange(n), key)))
    s = start.cpu().numpy()
    assert s[-1] == n and np.array_equal(np.diff(s), np.bincount(key, minlength=len(s) - 1))


@pytest.mark.parametrize("samples", [1, 255, 256, 257, 1500])
def test_samples_in_chunks(engine, samples):
    """A neighbor capacity whose lists would not fit the scratch (served by the
    list-free kernel) gives what lists give, bit for bit."""
    cn = scenes.make_const(np.float32, 0.01)
    h = float(cn.kernel_radius)
    x = scenes.fluid_block((12, 11, 10), (0, 0, 0), 0.01, np.float32, seed=1)
    rng = np.random.default_rng(samples)
    n = len(x)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    xd, vd = dev(x), dev(rng.normal(0, 1, (n, 3)))
    rho = dev(1000 + 20 * rng.random(n))
    sx = dev(rng.random((samples, 3)) * x.max(0))
    out = []
    for cap in (64, 1 << 18):
        cni = scenes.make_consti((0, 0, 0), x.max(0), h, 0, max_num_neighbors_per_particle=cap)
        den = torch.zeros(samples, device="cuda")
        vel, vort = (torch.zeros(samples, 3, device="cuda") for _ in range(2))
        req = _capi.SampleF32()
        req.sample_x, req.num_samples = _capi.ptr(sx).value, samples
        req.particle_density, req.particle_v = _capi.ptr(rho).value, _capi.ptr(vd).value
        req.sample_density, req.sample_v = _capi.ptr(den).value, _capi.ptr(vel).value
        req.sample_vorticity = _capi.ptr(vort).value
        _capi.check(_capi.lib().al_sample_fluid_f32(
            engine.handle, _capi.ptr(cn), _capi.ptr(cni), _capi.ptr(xd), n, None, _capi.ptr(req),
            None), "al_sample_fluid_f32")
        out.append([t.cpu().numpy() for t in (den, vel, vort)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert np.isfinite(out[0][2]).all()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("method,sp", [
    ("df", dict(max_divergence_solve=0)), ("df", dict(min_divergence_solve=3)),
    ("df", dict(enable_divergence_solve=0)), ("df", dict(max_density_solve=0)),
    ("ii", dict(max_density_solve=0)), ("ii", dict(min_density_solve=1, max_density_solve=1)),
    ("i", dict(max_density_solve=0)), ("i", dict(min_density_solve=1, max_density_solve=1)),
    ("i", dict(min_density_solve=4, max_density_solve=4))])
def test_loops_of_no_iteration_or_several(engine, dtype, method, sp):
    """The first divergence iteration runs before its loop and forms the
    viscosity sums; solves of no iteration, one and several agree with the
    oracle, eagerly and from the captured graph (same bounds as single steps)."""
    scene = _scene(engine, dtype)
    params = scenes.solver_params(**sp)
    ostate, _, odt, oreps = _oracle_run(scene, method, params, 1e-4, 4)
    dt, reps = 1e-4, []
    for _ in range(4):
        dt, rep = scene.step(method, params, dt)
        reps.append(rep)
    for r, o in zip(reps, oreps):
        assert r.num_density_solve == o.num_density_solve
        assert r.num_divergence_solve == o.num_divergence_solve
    g, tol = scene.state(), TOL[(dtype, 4)]
    assert dt == pytest.approx(odt, rel=tol["dt"])
    for key, bound in (("x", "x"), ("v", "v"), ("density", "density")):
        _close(g[key], ostate[key], tol[bound], key)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_boundary_stop_at_zero_cells_changes_nothing(engine, dtype):
    """A step that exports the dense boundary terms evaluates every pair, one that
    does not stops at map cells whose nodes are all 0: equal states, and as many
    active pairs as the dense terms have volumes."""
    out = []
    for dense in (False, True):
        sc = _scene(engine, dtype)
        nb = sc.num_boundaries
        terms = [torch.full((nb, sc.n, 4), -1.0, dtype=sc.tdtype, device="cuda")
                 for _ in range(2)]
        if dense:
            bufs = type(sc).fluid(sc, terms)
            sc.fluid = lambda: bufs
        dt = 1e-4
        for _ in range(3):
            dt, rep = sc.step("df", scenes.solver_params(), dt)
        out.append((dt, rep.num_active_boundary_pairs, sc.state(),
                    scenes.rigid_array(sc.dtype, [sc.rigid[b] for b in range(nb)])))
    (dt0, pairs0, a, rig0), (dt1, pairs1, b, rig1) = out
    volumes = terms[0][..., 3]
    assert pairs0 == pairs1 == int((volumes != 0).sum())
    assert 0 < pairs0 < volumes.numel()  # both kinds occur
    assert dt0 == dt1 and np.array_equal(rig0, rig1)
    for key in a:
        assert np.array_equal(a[key], b[key]), key
