"""Sizes at which the launch rules of the kernels change branch, against the
oracle (float64, 1e-12 relative: the parity tests' bound for one evaluation)."""
import numpy as np
import pytest

from ins2d_b200 import api
from oracle import ins2d_ref as R
from tests.cases_common import BC_COMBOS, grid_stretched, smooth_bc

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.max(np.abs(np.asarray(a) - np.asarray(b))) / np.max(np.abs(b)))


# walker runs of 2, 4, .. 32 rows per thread, with and without interior tiles,
# odd row lengths (global-memory walkers) and even ones (tiled walkers)
@pytest.mark.parametrize("bc", ["cavity", "channel", "per_x_walls"])
@pytest.mark.parametrize("shape", [(3, 2), (63, 31), (65, 33), (257, 130), (770, 515), (1025, 1024)])
def test_walker_runs(shape, bc):
    uBC, vBC = smooth_bc(3)
    kw = dict(Re=50.0, uBC=uBC, vBC=vBC)
    x, y = grid_stretched(shape[0], 0.0, 2.0), grid_stretched(shape[1])
    m = api.Options(x, y, BC_COMBOS[bc], poisson=4, precond="jacobi", **kw)
    o = R.make_options(x, y, BC_COMBOS[bc], poisson=4, **kw)
    rng = np.random.default_rng(shape[0])
    V, p = rng.standard_normal(m.NV), rng.standard_normal(m.Np)
    mr, F = m.F(V, None, p)
    mr_ref, F_ref = R.F(V, V, p, 0.0, o)
    assert _rel(F, F_ref) < 1e-12 and abs(mr - mr_ref) < 1e-12 * mr_ref
    m.close()


# one-cluster solves: slices of 1 .. 16 columns, empty blocks, both mode
# directions, cyclic systems, the basis in shared memory (up to about 112
# modes) and read through L1; 129: the multi-launch path.  The bound is the
# stopping rule's, 1e-12 relative, with a factor 2 for the residual's rounding.
@pytest.mark.parametrize("combo", ["cavity", "channel", "per_x_walls", "per_y_open", "periodic"])
@pytest.mark.parametrize("shape", [(4, 3), (9, 16), (16, 9), (64, 64), (65, 40), (112, 112), (113, 120), (128, 128),
                                   (128, 7), (7, 128), (129, 128)])
def test_small_grid_solve(shape, combo):
    bc = BC_COMBOS[combo]
    x, y = grid_stretched(shape[0], 0.0, 1.7), grid_stretched(shape[1], -0.5, 0.5, beta=1.2)
    m = api.Options(x, y, bc, poisson=4, CG_acc=1e-12, CG_maxit=50, precond="fdm")
    o = R.make_options(x, y, bc, poisson=1)
    M, A = o.discretization.M, o.discretization.A
    f = M @ np.random.default_rng(5).standard_normal(o.grid.NV)
    dp, st = m.pressure_poisson(f, return_stats=True)
    assert np.linalg.norm(A @ dp - f) <= 2e-12 * np.linalg.norm(f) and st["iters"] <= 4
    assert np.all(m.pressure_poisson(np.zeros(m.Np)) == 0.0)
    # the divergence formed inside the solve: one host-driven step and the
    # same step in a captured run against the oracle's
    V = R.initial_projection(0.3 * np.random.default_rng(6).standard_normal(o.grid.NV), 0.0, o)
    ref, pref = R.time_ERK(V, np.zeros(m.Np), 0.0, 1e-3, o)
    V1, p1 = m.time_ERK(V, np.zeros(m.Np), 0.0, 1e-3)
    assert _rel(V1, ref) < 1e-10
    ref, pref = R.time_ERK(ref, pref, 1e-3, 1e-3, o)
    assert _rel(m.time_ERK(V, np.zeros(m.Np), 0.0, 1e-3, nsteps=2)[0], ref) < 1e-10
    m.close()


# line transforms: every radix and leftover, primes by direct sums (up to 31)
# and by Bluestein's algorithm (37 and more, up to the longest length), odd
# lengths, one side a compile-time power of two; right-hand sides given, and
# formed from a velocity inside the first pass (FP64 and FP32 stages); (256, 256) to
# (4096, 32) take a quarter, half and all of the columns a block can hold, then
# the largest whole solve in one block and the first in three kernels, and lines
# of 3 by 500
@pytest.mark.parametrize("shape", [(2, 3), (6, 2), (12, 10), (40, 32), (31, 29), (49, 37), (125, 343), (74, 961), (64, 1009),
                                   (2039, 64), (2047, 17), (24, 2039), (1000, 600), (1536, 640), (375, 2000), (256, 256), (2048, 128),
                                   (4096, 32), (45, 40), (40, 46), (3, 500)])
def test_line_transforms(shape):
    nx, ny = shape
    x, y = np.arange(nx + 1) / nx * 1.5, np.arange(ny + 1) / ny
    bc = BC_COMBOS["periodic"]
    m = api.Options(x, y, bc, poisson=6)
    rng = np.random.default_rng(nx)
    f = rng.standard_normal((ny, nx))
    f -= f.mean()
    J, I = np.arange(ny)[:, None], np.arange(nx)[None, :]
    dx, dy = x[1], y[1]
    a = 4 * dx * dy * (np.sin(np.pi * I / nx) ** 2 / dx ** 2 + np.sin(np.pi * J / ny) ** 2 / dy ** 2)
    a[0, 0] = 1.0
    ref = np.real(np.fft.ifft2(-np.fft.fft2(f) / a)).ravel()
    assert _rel(m.pressure_poisson(f.ravel()), ref) < 1e-12
    assert np.all(m.pressure_poisson(np.zeros(nx * ny)) == 0.0)
    if min(shape) < 12 or max(shape) > 1000:
        return
    o = R.make_options(x, y, bc, poisson=6, Re=100.0)
    V = R.initial_projection(rng.standard_normal(o.grid.NV), 0.0, o)
    ref, pref = R.time_ERK(V, np.zeros(m.Np), 0.0, 1e-4, o)
    m = api.Options(x, y, bc, poisson=6, Re=100.0)
    V1, p1 = m.time_ERK(V, np.zeros(m.Np), 0.0, 1e-4)
    assert _rel(V1, ref) < 1e-11 and _rel(p1, pref) < 1e-9
    m = api.Options(x, y, bc, poisson=6, Re=100.0, precision="fp32")
    assert _rel(m.time_ERK(V, np.zeros(m.Np), 0.0, 1e-4)[0], ref) < 1e-5


# the network's layers and weight gradients: tile edges of 62, 64 and 16, strips
# of 128 columns (one row, one column over, several strips per block), one
# column or row left over, several fields; the learned tests' bounds
@pytest.mark.parametrize("path", ["tcgen05", "mma_sync"])
@pytest.mark.parametrize("shape", [(1, 1, 62), (1, 16, 63), (2, 17, 64), (1, 15, 65), (3, 33, 124), (1, 129, 130),
                                   (1, 1, 96), (2, 3, 128), (1, 40, 200), (300, 5, 97), (2, 150, 257)])
def test_network_tiles(shape, path):
    from oracle import cnn_ref as N
    from tests import test_gpu_learned as L
    net, w, scale = L._net(seed=11, scale=0.8, path=path)
    inp, tgt, ti, tt = L._inputs(9, *shape)
    acts = L._check_layers(net, w, scale, inp, net.forward(ti).cpu().numpy())
    loss, g = net.loss_grad(ti, tt)
    loss_ref, g_ref = N.loss_grad(w, scale, inp, tgt, bf16_mode=True, acts=acts)
    assert abs(loss - loss_ref) / loss_ref < 1e-5
    bounds = [0, N.OFF_WM] + [N.OFF_WM + (k + 1) * N.SZ_WM for k in range(N.NMID)] + [N.NPARAM]
    for a, b in zip(bounds[:-1], bounds[1:]):
        assert L._rel(g[a:b], g_ref[a:b]) < 1e-2, (a, b)
    assert L._rel(g[N.OFF_W6:], g_ref[N.OFF_W6:]) < 1e-5


# F's maximum and the conservation sums, written to the host by the last block
# of the last launch: no interior tile, interior and boundary tiles, interior
# tiles only; a later call's smaller maximum.  Sums of n terms: n rounding
# errors of the sum of their sizes at the most, far fewer in blocks of 256
@pytest.mark.parametrize("shape,bc", [((3, 2), "cavity"), ((64, 32), "periodic"), ((128, 64), "periodic"),
                                      ((300, 260), "cavity"), ((257, 321), "channel"), ((320, 96), "per_x_walls")])
def test_results_to_host(shape, bc):
    uBC, vBC = smooth_bc(3)
    kw = dict(Re=50.0) if bc == "periodic" else dict(Re=50.0, uBC=uBC, vBC=vBC)
    x, y = np.linspace(0.0, 2.0, shape[0] + 1), np.linspace(0.0, 1.0, shape[1] + 1)
    m = api.Options(x, y, BC_COMBOS[bc], poisson=6 if bc == "periodic" else 4, **kw)
    o = R.make_options(x, y, BC_COMBOS[bc], poisson=6 if bc == "periodic" else 4, **kw)
    rng = np.random.default_rng(shape[1])
    for scale in (1.0, 1e-2):
        V, p = scale * rng.standard_normal(m.NV), scale * rng.standard_normal(m.Np)
        mr, F = m.F(V, None, p)
        mr_ref, F_ref = R.F(V, V, p, 0.0, o)
        assert _rel(F, F_ref) < 1e-12 and abs(mr - mr_ref) < 1e-12 * mr_ref
        got, ref = m.check_conservation(V, 0.0), R.check_conservation(V, 0.0, o)
        top = np.max(np.abs(V)) + 2.0  # and the boundary values
        assert abs(got[0] - ref[0]) < 1e-12 * top
        for a, b, s in zip(got[1:], ref[1:], (top, top, top * top)):
            assert abs(a - b) < 2.0 * 2e-13 * s
    m.close()


# the fast diagonalization's systems of two and four warps per row and its
# products' ragged tiles; the stopping rule with a factor 2 for the residual's
# rounding (at 1e-10: rows of 1000 cells round at about 1e-12)
@pytest.mark.parametrize("combo", ["cavity", "per_x_walls", "per_y_open"])
@pytest.mark.parametrize("shape", [(257, 20), (20, 512), (513, 20), (24, 1024), (1024, 33), (130, 129)])
def test_long_rows(shape, combo):
    bc = BC_COMBOS[combo]
    x, y = grid_stretched(shape[0], 0.0, 1.7), grid_stretched(shape[1], -0.5, 0.5, beta=1.2)
    m = api.Options(x, y, bc, poisson=4, CG_acc=1e-10, CG_maxit=50, precond="fdm")
    o = R.make_options(x, y, bc, poisson=1)
    f = o.discretization.M @ np.random.default_rng(5).standard_normal(o.grid.NV)
    dp, st = m.pressure_poisson(f, return_stats=True)
    assert np.linalg.norm(o.discretization.A @ dp - f) <= 2e-10 * np.linalg.norm(f) and st["iters"] <= 4
    assert np.all(m.pressure_poisson(np.zeros(m.Np)) == 0.0)
    m.close()


# ensembles of members below a tile, of a ring of boundary points only, and of
# several tiles, against their own runs (solver tolerance 1e-12 per solve)
def test_ensemble_edges():
    import ins2d_b200
    from ins2d_b200 import cases
    members = []
    for k, (nx, ny) in enumerate([(4, 3), (5, 40), (33, 31), (65, 200), (32, 32), (140, 6)]):
        kw = dict(Re=200.0, poisson=4, CG_acc=1e-12, CG_maxit=200, RK="RK44")
        if k % 2 == 0:
            kw.update(x=cases.tanh_grid(nx, 0.0, 1.0, 1.05), y=cases.tanh_grid(ny, 0.0, 1.0, 1.05),
                      BC=cases.BC_CAVITY, uBC=cases.lid_uBC(1.0, 1.0))
        else:
            kw.update(x=cases.tanh_grid(nx, 0.0, 4.0, 1.05), y=cases.tanh_grid(ny, -0.5, 0.5, 1.05),
                      BC=cases.BC_CHANNEL, uBC=cases.channel_uBC(lambda yy: 1 - 4 * np.asarray(yy) ** 2))
        members.append(kw)
    ens = ins2d_b200.Ensemble(members)
    ens.set_solver(0)
    singles, V0 = [], []
    for k, kw in enumerate(members):
        m = ins2d_b200.Options(**kw)
        V = np.zeros(m.NV)
        p = m.pressure_additional_solve(V, np.zeros(m.Np), 0.0)
        ens.set_state(k, V, p)
        singles.append(m)
        V0.append((V, p))
    ens.time_ERK(0.0, 1e-4, 4)
    for k, m in enumerate(singles):
        V, p = ens.get_state(k)
        Vs, ps = m.time_ERK(V0[k][0], V0[k][1], 0.0, 1e-4, nsteps=4)
        assert _rel(V, Vs) < 1e-9 and _rel(p, ps) < 1e-7, (k, _rel(V, Vs), _rel(p, ps))
