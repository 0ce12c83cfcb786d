"""Behaviour at the edges of what the kernels accept."""
import functools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# A stage solve that does not converge leaves a member's velocity projected
# with the last field that did: none here, so the steps are the tableau's
# without a projection (p stays zero).  Rounding of a few evaluations: 1e-12.
@pytest.mark.parametrize("solver,nsteps", [(0, 1), (0, 3), (-1, 3)])
def test_unconverged_member_projection(solver, nsteps):
    import ins2d_b200
    from ins2d_b200 import cases
    from ins2d_b200.rk import getRKmethod
    from oracle import ins2d_ref as R
    members = [dict(x=cases.tanh_grid(nx, 0.0, 1.0, 1.05), y=cases.tanh_grid(ny, 0.0, 1.0, 1.05), BC=cases.BC_CAVITY,
                    uBC=cases.lid_uBC(0.0, 1.0), Re=100.0, poisson=4, CG_acc=1e-17, CG_maxit=1, RK="RK44")
               for nx, ny in [(33, 31), (20, 24), (70, 66)]]
    ens = ins2d_b200.Ensemble(members)
    ens.set_solver(solver)
    # at rest every right-hand side is zero: solved without a pass, dp = 0
    for m in range(3):
        o = ens.member(m)
        ens.set_state(m, np.zeros(o.NV), np.zeros(o.Np))
    ens.time_ERK(0.0, 1e-3, 2)
    dt, V0 = 1e-3, []
    for m in range(3):
        o = ens.member(m)
        V0.append(np.random.default_rng(m).standard_normal(o.NV))
        ens.set_state(m, V0[m], np.zeros(o.Np))
    with pytest.raises(ins2d_b200.Ins2dError) as ei:
        ens.time_ERK(0.0, dt, nsteps)
    assert ei.value.status == 2
    A, b, _ = getRKmethod("RK44")
    for m, kw in enumerate(members):
        o = R.make_options(kw["x"], kw["y"], kw["BC"], Re=kw["Re"], poisson=1, uBC=kw["uBC"])
        V = V0[m]
        for _ in range(nsteps):
            k, U = [], V
            for row in np.vstack([A[1:], b[None]]):
                k.append(o.grid.Om_inv * R.F(U, U, np.zeros(o.grid.Np), 0.0, o, nopressure=1)[1])
                U = V + dt * sum(a * q for a, q in zip(row, k))
            V = U
        Ve, pe = ens.get_state(m)
        assert np.max(np.abs(Ve - V)) <= 1e-12 * np.max(np.abs(V)), m
        assert np.all(pe == 0.0)


# A fast-diagonalization ensemble has one form of solve and times none: a first
# run in the tuned setting takes the steps of a second ensemble's with the form
# given, and its statistics count those solves only
def test_ensemble_without_tuning():
    import ins2d_b200
    from ins2d_b200 import ensembles
    states, ens = [], None
    for solver in (-1, 0):
        members = ensembles.random_members(3, seed=3, sizes=(24, 40), CG_acc=1e-12)
        ens = ins2d_b200.Ensemble(members)
        ens.set_solver(solver)
        for m in range(3):
            o = ens.member(m)
            ens.set_state(m, np.zeros(o.NV), np.zeros(o.Np))
        st = ens.time_ERK(0.0, 1e-4, 3)
        assert all(s["n_solves"] == 12 for s in st)
        shape = ens.solve_shape()
        assert shape["batched"] and all(v == 0.0 for v in shape["tuned_ms"].values())
        states.append([ens.get_state(m) for m in range(3)])
    for a, b in zip(*states):
        assert all(np.array_equal(p, q) for p, q in zip(a, b))


# Weights of two nonzero taps per output and per input channel: activations
# are whole numbers up to 64, gradients up to 16 times a power of two, so every
# value is exact in BF16 and every sum in FP32, and the device's result must
# equal the oracle's to the last bit.  Tiles of 62 to 128 columns, rows left
# over, several tiles per block, many small fields.
@functools.lru_cache(maxsize=1)
def _exact_case(shape):
    from oracle import cnn_ref as N
    rng = np.random.default_rng(shape[1])

    def signs(n):
        return rng.choice([-1.0, 1.0], n, p=[0.25, 0.75])

    W1, W6, Wm = np.zeros((N.C, N.TAPS)), np.zeros((N.TAPS, N.C)), []
    for c in range(N.C):
        W1[c, rng.choice(N.TAPS, 2, replace=False)] = signs(2)
    for _ in range(N.NMID):
        W = np.zeros((N.C, N.TAPS, N.C))
        for _ in range(2):
            W[np.arange(N.C), rng.integers(N.TAPS, size=N.C), rng.permutation(N.C)] += signs(N.C)
        Wm.append(W)
    W6[rng.integers(N.TAPS, size=N.C), np.arange(N.C)] = signs(N.C)
    w = N.join(W1, Wm, W6)
    inp = rng.integers(-1, 3, shape).astype(np.float32)
    y, acts = N.forward(w, 1.0, inp)
    tgt = (y - rng.integers(-1, 2, shape)).astype(np.float32)
    loss, g = N.loss_grad(w, 1.0, inp, tgt, acts=acts[1:])
    assert all(np.mean(q != 0.0) > 0.3 for q in [*N.split(g)[1], *N.split(g)[::2]])  # every layer takes part
    return w.astype(np.float32), inp, tgt, y, acts, loss, g


@pytest.mark.parametrize("shape", [(1, 8, 64), (2, 16, 32), (4, 64, 128), (2, 512, 256), (256, 8, 64)])
@pytest.mark.parametrize("path", ["tcgen05", "mma_sync"])
def test_network_exact_arithmetic(path, shape):
    import torch
    from ins2d_b200.learned import ConvNet
    w, inp, tgt, y, acts, loss, g = _exact_case(shape)
    net = ConvNet(device=0, seed=1)
    net.set_path(path)
    net.set_params(w, 1.0)
    ti, tt = torch.from_numpy(inp).cuda(), torch.from_numpy(tgt).cuda()
    assert np.array_equal(net.forward(ti).cpu().numpy(), y)
    for l in range(1, 6):
        assert np.array_equal(net.activations(l, y.size).reshape(shape + (32,)), acts[l]), l
    loss_d, g_d = net.loss_grad(ti, tt)
    assert loss_d == loss and np.array_equal(np.asarray(g_d, dtype=np.float64), g)


# The output layer's sums with activations that overflowed to infinity, and
# with weights beyond BF16's largest value: infinite where one sign of infinity
# reaches a pixel, NaN where both do, else FP32 sums (the learned tests' bound)
@pytest.mark.parametrize("path", ["tcgen05", "mma_sync"])
@pytest.mark.parametrize("what", ["positive", "mixed", "weight"])
@pytest.mark.parametrize("shape", [(2, 16, 32), (1, 9, 140), (1, 64, 16)])
def test_output_layer_overflow(shape, what, path):
    import torch
    from ins2d_b200.learned import ConvNet
    from oracle import cnn_ref as N
    w = _exact_case((2, 16, 32))[0].copy()
    rng = np.random.default_rng(shape[2])
    W6 = np.exp2(-100.0) * rng.uniform(0.5, 1.5, N.K)
    if what == "mixed":
        W6 *= rng.choice([-1.0, 1.0], N.K)
    # layer 5's whole numbers by 2^124: 16 and more are infinite
    w[N.OFF_W6 - N.SZ_WM:N.OFF_W6] *= np.float32(2.0 ** (-30 if what == "weight" else 124))
    if what == "weight":
        W6[rng.integers(N.K, size=4)] = 3.4e38
    w[N.OFF_W6:] = W6
    net = ConvNet(device=0, seed=1)
    net.set_path(path)
    net.set_params(w, 1.0)
    inp = rng.integers(-1, 3, shape).astype(np.float32)
    y = net.forward(torch.from_numpy(inp).cuda()).cpu().numpy().astype(np.float64)
    a5 = net.activations(5, y.size).reshape(shape + (N.C,)).astype(np.float64)
    with np.errstate(invalid="ignore"):
        ref = N.layer(w.astype(np.float64), 6, a5)
    inf = np.isinf(ref)
    assert np.array_equal(np.isnan(y), np.isnan(ref)) and np.array_equal(y[inf], ref[inf])
    assert what == "weight" or np.isinf(a5).any() and np.isfinite(ref).any()
    assert {"positive": inf.any(), "mixed": np.isnan(ref).any() and inf.any(), "weight": np.isfinite(ref).all()}[what]
    fin = np.isfinite(ref)
    assert np.max(np.abs(y[fin] - ref[fin])) <= 1e-5 * np.max(np.abs(ref[fin]))


# Layer 1's weight gradient where the data gradient overflowed at a corner, an
# edge or inside (identity layers: one pixel's gradient stays that pixel's): a
# tap outside the field takes no part, the others are infinite
@pytest.mark.parametrize("pixel", [(0, 0), (0, 69), (16, 33), (8, 0), (8, 68)])
def test_first_layer_gradient_overflow(pixel):
    import torch
    from ins2d_b200.learned import ConvNet
    from oracle import cnn_ref as N
    H, W = 17, 70
    W1, W6, eye = np.zeros((N.C, N.TAPS)), np.zeros((N.TAPS, N.C)), np.zeros((N.C, N.TAPS, N.C))
    W1[:, 4], W6[4] = 2.0 ** -60, 1.0
    eye[np.arange(N.C), 4, np.arange(N.C)] = 1.0
    w = N.join(W1, [eye * 2.0 ** 60, eye, eye, eye], W6)
    net = ConvNet(device=0, seed=1)
    net.set_params(w.astype(np.float32), 1.0)
    inp = torch.ones((1, H, W), device="cuda")
    tgt = net.forward(inp).clone()
    tgt[0, pixel[0], pixel[1]] = -2.0 ** 100
    g = np.asarray(net.loss_grad(inp, tgt)[1])
    ref = np.zeros((N.C, N.TAPS))
    for t in range(N.TAPS):
        y, x = pixel[0] + t // 3 - 1, pixel[1] + t % 3 - 1
        if 0 <= y < H and 0 <= x < W:
            ref[:, t] = np.inf
    assert np.array_equal(g[:N.OFF_WM].reshape(N.C, N.TAPS), ref)
    assert np.all(np.isfinite(g[N.OFF_WM:]))


# F's launches as counted by the profile: the tiled walkers, the table walkers
# around them, or both
@pytest.mark.parametrize("shape,bc,n", [((128, 64), "periodic", 1), ((300, 260), "cavity", 2), ((40, 30), "cavity", 1)])
def test_launch_count(shape, bc, n):
    import ins2d_b200
    from ins2d_b200 import cases
    from tests.cases_common import BC_COMBOS
    m = ins2d_b200.Options(cases.uniform_grid(shape[0], 0.0, 1.0), cases.uniform_grid(shape[1], 0.0, 1.0), BC_COMBOS[bc],
                           Re=100.0, poisson=6 if bc == "periodic" else 4, precond="jacobi")
    V, p = np.random.default_rng(1).standard_normal(m.NV), np.zeros(m.Np)
    m.profile()
    m.F(V, None, p)
    assert m.profile_read()["other"][1] == n
    # a step from its own first stage: four stages and the residual, then as
    # many without the first stage
    m.time_ERK(V, p, 0.0, 1e-6)
    fam = m.profile_read()
    assert fam["stage"][1] + fam["residual"][1] == 5 * n, fam


# Work arrays that only one solver reads are not allocated for the others: of
# the pressure-sized ones fast diagonalization holds five more than Jacobi
# (second direction, application's input and output, pivots, basis / 2)
def test_work_arrays():
    import ins2d_b200
    import torch
    from ins2d_b200 import cases
    from tests.cases_common import BC_COMBOS
    x, y = cases.uniform_grid(512, 0.0, 1.0), cases.uniform_grid(1024, 0.0, 2.0)

    def used(precond):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        m = ins2d_b200.Options(x, y, BC_COMBOS["cavity"], Re=100.0, poisson=4, precond=precond)
        n = free - torch.cuda.mem_get_info()[0]
        m.close()
        return n

    used("jacobi"), used("fdm")  # kernels and pools loaded
    assert used("fdm") - used("jacobi") >= 4 * 512 * 1024 * 8


# Transform solves on sides with primes above 31: direct sums up to 127 (alone,
# beside other radices, in one block and in three kernels), Bluestein's algorithm
# from 131 on; right-hand sides formed from a velocity as well.  The parity
# tests' bounds for one evaluation and for a step.
@pytest.mark.parametrize("shape", [(37, 37), (41, 41), (61, 29), (127, 8), (8, 127), (64, 113), (127, 64), (254, 67),
                                   (8, 381), (536, 201), (131, 64), (64, 137), (12, 131)])
def test_direct_sums(shape):
    import ins2d_b200
    from oracle import ins2d_ref as R
    from tests.cases_common import BC_COMBOS
    nx, ny = shape
    x, y = np.arange(nx + 1) / nx * 1.5, np.arange(ny + 1) / ny
    m = ins2d_b200.Options(x, y, BC_COMBOS["periodic"], poisson=6, Re=100.0)
    rng = np.random.default_rng(nx)
    f = rng.standard_normal((ny, nx))
    f -= f.mean()
    J, I = np.arange(ny)[:, None], np.arange(nx)[None, :]
    a = 4 * x[1] * y[1] * (np.sin(np.pi * I / nx) ** 2 / x[1] ** 2 + np.sin(np.pi * J / ny) ** 2 / y[1] ** 2)
    a[0, 0] = 1.0
    ref = np.real(np.fft.ifft2(-np.fft.fft2(f) / a)).ravel()
    assert np.max(np.abs(m.pressure_poisson(f.ravel()) - ref)) < 1e-12 * np.max(np.abs(ref))
    assert np.all(m.pressure_poisson(np.zeros(nx * ny)) == 0.0)
    o = R.make_options(x, y, BC_COMBOS["periodic"], poisson=6, Re=100.0)
    V = R.initial_projection(rng.standard_normal(o.grid.NV), 0.0, o)
    ref, _ = R.time_ERK(V, np.zeros(m.Np), 0.0, 1e-4, o)
    for precision, tol in (("fp64", 1e-11), ("fp32", 1e-5)):
        m = ins2d_b200.Options(x, y, BC_COMBOS["periodic"], poisson=6, Re=100.0, precision=precision)
        assert np.max(np.abs(m.time_ERK(V, np.zeros(m.Np), 0.0, 1e-4)[0] - ref)) < tol * np.max(np.abs(ref))


# The spectral preconditioner on sides that are no powers of two (one block,
# mixed radix, direct sums, one compile-time side): its solves against the
# transform solver's; a right-hand side near the zero threshold, where the
# preconditioner must not take the early return of a direct solve (a tolerance
# of 1e-18 takes it to residuals below 1e-26 in a second pass, met or not; a
# zero application would end as a breakdown); steps in a captured run
@pytest.mark.parametrize("shape", [(40, 40), (74, 60), (100, 60), (64, 45), (37, 61), (256, 134)])
def test_spectral_preconditioner_sides(shape):
    import ins2d_b200
    from ins2d_b200 import cases
    nx, ny = shape
    x, y = cases.uniform_grid(nx, 0.0, 1.0), cases.uniform_grid(ny, 0.0, ny / nx)
    kw = dict(Re=100.0, precond="fdm")
    m = ins2d_b200.Options(x, y, cases.BC_PERIODIC, poisson=4, CG_acc=1e-12, **kw)
    mf = ins2d_b200.Options(x, y, cases.BC_PERIODIC, poisson=6, Re=100.0)
    rng = np.random.default_rng(nx)
    f = rng.standard_normal(nx * ny)
    f -= f.mean()
    ref = mf.pressure_poisson(f)
    ref -= ref.mean()
    for scale in (1.0, 2.0 ** -43):
        dp, st = m.pressure_poisson(scale * f, return_stats=True)
        assert 1 <= st["iters"] <= 2
        assert np.max(np.abs(dp - dp.mean() - scale * ref)) < 1e-11 * scale * np.max(np.abs(ref))
    assert np.all(m.pressure_poisson(np.zeros(nx * ny)) == 0.0)
    never = ins2d_b200.Options(x, y, cases.BC_PERIODIC, poisson=4, CG_acc=1e-18, CG_maxit=3, **kw)
    try:
        assert never.pressure_poisson(2.0 ** -43 * f, return_stats=True)[1]["iters"] >= 2
    except ins2d_b200.Ins2dError as e:
        assert e.status == 2
    V, p = 0.1 * rng.standard_normal(m.NV), np.zeros(m.Np)
    V = mf.time_ERK(V, p, 0.0, 1e-4)[0]
    Va, pa = m.time_ERK(V, p, 0.0, 1e-4, nsteps=3)
    Vb, pb = mf.time_ERK(V, p, 0.0, 1e-4, nsteps=3)
    assert np.max(np.abs(Va - Vb)) < 1e-10 * np.max(np.abs(Vb))
    assert np.max(np.abs((pa - pa.mean()) - (pb - pb.mean()))) < 1e-8 * np.max(np.abs(pb))


# Right-hand sides outside the range of A (closed and periodic domains; their sum
# is what A cannot produce): a solve with fast diagonalization ends with an error,
# whichever form it takes (cluster, one to four warps per system, cyclic
# systems); steps from rest on small grids, whose pressure update's right-hand
# side is inconsistent by the rounding of its divergence, still end well
@pytest.mark.parametrize("combo", ["cavity", "per_x_walls", "periodic"])
@pytest.mark.parametrize("shape", [(12, 10), (7, 16), (64, 64), (128, 100), (200, 150), (20, 300), (600, 40)])
def test_inconsistent_right_hand_side(shape, combo):
    import ins2d_b200
    from tests.cases_common import BC_COMBOS, grid_stretched
    x, y = grid_stretched(shape[0], 0.0, 1.7), grid_stretched(shape[1], -0.5, 0.5, beta=1.2)
    m = ins2d_b200.Options(x, y, BC_COMBOS[combo], Re=100.0, poisson=4, CG_acc=1e-10, CG_maxit=300)
    rng = np.random.default_rng(shape[0])
    f = rng.standard_normal(m.Np)
    f -= f.mean()
    vol = np.kron(np.diff(y), np.diff(x))
    for g in (np.ones(m.Np), vol / vol.mean(), f + 1.0, f + 1e-3):
        with pytest.raises(ins2d_b200.Ins2dError) as ei:
            m.pressure_poisson(g)
        assert ei.value.status in (2, 4)
    dp = m.pressure_poisson(f)
    assert abs(vol @ dp) <= 1e-12 * vol.sum() * np.max(np.abs(dp))


@pytest.mark.parametrize("shape", [(3, 3), (4, 3), (8, 8), (140, 6), (33, 200)])
@pytest.mark.parametrize("form", ["single", "ensemble"])
def test_steps_from_rest(form, shape):
    import ins2d_b200
    from ins2d_b200 import cases
    kw = dict(x=cases.tanh_grid(shape[0], 0.0, 1.0, 1.05), y=cases.tanh_grid(shape[1], 0.0, 1.0, 1.05), BC=cases.BC_CAVITY,
              uBC=cases.lid_uBC(1.0, 1.0), Re=200.0, poisson=4, CG_acc=1e-12, CG_maxit=200, RK="RK44")
    m = ins2d_b200.Options(**kw)
    V, p = np.zeros(m.NV), np.zeros(m.Np)
    p = m.pressure_additional_solve(V, p, 0.0)
    scale = np.max(np.abs(p))
    for nsteps in (1, 4):
        if form == "single":
            V1, p1 = m.time_ERK(V, p, 0.0, 1e-4, nsteps=nsteps)
        else:
            e = ins2d_b200.Ensemble([kw])
            e.set_solver(0)
            e.set_state(0, V, p)
            e.time_ERK(0.0, 1e-4, nsteps)
            V1, p1 = e.get_state(0)
        assert np.max(np.abs(V1)) <= 1.0 and np.max(np.abs(p1)) <= 4.0 * scale  # no constant of the null space
        assert m.check_conservation(V1, 0.0)[0] < 1e-10
