"""Behaviour at the edges of what the kernels accept."""
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
