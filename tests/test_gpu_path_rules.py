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
