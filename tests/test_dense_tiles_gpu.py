"""Drop-in kernels at the edges of their tiles (32 cells along z, a few rows
in x and y): sizes around the tile sizes, single rows, and lists deeper than
one phase block, against the oracle.  nf, mf and status exact; phi within
1e-12 (float64) and 1e-6 (float32), the bounds of the golden comparisons."""
import numpy as np
import pytest

import oracle as O
from _helpers import valid_mf_equal
from test_dense_gpu import TOL, run_dropin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims,grains", [((1, 1, 1), 1), ((2, 1, 33), 2), ((5, 9, 31), 7), ((4, 8, 64), 8),
                                         ((3, 17, 65), 9), ((9, 7, 96), 17), ((68, 67, 63), 4)])
def test_dropin_tile_edges(dims, grains, dtype):
    from mpf3d import inputs
    N = grains + 1
    rng = np.random.default_rng(17)
    case = inputs.voronoi_case(8, 8, 16, grains, 8, seed=1, orientation_seed=2)
    # random sparse lists: every cell holds one to three phases
    phi = np.where(rng.random((N,) + dims) < 2.0 / N, rng.random((N,) + dims), 0.0)
    phi[0] += phi.sum(0) == 0.0
    phi = (phi / phi.sum(0)).astype(dtype)
    f32 = dtype == np.float32
    temp = (case.phys.T_melt - rng.uniform(0.0, 3.0, dims)).astype(dtype)
    sc = case.phys.kernel_scalars(f32=f32)
    hist = run_dropin(phi, temp, case.wij, case.aij, case.mij, case.n111, sc, 2, 0.0, checked=True, switchable=True,
                      cooling=False)
    _, _, _, _, want = O.run(phi, temp, case.wij, case.aij, case.mij, case.n111,
                             O.make_scalars([float(v) for v in sc], f32), 2, cooling=False, record=True)
    for (p, n, m, st, _), (op, on, om, ost, _) in zip(hist, want):
        assert np.array_equal(n, on) and valid_mf_equal(m, om, n) and np.array_equal(st, ost)
        assert np.abs(p.astype(np.float64) - op.astype(np.float64)).max() <= TOL[np.dtype(dtype)]
