"""Blocks of the drop-in update whose listed cells are all flat two-phase cells: the
block's warps must agree that there is work, however late one of them is.  Against
the oracle within the bounds of the golden comparisons, and the same bits from
every launch."""
import numpy as np
import pytest

import oracle as O
from test_dense_gpu import TOL, run_dropin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims", [(8, 12, 40), (68, 64, 66), (128, 130, 130)])
def test_flat_two_phase_cells(dims, dtype):
    from mpf3d import inputs
    case = inputs.voronoi_case(8, 8, 16, 2, 8, seed=1, orientation_seed=2)
    phi = np.zeros((3,) + dims, dtype)
    phi[0], phi[1] = 0.75, 0.25
    temp = np.full(dims, case.phys.T_melt - 1.0, dtype)
    f32 = dtype == np.float32
    sc = case.phys.kernel_scalars(f32=f32)
    mats = (case.wij, case.aij, case.mij, case.n111)
    runs = [run_dropin(phi, temp, *mats, sc, 1, 0.0, checked=True, switchable=True, cooling=False)[0][0]
            for _ in range(3)]
    small = tuple(min(d, 9) for d in dims)  # every cell sees the same surroundings
    cut = (slice(None),) + tuple(slice(0, n) for n in small)
    want, _, _, _ = O.run(phi[cut], temp[cut[1:]], *mats, O.make_scalars([float(v) for v in sc], f32), 1,
                          cooling=False)
    assert np.ptp(want[1]) == 0.0 and want[1].flat[0] != 0.25
    assert np.abs(runs[0].astype(np.float64) - want[:, :1, :1, :1].astype(np.float64)).max() <= TOL[np.dtype(dtype)]
    for r in runs[1:]:
        assert np.array_equal(r, runs[0])
