"""metrics() and interface_positions() at the edges of the kernel's column
groups (32 in x) and layer runs, against float64 sums of the dense field:
counts and extrema exact, sums within 1e-12 (float64 rounding of at most 1e5
terms), grain ids above the shared-memory histogram included."""
import numpy as np
import pytest

from test_observe_gpu import interface_positions_np, make_solver, metrics_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,grains,slots", [((1, 1, 24), 1, 4), ((31, 3, 25), 3, 8), ((33, 5, 31), 5, 8),
                                               ((64, 2, 40), 9, 16), ((37, 29, 64), 40, 16), ((8, 8, 24), 4100, 4)])
def test_metrics_column_groups(dims, grains, slots):
    from mpf3d import inputs
    used = min(grains, 40)
    case = inputs.voronoi_case(*dims, used, 8, seed=3, orientation_seed=4, undercooling=2.0)
    if grains > used:  # spread the ids beyond the histogram's size
        N = grains + 1
        phi = np.zeros((N,) + dims, np.float32)
        phi[0] = case.phi[0]
        for g in range(1, used + 1):
            phi[g * (grains // used)] = case.phi[g]
        case.phi = phi
        case.wij, case.aij, case.mij = inputs.matrices_for(case.phys, N)
        case.n111 = np.repeat(case.n111[1:2], N, 0)
    s = make_solver(case, slots=slots)
    if grains == used:
        s.step(3)
    phi = s.to_dense()
    got, want = s.metrics(), metrics_np(phi, s.active_count(), case.phys.dx)
    for k in ("phi_min", "phi_max", "nf_max", "nan_count", "surviving_grains", "interface_position_max"):
        assert got[k] == want[k], k
    for k in ("solid_fraction", "solid_volume", "interface_position_mean", "grain_volumes"):
        np.testing.assert_allclose(got[k], want[k], rtol=1e-12, atol=1e-30, err_msg=k)
    assert abs(got["phi_sum_error_max"] - want["phi_sum_error_max"]) <= 1e-15
    np.testing.assert_array_equal(s.interface_positions(), interface_positions_np(phi))
