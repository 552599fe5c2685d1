"""Dense fields from a compact state: every stored phase in its plane, zero elsewhere,
for z counts in and out of multiples of four, both types and unaligned fields."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("slots", [4, 8, 16])
@pytest.mark.parametrize("dims", [(5, 3, 4), (9, 6, 68), (33, 2, 7), (4, 5, 130), (1, 1, 1)])
def test_round_trip(dims, slots):
    from mpf3d import inputs
    from mpf3d.solver import CompactSolver
    rng = np.random.default_rng(sum(dims) + slots)
    N = 21
    phi = np.zeros((N, *dims), np.float32)
    cells = phi.reshape(N, -1)
    for c in range(cells.shape[1]):  # 1 to `slots` phases, the first and last ones among them
        ids = rng.choice(N, rng.integers(1, slots + 1), replace=False)
        cells[ids, c] = rng.uniform(0.01, 1.0, len(ids)) if len(ids) > 1 else 1.0
    wij, aij, mij = inputs.matrices_for(inputs.Physics(), N)
    s = CompactSolver(phi, np.zeros(dims), inputs.rotated_n111(inputs.random_quaternions(N - 1, 1)), wij, aij, mij,
                      slots=slots)
    for dtype in (torch.float32, torch.float64):
        for shift in (0, 1, 2):  # elements off the allocation's alignment
            flat = torch.full((phi.size + 2,), -1.0, dtype=dtype, device="cuda")
            out = flat[shift:shift + phi.size].view(phi.shape)
            s.to_dense(out=out, host=False)
            assert np.array_equal(out.cpu().numpy(), phi.astype(out.cpu().numpy().dtype))
            rest = torch.cat([flat[:shift], flat[shift + phi.size:]])
            assert bool((rest == -1.0).all())
