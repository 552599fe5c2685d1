"""The forms of a queued cell's update -- eight lanes per cell on small domains;
pairs, trios and what they leave on large ones -- give the same bits, for
antipodal and general normals and ragged boxes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def solver(dims, grains, antipodal=True, **kw):
    from mpf3d import inputs
    from mpf3d.solver import CompactSolver
    case = inputs.voronoi_case(*dims, grains, 8, seed=5, orientation_seed=6, undercooling=2.0)
    n111 = case.n111.copy()
    if not antipodal:
        rng = np.random.default_rng(1)
        n111 = rng.standard_normal(n111.shape).astype(np.float32)
        n111 /= np.linalg.norm(n111, axis=2, keepdims=True)
    return CompactSolver(case.phi, case.temp, n111, case.wij, case.aij, case.mij, case.phys, **kw)


@pytest.mark.parametrize("antipodal", [True, False])
@pytest.mark.parametrize("slots", [8, 16])
def test_pair_kernel_equals_merge(monkeypatch, slots, antipodal):
    """With the multi-solid list the sweep keeps list 1 to pairs; without it every
    interface cell goes through the merge."""
    from mpf3d import solver as mod
    a = solver((131, 127, 64), 40, antipodal, slots=slots)
    b = solver((131, 127, 64), 40, antipodal, slots=slots)
    for steps in (1, 7, 12):
        a.step(steps)
        with monkeypatch.context() as m:
            m.setattr(mod._lib, "STEP_MULTI_LIST", 0)
            b.step(steps)
        assert torch.equal(a.to_dense(host=False), b.to_dense(host=False))


@pytest.mark.parametrize("slots,torque", [(4, True), (8, False), (16, True)])
def test_octets_equal_threads(slots, torque):
    """The first instance's interface list alone is short (octets), in the batch long (threads, pairs)."""
    from mpf3d.batched import BatchedBicrystals
    rng = np.random.default_rng(2)
    dims = [(19, 9, 30), (33, 20, 41), (1, 1, 24)] + [(96, 64, 72)] * 3
    q = rng.standard_normal((len(dims), 2, 4))
    q /= np.linalg.norm(q, axis=2, keepdims=True)
    dt, da = rng.uniform(0.25, 3.0, len(dims)), rng.uniform(0.0, 1.0, len(dims))
    kw = dict(base_height=8.0, slots=slots, torque=torque)
    whole = BatchedBicrystals(dims, q, dt, da, **kw)
    alone = BatchedBicrystals(dims[:3], q[:3], dt[:3], da[:3], **kw)
    whole.step(25)
    alone.step(25)
    whole.check()
    alone.check()
    for i in range(3):
        assert np.array_equal(whole.dense(i), alone.dense(i)), f"instance {i}"


@pytest.mark.parametrize("slots,anisotropy", [(8, True), (16, True), (8, False), (16, False)])
def test_tiled_domain_equals_its_period(slots, anisotropy):
    """x and y are periodic: 2 x 2 copies of a box (large: pairs, trios, rest) step as the box does (octets)."""
    from mpf3d import inputs
    from mpf3d.solver import CompactSolver
    case = inputs.voronoi_case(62, 66, 60, 24, 8, seed=9, orientation_seed=3, undercooling=2.0)
    kw = dict(slots=slots, anisotropy=anisotropy)
    rest = (case.temp, case.n111, case.wij, case.aij, case.mij, case.phys)
    box = CompactSolver(case.phi, *rest, **kw)
    tiled = CompactSolver(np.tile(case.phi, (1, 2, 2, 1)), np.tile(case.temp, (2, 2, 1)), *rest[1:], **kw)
    for steps in (1, 9):
        box.step(steps)
        tiled.step(steps)
        assert torch.equal(tiled.to_dense(host=False), box.to_dense(host=False).repeat(1, 2, 2, 1))
