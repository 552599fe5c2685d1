"""Long work lists and cells of many phases: the forms by one thread per cell of any
neighbourhood give the bits of the octets.  x and y are periodic, so copies of a box
side by side step as the box does; the copies make its lists long."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BOX, GRAINS, STEPS = (22, 20, 40), 8, 40


def solver(copies, antipodal=True, box=BOX, **kw):
    """A melt undercooled so far that every grain's phase grows everywhere."""
    from mpf3d import inputs
    from mpf3d.solver import CompactSolver
    case = inputs.voronoi_case(*box, GRAINS, 8, seed=9, orientation_seed=3, undercooling=2.0)
    n111 = case.n111
    if not antipodal:
        n111 = np.random.default_rng(1).standard_normal(n111.shape).astype(np.float32)
        n111 /= np.linalg.norm(n111, axis=2, keepdims=True)
    phi, temp = np.tile(case.phi, (1,) + copies + (1,)), np.tile(case.temp, copies + (1,))
    return CompactSolver(phi, temp, n111, case.wij, case.aij, case.mij, case.phys, **kw)


def lists(s):
    c, p = s.work_count.cpu().numpy(), s.step_count & 1
    return int(c[2 * p]), int(c[2 * p + 1]), int(c[4 + p])


@pytest.mark.parametrize("slots,antipodal,anisotropy", [(8, True, True), (16, True, True), (16, False, True),
                                                        (16, True, False)])
@pytest.mark.parametrize("copies", [(3, 3), (8, 7)])
def test_copies_step_as_the_box(copies, slots, antipodal, anisotropy):
    """3 x 3: octet_kernel's lists are long; 8 x 7: kernels by kind, several solids everywhere
    (isotropic: blocks left with many cells, either way)."""
    kw = dict(slots=slots, anisotropy=anisotropy)
    box, many = solver((1, 1), antipodal, **kw), solver(copies, antipodal, **kw)
    for steps in (1, STEPS - 1):
        box.step(steps)
        many.step(steps)
        assert torch.equal(many.to_dense(host=False), box.to_dense(host=False).repeat(1, *copies, 1))
    assert int(box.active_count(host=False).max()) >= 8
    if anisotropy:
        assert sum(lists(box)) < 40000 and lists(box)[2] < 16384  # octets
        _, one, several = lists(many)
        assert several > (60000 if copies == (8, 7) else 16384) and several > 8 * one


def test_long_isotropic_lists_of_a_narrow_domain():
    """Too small a plane for isotropic_kernel: octet_kernel's threads on list 0 alone."""
    kw = dict(box=(22, 20, 90), slots=16, anisotropy=False)
    box, many = solver((1, 1), **kw), solver((2, 2), **kw)
    for steps in (1, 79):
        box.step(steps)
        many.step(steps)
        assert torch.equal(many.to_dense(host=False), box.to_dense(host=False).repeat(1, 2, 2, 1))
    assert lists(box)[0] < 49152 < lists(many)[0]


@pytest.mark.parametrize("copies", [(3, 3), (8, 7)])
def test_overflow_widens_where_lists_are_long(copies):
    """A step that needs more slots leaves its cells as they were and is redone with wider ones."""
    a, b = solver(copies, slots=4), solver(copies, slots=16)
    a.step(STEPS)
    b.step(STEPS)
    assert a.slots > 4
    assert torch.equal(a.to_dense(host=False), b.to_dense(host=False))


def test_without_the_multi_solid_list(monkeypatch):
    """All interface cells in one list, long enough for the threads."""
    from mpf3d import solver as mod
    a, b = solver((3, 3), slots=16), solver((3, 3), slots=16)
    a.step(STEPS)
    with monkeypatch.context() as m:
        m.setattr(mod._lib, "STEP_MULTI_LIST", 0)
        b.step(STEPS)
    assert torch.equal(a.to_dense(host=False), b.to_dense(host=False))


@pytest.mark.parametrize("anisotropy", [True, False])
def test_batch_with_long_lists_equals_its_instances(anisotropy):
    """Bicrystals whose lists together are long (threads), and alone are not (octets)."""
    from mpf3d.batched import BatchedBicrystals
    rng = np.random.default_rng(2)
    dims = [(33, 21, 41), (19, 9, 30)] + [(48, 48, 64)] * 3
    q = rng.standard_normal((len(dims), 2, 4))
    q /= np.linalg.norm(q, axis=2, keepdims=True)
    dt, da = rng.uniform(1.0, 3.0, len(dims)), rng.uniform(0.0, 1.0, len(dims))
    kw = dict(base_height=8.0, anisotropy=anisotropy)
    whole = BatchedBicrystals(dims, q, dt, da, **kw)
    alone = BatchedBicrystals(dims[:2], q[:2], dt[:2], da[:2], **kw)
    long = 0
    for _ in range(8):
        whole.step(10)
        alone.step(10)
        p = whole.step_count & 1
        c = whole.work_count.cpu().numpy()
        long = max(long, int(c[2 * p] + c[2 * p + 1] + c[4 + p]))
        for i in range(2):
            assert np.array_equal(whole.dense(i), alone.dense(i)), f"instance {i}"
    whole.check()
    alone.check()
    assert long > 49152
