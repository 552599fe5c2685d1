"""The compact step's results bit for bit: states of small runs against those
recorded from the one-thread-per-cell kernels that came before the forms by kind of
cell.  The order and fusing of the solid-liquid sums is part of the results: a last
bit of lap_sl decides now and then which phases of a cell are clipped."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")

FIXTURE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "compact_bits.npz")
MODELS = {"full": (True, True), "no_torque": (True, False), "isotropic": (False, False)}


def box(model):
    """A box of grains of general orientation (multi-solid cells, octets on this size)."""
    from mpf3d import inputs
    from mpf3d.solver import CompactSolver
    case = inputs.voronoi_case(20, 13, 26, 6, 8, seed=2, orientation_seed=7, undercooling=2.0)
    aniso, torque = MODELS[model]
    s = CompactSolver(case.phi, case.temp, case.n111, case.wij, case.aij, case.mij, case.phys, slots=8,
                      anisotropy=aniso, torque=torque)
    s.step(16)
    return s.to_dense()


def plane(model):
    """Two grains under a wide plane: one-solid cells, by kind of cell; the layers about the front."""
    from mpf3d import inputs
    from mpf3d.solver import CompactSolver
    case = inputs.voronoi_case(80, 72, 24, 3, 8, seed=4, orientation_seed=11, undercooling=1.5)
    aniso, torque = MODELS[model]
    s = CompactSolver(case.phi, case.temp, case.n111, case.wij, case.aij, case.mij, case.phys, slots=8,
                      anisotropy=aniso, torque=torque)
    s.step(12)
    return s.to_dense()[:, ::5, ::3]


def bicrystals(model):
    from mpf3d.batched import BatchedBicrystals
    rng = np.random.default_rng(8)
    dims = [(24, 8, 28), (17, 5, 24)]
    q = rng.standard_normal((len(dims), 2, 4))
    q /= np.linalg.norm(q, axis=2, keepdims=True)
    aniso, torque = MODELS[model]
    b = BatchedBicrystals(dims, q, [2.5, 1.25], [0.36, 0.9], base_height=8.0, anisotropy=aniso, torque=torque)
    b.step(20, use_graph=False)
    b.check()
    return np.concatenate([b.dense(i).ravel() for i in range(len(dims))])


@pytest.mark.parametrize("model", list(MODELS))
@pytest.mark.parametrize("run", [box, plane, bicrystals])
def test_states_equal_the_recorded_ones(run, model):
    want = np.load(FIXTURE)[f"{run.__name__}_{model}"]
    got = run(model)
    n = int((got != want).sum())
    assert n == 0, f"{n} of {got.size} values differ, by up to {np.abs(got - want).max():.3g}"
