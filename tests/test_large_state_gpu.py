"""Cells whose records lie beyond 2^32 entries of the slot arrays: the same step as of
the same cells at the start of small arrays, bit for bit.  One small instance of a batch
stands at the end of state arrays of 1.45e9 cells (about 52 GB, hardly any of it
touched); the arrays written to are the same allocation, shifted."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SLOTS, AMAX, SHIFT = 4, 8, 8192


def one_step(s, cells, offset):
    """One batched step of the state of solver s at `offset` in arrays of `cells` cells; its dense field."""
    from mpf3d import _lib
    from mpf3d.batched import TILE, Instance, _e2_flat
    head = torch.empty(cells + SHIFT, dtype=torch.int32, device="cuda")
    idx = torch.empty(SLOTS * cells + SHIFT, dtype=torch.int16, device="cuda")
    val = torch.empty(SLOTS * cells + SHIFT, dtype=torch.float32, device="cuda")
    items = torch.empty(2 * cells, dtype=torch.int32, device="cuda")
    count = torch.zeros(6, dtype=torch.int32, device="cuda")
    n = s.cells
    assert n <= SHIFT and offset + SHIFT <= cells
    h, i, v = s.buf[s.cur]
    head[offset:offset + n] = h
    for k in range(SLOTS):
        idx[k * cells + offset:k * cells + offset + n] = i[k * n:(k + 1) * n]
        val[k * cells + offset:k * cells + offset + n] = v[k * n:(k + 1) * n]
    I = Instance()
    I.nx, I.ny, I.nz, I.offset = s.nx, s.ny, s.nz, offset
    I.delta_a, I.mu_da = s.phys.delta_a, float(np.float32(s.phys.mu_a * s.phys.delta_a))
    I.e2_flat, I.undercooling = _e2_flat(s.phys, s.phys.delta_a), 2.0
    inst = torch.frombuffer(bytearray(bytes(I)), dtype=torch.uint8).cuda()
    tiles = -(-s.nx // TILE[0]) * -(-s.ny // TILE[1]) * -(-s.nz // TILE[2])
    out = [head.data_ptr() + 4 * SHIFT, idx.data_ptr() + 2 * SHIFT, val.data_ptr() + 4 * SHIFT]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    lib = _lib.lib()
    _lib.check(lib.mpf3d_batched_step_tuned(
        head.data_ptr(), idx.data_ptr(), val.data_ptr(), *out, SLOTS, AMAX, inst.data_ptr(), 1, tiles, cells,
        s.wij.data_ptr(), s.a2ij.data_ptr(), s.mij.data_ptr(), s.n111.data_ptr(), s.N, ctypes.byref(s.scalars),
        int(s.anisotropy), int(s.torque), int(s.symmetric_normals), items.data_ptr(), count.data_ptr(), 1,
        err.data_ptr(), None, _lib.STEP_MULTI_LIST, None, None), "batched_step_tuned")
    phi = torch.empty((s.N, s.nx, s.ny, s.nz), device="cuda")
    _lib.check(lib.mpf3d_compact_to_dense_view(*out, SLOTS, cells, offset, s.N, s.nx, s.ny, s.nz, phi.data_ptr(), 0,
                                               None), "to_dense_view")
    assert int(err.item()) == 0
    return phi


@pytest.mark.parametrize("anisotropy", [True, False])
def test_records_beyond_32_bits(anisotropy):
    if torch.cuda.mem_get_info()[0] < 70e9:
        pytest.skip("needs 52 GB of free device memory")
    from mpf3d import inputs
    from mpf3d.solver import CompactSolver
    case = inputs.voronoi_case(20, 13, 26, 3, 8, seed=2, orientation_seed=7, undercooling=2.0)
    s = CompactSolver(case.phi, case.temp, case.n111, case.wij, case.aij, case.mij, case.phys, slots=SLOTS,
                      anisotropy=anisotropy)
    s.step(6)
    assert s.slots == SLOTS
    act = s.active_count(host=False)
    assert int((s.stored_counts() >= 3).sum()) > 50 and int((act > 3).sum()) > 20
    near = one_step(s, 1 << 18, 0)
    cells = 1_450_000_000
    assert 2 * cells + (cells - SHIFT) > 2 ** 32
    far = one_step(s, cells, cells - SHIFT)
    assert torch.equal(near, far)
    del far
    torch.cuda.empty_cache()
