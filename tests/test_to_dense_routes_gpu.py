"""The converters to dense fields by destination: device and pinned host memory, both
types, sizes on both sides of the rule that picks four cells a thread, fields off the 16
bytes, and in a captured graph.  Each value against the state's own slots."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def solver(dims, grains):
    from mpf3d import inputs
    from mpf3d.solver import CompactSolver
    phys = inputs.Physics()
    slab = min(6, dims[2])
    owner = inputs.voronoi_slab_owner(dims[0], dims[1], slab, grains, slab, seed=3)
    prof = inputs.tanh_profile(dims[2], 4.0, phys.dx, phys.derived()["delta"])
    s = CompactSolver.from_owner(owner, prof, np.full(dims[2], phys.T_melt - 1.0),
                                 inputs.rotated_n111(inputs.random_quaternions(grains, 4)),
                                 *inputs.matrices_for(phys, grains + 1), phys)
    s.step(3)
    return s


def from_slots(s):
    """The dense field gathered from heads, ids and values with torch."""
    head, idx, val = s.buf[s.cur]
    n, first, cells = head & 0x7F, head >> 8, s.cells
    phi = torch.zeros((s.N, cells), device=head.device)
    at = torch.arange(cells, device=head.device)
    alone = (n == 1) & ((head & 0x80) == 0)
    phi[first.long(), at] = torch.where(alone, 1.0, val[:cells])
    for k in range(1, s.slots):
        has = n > k
        phi[(idx[k * cells:(k + 1) * cells].long() & 0xFFFF)[has], at[has]] = val[k * cells:(k + 1) * cells][has]
    return phi.view(s.N, s.nz, s.ny, s.nx).permute(0, 3, 2, 1).contiguous()


@pytest.mark.parametrize("dims,grains", [((32, 17, 64), 5), ((130, 128, 64), 62), ((130, 128, 68), 62), ((40, 9, 8), 3),
                                         ((33, 5, 30), 4)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_every_destination(dims, grains, dtype):
    s = solver(dims, grains)
    want = from_slots(s).to(dtype)
    for shift in (0, 1):
        flat = torch.full((want.numel() + 1,), -1.0, dtype=dtype, device="cuda")
        out = flat[shift:shift + want.numel()].view(want.shape)
        s.to_dense(out=out, host=False)
        assert torch.equal(out, want)
    host = torch.full(want.shape, -1.0, dtype=dtype, pin_memory=True)
    s.to_dense(out=host)
    torch.cuda.synchronize()
    assert torch.equal(host, want.cpu())


@pytest.mark.parametrize("pinned", [False, True])
def test_in_a_captured_graph(pinned):
    s = solver((32, 17, 64), 5)
    want = from_slots(s)
    out = torch.zeros(want.shape, pin_memory=True) if pinned else torch.zeros(want.shape, device="cuda")
    g = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=stream):
        s.to_dense(out=out, host=False)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out.cuda(), want)
