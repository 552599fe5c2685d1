"""The sweep's quiet-tile flags: one byte per tile of 32 x 1 x zb cells, 1 where
every cell of the tile was uniform with its neighbours in the step.  Boxes whose
last block of rows is not full (y extents that are no multiple of the sweep's
block height) must write the flags of their own tiles only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def owner_solver(nx, ny, nz, grains, slab, **kw):
    """A Voronoi slab under a tanh front, without a dense field."""
    from mpf3d import inputs
    from mpf3d.solver import CompactSolver
    phys = inputs.Physics()
    d = phys.derived()
    owner = inputs.voronoi_slab_owner(nx, ny, slab, grains, slab, seed=3)
    n111 = inputs.rotated_n111(inputs.random_quaternions(grains, 4))
    assert n111.shape[0] == grains + 1
    prof = inputs.tanh_profile(nz, slab, phys.dx, d["delta"]).astype(np.float32)
    temp = np.full(nz, phys.T_melt - 2.0)
    return CompactSolver.from_owner(owner, prof, temp, n111, *inputs.matrices_for(phys, grains + 1), phys, **kw)


def expected_flags(head, nx, ny, nz, zb):
    """Per tile, in the flags' order (x fastest, then y, then z): whether all its cells are uniform."""
    h = head.view(nz, ny, nx)
    up, down = torch.cat([h[1:], h[-1:]]), torch.cat([h[:1], h[:-1]])
    same = (h & 0xFF) == 1
    for q in (h.roll(1, 2), h.roll(-1, 2), h.roll(1, 1), h.roll(-1, 1), up, down):
        same &= q == h
    pad = (0, -nx % 32, 0, 0, 0, -nz % zb)
    same = torch.nn.functional.pad(same, pad, value=True)
    return same.view(-1, zb, ny, same.shape[2] // 32, 32).all(4).all(1).reshape(-1).to(torch.uint8)


@pytest.mark.parametrize("zb,by", [(2, 4), (2, 8), (2, 16), (4, 8), (8, 4), (8, 16)])
@pytest.mark.parametrize("nx,ny,nz", [(40, 1, 12), (33, 5, 24), (64, 13, 30), (36, 117, 22), (20, 361, 9)])
def test_flags_are_those_of_the_domains_tiles(nx, ny, nz, zb, by):
    from mpf3d import autotune
    s = owner_solver(nx, ny, nz, 3, min(6, nz - 3))
    s.tuning = autotune.make((zb, by) + autotune.DEFAULT[2:])
    n = -(-nx // 32) * ny * -(-nz // zb)
    guard = 16 * -(-nx // 32) + 64
    s.tile_flags = torch.zeros(2 * n + guard, dtype=torch.uint8, device=s.device)
    s.tile_flags[2 * n:] = 0xA5
    s._tiles_zb = zb  # the flags are for this shape: keep the guard
    halves = [torch.zeros(n, dtype=torch.uint8, device=s.device) for _ in range(2)]
    for step in range(1, 9):
        halves[step & 1] = expected_flags(s.buf[s.cur][0], nx, ny, nz, zb)
        s.step(1)
        assert torch.equal(s.tile_flags[:2 * n].view(2, n), torch.stack(halves)), f"step {step}"
        assert bool((s.tile_flags[2 * n:] == 0xA5).all()), f"step {step}: written past the flags"


@pytest.mark.parametrize("zb,by", [(4, 8), (2, 16)])
def test_large_box_equals_the_sweep_of_every_tile(zb, by):
    """Several chunks of tiles per block, and rows past the last band."""
    from mpf3d import autotune
    a, b = (owner_solver(400, 403, 100, 12, 16) for _ in range(2))
    a.tuning = b.tuning = autotune.make((zb, by) + autotune.DEFAULT[2:])
    b.skip_quiet_tiles = False
    for _ in range(5):
        a.step(10)
        b.step(10)
        assert torch.equal(a.to_dense(host=False), b.to_dense(host=False))
