"""The step's two routes -- all lists to octet_kernel, or kernels by kind of cell on two
streams -- under everything a caller does with a step: graphs, several streams, the device
clock, launch shapes, the entry without scratch; and both routes against each other where
the dispatch rule changes over.  x and y are periodic, so copies of a box step as it does."""
import ctypes

import numpy as np
import pytest

from test_quiet_flags_gpu import owner_solver

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SMALL, LARGE = (40, 36, 40), (128, 64, 112)
ROUTES = [pytest.param(SMALL, id="octets"), pytest.param(LARGE, id="by_kind")]


def by_kind(dims, anisotropy=True):
    from mpf3d import _lib
    return bool(_lib.lib().mpf3d_compact_step_by_kind(*dims, int(anisotropy)))


def make(dims, **kw):
    assert by_kind(dims) == (dims == LARGE)
    return owner_solver(*dims, 10, 12, **kw)


def same(a, b):
    for s in (a, b):
        s.check()
    return torch.equal(a.to_dense(host=False), b.to_dense(host=False))


@pytest.mark.parametrize("dims", ROUTES)
@pytest.mark.parametrize("prepared", [True, False])
def test_steps_captured_by_the_caller(dims, prepared):
    """Two steps in a graph of the caller's: after mpf3d_streams_prepare with the second
    stream, without it (the stream's first call is inside the capture) all on one."""
    from mpf3d import _lib
    a, b = make(dims), make(dims)
    a.step(2, check=False)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    if prepared:
        _lib.check(_lib.lib().mpf3d_streams_prepare(stream.cuda_stream), "streams_prepare")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        b.launch_step(1)
        b.launch_step(2)
    torch.cuda.current_stream().wait_stream(stream)
    g.replay()
    torch.cuda.synchronize()
    b.step_count = 2
    assert same(a, b)


@pytest.mark.parametrize("dims", ROUTES)
@pytest.mark.parametrize("tma", [True, False])
def test_replays_keep_cooling(dims, tma):
    """Three replays of four captured steps and eager ones around them, under fast cooling."""
    a, b = make(dims, cooling_rate=0.21), make(dims, cooling_rate=0.21)
    a.sweep_tma = b.sweep_tma = tma
    a.step(14, check=False)
    b.step(1, check=False)
    b.capture(4)
    b.step(13)
    torch.cuda.synchronize()
    assert b.step_count == 14 and same(a, b)


@pytest.mark.parametrize("dims", ROUTES)
def test_two_caller_streams(dims):
    ref, a, b = make(dims), make(dims), make(dims)
    ref.step(6, check=False)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for st in streams:
        st.wait_stream(torch.cuda.current_stream())
    for _ in range(6):
        for s, st in ((a, streams[0]), (b, streams[1])):
            with torch.cuda.stream(st):
                s.step(1, check=False)
    torch.cuda.synchronize()
    assert same(a, ref) and same(b, ref)


@pytest.mark.parametrize("dims", ROUTES)
def test_temperature_by_value(dims):
    from mpf3d import _lib
    a, b = make(dims, cooling_rate=0.21), make(dims, cooling_rate=0.21)
    a.step(7, check=False)
    for s in range(1, 8):
        src, dst = b.buf[b.cur], b.buf[1 - b.cur]
        _lib.check(_lib.lib().mpf3d_compact_step_tuned(
            *(t.data_ptr() for t in src), *(t.data_ptr() for t in dst), b.slots, b.amax, b.T0z.data_ptr(),
            b.T_melt + s * b.cooling_rate, b.wij.data_ptr(), b.a2ij.data_ptr(), b.mij.data_ptr(), b.n111.data_ptr(), b.N,
            b.nx, b.ny, b.nz, ctypes.byref(b.scalars), 1, 1, int(b.symmetric_normals), b.work_items.data_ptr(),
            b.work_count.data_ptr(), s & 1, b.err.data_ptr(), b._stream(), None, b.tile_flags.data_ptr(),
            _lib.STEP_MULTI_LIST), "compact_step_tuned")
        b.cur = 1 - b.cur
    assert same(a, b)


@pytest.mark.parametrize("dims", ROUTES)
@pytest.mark.parametrize("cfg", [(2, 4, 4, 256, 4, 128), (8, 16, 32, 128, 32, 64), (4, 8, 8, 256, 16, 64), (2, 16, 64, 128, 1, 128)])
def test_launch_shapes(dims, cfg):
    from mpf3d import autotune
    ref, s = make(dims), make(dims)
    s.tuning = autotune.make(cfg)
    for _ in range(2):
        ref.step(6)
        s.step(6)
        assert same(ref, s), cfg


@pytest.mark.parametrize("dims", ROUTES)
@pytest.mark.parametrize("captured", [False, True])
def test_step_without_scratch(dims, captured):
    from mpf3d import _lib
    ref, s = make(dims), make(dims)
    ref.step(2, check=False)
    bufs = [s.buf[s.cur], s._alloc(), s._alloc()]

    def steps(stream):
        for i in (1, 2):
            _lib.check(_lib.lib().mpf3d_compact_step_noalloc(
                *(t.data_ptr() for t in bufs[i - 1]), *(t.data_ptr() for t in bufs[i]), s.slots, s.amax,
                s.T0z.data_ptr(), s.T_melt + i * s.cooling_rate, s.wij.data_ptr(), s.a2ij.data_ptr(), s.mij.data_ptr(),
                s.n111.data_ptr(), s.N, s.nx, s.ny, s.nz, ctypes.byref(s.scalars), 1, 1, int(s.symmetric_normals),
                s.err.data_ptr(), stream), "compact_step_noalloc")

    if captured:
        stream, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.graph(g, stream=stream):
            steps(stream.cuda_stream)
        torch.cuda.current_stream().wait_stream(stream)
        g.replay()
    else:
        steps(None)
    torch.cuda.synchronize()
    s.buf[s.cur] = bufs[2]
    assert same(ref, s)


@pytest.mark.parametrize("slots,torque", [(8, True), (16, False)])
def test_change_over_of_a_domain(slots, torque):
    from mpf3d.solver import CompactSolver
    copies_of(CompactSolver, (128, 32, 112), (1, 2), slots=slots, torque=torque)


@pytest.mark.parametrize("slots", [8, 16])
def test_change_over_of_an_isotropic_plane(slots):
    from mpf3d.solver import CompactSolver
    copies_of(CompactSolver, (40, 44, 40), (1, 2), slots=slots, anisotropy=False)


def copies_of(cls, dims, copies, **kw):
    from mpf3d import inputs
    case = inputs.voronoi_case(*dims, 12, 10, seed=5, orientation_seed=8, undercooling=1.0)
    rest = (case.n111, case.wij, case.aij, case.mij, case.phys)
    aniso = kw.get("anisotropy", True)
    large = (dims[0] * copies[0], dims[1] * copies[1], dims[2])
    assert not by_kind(dims, aniso) and by_kind(large, aniso)
    box = cls(case.phi, case.temp, *rest, **kw)
    tiled = cls(np.tile(case.phi, (1,) + copies + (1,)), np.tile(case.temp, copies + (1,)), *rest, **kw)
    for steps in (1, 11):
        box.step(steps)
        tiled.step(steps)
        assert torch.equal(tiled.to_dense(host=False), box.to_dense(host=False).repeat(1, *copies, 1))


def batch(n, **kw):
    from mpf3d.batched import BatchedBicrystals
    rng = np.random.default_rng(7)
    q = rng.standard_normal((3, 2, 4))
    q /= np.linalg.norm(q, axis=2, keepdims=True)
    dt, da = rng.uniform(0.5, 3.0, 3), rng.uniform(0.0, 1.0, 3)
    return BatchedBicrystals([(96, 63, 72)] * n, q[:n], dt[:n], da[:n], base_height=10.0, **kw)


def test_change_over_of_a_batch():
    """Two instances below the rule, the same two among three above it; the latter also from a
    graph and with every kind of list shape."""
    from mpf3d import _lib, autotune
    two, three, graphed = batch(2), batch(3), batch(3)
    kind = _lib.lib().mpf3d_batched_step_by_kind
    assert not kind(two.total_cells, 1) and kind(three.total_cells, 1)
    graphed.capture(4)
    for b in (two, three, graphed):
        b.step(12)
        b.check()
    for cfg in ((4, 8, 4, 256, 4, 128), (4, 8, 32, 128, 32, 64)):
        s = batch(3)
        s.tuning = autotune.make(cfg)
        s.step(12)
        assert np.array_equal(s.dense(1), three.dense(1)), cfg
    for i in range(2):
        assert np.array_equal(two.dense(i), three.dense(i)) and np.array_equal(two.dense(i), graphed.dense(i))
    assert np.array_equal(three.dense(2), graphed.dense(2))
