"""The surrogate's chain kernels at row counts around their tiles (128 rows,
64-row reduction chunks), against the float64 restatement with the same BF16
rounding points.  Values whose FP32 sum rounds to the other BF16 neighbour
(about one in a thousand, each off by 2^-9) stay within 1e-4 of a norm; one
wrong row of the largest case would be 3%.  Bound: 2e-3."""
import numpy as np
import pytest

from test_surrogate_gpu import bf16_round, cpu_forward_backward

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("M", [1, 2, 63, 65, 127, 128, 129, 300, 1000])
def test_chain_kernels_row_counts(M):
    from mpf3d.surrogate import Surrogate, LAYERS, IN_FEATURES, DERIVED, K1
    s = Surrogate(seed=7)
    rng = np.random.default_rng(M)
    live = IN_FEATURES + DERIVED
    X = np.zeros((M, K1))
    X[:, :live] = bf16_round(rng.uniform(-1, 1, (M, live)).astype(np.float32))
    T = rng.standard_normal((M, 2)).astype(np.float32)
    x16 = s.prepare(X.astype(np.float32))
    s.loss_and_grad(x16, torch.from_numpy(T).to("cuda:0"))
    s.check()
    out, grads = cpu_forward_backward(s.bf16_weights(), X, T.astype(np.float64), np.ones(2))
    near = lambda got, ref: np.linalg.norm(got - ref) <= 2e-3 * np.linalg.norm(ref)
    got = s.forward(x16)
    assert near(got.cpu().numpy(), out)
    assert torch.equal(got, s.forward(x16, keep=True))
    g = s.g.cpu().numpy().astype(np.float64)
    for layer, (K, N, _) in enumerate(LAYERS):
        o, ob = s.offsets[layer]
        assert near(g[o:o + N * K].reshape(N, K), grads[layer][0]), f"weights of layer {layer}"
        assert near(g[ob:ob + N], grads[layer][1]), f"biases of layer {layer}"


def test_many_tiles_per_block_and_padding_columns():
    """More row tiles than resident CTAs; gradients of the input's padding stay zero whatever it holds."""
    from mpf3d.surrogate import Surrogate, HIDDEN, IN_FEATURES, DERIVED, K1
    s = Surrogate(seed=8)
    rng = np.random.default_rng(0)
    X = rng.uniform(-1, 1, (128 * 701 + 5, K1)).astype(np.float32)
    x16 = s.prepare(X)
    whole = s.forward(x16)
    parts = torch.cat([s.forward(x16[a:a + 1000]) for a in range(0, len(X), 1000)])
    assert torch.equal(whole, parts)
    s.loss_and_grad(x16[:640], torch.zeros((640, 2), device="cuda:0"))
    s.check()
    assert not s.g[:HIDDEN * K1].view(HIDDEN, K1)[:, IN_FEATURES + DERIVED:].any()
