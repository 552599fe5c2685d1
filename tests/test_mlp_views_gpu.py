"""Surrogate passes on views: gradients of the first rows of a forward pass, and arrays
that start at an odd offset."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def net_and_rows(rows):
    from mpf3d.surrogate import Surrogate
    s = Surrogate(seed=3)
    X = np.random.default_rng(4).uniform(-1, 1, (rows, 14)).astype(np.float32)
    return s, s.prepare(X)


@pytest.mark.parametrize("rows,first", [(640, 128), (300, 129), (300, 1)])
def test_gradient_of_the_first_rows(rows, first):
    """Equal to the gradients of a forward pass of these rows alone, up to the order of FP32 sums."""
    s, x = net_and_rows(rows)
    dout = torch.randn((first, 2), generator=torch.Generator("cuda").manual_seed(1), device="cuda")
    s.forward(x[:first].contiguous(), keep=True)
    s.backward(dout)
    want = s.g.clone()
    s.g.fill_(float("nan"))
    s.forward(x, keep=True)
    s.backward(dout)
    s.check()
    assert float((s.g - want).abs().max()) <= 1e-5 * float(want.abs().max())
    with pytest.raises(ValueError):
        s.backward(torch.zeros((rows + 1, 2), device="cuda"))


def test_arrays_at_an_odd_offset():
    s, x = net_and_rows(200)
    dout = torch.randn((200, 2), generator=torch.Generator("cuda").manual_seed(2), device="cuda")
    want = s.forward(x, keep=True)
    s.backward(dout)
    g = s.g.clone()
    shifted = torch.cat([torch.zeros(3, dtype=x.dtype, device="cuda"), x.reshape(-1)])[3:].view(x.shape)
    odd = torch.cat([torch.zeros(1, device="cuda"), dout.reshape(-1)])[1:].view(dout.shape)
    assert shifted.data_ptr() % 16 and odd.data_ptr() % 8
    assert torch.equal(s.forward(shifted, keep=True), want)
    s.backward(odd)
    s.check()
    assert torch.equal(s.g, g)
