"""`ops.linear` and `ops.dense_swiglu`: whatever the number of rows, the same calls are
taken and the same are refused."""
import pytest
import torch
import torch.nn.functional as F

from sparse_b200 import ops

BF = torch.bfloat16
gpu = pytest.mark.gpu


def _pair(t, k, n, dtype, device):
    torch.manual_seed(t + k + n)
    return torch.randn(t, k, device=device).to(dtype), (torch.randn(n, k, device=device) / k ** 0.5).to(dtype)


@pytest.mark.parametrize("t", [0, 1, 16, 17])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, BF])
def test_linear_on_the_host_is_the_library(t, dtype):
    x, w = _pair(t, 64, 24, dtype, "cpu")
    assert torch.equal(ops.linear(x, w), F.linear(x, w))
    with pytest.raises(RuntimeError):
        ops.linear(x, w[:, :32])


def test_linear_keeps_the_gradient():
    x, w = _pair(3, 64, 24, torch.float32, "cpu")
    w.requires_grad_()
    ops.linear(x, w).sum().backward()
    assert torch.equal(w.grad, x.sum(0).expand_as(w))


@gpu
@pytest.mark.parametrize("t", [1, 16, 17])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, BF])
def test_linear_takes_what_the_library_takes(t, dtype):
    x, w = _pair(t, 96, 40, dtype, "cuda")
    b = torch.randn(40, device="cuda").to(dtype)
    # fp32 sums of 96 products of order 0.1 (1e-4), one rounding of the result and, where the
    # library adds the bias afterwards, one of the product: u (2 |want| + |b|)
    u = {torch.float32: 2.0 ** -24, torch.float16: 2.0 ** -11, BF: 2.0 ** -8}[dtype]
    want = F.linear(x.double(), w.double(), b.double())

    def close(got):
        return bool(((got.double() - want).abs() <= u * (2 * want.abs() + b.double().abs()) + 1e-4).all())

    turned = torch.randn(96, 40, device="cuda").to(dtype)
    turned.copy_(w.t())
    shifted = torch.empty(40 * 96 + 1, dtype=dtype, device="cuda")[1:].view(40, 96)  # off a 16-byte boundary
    shifted.copy_(w)
    padded = torch.zeros(40, 104, dtype=dtype, device="cuda")[:, :96]
    padded.copy_(w)
    spread = torch.empty(80, dtype=dtype, device="cuda")[::2]
    spread.copy_(b)
    for weight in (w, turned.t(), shifted, padded):
        for bias in (b, spread):
            assert close(ops.linear(x, weight, bias))
    rows = torch.empty(t * 96 + 1, dtype=dtype, device="cuda")[1:].view(t, 96)
    rows.copy_(x)
    assert close(ops.linear(rows, w, b))


@gpu
@pytest.mark.parametrize("t", [1, 16, 17])
def test_linear_refuses_what_the_library_refuses(t):
    x, w = _pair(t, 96, 40, BF, "cuda")
    for weight, bias in ((w[:, :64].contiguous(), None), (w.float(), None), (w, torch.zeros(39, device="cuda", dtype=BF)),
                         (w.cpu(), None), (w, torch.zeros(40, device="cuda"))):
        with pytest.raises(RuntimeError):
            ops.linear(x, weight, bias)


@gpu
@pytest.mark.parametrize("t", [1, 16, 17])
def test_dense_swiglu_refuses_operands_that_do_not_fit(t):
    h, i = 128, 192
    x = torch.randn(t, h, device="cuda").to(BF)
    w13, w2 = torch.zeros(1, 2 * i, h, device="cuda", dtype=BF), torch.zeros(1, h, i, device="cuda", dtype=BF)
    assert ops.dense_swiglu(x, w13, w2).shape == (t, h)

    def off(v):                                           # the same values, off a 16-byte boundary
        moved = torch.empty(v.numel() + 1, device="cuda", dtype=v.dtype)[1:].view(v.shape)
        return moved.copy_(v)

    bad = [(x.float(), w13, w2), (x, w13.half(), w2), (x, w13, w2.float()), (x[:, :64].contiguous(), w13, w2),
           (x, w13, w2[:, :, :64].contiguous()), (x, w13, w2[:, :64].contiguous()),
           (x, w13, w2.transpose(1, 2)), (x.cpu(), w13, w2), (off(x), w13, w2), (x, off(w13), w2), (x, w13, off(w2))]
    for args in bad:
        with pytest.raises(RuntimeError):
            ops.dense_swiglu(*args)
