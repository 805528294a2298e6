"""GPU: the decode-loop kernels at the edges of their vector paths, against the same
call on tensors that take the other path (bits where the arithmetic is the same)
or against plain PyTorch fp32."""
import pytest
import torch

from sparse_b200._lib import lib, check

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
BF = torch.bfloat16


def _stream():
    return torch.cuda.current_stream(torch.device(DEV)).cuda_stream


def _shifted(t: torch.Tensor, elements: int) -> torch.Tensor:
    """The same values at an address `elements` bf16 past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    view = buf[elements:elements + t.numel()].view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.parametrize("t,heads,dk,dv,rope_dim", [(1, 16, 128, 128, 128), (5, 3, 40, 24, 16), (3, 2, 192, 128, 64),
                                                   (2, 2, 64, 64, 0), (1000, 1, 16, 8, 16)])
def test_rope_vectors_give_the_bits_of_single_elements(t, heads, dk, dv, rope_dim):
    torch.manual_seed(dk + t)
    s_max = t + 3
    q, k, v = (torch.randn(t, heads * d, device=DEV).to(BF) for d in (dk, dk, dv))
    seq = torch.zeros(t, dtype=torch.int32, device=DEV)
    pos = torch.arange(t, dtype=torch.int32, device=DEV)
    pos[0] = s_max                                    # past the cache: q turns, nothing is stored
    got = []
    for move in (lambda x: x.clone(), lambda x: _shifted(x, 1)):
        qq, kk, vv = move(q), move(k), move(v)
        ck, cv = (torch.zeros(1, s_max, heads, d, dtype=BF, device=DEV) for d in (dk, dv))
        check(lib.sb_rope_append(qq.data_ptr(), kk.data_ptr(), vv.data_ptr(), seq.data_ptr(), pos.data_ptr(), t, heads,
                                 heads, dk, dv, rope_dim, 1.0e4, s_max, ck.data_ptr(), cv.data_ptr(), 0, 0, 0,
                                 _stream()), "sb_rope_append")
        got.append((qq, ck, cv))
    torch.cuda.synchronize()
    for a, b in zip(*got):
        assert torch.equal(a, b)
    assert torch.equal(got[0][2][0, 1:t].reshape(t - 1, -1), v[1:])
