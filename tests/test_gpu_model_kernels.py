"""GPU: the decode-loop kernels at the edges of their vector paths, against the same
call on tensors that take the other path (bits where the arithmetic is the same)
or against plain PyTorch fp32."""
import math

import pytest
import torch

from sparse_b200 import ops
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
    assert torch.equal(got[0][2][0, 1:t].flatten(), v[1:].flatten())


@pytest.mark.parametrize("t,h,with_delta", [(3, 8, True), (2, 504, True), (1, 2056, False), (2, 16384, True)])
def test_rmsnorm_vectors_give_the_bits_of_single_elements(t, h, with_delta):
    torch.manual_seed(h)
    resid, delta = (torch.randn(t, h, device=DEV).to(BF) for _ in range(2))
    w = torch.randn(h, device=DEV).to(BF)
    got = []
    for off in (0, 1):
        r, d, o = _shifted(resid, off), _shifted(delta, off), _shifted(resid, off)
        check(lib.sb_add_rmsnorm(r.data_ptr(), d.data_ptr() if with_delta else None, None, w.data_ptr(), 1e-6, t, h,
                                 o.data_ptr(), _stream()), "sb_add_rmsnorm")
        got.append((r, o))
    torch.cuda.synchronize()
    for r, o in got[1:]:
        assert torch.equal(r, got[0][0]) and torch.equal(o, got[0][1])
    x = (resid.float() + delta.float()).to(BF).float() if with_delta else resid.float()
    want = w.float() * (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6)).to(BF).float()
    # rsqrt and the fp32 mean may round differently: one bf16 step of the largest value
    assert float((got[0][1].float() - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max())


@pytest.mark.parametrize("n_q,n_kv,dk,dv", [(4, 4, 128, 128), (2, 2, 192, 128), (4, 2, 64, 64)])
@pytest.mark.parametrize("n_split,shift", [(1, 0), (3, 2), (256, 0)])
def test_attn_decode_key_group_edges(n_q, n_kv, dk, dv, n_split, shift):
    """Lengths around the 16 keys of a CTA's groups and its 32 per iteration, more splits
    than keys, caches on 4-byte boundaries."""
    torch.manual_seed(dk + n_split)
    lens = [0, 1, 15, 16, 17, 31, 32, 33, 97]
    b, s_max = len(lens), max(lens)
    q = torch.randn(b, n_q, dk, device=DEV).to(BF)
    ck = _shifted(torch.randn(b, s_max, n_kv, dk, device=DEV).to(BF), shift)
    cv = _shifted(torch.randn(b, s_max, n_kv, dv, device=DEV).to(BF), shift)
    cv[2, 15:] = float("inf")                         # past the length: read by nobody's sum
    seq_lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    ws = torch.empty(lib.sb_attn_decode_workspace_bytes(b, n_q, dv, n_split), dtype=torch.uint8, device=DEV)
    out = torch.empty(b, n_q, dv, dtype=BF, device=DEV)
    check(lib.sb_attn_decode(q.data_ptr(), 0, ck.data_ptr(), cv.data_ptr(), seq_lens.data_ptr(), b, n_q, n_kv, dk, dv,
                             s_max, 1.0 / math.sqrt(dk), n_split, ws.data_ptr(), ws.numel(), out.data_ptr(), _stream()),
          "sb_attn_decode")
    torch.cuda.synchronize()
    assert float(out[0].abs().max()) == 0.0
    for i, n in enumerate(lens[1:], 1):
        kk = ck[i, :n].float().repeat_interleave(n_q // n_kv, dim=1)
        vv = cv[i, :n].float().repeat_interleave(n_q // n_kv, dim=1)
        p = torch.softmax(torch.einsum("hd,nhd->hn", q[i].float(), kk) / math.sqrt(dk), dim=-1)
        want = torch.einsum("hn,nhd->hd", p, vv)
        # fp32 sums, one rounding to bf16: half a step of 2^-8 of a value, and __expf's 2^-21
        assert float(((out[i].float() - want).abs() - 2.0 ** -8 * want.abs()).max()) < 1e-4


@pytest.mark.parametrize("t,heads,rope,nope,dv,lora", [(1, 16, 64, 128, 128, 512), (5, 3, 16, 20, 12, 40)])
def test_mla_append_and_strided_norm_give_the_bits_of_assembled_rows(t, heads, rope, nope, dv, lora):
    torch.manual_seed(t + lora)
    dk, s_max = rope + nope, t + 2
    kv_a = torch.randn(t, lora + rope, device=DEV).to(BF)
    kv = torch.randn(t, heads, nope + dv, device=DEV).to(BF)
    q = torch.randn(t, heads * dk, device=DEV).to(BF)
    w = torch.randn(lora, device=DEV).to(BF)
    seq, pos = torch.zeros(t, dtype=torch.int32, device=DEV), torch.arange(t, dtype=torch.int32, device=DEV)
    k = torch.cat([kv_a[:, lora:].unsqueeze(1).expand(t, heads, rope), kv[:, :, :nope]], dim=2).contiguous()
    v = kv[:, :, nope:].contiguous()
    caches = [[torch.zeros(1, s_max, heads, d, dtype=BF, device=DEV) for d in (dk, dv)] for _ in range(2)]
    q1, q2 = q.clone(), q.clone()
    check(lib.sb_rope_append(q1.data_ptr(), k.data_ptr(), v.data_ptr(), seq.data_ptr(), pos.data_ptr(), t, heads, heads,
                             dk, dv, rope, 1.0e4, s_max, caches[0][0].data_ptr(), caches[0][1].data_ptr(), 0, 0, 0,
                             _stream()), "sb_rope_append")
    check(lib.sb_rope_append_mla(q2.data_ptr(), kv_a[:, lora:].data_ptr(), kv.data_ptr(), seq.data_ptr(), pos.data_ptr(),
                                 t, heads, rope, nope, dv, 1.0e4, s_max, caches[1][0].data_ptr(),
                                 caches[1][1].data_ptr(), heads * dk, lora + rope, heads * (nope + dv), _stream()),
          "sb_rope_append_mla")
    latent, a, b = kv_a[:, :lora].contiguous(), *(torch.empty(t, lora, dtype=BF, device=DEV) for _ in range(2))
    check(lib.sb_add_rmsnorm(latent.data_ptr(), None, None, w.data_ptr(), 1e-6, t, lora, a.data_ptr(), _stream()), "norm")
    check(lib.sb_rmsnorm_rows(kv_a.data_ptr(), lora + rope, w.data_ptr(), 1e-6, t, lora, b.data_ptr(), _stream()), "rows")
    torch.cuda.synchronize()
    assert torch.equal(q1, q2) and torch.equal(a, b)
    assert all(torch.equal(x, y) for x, y in zip(*caches))


@pytest.mark.parametrize("t", [1, 8, 9, 16, 17])
def test_dense_swiglu_on_either_side_of_the_streaming_limit(t):
    torch.manual_seed(t)
    h, i = 256, 1216
    x = torch.randn(t, h, device=DEV).to(BF)
    w13 = (0.05 * torch.randn(1, 2 * i, h, device=DEV)).to(BF)
    w2 = (0.05 * torch.randn(1, h, i, device=DEV)).to(BF)
    got = ops.dense_swiglu(x, w13, w2).float()
    want = ops.grouped_swiglu(x, w13, w2, dense_rows=t)[0].float()
    # fp32 sums in another order: the two differ where a bf16 rounding falls the other way
    assert got.shape == (t, h)
    assert float((got - want).norm() / want.norm()) < 5e-3


@pytest.mark.parametrize("b,v", [(1, 1), (3, 4096), (2, 102400), (8, 151936), (2, 1003)])
def test_argmax_rows_is_torch_argmax(b, v):
    torch.manual_seed(v)
    logits = (torch.randn(b, v, device=DEV) * 0.5).to(BF)          # coarse values: many ties
    logits[0, v // 2] = -0.0
    if b > 1:
        logits[1] = -float("inf")
        logits[1, v - 1] = float("nan") if v == 4096 else -float("inf")
    if b > 2:
        logits[2] = 0.0
        logits[2, ::2] = -0.0
    ids = torch.empty(b, dtype=torch.int64, device=DEV)
    check(lib.sb_argmax_rows(logits.data_ptr(), b, v, ids.data_ptr(), _stream()), "sb_argmax_rows")
    torch.cuda.synchronize()
    assert torch.equal(ids.cpu(), torch.argmax(logits.float().cpu(), dim=-1))


@pytest.mark.parametrize("t", [1, 8, 9, 16, 17])
@pytest.mark.parametrize("n,k,with_bias", [(1, 32, True), (130, 96, False), (2048, 2048, True), (6144, 512, False)])
def test_linear_on_either_side_of_the_streaming_limit(t, n, k, with_bias):
    torch.manual_seed(t + n)
    x = torch.randn(t, k, device=DEV).to(BF)
    w = (torch.randn(n, k, device=DEV) / math.sqrt(k)).to(BF)
    b = torch.randn(n, device=DEV).to(BF) if with_bias else None
    got = ops.linear(x, w, b)
    want = x.double() @ w.double().T + (b.double() if with_bias else 0.0)
    # fp32 sums of at most 2048 products of order 1 / sqrt(k), one rounding to bf16
    assert got.shape == (t, n)
    assert float(((got.double() - want).abs() - 2.0 ** -8 * want.abs()).max()) < 1e-4


@pytest.mark.parametrize("n_q,n_kv,dk,dv", [(2, 2, 128, 128), (2, 1, 192, 128), (2, 2, 64, 64)])
@pytest.mark.parametrize("n_split", [1, 4])
def test_attn_decode_scores_of_minus_infinity_weigh_nothing(n_q, n_kv, dk, dv, n_split):
    """Keys with a score of -inf alone in a group's first turn, in a warp, in a split; a
    sequence of nothing else gives zeros, as an empty one does."""
    torch.manual_seed(dk + n_split)
    lens = [5, 17, 40, 97, 33, 6]
    dead = [[0], [16], [0, 1, 2, 3, 20], [0, 31, 32, 96], list(range(0, 33, 2)), list(range(6))]
    b, s_max = len(lens), max(lens)
    q = (torch.rand(b, n_q, dk, device=DEV) + 0.1).to(BF)
    ck = torch.randn(b, s_max, n_kv, dk, device=DEV).to(BF)
    cv = torch.randn(b, s_max, n_kv, dv, device=DEV).to(BF)
    for i, keys in enumerate(dead):
        ck[i, keys, :, 3] = float("-inf")
    seq_lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    ws = torch.empty(lib.sb_attn_decode_workspace_bytes(b, n_q, dv, n_split), dtype=torch.uint8, device=DEV)
    out = torch.empty(b, n_q, dv, dtype=BF, device=DEV)
    check(lib.sb_attn_decode(q.data_ptr(), 0, ck.data_ptr(), cv.data_ptr(), seq_lens.data_ptr(), b, n_q, n_kv, dk, dv,
                             s_max, 1.0 / math.sqrt(dk), n_split, ws.data_ptr(), ws.numel(), out.data_ptr(), _stream()),
          "sb_attn_decode")
    torch.cuda.synchronize()
    assert float(out[5].abs().max()) == 0.0
    for i, n in enumerate(lens[:5]):
        kk = ck[i, :n].float().repeat_interleave(n_q // n_kv, dim=1)
        vv = cv[i, :n].float().repeat_interleave(n_q // n_kv, dim=1)
        p = torch.softmax(torch.einsum("hd,nhd->hn", q[i].float(), kk) / math.sqrt(dk), dim=-1)
        want = torch.einsum("hn,nhd->hd", p, vv)
        # fp32 sums, one rounding to bf16: half a step of 2^-8 of a value, and __expf's 2^-21
        assert float(((out[i].float() - want).abs() - 2.0 ** -8 * want.abs()).max()) < 1e-4


@pytest.mark.parametrize("h", [12288, 12296, 16384])
def test_wide_rows_off_a_vector_boundary(h):
    """Rows whose fp32 copy is larger than 48 KB, on addresses that are no whole vectors."""
    torch.manual_seed(h)
    rows, w = torch.randn(2, h, device=DEV).to(BF), torch.randn(h, device=DEV).to(BF)
    got = []
    for off in (0, 1):
        r, o = _shifted(rows, off), _shifted(rows, off)
        check(lib.sb_rmsnorm_rows(r.data_ptr(), h, w.data_ptr(), 1e-6, 2, h, o.data_ptr(), _stream()), "sb_rmsnorm_rows")
        check(lib.sb_add_rmsnorm(r.data_ptr(), rows.data_ptr(), None, w.data_ptr(), 1e-6, 2, h, o.data_ptr(), _stream()),
              "sb_add_rmsnorm")
        got.append((r, o))
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(*got))
