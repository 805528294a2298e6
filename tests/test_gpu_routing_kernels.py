"""GPU: the routing kernels at the edges of their launch shapes."""
import pytest
import torch

from oracle import moe_oracle as mo
from sparse_b200 import ops

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("n,e", [(1, 3), (31, 60), (2048, 60), (2049, 256), (4097, 7), (262144, 64), (262145, 64)])
def test_expert_sort_at_its_size_limits(n, e):
    """One warp's items, one CTA, the cluster of eight, the three-kernel path."""
    torch.manual_seed(n)
    ids = (torch.rand(n).pow(3) * e).to(torch.int32).clamp_(max=e - 1)
    slot, item, offs = mo.expert_sorted_permutation(ids.view(n, 1), e)
    p = ops.permute(torch.zeros(n, 8, dtype=torch.bfloat16, device=DEV), ids.to(DEV), e, 1)
    assert torch.equal(p.expert_offsets.cpu().long(), offs)
    assert torch.equal(p.slot_of_item.cpu().long()[:n], slot)
    assert torch.equal(p.item_of_slot.cpu().long()[:n], item)
    tt, want = p.tile_table.cpu(), []
    for x in range(e):
        want += [[x, b, min(b + 256, int(offs[x + 1])), 0] for b in range(int(offs[x]), int(offs[x + 1]), 256)]
    assert int(tt[0]) == len(want) and tt[4:4 + 4 * len(want)].view(-1, 4).tolist() == want


@pytest.mark.parametrize("h,e,k,dtype", [(2048, 60, 4, torch.bfloat16), (264, 256, 8, torch.bfloat16),
                                         (2048, 64, 6, torch.float32), (16384, 8, 2, torch.bfloat16)])
def test_router_rows_do_not_depend_on_the_tile_shape(h, e, k, dtype):
    """Every tile shape of the router alone (tokens per CTA, CTAs per tile), ragged last tiles: the bits
    of one token alone.  (The shapes beside a GEMM, from 593 tokens on: test_gpu_layer_calls.py.)"""
    torch.manual_seed(h + e)
    total = 1100
    x = torch.randn(total, h, device=DEV).to(dtype)
    wg, ws = (torch.randn(e, h, device=DEV) * 0.02).to(dtype), (torch.randn(h, device=DEV) * 0.02).to(dtype)
    bias = torch.randn(e, device=DEV)
    whole = ops.router_topk(x, wg, k, bias, ws)
    for t in (1, 2, 73, 75, 147, 149, 295, 297, 591, 593, 887, 889, 1035, 1037):
        part = ops.router_topk(x[:t].contiguous(), wg, k, bias, ws)
        for a, b in zip(whole, part):
            assert torch.equal(a[:t], b)
    one = ops.router_topk(x[total - 1:].contiguous(), wg, k, bias, ws)
    for a, b in zip(whole, one):
        assert torch.equal(a[total - 1:], b)


@pytest.mark.parametrize("h,i", [(64, 64), (128, 192), (192, 320), (256, 448), (448, 64)])
@pytest.mark.parametrize("t", [1, 17, 32, 33])
def test_light_tiles_of_any_depth(h, i, t):
    """K steps that fill the last stage of a light tile once, twice or wholly."""
    torch.manual_seed(h + i + t)
    x = torch.randn(t, h, device=DEV).to(torch.bfloat16)
    w13 = (torch.randn(1, 2 * i, h, device=DEV) * 0.1).to(torch.bfloat16)
    w2 = (torch.randn(1, h, i, device=DEV) * 0.1).to(torch.bfloat16)
    out, hid = ops.grouped_swiglu(x, w13, w2, dense_rows=t)
    g, u = (x.float() @ w13[0, j::2].float().T for j in (0, 1))
    bf = torch.bfloat16
    want_h = (torch.nn.functional.silu(g.to(bf).float()).to(bf) * u.to(bf)).float()
    # fp32 sums in another order move a bf16 rounding now and then: a few steps of 2^-8 of a value
    assert float((hid[:t].float() - want_h).norm() / want_h.norm()) < 5e-3
    want = hid[:t].float() @ w2[0].float().T
    assert float((out[:t].float() - want).norm() / want.norm()) < 5e-3
