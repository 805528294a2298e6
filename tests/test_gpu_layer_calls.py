"""GPU: the layer pass as programs call it: rows made just before a pass, buffers used again."""
import pytest
import torch

from sparse_b200 import ops, synth
from sparse_b200._lib import lib, check
from sparse_b200.block import B200MoeBlock
from sparse_b200.layer import LayerRunner
from sparse_b200.model import random_layer_weights

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")
BF = torch.bfloat16
_WEIGHTS = {}


def _weights(name):
    if name not in _WEIGHTS:
        shape = getattr(synth, name)
        _WEIGHTS[name] = random_layer_weights(shape, DEV, 5, range(shape.num_experts))
    return _WEIGHTS[name]


def _rows(tokens, hidden, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn((tokens, hidden), generator=gen, device=DEV).to(BF)


@pytest.mark.parametrize("t", [1, 2, 8, 16])
def test_rows_written_just_before_a_pass_are_the_ones_it_reads(t):
    """One input buffer, rewritten by a kernel right in front of every pass."""
    runner = LayerRunner(_weights("QWEN_MOE"), synth.QWEN_MOE.top_k, t)
    batches = [_rows(t, synth.QWEN_MOE.hidden, s) for s in range(3)]
    want = []
    for b in batches:
        want.append(runner.forward(b)[0].clone())
        torch.cuda.synchronize()
    x = torch.empty_like(batches[0])
    out = [torch.empty_like(x) for _ in range(24)]
    for i, o in enumerate(out):
        x.copy_(batches[i % 3])
        runner.forward(x, o)
    torch.cuda.synchronize()
    for i, o in enumerate(out):
        assert torch.equal(o, want[i % 3])
    runner.check_status()


@pytest.mark.parametrize("t", [1, 2, 3, 4, 5, 16])
def test_decode_rows_do_not_depend_on_how_the_experts_are_called(t):
    """The Qwen shape's rows through the one-GPU layer, and through the calls that the
    expert-parallel step, the local expert cache and the offloaded layer make: the same bits."""
    shape, w = synth.QWEN_MOE, _weights("QWEN_MOE")
    h, i, e, k = shape.hidden, shape.inter, shape.num_experts, shape.top_k
    runner = LayerRunner(w, k, t)
    x = _rows(t, h, 70 + t)
    want, idx, wts, _ = runner.forward(x)
    gate = ops.router_topk(x, w.router_w, k, bias=w.router_bias, w_shared_gate=w.shared_gate_w)[3]
    p = ops.permute(x, idx.reshape(-1), e, k, item_scale=wts.reshape(-1))
    hbuf = torch.empty((p.r_cap, i), dtype=BF, device=DEV)
    status = torch.zeros((1,), dtype=torch.int32, device=DEV)
    stream = torch.cuda.current_stream(DEV).cuda_stream
    shared_h = torch.empty((t, shape.shared_inter), dtype=BF, device=DEV)

    def experts(y, slots, shared_out):
        on = shared_out is not None
        check(lib.sb_decode_experts(
            x.data_ptr(), p.item_of_slot.data_ptr(), k, p.tile_table.data_ptr(), slots.data_ptr(), w.w13.data_ptr(),
            w.w2.data_ptr(), p.slot_scale.data_ptr(), h, i, w.n_slots, hbuf.data_ptr(), y.data_ptr(),
            w.shared_w13.data_ptr() if on else None, w.shared_w2.data_ptr() if on else None,
            gate.data_ptr() if on else None, shape.shared_inter if on else 0, t,
            shared_h.data_ptr() if on else None, shared_out.data_ptr() if on else None, status.data_ptr(), stream),
            "sb_decode_experts")

    def mixed(y, dst):
        check(lib.sb_grouped_swiglu_mixed(
            p.rows.data_ptr(), p.tile_table.data_ptr(), w.w13.data_ptr(), w.w2.data_ptr(), w.slot_of_expert.data_ptr(),
            p.slot_scale.data_ptr(), p.r_cap, h, i, w.n_slots, hbuf.data_ptr(), y.data_ptr(), 0, None, None, None,
            None, 0, 0, None, None, dst.data_ptr() if dst is not None else None, status.data_ptr(), stream),
            "sb_grouped_swiglu_mixed")

    # the shared expert by itself, as the expert-parallel step calls it
    alone = torch.empty((t, h), dtype=BF, device=DEV)
    check(lib.sb_decode_experts(
        x.data_ptr(), None, 1, None, None, None, None, None, h, i, 1, None, None, w.shared_w13.data_ptr(),
        w.shared_w2.data_ptr(), gate.data_ptr(), shape.shared_inter, t, shared_h.data_ptr(), alone.data_ptr(),
        status.data_ptr(), stream), "sb_decode_experts(shared)")
    got = {}
    y = {name: torch.full((p.r_cap, h), float("nan"), dtype=BF, device=DEV)
         for name in ("waves", "received", "scattered", "cached")}
    beside = torch.empty((t, h), dtype=BF, device=DEV)
    # the offloaded layer: the experts in two launches, the shared one in the first of them
    even = torch.arange(e, device=DEV) % 2 == 0
    skip = torch.full_like(w.slot_of_expert, -2)
    experts(y["waves"], torch.where(even, w.slot_of_expert, skip), beside)
    experts(y["waves"], torch.where(even, skip, w.slot_of_expert), None)
    mixed(y["received"], None)
    row_dst = {name: y[name].data_ptr() + 2 * h * torch.arange(p.r_cap, dtype=torch.int64, device=DEV)
               for name in ("scattered", "cached")}
    mixed(y["scattered"], row_dst["scattered"])
    check(lib.sb_decode_experts_to(
        x.data_ptr(), p.item_of_slot.data_ptr(), k, p.tile_table.data_ptr(), w.slot_of_expert.data_ptr(),
        w.w13.data_ptr(), w.w2.data_ptr(), p.slot_scale.data_ptr(), h, i, w.n_slots, hbuf.data_ptr(),
        row_dst["cached"].data_ptr(), t, status.data_ptr(), stream), "sb_decode_experts_to")
    got["waves"] = ops.combine(y["waves"], p.slot_of_item, idx, beside, t)
    for name in ("received", "scattered", "cached"):
        got[name] = ops.combine(y[name], p.slot_of_item, idx, alone, t)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert {name: torch.equal(o, want) for name, o in got.items()} == dict.fromkeys(got, True)


def test_recorded_passes_end_with_the_buffers_they_write_to():
    """A pass is recorded, a batch above `max_tokens` replaces the scratch and the result
    buffers, the first buffers come again: their pass writes to the new ones."""
    shape, w = synth.TINY, _weights("TINY")
    block = B200MoeBlock(w, shape.top_k, 64, use_graphs=True)
    plain = B200MoeBlock(w, shape.top_k, 200)
    x, out = _rows(48, shape.hidden, 1), torch.empty((48, shape.hidden), dtype=BF, device=DEV)
    for seed in (2, 3, 4):
        x.copy_(_rows(48, shape.hidden, seed))
        block.forward_device(x, out)
    assert len(block._graphs) == 1
    big = _rows(200, shape.hidden, 5)
    assert torch.equal(block.forward_device(big), plain.forward_device(big))
    for seed in (6, 7):
        x.copy_(_rows(48, shape.hidden, seed))
        block.forward_device(x, out)
        assert torch.equal(out, plain.forward_device(x))
        for a, b in zip((*block.topk(48), block.router_logits(48)), (*plain.topk(48), plain.router_logits(48))):
            assert torch.equal(a, b)
    block.check_status()


def test_replaced_scratch_is_not_given_away_while_a_pass_uses_it():
    """Passes wait in a stream of their own; the scratch that a larger batch replaces must not
    serve another stream's tensor before they are through."""
    shape = synth.TINY
    runner = LayerRunner(_weights("TINY"), shape.top_k, 64)
    small, big = _rows(64, shape.hidden, 1), _rows(300, shape.hidden, 2)
    stream = torch.cuda.Stream(device=DEV)
    with torch.cuda.stream(stream):                       # kernels loaded, the stream's memory at hand
        first = LayerRunner(_weights("TINY"), shape.top_k, 300)
        first.forward(small), first.forward(big)
        del first
        torch.cuda._sleep(1)
    torch.full((8,), 255, dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(400_000_000)                    # some 200 ms of the stream
        runner.forward(small)
        sizes = [runner._ws_raw.numel(), runner.out.numel() * 2]
        runner.forward(big)
    others = [torch.full((n,), 255, dtype=torch.uint8, device=DEV) for n in sizes for _ in range(4)]
    torch.cuda.synchronize()
    assert all(bool((o == 255).all()) for o in others)


@pytest.mark.parametrize("name", ["TINY", "QWEN_MOE"])
@pytest.mark.parametrize("t", [592, 593, 594, 599, 700, 887, 888, 889, 890, 895])
def test_routing_beside_the_shared_pass_gives_the_bits_of_the_router_alone(name, t):
    """The layer pass's own router tiles (six tokens, shared by two CTAs up to 888 tokens),
    ragged last tiles among them."""
    shape, w = getattr(synth, name), _weights(name)
    runner = LayerRunner(w, shape.top_k, t)
    x = _rows(t, shape.hidden, t)
    _, *got = runner.forward(x)
    want = ops.router_topk(x, w.router_w, shape.top_k, bias=w.router_bias, w_shared_gate=w.shared_gate_w)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
