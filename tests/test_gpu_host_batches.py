"""GPU: batches that live in host memory (`B200MoeBlock.forward_host`), whole and in parts."""
import pytest
import torch

from sparse_b200 import synth
from sparse_b200.block import B200MoeBlock
from sparse_b200.model import random_layer_weights

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")
BF = torch.bfloat16
SHAPE = synth.TINY


@pytest.fixture(scope="module")
def weights():
    return random_layer_weights(SHAPE, DEV, 3, range(SHAPE.num_experts))


def _rows(tokens, seed):
    return torch.randn((tokens, SHAPE.hidden), generator=torch.Generator().manual_seed(seed)).to(BF)


def _pinned(*shape):
    return torch.empty(shape, dtype=BF).pin_memory()


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("t", [3071, 3072, 3073, 12289])
def test_host_batches_equal_device_batches(weights, t, graphs):
    """Either side of the split, ragged parts, the same pinned buffers with other rows each time."""
    block = B200MoeBlock(weights, SHAPE.top_k, t, use_graphs=graphs)
    other = B200MoeBlock(weights, SHAPE.top_k, t)
    x, out = _pinned(t, SHAPE.hidden), _pinned(t, SHAPE.hidden)
    for call in range(4):
        rows = _rows(t, 10 * t + call)
        x.copy_(rows)
        out.fill_(float("nan"))
        block.forward_host(x, out)
        want = other.forward_device(rows.to(DEV))
        assert torch.equal(out, want.cpu())
        for a, b in zip((*block.topk(t), block.router_logits(t)), (*other.topk(t), other.router_logits(t))):
            assert torch.equal(a, b)
        if call == 0:                         # the first pass on new buffers records nothing
            assert not block._graphs and not any(block._part_graphs.values())
    block.check_status()


def test_a_recorded_part_takes_no_place_of_a_recorded_batch(weights):
    """Split batches of many sizes leave the graphs of a serving loop's own buffers alone."""
    t = 4096
    block = B200MoeBlock(weights, SHAPE.top_k, t, use_graphs=True)
    x = _rows(64, 1).to(DEV)
    y = torch.empty_like(x)
    block.forward_device(x, y)
    block.forward_device(x, y)
    kept = dict(block._graphs)
    assert len(kept) == 1
    for n in range(3072, 3072 + 20):
        rows, out = _rows(n, n), _pinned(n, SHAPE.hidden)
        for _ in range(2):
            block.forward_host(rows.pin_memory(), out)
        assert torch.equal(out, block.runner.forward(rows.to(DEV))[0].cpu())
    assert all(block._graphs.get(k) is v for k, v in kept.items())


@pytest.mark.parametrize("t", [2048, 3072])
def test_result_buffers_of_another_shape(weights, t):
    """What a copy of the whole result takes or refuses, at any size."""
    block = B200MoeBlock(weights, SHAPE.top_k, t)
    x = _rows(t, t).pin_memory()
    h = SHAPE.hidden
    want = block.forward_device(x.to(DEV)).cpu()
    for shape in ((t + 1, h), (t - 1, h), (t, h + 8)):
        with pytest.raises(RuntimeError):
            block.forward_host(x, _pinned(*shape))
        torch.cuda.synchronize()
    for shape in ((1, t, h), (2, t, h)):
        out = _pinned(*shape)
        block.forward_host(x, out)
        assert all(torch.equal(o, want) for o in out)


@pytest.mark.parametrize("shift", [0, 48])
def test_result_rows_over_the_input_rows(weights, shift):
    """The result may go where the input lay, also some rows further on."""
    t = 3072
    block = B200MoeBlock(weights, SHAPE.top_k, t)
    rows = _rows(t, 5)
    want = block.forward_device(rows.to(DEV)).cpu()
    buf = _pinned(t + shift, SHAPE.hidden)
    for _ in range(3):
        buf[:t] = rows
        block.forward_host(buf[:t], buf[shift:])
        assert torch.equal(buf[shift:], want)
