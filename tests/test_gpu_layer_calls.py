"""GPU: the layer pass as programs call it: rows made just before a pass, buffers used again."""
import pytest
import torch

from sparse_b200 import synth
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
