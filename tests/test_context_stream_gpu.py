"""torch's current stream beside several contexts: each one orders uploads, torch's own work and its launches on the stream
that it made current, so closing another one must not take that stream away."""
import pytest
import torch

from diffgemma_b200.step_attn import Context

pytestmark = pytest.mark.gpu


def test_closing_a_context_leaves_the_others_stream_current(ctx):
    before = torch.cuda.current_stream()
    a = Context(0)
    b = Context(0)
    assert torch.cuda.current_stream() == b.torch_stream
    a.close()
    assert torch.cuda.current_stream() == b.torch_stream
    c = Context(0)
    c.close()
    assert torch.cuda.current_stream() == b.torch_stream
    b.close()
    assert torch.cuda.current_stream() == a.torch_stream
    torch.cuda.set_stream(before)
    d = Context(0)
    d.close()
    assert torch.cuda.current_stream() == before
