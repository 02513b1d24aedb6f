"""Argmax over rows that several CTAs share, at the edges
of their pieces, against numpy."""
import numpy as np
import pytest
import torch

from engine_b200 import _lib, decode

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ops(ctx):
    return decode.CudaDenseOps(ctx)


@pytest.mark.parametrize("members,length", [(1, 1), (3, 255), (2, 4095), (2, 4096), (2, 4097), (1, 151936), (700, 12289)])
def test_argmax_of_shared_rows(ctx, ops, members, length):
    generator = torch.Generator(device=ctx.device)
    generator.manual_seed(length)
    logits = torch.randint(-500, 500, (members, length), device=ctx.device, generator=generator).float()   # many ties
    out = torch.full((members,), -1, dtype=torch.int32, device=ctx.device)
    for _ in range(2):                                # the second call finds the counters as the first left them
        ops.argmax(logits, members, out)
        ctx.synchronize()
        assert np.array_equal(out.cpu().numpy(), np.argmax(logits.cpu().numpy(), axis=1))
