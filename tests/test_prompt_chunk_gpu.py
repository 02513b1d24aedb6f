"""The attention of a prompt chunk (consecutive tokens of one sequence) and argmax over rows that several CTAs share, at the
edges of their tiles, against plain float64 / integer references."""
import numpy as np
import pytest
import torch

from engine_b200 import _lib, decode

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ops(ctx):
    return decode.CudaDenseOps(ctx)


# rows = tokens * heads per KV head in tiles of 48: whole tiles, a ragged last one, a group that does not divide a tile, eight
# heads, one head; chunks just below and above what the tile kernel takes on 148 SMs
@pytest.mark.parametrize("count,start,q_heads,kv_heads,out_dtype", [
    (112, 47, 32, 8, torch.float32), (108, 0, 32, 8, torch.float32), (160, 30, 24, 8, torch.float32), (161, 64, 24, 8, torch.float32),
    (75, 250, 64, 8, torch.bfloat16), (600, 0, 8, 8, torch.float32), (130, 1000, 32, 8, torch.float32), (74, 70, 64, 8, torch.float32),
    (15, 70, 4, 1, torch.float32),
])
def test_chunk_attention(ctx, ops, count, start, q_heads, kv_heads, out_dtype):
    d, max_context = 128, start + count + 5
    generator = torch.Generator(device=ctx.device)
    generator.manual_seed(count + start)
    q = 3 * torch.randn(count, q_heads, d, device=ctx.device, generator=generator)
    k_cache = torch.randn(1, kv_heads, max_context, d, device=ctx.device, generator=generator).to(torch.float16)
    v_cache = torch.randn(1, kv_heads, max_context, d, device=ctx.device, generator=generator).to(torch.float16)
    k_cache[:, :, start + count:] = float("nan")     # past the last token: must not be looked at
    v_cache[:, :, start + count:] = float("nan")
    positions = torch.arange(start, start + count, dtype=torch.int32, device=ctx.device)
    code = _lib.RIBN_F32 if out_dtype == torch.float32 else _lib.RIBN_BF16
    attention = _lib.Attention(count, q_heads, kv_heads, d, d, 1e6, 1e-6, None, None, positions.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(),
                               max_context, start + count, 1, code)
    out = torch.zeros(count, q_heads, d, dtype=out_dtype, device=ctx.device)
    ops.attention_decode(attention, q, out)
    ctx.synchronize()
    keys = k_cache[0, :, :start + count].double().repeat_interleave(q_heads // kv_heads, 0)
    values = v_cache[0, :, :start + count].double().repeat_interleave(q_heads // kv_heads, 0)
    scores = torch.einsum("thd,hsd->hts", q.double(), keys) / d ** 0.5
    visible = torch.arange(start + count, device=ctx.device)[None, :] <= positions[:, None]
    expected = torch.einsum("hts,hsd->thd", torch.softmax(scores.masked_fill(~visible[None], float("-inf")), -1), values)
    error = (out.double() - expected).abs()
    bound = 2e-5 if out_dtype == torch.float32 else 2e-5 + 2.0 ** -8 * expected.abs()
    assert torch.all(error <= bound), float(error.max())


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
