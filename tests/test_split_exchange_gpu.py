"""Split-K calls whose CTAs share the sum of their partial tiles: whoever waits, gives up or comes last, and whatever runs beside them,
the result has the same bits, and the counters are ready for the next call."""
import numpy as np
import pytest
import torch

import engine_b200
from engine_b200 import synth

pytestmark = pytest.mark.gpu


def weight_of(ctx, vt, n, k):
    data = torch.from_numpy(synth.random_weight(vt, k, n, seed=n + k).reshape(-1).view(np.uint8)).to(ctx.device)
    return engine_b200.CudaQuantizedWeight(engine_b200.WeightTensorSpec.new("w", [k, n]), vt, data)


def call(ctx, weight, x, y):
    if x.shape[0] > 64:
        engine_b200.gemm(ctx, weight, x, y)
    else:
        engine_b200.QwenGemvKernel.from_value_type(weight.value_type(), ctx).execute_warp_batch(weight, x, y, x.shape[0])


# batch GEMV (up to 64 rows) and GEMM; splits chosen and forced, one round of tiles and more (nobody waits there), ragged row counts,
# more slices than shares
@pytest.mark.parametrize("vt,n,k,rows,split", [(12, 1024, 4096, 16, 0), (14, 333, 8192, 64, 0), (13, 1022, 4096, 33, 3), (12, 128, 8192, 9, 32),
                                               (12, 256, 7168, 17, 25), (12, 16000, 1024, 16, 4), (14, 512, 4096, 65, 0), (13, 1000, 5120, 173, 0),
                                               (12, 130, 8192, 100, 32), (8, 512, 6400, 300, 25), (12, 8000, 1024, 700, 3)])
@pytest.mark.parametrize("y_dtype", [torch.float32, torch.bfloat16])
def test_the_sum_does_not_depend_on_who_adds_it(ctx, vt, n, k, rows, split, y_dtype):
    weight = weight_of(ctx, vt, n, k)
    x = torch.from_numpy(synth.random_activations(rows, k, seed=rows)).to(ctx.device).to(torch.bfloat16)
    results = []
    try:
        ctx.set_option("tc_ksplit", split)
        for wait_ns in (0, 1, 2000, 100000):
            ctx.set_option("exchange_wait_ns", wait_ns)
            for _ in range(4):
                y = torch.full((rows, n), float("nan"), device=ctx.device, dtype=y_dtype)
                call(ctx, weight, x, y)
                results.append(y)
    finally:
        ctx.set_option("tc_ksplit", 0)
        ctx.set_option("exchange_wait_ns", 100000)
    ctx.synchronize()
    assert torch.isfinite(results[0]).all()
    assert all(torch.equal(y, results[0]) for y in results)


def test_calls_of_two_contexts_overlap(ctx):
    """Two owners with a stream each, as two models in one process: their split-K calls share the GPU."""
    cases = [(12, 1024, 4096, 16), (14, 4096, 12288, 64), (13, 5120, 5120, 173), (12, 512, 4096, 65), (14, 1024, 5120, 33)]
    weights = [weight_of(ctx, vt, n, k) for vt, n, k, _ in cases]
    xs = [torch.from_numpy(synth.random_activations(rows, k, seed=rows)).to(ctx.device).to(torch.bfloat16) for _, _, k, rows in cases]
    outputs = lambda: [torch.full((rows, n), float("nan"), device=ctx.device) for _, n, _, rows in cases]
    alone = outputs()
    for w, x, y in zip(weights, xs, alone):
        call(ctx, w, x, y)
    ctx.synchronize()
    owners = [engine_b200.RibnContext(0, torch.cuda.Stream()) for _ in range(2)]
    try:
        rounds = [[outputs() for _ in range(12)] for _ in owners]
        torch.cuda.synchronize()
        for step in range(12):
            for i in range(len(cases)):
                for owner, made in zip(owners, rounds):
                    j = i if owner is owners[0] else len(cases) - 1 - i   # different calls side by side
                    call(owner, weights[j], xs[j], made[step][j])
        for owner in owners:
            owner.synchronize()
        assert all(torch.equal(y, reference) for made in rounds for one in made for y, reference in zip(one, alone))
    finally:
        for owner in owners:
            owner.close()
