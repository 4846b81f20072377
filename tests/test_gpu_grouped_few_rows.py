"""The grouped product where experts get a few rows: streamed in tiles of 8 and 16 pairs (and, from 16 pairs an expert on, tiles of 64), and
on tcgen05, which serves many experts from the first row on; experts with no, one and one more row than a tile, more experts than a
warp looks at in one go, odd sizes; against 64 bits."""
import pytest
import torch

from llmengine_b200.engine.batch import StepBatch
from llmengine_b200.engine.plan import Plan

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rows,top,n,k", [
    ([1], 1, 16, 8), ([0, 8, 0, 9, 1, 0], 2, 34, 72), ([3] * 40 + [9] + [0] * 30 + [1], 1, 18, 64), ([16, 17, 0, 15], 4, 64, 520),
    ([5, 2, 0, 7], 2, 2048, 2048), ([20, 33, 64, 65], 2, 130, 200)])
@pytest.mark.parametrize("act", [None, "silu", "relu2", "gelu"])
@pytest.mark.parametrize("gather,scatter", [(True, False), (False, True)])
@pytest.mark.parametrize("kernel", ["mma", "tcgen05"])
def test_few_rows(rows, top, n, k, act, gather, scatter, kernel):
    from llmengine_b200.kernels.ops import CudaOps
    ops, g = CudaOps(torch.device(DEV)), torch.Generator(device=DEV).manual_seed(sum(rows) + n)
    ops.choose("grouped_linear", kernel)
    E, pairs = len(rows), -(-sum(rows) // top) * top
    rows = rows[:-1] + [rows[-1] + pairs - sum(rows)]                    # whole tokens
    T = pairs // top
    offsets = torch.tensor([sum(rows[:e]) for e in range(E + 1)], dtype=torch.int32, device=DEV)
    order = torch.randperm(pairs, generator=g, device=DEV).to(torch.int32)
    x = torch.randn(T if gather else pairs, k, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(E, n, k, generator=g, device=DEV) / k ** 0.5).to(torch.bfloat16)
    n_out = n // 2 if act == "silu" else n
    dtype = torch.bfloat16 if gather else torch.float32
    out, mid, plan = torch.full((pairs, n_out), 7.0, dtype=dtype, device=DEV), torch.empty(pairs, n, dtype=torch.bfloat16, device=DEV), Plan()
    plan.grouped_linear(x=x, w=w, out=out, offsets=offsets, order=order, top_k=top, gather=gather, scatter=scatter, mid=mid, act=act,
                        rows=torch.empty(pairs, k, dtype=torch.bfloat16, device=DEV) if gather else None)
    ops.compile(plan).run(StepBatch.bare(T, torch.device(DEV)))
    torch.cuda.synchronize()
    for e in range(E):
        at = torch.arange(int(offsets[e]), int(offsets[e + 1]), device=DEV)
        pair = order[at].long()
        z = x[pair // top if gather else at].double() @ w[e].double().t()
        got = out[pair if scatter else at].double()
        err = k * 2.0 ** -24 * (x.double().abs().max() * w.double().abs().max())          # 32-bit sums of k products in any order
        slope = 2.0 * z.abs() + 1.2                                                       # of every activation
        if act == "silu":
            b = z.to(torch.bfloat16).double()
            gate, up = b[:, :n_out], b[:, n_out:]
            want = gate * torch.sigmoid(gate) * up
            # a neighbouring bfloat16 (2^-8) of either argument; the gate's slope is below 1.1
            bound = 2.0 ** -8 * (1.1 * gate.abs() * up.abs() + gate.abs() * up.abs()) + 1e-5
        else:
            want = z if act is None else z.clamp(min=0) ** 2 if act == "relu2" else torch.nn.functional.gelu(z)
            bound = err * slope + 1e-5 * want.abs()
        bound = bound + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0.0) + 1e-6
        assert bool(((got - want).abs() <= bound).all()), (e, float(((got - want).abs() / bound).max()))
