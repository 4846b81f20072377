"""Prompt portions of the latent attention on tcgen05, alone: sizes at the edges of its tiles (128 rows of (token, head), 128 keys,
pages, chunks of 64 columns) against the softmax written out in 64 bits over the same queries and cache rows."""
import pytest
import torch

from llmengine_b200.engine.batch import GroupView, StepBatch
from llmengine_b200.engine.plan import Plan

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rank,rot,heads,page,window,sink,lens", [
    # lens: (cached, new) per request
    (512, 64, 16, 16, 0, False, [(0, 2), (0, 8), (0, 9), (120, 8), (127, 2), (128, 130), (0, 1), (300, 257)]),
    (512, 64, 32, 64, 0, True, [(0, 4), (61, 5), (0, 129), (255, 2), (900, 40)]),
    (512, 0, 5, 8, 0, True, [(0, 25), (0, 26), (0, 52), (7, 100)]),
    (512, 64, 16, 32, 100, False, [(0, 300), (250, 130), (99, 3), (400, 2)]),
    (512, 32, 3, 128, 7, True, [(0, 43), (130, 90)]),
    (384, 64, 8, 16, 130, True, [(0, 200), (333, 17)]),
    (256, 8, 8, 16, 0, False, [(0, 16), (5, 17), (40, 128)]),
    (128, 64, 16, 16, 0, True, [(0, 8), (3, 300), (0, 1)]),
    (128, 0, 1, 64, 33, False, [(0, 127), (0, 128), (0, 129), (64, 2)]),
])
def test_portions(rank, rot, heads, page, window, sink, lens):
    run(rank, rot, heads, page, window, sink, lens)


@pytest.mark.parametrize("page,window", [(8, 0), (16, 50), (32, 0), (64, 0), (64, 90), (128, 0)])
def test_value_rows_written_by_hand(page, window):
    """Requests that end inside a load of value rows, and windows that begin inside one, at many places at once: what lies behind the last
    token is NaN, and both blocks of a pair must see the zeros written over it, every time."""
    lens = [(37 * i % 211, 2 + (29 * i) % 70) for i in range(40)]
    first = run(512, 64, 16, page, window, False, lens)
    for _ in range(3):
        assert torch.equal(run(512, 64, 16, page, window, False, lens), first)


def run(rank, rot, heads, page, window, sink, lens):
    """Runs the step over these requests, compares every row with its 64-bit result and returns the outputs."""
    from llmengine_b200.kernels.ops import CudaOps
    ops, g = CudaOps(torch.device(DEV)), torch.Generator().manual_seed(rank + rot + heads)
    width, R, T = rank + rot, len(lens), sum(n for _, n in lens)
    need = [-(-(c + n) // page) for c, n in lens]
    perm = torch.randperm(sum(need) + 3, generator=g).tolist()
    tables, slots, positions = torch.full((R, max(need)), -1, dtype=torch.int32), [], []
    cache = torch.full((sum(need) + 3, page, width), float("nan"))
    for r, (c, n) in enumerate(lens):
        pages = [perm.pop() for _ in range(need[r])]
        gone = max(0, c + 1 - window) // page if window else 0        # pages the window has passed are not held any more
        tables[r, gone:need[r]] = torch.tensor(pages[gone:], dtype=torch.int32)
        for p in range(gone * page, c):
            cache[pages[p // page], p % page] = torch.randn(width, generator=g)
        slots += [pages[p // page] * page + p % page for p in range(c, c + n)]
        positions += range(c, c + n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    q_len = [n for _, n in lens]
    cu = [sum(q_len[:r]) for r in range(R + 1)]
    cache, q = cache.to(torch.bfloat16).to(DEV), (torch.randn(T, heads * width, generator=g) * 0.7).to(torch.bfloat16).to(DEV)
    batch = StepBatch(
        num_tokens=T, num_requests=R, q_lens=q_len, start_positions=[c for c, _ in lens], token_ids=i32([0] * T), positions=i32(positions),
        token_request=i32([r for r in range(R) for _ in range(q_len[r])]), cu_q_lens=i32(cu), ctx_lens=i32([c + n for c, n in lens]),
        state_slots=i32(list(range(R))), first_portion=i32([0] * R), logit_rows=i32([]), decode_rows=i32([r for r in range(R) if q_len[r] == 1]),
        portion_rows=i32([r for r in range(R) if q_len[r] != 1]), groups=[GroupView(page, window, tables.to(DEV), i32(slots), max(need))])
    kv_in = torch.randn(T, width, generator=g).to(torch.bfloat16).to(DEV)
    q_rot = torch.randn(T, heads, rot, generator=g).to(torch.bfloat16).to(DEV) if rot else None
    out = torch.full((T, heads * rank), 7.0, dtype=torch.bfloat16, device=DEV)
    sinks = (torch.randn(heads, generator=g) * 3).to(DEV) if sink else None
    plan, scale = Plan(), width ** -0.5
    plan.latent_attention(q_rot=q_rot, kv_in=kv_in, c_gain=torch.ones(rank, device=DEV), eps=1e-6, inv_freq=torch.linspace(1.0, 0.01, rot // 2).to(DEV) if rot else None,
                          rot_dims=rot, q=q, out=out, cache=cache, group=0, num_heads=heads, kv_rank=rank, rot_dim=rot, scale=scale, sink=sinks, window=window,
                          scratch=None)
    compiled = ops.compile(plan)
    assert f"attention_latent_tcgen05@RANK={rank}" in ops._libs
    compiled.run(batch)
    torch.cuda.synchronize()
    assert int(ops._libs[f"attention_latent_tcgen05@RANK={rank}"].llme_latent_pair_status()) == 0
    rows, qd, got = cache.double().view(-1, width), q.double().view(T, heads, width), out.double().view(T, heads, rank)
    for r, (c, n) in enumerate(lens):
        lo = max(0, c + 1 - window) if window else 0
        keys = torch.stack([rows[int(tables[r, p // page]) * page + p % page] for p in range(lo, c + n)])
        i, j = torch.arange(c, c + n, device=DEV)[:, None], torch.arange(lo, c + n, device=DEV)[None, :]
        seen = (j <= i) & ((i - j < window) if window else (j >= 0))
        s = (torch.einsum("thw,kw->htk", qd[cu[r]:cu[r + 1]], keys) * scale).masked_fill(~seen[None], float("-inf"))
        if sink:
            s = torch.cat([s, sinks.double()[:, None, None].expand(heads, n, 1)], -1)
        p = torch.softmax(s, -1)[..., :keys.shape[0]]
        want = torch.einsum("htk,kr->thr", p, keys[:, :rank])
        # probabilities are rounded to bfloat16 once (8 digits: up to 2^-8 of each, and they sum to at most one), and so is the result
        bound = 2.0 ** -8 * (float(keys[:, :rank].abs().max()) + want.abs()) * 1.05 + 1e-4
        err = (got[cu[r]:cu[r + 1]] - want).abs()
        assert bool((err <= bound).all()), f"request {r}: {float(err.max()):.3e}, {float((err / bound).max()):.3f} of the bound"
    return out
