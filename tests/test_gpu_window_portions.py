"""The window attention with a sink, kept first positions and a cap in the grouped-query kernels (prompt portions on tcgen05, single
tokens in shares of the context), behind the norm over the whole projection: sizes at the edges of tiles (128 keys, 128 rows of a
group, 16 keys, pages), against the formulas in 64 bits."""
import pytest
import torch

from llmengine_b200.engine.batch import GroupView, StepBatch
from llmengine_b200.engine.plan import Plan

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 1e-6


@pytest.mark.parametrize("H,G,d,page,window,first,sink,cap,norm,rot,interleaved,lens", [
    # lens: (cached, new) per request
    (16, 4, 128, 16, 100, 4, True, 0.0, True, 64, False, [(0, 300), (250, 131), (0, 2), (700, 3)]),
    (8, 8, 128, 64, 128, 130, True, 0.0, False, 128, True, [(0, 129), (600, 140), (257, 2)]),
    (6, 3, 64, 8, 0, 0, True, 0.0, True, 10, False, [(0, 64), (127, 65), (128, 128)]),
    (8, 1, 64, 32, 33, 1, False, 2.0, True, 0, False, [(0, 17), (500, 33), (31, 97)]),
    (4, 2, 128, 128, 257, 3, False, 0.0, False, 32, False, [(0, 513), (385, 2)]),
    (16, 16, 64, 16, 0, 0, False, 30.0, True, 64, True, [(0, 257), (5, 128)]),
    # single tokens
    (16, 4, 128, 16, 100, 4, True, 0.0, True, 64, False, [(0, 1), (15, 1), (16, 1), (98, 1), (99, 1), (100, 1), (103, 1), (115, 1), (116, 1), (3000, 1)]),
    (34, 2, 64, 4, 33, 19, True, 0.0, False, 16, False, [(0, 1), (35, 1), (50, 1), (52, 1), (55, 1), (70, 1), (1000, 1)]),
    (8, 8, 64, 8, 250, 130, True, 3.0, False, 64, True, [(249, 1), (379, 1), (381, 1), (2047, 1)]),
    (32, 8, 128, 64, 0, 0, True, 0.0, False, 0, False, [(5999, 1), (63, 1)]),
    (4, 4, 128, 128, 17, 600, False, 0.0, True, 128, False, [(616, 1), (617, 1), (5000, 1)]),
    (16, 2, 64, 16, 0, 0, False, 20.0, False, 64, False, [(10 * i, 1) for i in range(70)] + [(40, 90)]),
])
def test_window_attention(H, G, d, page, window, first, sink, cap, norm, rot, interleaved, lens):
    from llmengine_b200.kernels.ops import CudaOps
    ops, g = CudaOps(torch.device(DEV)), torch.Generator().manual_seed(H + d + window)
    R, T, D2 = len(lens), sum(n for _, n in lens), H * d + 2 * G * d
    need = [-(-(c + n) // page) for c, n in lens]
    perm = torch.randperm(sum(need) + 3, generator=g).tolist()
    tables, slots, positions = torch.full((R, max(need)), -1, dtype=torch.int32), [], []
    cache = torch.full((sum(need) + 3, 2, G, page, d), float("nan"))
    for r, (c, n) in enumerate(lens):
        pages = [perm.pop() for _ in range(need[r])]
        lo = max(0, c + 1 - window) if window else 0
        for b in range(need[r]):                                     # a page is held if a key that may be seen lies in it
            if (b + 1) * page > lo or b * page < first:
                tables[r, b] = pages[b]
                for p in range(b * page, min((b + 1) * page, c)):
                    cache[pages[b], :, :, p % page] = torch.randn(2, G, d, generator=g)
        slots += [pages[p // page] * page + p % page for p in range(c, c + n)]
        positions += range(c, c + n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    q_len = [n for _, n in lens]
    cu = [sum(q_len[:r]) for r in range(R + 1)]
    cache = cache.to(torch.bfloat16).to(DEV).view(cache.shape[0], -1).contiguous()
    batch = StepBatch(
        num_tokens=T, num_requests=R, q_lens=q_len, start_positions=[c for c, _ in lens], token_ids=i32([0] * T), positions=i32(positions),
        token_request=i32([r for r in range(R) for _ in range(q_len[r])]), cu_q_lens=i32(cu), ctx_lens=i32([c + n for c, n in lens]),
        state_slots=i32(list(range(R))), first_portion=i32([0] * R), logit_rows=i32([]), decode_rows=i32([r for r in range(R) if q_len[r] == 1]), portion_rows=i32([r for r in range(R) if q_len[r] != 1]),
        groups=[GroupView(page, window, tables.to(DEV), i32(slots), max(need))])
    proj = torch.randn(T, D2 + 8, generator=g).to(torch.bfloat16).to(DEV)
    qs, ks = H * d, G * d
    q, out = torch.zeros(T, qs, dtype=torch.bfloat16, device=DEV), torch.full((T, qs), 7.0, dtype=torch.bfloat16, device=DEV)
    sinks = (torch.randn(H, generator=g) * 3).to(DEV) if sink else None
    gains = [(1 + 0.1 * torch.randn(n, generator=g)).to(DEV) if norm else None for n in (qs, ks)]
    freq = torch.linspace(1.0, 0.01, rot // 2).to(DEV) if rot else None
    plan, scale = Plan(), d ** -0.5
    plan.window_attention(q_in=proj[:, :qs], k_in=proj[:, qs:qs + ks], v_in=proj[:, qs + ks:D2], q_gain=gains[0], k_gain=gains[1], eps=EPS, inv_freq=freq,
                          rot_dims=rot, amplitude=1.1, q=q, out=out, cache=cache, group=0, num_heads=H, num_kv_heads=G, qk_dim=d, v_dim=d, window=window,
                          keep_first=first, scale=scale, sink=sinks, softcap=cap, interleaved=interleaved,
                          decode_scratch=torch.zeros(ops.attention_scratch_floats(R, H, G, d), device=DEV))
    compiled = ops.compile(plan)
    assert f"attention_tc@HEAD_DIM={d}" in ops._libs
    compiled.run(batch)
    torch.cuda.synchronize()
    assert int(ops._libs[f"attention_tc@HEAD_DIM={d}"].llme_attention_tc_status()) == 0
    kv = cache.view(-1, 2, G, page, d).double()

    # the step in front: rounded to bfloat16 once (8 digits), from 32-bit angles (half a digit of up to 6,000: 2.5e-4 in their sine)
    def finished(x, gain, heads):
        x = x.double()
        if gain is not None:
            x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * gain.double()
        x = x.view(T, heads, d)
        if not rot:
            return x
        a = i32(positions).double()[:, None, None] * freq.double()
        c, s = torch.cos(a) * 1.1, torch.sin(a) * 1.1
        y = x.clone()
        u, w = (x[..., 0:rot:2], x[..., 1:rot:2]) if interleaved else (x[..., :rot // 2], x[..., rot // 2:rot])
        lo, hi = u * c - w * s, w * c + u * s
        if interleaved:
            y[..., 0:rot:2], y[..., 1:rot:2] = lo, hi
        else:
            y[..., :rot // 2], y[..., rot // 2:rot] = lo, hi
        return y
    at = i32(slots).long()
    for got, want in ((q.double().view(T, H, d), finished(proj[:, :qs], gains[0], H)),
                      (kv[at // page, 0, :, at % page], finished(proj[:, qs:qs + ks], gains[1], G)),
                      (kv[at // page, 1, :, at % page], proj[:, qs + ks:D2].double().view(T, G, d))):
        assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + (2e-3 if max(positions) > 1000 else 5e-4)).all()), float((got - want).abs().max())

    for r, (c, n) in enumerate(lens):
        where = [p for p in range(c + n) if not window or p > c - window or p < first]
        page_of, slot_of = tables[r, torch.tensor(where) // page].long().to(DEV), torch.tensor(where, device=DEV) % page
        k, v = kv[page_of, 0, :, slot_of].repeat_interleave(H // G, 1), kv[page_of, 1, :, slot_of].repeat_interleave(H // G, 1)
        i, j = torch.arange(c, c + n, device=DEV)[:, None], torch.tensor(where, device=DEV)[None, :]
        seen = (j <= i) & (((i - j < window) | (j < first)) if window else (j >= 0))
        s = torch.einsum("thd,khd->htk", q[cu[r]:cu[r + 1]].double().view(n, H, d), k) * scale
        s = (cap * torch.tanh(s / cap) if cap else s).masked_fill(~seen[None], float("-inf"))
        if sink:
            s = torch.cat([s, sinks.double()[:, None, None].expand(H, n, 1)], -1)
        want = torch.einsum("htk,khd->thd", torch.softmax(s, -1)[..., :len(where)], v)
        # probabilities are rounded to bfloat16 once (8 digits: up to 2^-8 of each, and they sum to at most one), and so is the result
        bound = 2.0 ** -8 * (float(v.abs().max()) + want.abs()) * 1.05 + 1e-4
        err = (out[cu[r]:cu[r + 1]].double().view(n, H, d) - want).abs()
        assert bool((err <= bound).all()), f"request {r}: {float(err.max()):.3e}, {float((err / bound).max()):.3f} of the bound"
