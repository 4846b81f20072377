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
    # many kept first positions: more shares than three, the kept ones' pages in a block's table behind the window's
    (16, 4, 128, 16, 128, 4096, True, 0.0, False, 0, False, [(8000, 1), (4223, 1), (4224, 1), (4100, 1)]),
    (8, 8, 64, 8, 20, 1003, True, 0.0, False, 0, False, [(1003, 1), (1022, 1), (1023, 1), (1040, 1), (2500, 1)]),
    # pages that do not fit the table: the window's alone, the kept ones' alone, neither (one share a request)
    (40, 40, 64, 1, 700, 40, False, 0.0, False, 0, False, [(1500, 1)] + [(60, 1)] * 9),
    (40, 40, 64, 1, 100, 600, False, 0.0, False, 0, False, [(1500, 1)] + [(60, 1)] * 9),
    (40, 40, 64, 1, 600, 600, False, 0.0, False, 0, False, [(1500, 1)] + [(60, 1)] * 9),
    (16, 4, 128, 16, 30, 700, True, 0.0, False, 0, False, [(0, 900), (1500, 70)]),
])
def test_window_attention(H, G, d, page, window, first, sink, cap, norm, rot, interleaved, lens):
    run(H, G, d, page, window, first, sink, cap, norm, rot, interleaved, lens)


@pytest.mark.parametrize("lens", [[(0, 64), (30, 2), (0, 1)], [(0, 65)], [(0, 3)], [(0, 64), (900, 1)]])
def test_short_portions(lens):
    """Up to 64 keys the warp-level kernel serves them, whatever single tokens beside them see."""
    run(16, 4, 128, 16, 40, 3, True, 0.0, True, 64, False, lens)


@pytest.mark.parametrize("floats", [0, 1, 65536 + 4 * 16 * 2 * 130])
def test_any_scratch_memory_is_enough(floats):
    """As many shares of a context as their partial results find room for, one at least."""
    run(16, 4, 128, 16, 0, 0, True, 0.0, False, 0, False, [(3000, 1), (100, 1), (5, 1), (4000, 1)], scratch_floats=max(floats, 1))


@pytest.mark.parametrize("window,first,sink,cap", [(1024, 4, True, 0.0), (0, 0, True, 0.0), (200, 2, False, 0.0), (0, 0, True, 5.0)])
def test_portions_are_no_further_off_than_the_warp_level_kernel(window, first, sink, cap):
    """Both round the probabilities to bfloat16.  The warp-level kernel takes them relative to the row's true maximum, whose probability is
    then exactly one; a reference that stays at the sink or far below the maximum rounds the largest one too (up to 13 % more error)."""
    err = [run(16, 4, 128, 16, window, first, sink, cap, True, 0, False, [(0, 700), (300, 900), (0, 60)], portion=portion, error=True) for portion in ("tcgen05", "mma")]
    assert err[0] <= 1.01 * err[1], err


@pytest.mark.parametrize("d,cap", [(64, 0.0), (128, 0.0), (128, 3.0)])
def test_a_single_key_beside_a_sink(d, cap):
    """A row of one key: its probability is 1 / (1 + exp(sink - score)), and nothing but the result is rounded where the key leads."""
    out, want, lead = run(16, 4, d, 16, 1, 0, True, cap, True, 0, False, [(0, 200)], single=True)
    assert int(lead.sum()) > 400
    bound = (2.0 ** -8 + 1e-4) * want.abs()                  # half a unit of the last of eight digits, and the 32-bit exponentials
    assert bool(((out - want).abs() <= bound)[lead].all()), float(((out - want).abs() / want.abs())[lead].max())


def run(H, G, d, page, window, first, sink, cap, norm, rot, interleaved, lens, portion="tcgen05", scratch_floats=None, error=False, single=False):
    """Runs the step over these requests and compares every row with its 64-bit result.  `error`: returns the relative error of the
    heads; `single`: (outputs, 64-bit results, where a row's one key leads its sink)."""
    from llmengine_b200.kernels.ops import CudaOps
    ops, g = CudaOps(torch.device(DEV)), torch.Generator().manual_seed(H + d + window)
    ops.choose("attention.portion", portion)
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
                          decode_scratch=torch.zeros(scratch_floats or max(1, ops.attention_scratch_floats(R, H, G, d)), device=DEV))
    compiled = ops.compile(plan)
    assert (f"attention_tc@HEAD_DIM={d}" in ops._libs) == (portion == "tcgen05")
    compiled.run(batch)
    torch.cuda.synchronize()
    assert portion != "tcgen05" or int(ops._libs[f"attention_tc@HEAD_DIM={d}"].llme_attention_tc_status()) == 0
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

    square, square_want, wants, leads = 0.0, 0.0, [], []
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
        diff = out[cu[r]:cu[r + 1]].double().view(n, H, d) - want
        err = diff.abs()
        assert bool((err <= bound).all()), f"request {r}: {float(err.max()):.3e}, {float((err / bound).max()):.3f} of the bound"
        # Every rounding is half a unit of the last of eight digits at most, 2^-8 (1.6e-3 in the mean square), and those of a row's
        # probabilities are independent of one another: in the 2-norm of a row of independent values the two roundings add up to a
        # share of 2.3e-3 in the mean, and of 2^-7 at most.  One key too many or
        # too few of n is a share of n^-1/2 or so.
        share = diff.norm(dim=-1) / want.norm(dim=-1)
        assert float(share.max()) <= 2.0 ** -7, f"request {r}: a row is {float(share.max()):.3e} off"
        square, square_want = square + float(diff.square().sum()), square_want + float(want.square().sum())
        wants.append(want)
        if sink:
            leads.append(s[..., :-1].max(-1).values.t() > s[..., -1].t())
    if single:
        return out.double().view(T, H, d), torch.cat(wants), torch.cat(leads)
    return (square / square_want) ** 0.5 if error else None
