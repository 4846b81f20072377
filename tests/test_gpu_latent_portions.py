"""The latent attention, alone: prompt portions on tcgen05 and single tokens, at the edges of their tiles (128 rows of (token, head), 128 or
64 keys, pages, chunks of 64 columns, key ranges), against the softmax written out in 64 bits over the same queries and cache rows; and
the step in front of it (norm of the latent, rotations, cache write) against its formulas in 64 bits."""
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


@pytest.mark.parametrize("heads,page,window,sink,lens", [
    # tiles of 64 keys with up to 32 heads, of 32 with more; one, two and three tiles, their edges, many; requests of few keys beside
    # long ones get more key ranges than they have tiles
    (16, 16, 0, False, [0, 62, 63, 64, 126, 127, 128, 129, 191, 3999]),
    (16, 16, 0, True, [0, 1, 4000]),
    (20, 64, 0, True, [5, 63, 64, 700, 2047]),
    (40, 8, 0, True, [0, 30, 31, 32, 33, 64, 65, 1500]),
    (16, 16, 100, True, [50, 98, 99, 100, 130, 163, 2000]),
    (32, 4, 1000, False, [999, 1000, 1030, 3001]),
    # a block's range of more pages than its table holds (512), with and without a last tile that is not full
    (16, 4, 0, False, [4000, 2111, 7, 2048]),
    (16, 1, 0, True, [700, 511, 512, 513]),
    (16, 3, 0, False, [2500, 1536]),
])
@pytest.mark.parametrize("ranges", [True, False])
def test_single_tokens(heads, page, window, sink, lens, ranges):
    run(512, 64, heads, page, window, sink, [(c, 1) for c in lens], ranges=ranges)


@pytest.mark.parametrize("rank,rot,heads,ctx", [(64, 64, 8, 300), (128, 0, 32, 1000), (256, 64, 17, 500), (512, 0, 16, 777)])
def test_single_tokens_of_other_sizes(rank, rot, heads, ctx):
    run(rank, rot, heads, 16, 0, True, [(ctx, 1), (0, 1), (ctx // 2, 1)], ranges=True)


@pytest.mark.parametrize("lens", [[(0, 64), (30, 2), (0, 1)], [(0, 65)], [(0, 3)], [(0, 64), (900, 1)]])
@pytest.mark.parametrize("sink", [True, False])
def test_short_portions(lens, sink):
    """Up to 64 keys the warp-level kernel serves them, whatever single tokens beside them see."""
    run(512, 64, 16, 16, 0, sink, lens)


@pytest.mark.parametrize("heads,sink", [(16, True), (16, False), (32, True)])
def test_portions_are_no_further_off_than_the_warp_level_kernel(heads, sink):
    """Both round the probabilities to bfloat16.  The warp-level kernel takes them relative to the row's true maximum, whose probability is
    then exactly one; a reference that stays at the sink or far below the maximum rounds the largest one too (12 % more error)."""
    lens = [(0, 300), (100, 500), (0, 40)]
    err = [run(512, 64, heads, 16, 0, sink, lens, portion=portion, spread=0.4, error=True) for portion in ("tcgen05", "mma")]
    assert err[0] <= 1.01 * err[1], err


def test_a_single_key_beside_a_sink():
    """A row of one key: its probability is 1 / (1 + exp(sink - score)), and nothing but the result is rounded where the key leads."""
    heads, T = 16, 100
    out, want, lead = run(512, 64, heads, 16, 1, True, [(0, T)], single=True)
    assert int(lead.sum()) > 100
    bound = (2.0 ** -8 + 1e-4) * want.abs()                  # half a unit of the last of eight digits, and the 32-bit exponentials
    assert bool(((out - want).abs() <= bound)[lead].all()), float(((out - want).abs() / want.abs())[lead].max())


@pytest.mark.parametrize("T,rot,rot_dims,interleaved,gain_dtype", [
    (256, 64, 64, False, torch.float32), (257, 64, 64, False, torch.float32), (600, 64, 64, True, torch.bfloat16), (300, 64, 32, False, torch.bfloat16),
    (300, 64, 24, True, torch.float32), (1000, 32, 32, False, torch.float32), (300, 64, 20, False, torch.float32), (257, 0, 0, False, torch.float32)])
def test_norm_rotation_and_cache_write(T, rot, rot_dims, interleaved, gain_dtype):
    """The step in front, in pieces of 16 bytes (many tokens) and value by value (few, or counts that are not whole pieces): a row is stored
    only where the token has a slot."""
    from llmengine_b200.kernels.ops import CudaOps
    ops, g = CudaOps(torch.device(DEV)), torch.Generator().manual_seed(T + rot_dims)
    rank, heads, page, amplitude = 512, 5, 16, 1.2
    width, pages = rank + rot, -(-T // page)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    table = torch.randperm(pages, generator=g).tolist()
    slots = [-1 if t % 7 == 3 else table[t // page] * page + t % page for t in range(T)]
    before = torch.randn(pages, page, width, generator=g).to(torch.bfloat16).to(DEV)
    cache, q = before.clone(), torch.randn(T, heads * width, generator=g).to(torch.bfloat16).to(DEV)
    kv_in = torch.randn(T, width + 8, generator=g).to(torch.bfloat16).to(DEV)[:, :width]
    q_rot = torch.randn(T, heads, rot + 16, generator=g).to(torch.bfloat16).to(DEV)[:, :, :rot] if rot else None
    gain = (1 + 0.2 * torch.randn(rank, generator=g)).to(gain_dtype).to(DEV)
    freq = torch.linspace(1.0, 0.01, rot_dims // 2).to(DEV) if rot else None
    batch = StepBatch(
        num_tokens=T, num_requests=1, q_lens=[T], start_positions=[0], token_ids=i32([0] * T), positions=i32(range(T)), token_request=i32([0] * T), cu_q_lens=i32([0, T]),
        ctx_lens=i32([T]), state_slots=i32([0]), first_portion=i32([1]), logit_rows=i32([]), decode_rows=i32([]), portion_rows=i32([0]),
        groups=[GroupView(page, 0, i32([table]), i32(slots), pages)])
    plan, q0 = Plan(), q.clone().view(T, heads, width)
    plan.latent_attention(q_rot=q_rot, kv_in=kv_in, c_gain=gain, eps=1e-6, inv_freq=freq, rot_dims=rot_dims, q=q, out=torch.zeros(T, heads * rank, dtype=torch.bfloat16, device=DEV),
                          cache=cache, group=0, num_heads=heads, kv_rank=rank, rot_dim=rot, scale=0.05, interleaved=interleaved, amplitude=amplitude)
    ops.compile(plan).run(batch)
    torch.cuda.synchronize()

    def rotated(x):                                          # [T, n, rot]
        a = torch.arange(T, device=DEV).double()[:, None, None] * freq.double()
        c, s, y = torch.cos(a) * amplitude, torch.sin(a) * amplitude, x.clone()
        first, second = (slice(0, rot_dims, 2), slice(1, rot_dims, 2)) if interleaved else (slice(0, rot_dims // 2), slice(rot_dims // 2, rot_dims))
        y[..., first], y[..., second] = x[..., first] * c - x[..., second] * s, x[..., second] * c + x[..., first] * s
        return y
    c = kv_in[:, :rank].double()
    row = c / torch.sqrt((c * c).mean(-1, keepdim=True) + 1e-6) * gain.double()
    if rot:
        row = torch.cat([row, rotated(kv_in[:, None, rank:].double())[:, 0]], 1)
    at = torch.tensor(slots, device=DEV)
    held = at >= 0
    # rounded to bfloat16 once (half a unit of the last of eight digits); angles are 32-bit, up to 1,000 in size: 6e-5 in their sine, of values up to five
    close = lambda got, want: bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 5e-4).all())
    assert close(cache.view(-1, width)[at[held]], row[held])
    untouched = torch.ones(pages * page, dtype=torch.bool, device=DEV)
    untouched[at[held]] = False
    assert torch.equal(cache.view(-1, width)[untouched], before.view(-1, width)[untouched])
    assert torch.equal(q.view(T, heads, width)[..., :rank], q0[..., :rank])
    if rot:
        assert close(q.view(T, heads, width)[..., rank:], rotated(q_rot.double()))


def run(rank, rot, heads, page, window, sink, lens, ranges=False, portion="tcgen05", spread=0.7, error=False, single=False):
    """Runs the step over these requests, compares every row with its 64-bit result and returns the outputs.  `ranges`: with the scratch
    memory for key ranges.  `error`: returns the relative error instead; `single`: (outputs, 64-bit results, where a row's one key leads
    its sink)."""
    from llmengine_b200.kernels.ops import CudaOps
    ops, g = CudaOps(torch.device(DEV)), torch.Generator().manual_seed(rank + rot + heads)
    ops.choose("attention.portion", portion)
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
    cache, q = cache.to(torch.bfloat16).to(DEV), (torch.randn(T, heads * width, generator=g) * spread).to(torch.bfloat16).to(DEV)
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
                          scratch=torch.full((ops.latent_scratch_floats(heads, rank),), float("nan"), device=DEV) if ranges else None)
    compiled = ops.compile(plan)
    pair = f"attention_latent_tcgen05@RANK={rank}"
    assert pair in ops._libs or portion != "tcgen05" or rank % 128
    compiled.run(batch)
    torch.cuda.synchronize()
    assert pair not in ops._libs or int(ops._libs[pair].llme_latent_pair_status()) == 0
    assert int(ops._libs[f"attention_latent_tc@RANK={rank}"].llme_latent_attention_tc_status()) == 0
    rows, qd, got = cache.double().view(-1, width), q.double().view(T, heads, width), out.double().view(T, heads, rank)
    square, square_want, wants, leads = 0.0, 0.0, [], []
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
        diff = got[cu[r]:cu[r + 1]] - want
        err = diff.abs()
        assert bool((err <= bound).all()), f"request {r}: {float(err.max()):.3e}, {float((err / bound).max()):.3f} of the bound"
        # Every rounding is half a unit of the last of eight digits at most, 2^-8 (1.6e-3 in the mean square), and those of a row's
        # probabilities are independent of one another: in the 2-norm of a row of independent values the two roundings add up to a
        # share of 2.3e-3 in the mean, and of 2^-7 at most.  One key too many or
        # too few of n is a share of n^-1/2 or more.
        share = diff.norm(dim=-1) / want.norm(dim=-1)
        assert float(share.max()) <= 2.0 ** -7, f"request {r}: a row is {float(share.max()):.3e} off"
        square, square_want = square + float(diff.square().sum()), square_want + float(want.square().sum())
        wants.append(want)
        if sink:
            leads.append(s[..., :-1].max(-1).values.t() > s[..., -1].t())
    if single:
        return got, torch.cat(wants), torch.cat(leads)
    return (square / square_want) ** 0.5 if error else out
