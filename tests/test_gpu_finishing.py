"""What stands between a product and an attention kernel over many tokens (norm, rotation, cache write), at the edges of the forms that keep
whole pieces of the rows in registers: against 64 bits, and rows that begin on 8 bytes against rows that begin on 16."""
import ctypes
from ctypes import c_float, c_int, c_longlong, c_void_p

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF16_STEP = 2.0 ** -8                      # the largest relative error of a rounding to bfloat16


class _Post(ctypes.Structure):             # LlmeWindowPostArgs
    _fields_ = [("q_in", c_void_p), ("k_in", c_void_p), ("v_in", c_void_p), ("q_stride", c_longlong), ("k_stride", c_longlong), ("v_stride", c_longlong),
                ("q_gain", c_void_p), ("k_gain", c_void_p), ("eps", c_float), ("inv_freq", c_void_p), ("rot_dims", c_int), ("amplitude", c_float),
                ("positions", c_void_p), ("q_out", c_void_p), ("cache", c_void_p), ("slot_mapping", c_void_p)] + \
               [(n, c_int) for n in ("tokens", "nh", "nkv", "dk", "dv", "page_size")] + [("q_bias", c_void_p), ("k_bias", c_void_p), ("v_bias", c_void_p)] + \
               [(n, c_int) for n in ("head_norm", "interleaved", "in_f32", "unit_norm", "value_share")]


@pytest.mark.parametrize("T", [1, 9, 150, 2001])
@pytest.mark.parametrize("nh,nkv,dk,dv,rot,interleaved,wide_in,gains,share,pad", [
    (16, 4, 128, 128, 64, 0, False, True, 1, 0), (32, 8, 128, 128, 128, 0, False, True, 1, 8), (5, 1, 64, 64, 16, 0, True, True, 1, 4), (3, 2, 256, 64, 64, 1, False, True, 1, 0),
    (64, 16, 256, 256, 128, 0, False, True, 1, 0), (4, 4, 64, 128, 0, 0, False, False, 2, 0), (7, 1, 128, 40, 8, 1, True, True, 1, 0), (6, 3, 128, 128, 48, 0, False, True, 1, 0)])
def test_rows_of_window_layers(T, nh, nkv, dk, dv, rot, interleaved, wide_in, gains, share, pad):
    from llmengine_b200.kernels.ops import CudaOps
    ops, g, ps, nv = CudaOps(torch.device(DEV)), torch.Generator(device=DEV).manual_seed(T + nh), 16, nkv // share
    kind, eps, amp = (torch.float32 if wide_in else torch.bfloat16), 1e-5, 1.25
    rows = torch.randn(T, nh * dk + nkv * dk + nv * dv + pad, generator=g, device=DEV).to(kind)
    q, k, v = rows[:, :nh * dk], rows[:, nh * dk:(nh + nkv) * dk], rows[:, (nh + nkv) * dk:(nh + nkv) * dk + nv * dv]
    qg, kg = [1 + 0.1 * torch.randn(n * dk, generator=g, device=DEV) for n in (nh, nkv)]
    freq = torch.tensor([1000.0 ** (-2.0 * i / max(rot, 1)) for i in range(rot // 2)], device=DEV)
    positions = torch.randint(0, 5000, (T,), generator=g, device=DEV, dtype=torch.int32)
    pages = -(-T // ps) + 2
    slots = torch.randperm(pages * ps, generator=g, device=DEV)[:T].to(torch.int32)
    if T > 3:
        slots[3] = -1                      # a token that is not stored
    width = ps * (nkv * dk + nv * dv)
    cache, out = torch.full((pages, width), 7.0, device=DEV, dtype=torch.bfloat16), torch.zeros(T, nh * dk, device=DEV, dtype=torch.bfloat16)
    p = lambda t: c_void_p(t.data_ptr())
    args = _Post(p(q), p(k), p(v), rows.stride(0), rows.stride(0), rows.stride(0), p(qg) if gains else None, p(kg) if gains else None, eps, p(freq) if rot else None, rot, amp,
                 p(positions), p(out), p(cache), p(slots), T, nh, nkv, dk, dv, ps, None, None, None, 0, interleaved, int(wide_in), 0, share)
    ops.require("attention_window")
    assert ops._lib("attention_window").llme_window_post(ctypes.byref(args), c_int(1), c_void_p(torch.cuda.current_stream().cuda_stream)) == 0

    def finished(x, gain, n):
        x = x.double()
        if gains:
            x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * gain.double()
        x = x.view(T, n, dk)
        if rot:
            # the angle as the kernel forms it, in 32 bits
            a = (positions.float()[:, None] * freq).double()[:, None]
            c, s = torch.cos(a) * amp, torch.sin(a) * amp
            u, w = (x[..., 0:rot:2], x[..., 1:rot:2]) if interleaved else (x[..., :rot // 2], x[..., rot // 2:rot])
            pair = (u * c - w * s, w * c + u * s)
            x = torch.cat([torch.stack(pair, -1).flatten(-2) if interleaved else torch.cat(pair, -1), x[..., rot:]], -1)
        return x
    want_q, want_k = finished(q, qg, nh), finished(k, kg, nkv)
    # one rounding to bfloat16, and 32-bit sines and sums before it
    near = lambda a, b: bool(((a.double() - b).abs() <= BF16_STEP * b.abs() + 1e-5 * (1 + b.abs().amax(-1, keepdim=True))).all())
    assert near(out.view(T, nh, dk), want_q)
    stored = torch.nonzero(slots >= 0)[:, 0]
    page, off = slots[stored].long() // ps, slots[stored].long() % ps
    keys = cache[:, :ps * nkv * dk].view(pages, nkv, ps, dk)[page, :, off]
    values = cache[:, ps * nkv * dk:].view(pages, nv, ps, dv)[page, :, off]
    assert near(keys, want_k[stored]) and torch.equal(values, v.to(torch.bfloat16).view(T, nv, dv)[stored])
    untouched = torch.ones(pages, ps, dtype=torch.bool, device=DEV)
    untouched[page, off] = False
    left = cache[:, :ps * nkv * dk].view(pages, nkv, ps, dk).transpose(1, 2)[untouched]
    assert bool((left == 7.0).all())


@pytest.mark.parametrize("nh,nkv,hd", [(32, 8, 128), (3, 1, 64), (5, 5, 32), (2, 1, 256)])
def test_rows_that_begin_on_eight_bytes(nh, nkv, hd):
    from llmengine_b200.kernels.ops import CudaOps
    ops, g, T, page = CudaOps(torch.device(DEV)), torch.Generator(device=DEV).manual_seed(hd), 3001, 16
    n = (nh + 2 * nkv) * hd
    whole = torch.randn(T, n, generator=g, device=DEV).to(torch.bfloat16)
    odd = torch.zeros(T, n + 4, device=DEV, dtype=torch.bfloat16)
    odd[:, :n] = whole
    gain = 1 + 0.1 * torch.randn(hd, generator=g, device=DEV)
    table = torch.randn(T, hd, generator=g, device=DEV)
    positions = torch.arange(T, dtype=torch.int32, device=DEV)
    x = whole.double().view(T, nh + 2 * nkv, hd)
    u = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6) * gain.double()
    a, b, c, s = u[..., :hd // 2], u[..., hd // 2:], table[:, None, :hd // 2].double(), table[:, None, hd // 2:].double()
    want = torch.cat([a * c - b * s, a * s + b * c], -1)
    # one rounding to bfloat16, and 32-bit sums and products before it
    near = lambda got, to: bool(((got.double() - to).abs() <= BF16_STEP * to.abs() + 1e-5 * (1 + to.abs().amax(-1, keepdim=True))).all())
    outs = []
    for rows in (whole, odd[:, :n]):
        cache, out = torch.zeros(-(-T // page), 2, nkv, page, hd, device=DEV, dtype=torch.bfloat16), torch.zeros(T, nh * hd, device=DEV, dtype=torch.bfloat16)
        ops.qkv_post(q_in=rows[:, :nh * hd], k_in=rows[:, nh * hd:(nh + nkv) * hd], v_in=rows[:, (nh + nkv) * hd:], num_heads=nh, num_kv_heads=nkv, head_dim=hd, q_gain=gain,
                     k_gain=gain, eps=1e-6, cos_sin=table, positions=positions, q_out=out, cache=cache, slot_mapping=positions, page_size=page)
        outs.append((out, cache))
        stored = cache.permute(0, 3, 1, 2, 4).reshape(-1, 2, nkv, hd)[:T]
        assert near(out.view(T, nh, hd), want[:, :nh]) and near(stored[:, 0], want[:, nh:nh + nkv]) and torch.equal(stored[:, 1], whole.view(T, -1, hd)[:, nh + nkv:])
    assert float(outs[0][0].abs().max()) > 0 and torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("nh,nkv,hd", [(32, 8, 128), (16, 4, 256), (40, 20, 64), (60, 30, 32)])
def test_the_squares_of_a_head_are_added_in_their_order(nh, nkv, hd):
    """Sums of four pairs (d, hd / 2 + d), then over neighbouring fours from the farthest to the nearest: the order decides some roundings to
    bfloat16, and with them every output behind the layer.  (Squares of bfloat16 values are exact in 32 bits.)"""
    from llmengine_b200.kernels.ops import CudaOps
    ops, g, T, eps = CudaOps(torch.device(DEV)), torch.Generator(device=DEV).manual_seed(hd), 3000, 1e-6
    n, lanes = (nh + 2 * nkv) * hd, hd // 8
    rows = torch.randn(T, n, generator=g, device=DEV).to(torch.bfloat16)
    gain, out = 1 + 0.1 * torch.randn(hd, generator=g, device=DEV), torch.zeros(T, nh * hd, device=DEV, dtype=torch.bfloat16)
    ops.qkv_post(q_in=rows[:, :nh * hd], k_in=rows[:, nh * hd:(nh + nkv) * hd], v_in=rows[:, (nh + nkv) * hd:], num_heads=nh, num_kv_heads=nkv, head_dim=hd, q_gain=gain,
                 k_gain=gain, eps=eps, cos_sin=None, positions=torch.arange(T, dtype=torch.int32, device=DEV), q_out=out, cache=None, slot_mapping=None, page_size=16)
    x = rows[:, :nh * hd].float().view(T, nh, hd)
    pairs = (x[..., :hd // 2] ** 2 + x[..., hd // 2:] ** 2).view(T, nh, lanes, 4)
    s = ((pairs[..., 0] + pairs[..., 1]) + pairs[..., 2]) + pairs[..., 3]
    while s.shape[-1] > 1:
        half = s.shape[-1] // 2
        s = s[..., :half] + s[..., half:]
    want = (x * (1.0 / torch.sqrt(s / hd + torch.tensor(eps, device=DEV)))) * gain
    assert torch.equal(out, want.to(torch.bfloat16).view(T, nh * hd))


@pytest.mark.parametrize("nh,nkv,dk,wide_in", [(16, 4, 128, False), (32, 8, 64, True), (64, 16, 256, False)])
def test_a_row_of_a_window_layer_does_not_depend_on_how_many_there_are(nh, nkv, dk, wide_in):
    from llmengine_b200.kernels.ops import CudaOps
    ops, g, ps, most = CudaOps(torch.device(DEV)), torch.Generator(device=DEV).manual_seed(nh), 16, 2500
    rows = 3 * torch.randn(most, (nh + 2 * nkv) * dk, generator=g, device=DEV).to(torch.float32 if wide_in else torch.bfloat16)
    qg, kg = [1 + 0.1 * torch.randn(n * dk, generator=g, device=DEV) for n in (nh, nkv)]
    positions, outs = torch.arange(most, dtype=torch.int32, device=DEV), []
    p = lambda t: c_void_p(t.data_ptr())
    for T in (most, 700, 250, 100, 3):
        kind = torch.float32 if wide_in else torch.bfloat16
        cache, out = torch.zeros(-(-most // ps), 2 * ps * nkv * dk, device=DEV, dtype=kind), torch.zeros(most, nh * dk, device=DEV, dtype=kind)
        args = _Post(p(rows), p(rows[:, nh * dk:]), p(rows[:, (nh + nkv) * dk:]), rows.stride(0), rows.stride(0), rows.stride(0), p(qg), p(kg), 1e-5, None, 0, 1.0,
                     p(positions), p(out), p(cache), p(positions), T, nh, nkv, dk, dk, ps, None, None, None, 0, 0, int(wide_in), 0, 1)
        ops.require("attention_window")
        assert ops._lib("attention_window").llme_window_post(ctypes.byref(args), c_int(0 if wide_in else 1), c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        outs.append((out[:T].clone(), cache[:, :ps * nkv * dk].view(-1, nkv, ps, dk).transpose(1, 2).flatten(0, 1)[:T].clone()))
    for q, k in outs[1:]:
        assert torch.equal(q, outs[0][0][:len(q)]) and torch.equal(k, outs[0][1][:len(k)])
