"""What stands between a product and an attention kernel over many tokens (norm, rotation, cache write), at the edges of the forms that keep
whole pieces of the rows in registers: against 64 bits, and rows that begin on 8 bytes against rows that begin on 16."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


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
    outs = []
    for rows in (whole, odd[:, :n]):
        cache, out = torch.zeros(-(-T // page), 2, nkv, page, hd, device=DEV, dtype=torch.bfloat16), torch.zeros(T, nh * hd, device=DEV, dtype=torch.bfloat16)
        ops.qkv_post(q_in=rows[:, :nh * hd], k_in=rows[:, nh * hd:(nh + nkv) * hd], v_in=rows[:, (nh + nkv) * hd:], num_heads=nh, num_kv_heads=nkv, head_dim=hd, q_gain=gain,
                     k_gain=gain, eps=1e-6, cos_sin=table, positions=positions, q_out=out, cache=cache, slot_mapping=positions, page_size=page)
        outs.append((out, cache))
    assert float(outs[0][0].abs().max()) > 0 and torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
