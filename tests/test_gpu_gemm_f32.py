"""The 32-bit product in each of its forms (weights streamed for up to 2, 4, 8, 16 and 32 rows, tiles of 128, 64 and 16 rows, whole and shared by a cluster) at sizes around their edges:
against 64 bits, and bit for bit the same row whatever else is in the launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("N,K,w_dtype,pad", [
    (2048, 5504, torch.float32, 0), (1000, 1023, torch.float32, 0), (130, 2049, torch.bfloat16, 0), (64, 9001, torch.float32, 3), (11008, 2048, torch.float32, 0),
    (300, 17, torch.bfloat16, 5), (4096, 16400, torch.bfloat16, 8), (50, 1030, torch.float32, 2), (4096, 16400, torch.float32, 4), (33, 6, torch.bfloat16, 2)])
def test_every_form(N, K, w_dtype, pad):
    from llmengine_b200.kernels.ops import CudaOps
    ops, g = CudaOps(torch.device(DEV)), torch.Generator(device=DEV).manual_seed(N + K)
    x = torch.randn(601, K + pad, generator=g, device=DEV)[:, :K]
    w = torch.randn(N, K + pad, generator=g, device=DEV).to(w_dtype)[:, :K]
    outs = {}
    for M in (1, 2, 3, 5, 8, 9, 16, 17, 32, 33, 65, 129, 300, 601):
        out = torch.full((M, N + pad), 5.0, device=DEV)
        ops.linear(x[:M], w, out[:, :N])
        assert bool((out[:, N:] == 5.0).all())
        outs[M] = out[:, :N]
    want = x.double() @ w.double().t()
    # segments of at most K / min(8, K / 1024) products in a row, then up to 8 sums: gamma_n |x| |w| with n = that and u = 2^-24
    n = K / max(1, min(8, K // 1024)) + 24
    bound = n * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
    assert bool(((outs[601].double() - want).abs() <= bound).all())
    for M, out in outs.items():
        assert torch.equal(out, outs[601][:M]), M


def test_a_batch_of_products():
    from llmengine_b200.engine.batch import StepBatch
    from llmengine_b200.engine.plan import Plan
    from llmengine_b200.kernels.ops import CudaOps
    ops, g = CudaOps(torch.device(DEV)), torch.Generator(device=DEV).manual_seed(1)
    for T, B, k, n in ((5, 3, 2100, 70), (150, 4, 1024, 130)):
        x, w = torch.randn(T, B, k, generator=g, device=DEV), torch.randn(B, n, k, generator=g, device=DEV)
        out, plan = torch.zeros(T, B, n, device=DEV), Plan()
        plan.batched_linear(x, w, out)
        ops.compile(plan).run(StepBatch.bare(T, torch.device(DEV)))
        want = torch.einsum("tbk,bnk->tbn", x.double(), w.double())
        assert float((out.double() - want).norm() / want.norm()) < 1e-6
