"""The 32-bit product in each of its forms (on the tensor cores; weights streamed for up to 2, 4, 8, 16 and 32 rows; tiles of 128, 64 and 16 rows, whole and shared by a cluster) at sizes
around their edges: against 64 bits, and bit for bit the same row whatever else is in the launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("N,K,w_dtype,pad", [
    (2048, 5504, torch.float32, 0), (1000, 1023, torch.float32, 0), (130, 2049, torch.bfloat16, 0), (64, 9001, torch.float32, 3), (11008, 2048, torch.float32, 0),
    (300, 17, torch.bfloat16, 5), (50, 4100, torch.float32, 4), (63, 2052, torch.float32, 0), (300, 3001, torch.float32, 2), (4096, 16400, torch.bfloat16, 8), (50, 1030, torch.float32, 2), (4096, 16400, torch.float32, 4), (33, 6, torch.bfloat16, 2)])
def test_every_form(N, K, w_dtype, pad):
    from llmengine_b200.kernels.ops import CudaOps
    # (float weights of 64 rows and 512 values or more whose rows begin on 16 bytes go to the tensor cores, all others to the multiply-adds)
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


@pytest.mark.parametrize("N,K,pad", [(64, 512, 0), (65, 577, 3), (129, 1030, 2), (300, 1024, 0), (2048, 5500, 4), (11008, 640, 0), (19000, 512, 0)])
def test_float_weights_on_the_tensor_cores(N, K, pad):
    """Around the edges of tiles, chunks of 64 values and segments.  An output's chunk is 24 instructions that may each cut off a last place of
    what has been added so far, 2^-23 of sum |x w| at most; the chunks' and segments' sums round once each, 2^-24, and the pieces leave out
    less than 2^-25 of each product, three times."""
    from llmengine_b200.kernels.ops import CudaOps
    ops, g = CudaOps(torch.device(DEV)), torch.Generator(device=DEV).manual_seed(N + K)
    x = torch.randn(260, K + pad, generator=g, device=DEV)[:, :K]
    w = torch.randn(N, K + pad, generator=g, device=DEV)[:, :K]
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    bound = (2 * 24 + K / 64 + 5 + 1.5) * 2.0 ** -24 * size
    full = None
    for M in (260, 1, 8, 16, 17, 32, 33, 48, 112, 113, 225):
        out = torch.full((M, N + 4), 5.0, device=DEV)
        ops.linear(x[:M], w, out[:, :N])
        assert bool((out[:, N:] == 5.0).all())
        full = out[:, :N] if full is None else full
        assert bool(((out[:, :N].double() - want[:M]).abs() <= bound[:M]).all()), M
        assert torch.equal(out[:, :N], full[:M]), M
    assert int(ops._lib("gemm_f32").llme_gemm_f32_status()) == 0


def test_no_number_where_32_bits_give_none_and_only_there():
    """Infinities, NaN, values next to the largest (which bfloat16 rounds up to infinity), sums that overflow, and tiny rows."""
    from llmengine_b200.kernels.ops import CudaOps
    ops, g = CudaOps(torch.device(DEV)), torch.Generator(device=DEV).manual_seed(3)
    for M in (20, 150):
        x, w = torch.randn(M, 1024, generator=g, device=DEV), torch.randn(256, 1024, generator=g, device=DEV) * 0.02
        x[3, 5], x[4, 7], x[5, 9], w[7, 11], w[8, 12] = float("inf"), float("nan"), 3.4e38, -float("inf"), 3.4e38
        x[6] *= 1e-30
        x[9] = 0.0
        x[10] *= 1e36
        x[11, 20], x[11, 21], w[9, 20], w[9, 21] = 3e38, 3e38, 1.0, 1.0
        out = torch.empty(M, 256, device=DEV)
        ops.linear(x, w, out)
        exact = x.double() @ w.double().t()
        large = exact.abs() >= (2 - 2.0 ** -24) * 2.0 ** 127               # from here on a value rounds to infinity in 32 bits
        assert torch.equal(out.isnan(), exact.isnan())
        assert torch.equal(out.isinf(), exact.isinf() | large) and bool((torch.sign(out) == torch.sign(exact))[large].all())
        rest = torch.isfinite(exact) & ~large
        size = x.double().abs() @ w.double().abs().t()
        assert bool(((out.double() - exact).abs() <= (2 * 24 + 1024 + 8) * 2.0 ** -24 * size)[rest].all())


@pytest.mark.parametrize("M,N,K", [(1, 4096, 2048), (40, 2048, 1024), (3, 64, 512)])
def test_weights_that_the_kernel_before_has_just_written(M, N, K):
    """The norm in front lets its successor in early: what it writes is there all the same when it is taken for weights."""
    from llmengine_b200.kernels.ops import CudaOps
    ops, g = CudaOps(torch.device(DEV)), torch.Generator(device=DEV).manual_seed(N)
    x, gain = torch.randn(M, K, generator=g, device=DEV), torch.ones(K, device=DEV)
    w, out = torch.zeros(N, K, device=DEV), torch.empty(M, N, device=DEV)
    for scale in (1.0, -1.0, 2.0, -3.0):
        rows = torch.randn(N, K, generator=g, device=DEV)
        want = scale * torch.nn.functional.rms_norm(rows.double(), (K,), eps=1e-6)
        torch.cuda.synchronize()
        ops.rmsnorm(rows, gain * scale, 1e-6, w)
        ops.linear(x, w, out)
        exact = x.double() @ want.t()
        assert float((out.double() - exact).norm()) < 2e-6 * float(exact.norm()), scale


@pytest.mark.parametrize("x_power,w_power", [(-112, 0), (-118, 0), (-130, 0), (-140, 0), (0, -124), (0, -138), (-118, 100), (-128, 100), (120, -126), (-60, -60), (-63, -64), (-70, -72)])
def test_operands_and_results_at_the_small_end(x_power, w_power):
    """Operands keep all their bits as far as 32-bit numbers have them.  To the bound of ordinary products (above) comes what 32 bits cannot hold
    of a small result: every addition may be off by 2^-149, the smallest number, 24 in a chunk and one for each chunk and segment."""
    from llmengine_b200.kernels.ops import CudaOps
    ops, g, N, K = CudaOps(torch.device(DEV)), torch.Generator(device=DEV).manual_seed(3), 256, 1024
    x = (torch.randn(40, K, generator=g, device=DEV).double() * 2.0 ** x_power).float()
    w = (torch.randn(N, K, generator=g, device=DEV).double() * 2.0 ** w_power).float()
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    bound = (2 * 24 + K / 64 + 5 + 1.5) * 2.0 ** -24 * size + (24 * (K / 64) + K / 64 + 5) * 2.0 ** -149
    for M in (3, 40):
        out = torch.empty(M, N, device=DEV)
        ops.linear(x[:M], w, out)
        assert bool(((out.double() - want[:M]).abs() <= bound[:M]).all()), M


@pytest.mark.parametrize("N,K", [(1000, 517), (11008, 2048)])
def test_rows_that_are_no_numbers_do_not_hold_up_the_launch(N, K):
    """A row of NaN, rows with one in their last place, an infinity: the outputs of 64 bits, at no more than forty times a launch of numbers (as
    a serial sum a thread they took 260 times that)."""
    from llmengine_b200.kernels.ops import CudaOps
    ops, g = CudaOps(torch.device(DEV)), torch.Generator(device=DEV).manual_seed(N)
    pad = -K % 4
    clean, w = torch.randn(300, K + pad, generator=g, device=DEV), torch.randn(N, K + pad, generator=g, device=DEV)
    every, some = clean.clone(), clean.clone()
    every[:, :] = float("nan")
    some[::3, K - 1], some[1, 5], some[2, 7] = float("nan"), float("inf"), 3.4e38
    times = []
    for x in (clean, every, some):
        out = torch.empty(300, N, device=DEV)
        took = []
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ops.linear(x[:, :K], w[:, :K], out)
            b.record()
            torch.cuda.synchronize()
            took.append(a.elapsed_time(b))
        times.append(min(took[1:]))
        exact = x[:, :K].double() @ w[:, :K].double().t()
        want = exact.float()
        assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out[want.isinf()], want[want.isinf()])
    assert max(times[1:]) < 40 * times[0], times
