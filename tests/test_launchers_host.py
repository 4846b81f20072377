"""Launchers against a stand-in for the CUDA runtime (`fake_cuda_runtime.cpp`): several devices in one process, and the flags that tell
of a wait that gave up; and what the step executor hands to the kernels that it chooses."""
import ctypes
import os
import subprocess
from ctypes import c_float, c_int, c_longlong, c_void_p

import pytest

from llmengine_b200.kernels import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def compiled(tmp_path_factory):
    """key of a library -> the library, compiled with the stand-in in the runtime's place."""
    folder, done = tmp_path_factory.mktemp("launchers"), {}

    def get(key):
        if key not in done:
            name, defines = build.split_key(key)
            at = os.path.join(str(folder), f"lib{len(done)}.so")
            subprocess.run([build.find_nvcc(), "-gencode", "arch=compute_100a,code=compute_100a", "-std=c++17", "-O1", "--shared", "-cudart", "none", "-Xcompiler", "-fPIC",
                            "-Xlinker", "-Bsymbolic", *defines, os.path.join(build.CSRC, build.SOURCES[name]), os.path.join(HERE, "fake_cuda_runtime.cpp"), "-I", build.INCLUDE, *build.LINK.get(name, []), "-o", at], check=True)
            done[key] = ctypes.CDLL(at)
        return done[key]
    return get


@pytest.mark.parametrize("M", [1, 2, 4, 8, 16, 32, 33, 64, 129, 300])
@pytest.mark.parametrize("w_dtype", [0, 1])
def test_32_bit_products_on_a_second_device(compiled, M, w_dtype):
    """Every form that takes more than 48 KB asks for it on the device that it is launched on."""
    lib = compiled("gemm_f32")
    for N, K in ((2048, 9000), (64, 2048), (11008, 2048)):
        for device in (0, 1, 0, 63, 64, 65):
            lib.fake_device(device)
            before = lib.fake_launches()
            rc = lib.llme_gemm_nt_f32(c_void_p(1 << 20), c_void_p(1 << 21), c_int(w_dtype), c_void_p(1 << 22), c_int(M), c_int(N), c_int(K), c_longlong(K), c_longlong(K),
                                      c_longlong(N), c_void_p(0))
            assert rc == 0 and lib.fake_launches() == before + 1, (device, N, K)


class _Fast(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in ("q", "cache", "out", "rows", "cu_q_lens", "ctx_lens", "table_rows", "block_tables", "scratch")] + \
               [(n, c_int) for n in ("max_blocks", "n_rows", "nh", "nkv", "page_size", "window", "splits")] + [("scale", c_float)]


def test_latent_attention_on_a_second_device(compiled):
    args = _Fast(*[1 << (20 + i) for i in range(9)], 4, 1, 16, 1, 16, 0, 1, 1.0)
    tc, pair = compiled("attention_latent_tc@RANK=512"), compiled("attention_latent_tcgen05@RANK=512")
    for rot in (0, 64, 0, 64):
        for device in (1, 0, 1):
            tc.fake_device(device)
            pair.fake_device(device)
            for q_len in (1, 2, 100):
                assert tc.llme_latent_attention_tc(ctypes.byref(args), None, c_int(rot), c_int(q_len), None) == 0
            assert pair.llme_latent_pair(ctypes.byref(args), c_longlong(1600), c_longlong(640), None, c_int(rot), c_int(100), None) == 0


STATUS = {"gemm_tcgen05": "llme_gemm_tc_status", "moe_tcgen05": "llme_grouped_tcgen05_status", "attention_tc@HEAD_DIM=64": "llme_attention_tc_status",
          "attention_latent_tc@RANK=128": "llme_latent_attention_tc_status", "attention_latent_tcgen05@RANK=128": "llme_latent_pair_status"}


@pytest.mark.parametrize("key", sorted(STATUS))
def test_a_status_is_told_once(compiled, key):
    lib = compiled(key)
    status = getattr(lib, STATUS[key])
    assert status() == 0
    lib.fake_flag(21, 0, 0)
    assert status() == 21 and status() == 0                # told, and forgotten
    lib.fake_flag(0, 7, 0)                                 # by a kernel that still runs: the device is waited for
    assert status() == 7 and status() == 0
    lib.fake_flag(0, 0, 1)                                 # a flag that cannot be read is not "fine"
    assert status() == -1
    lib.fake_flag(0, 0, 0)


def test_every_flag_is_read_when_one_is_set():
    """The engine reads (and thereby clears) all of them, names what gave up, and says nothing the next time."""
    from types import SimpleNamespace

    from llmengine_b200.engine.engine import Engine
    flags = {"gemm_tcgen05": 0, "attention_latent_tc@RANK=64": 1, "attention_latent_tcgen05@RANK=512": 22, "elementwise": 0}

    def lib(key):
        def take():
            v, flags[key] = flags[key], 0
            return v
        return SimpleNamespace(**{name: take for name in STATUS.values()})
    eng = SimpleNamespace(ops=SimpleNamespace(_libs={k: lib(k) for k in flags}, linear_tc_status=lambda: 0), _STATUS=getattr(Engine, "_STATUS", None))
    with pytest.raises(RuntimeError) as e:
        Engine.check_kernels(eng)
    assert "attention_latent_tc@RANK=64" in str(e.value) and "attention_latent_tcgen05@RANK=512" in str(e.value)
    Engine.check_kernels(eng)


class _Executor:
    """The step executor with stand-ins for its kernels, which keep what they were given."""

    def __init__(self, lib):
        from llmengine_b200.kernels import executor as ex
        self.lib, self.ex, self.given, self._keep = lib, ex, {}, []
        lib.llme_executor_create.restype = lib.llme_plan_create.restype = c_void_p
        lib.llme_executor_error.restype = ctypes.c_char_p
        self.handle = c_void_p(lib.llme_executor_create(0))

    def kernel(self, name, *types, takes=0, result=0, restype=c_int):
        """Registers a kernel of these argument types; argument `takes`, a structure's address, is kept under its name."""
        def called(*args):
            self.given[name] = args[takes].contents if hasattr(args[takes], "contents") else args
            return result(*args) if callable(result) else result
        fn = ctypes.CFUNCTYPE(restype, *types)(called)
        self._keep.append(fn)
        assert self.lib.llme_executor_register(self.handle, name.encode(), ctypes.cast(fn, c_void_p)) == 0

    def run(self, kind, record, step):
        plan = c_void_p(self.lib.llme_plan_create(self.handle))
        assert self.lib.llme_plan_add(plan, c_int(kind), ctypes.byref(record), ctypes.c_size_t(ctypes.sizeof(record))) == 0
        rc = self.lib.llme_plan_run(plan, ctypes.byref(step), c_int(0), c_int(1), None)
        assert rc == 0, self.lib.llme_executor_error(self.handle)


def _window_step(compiled, requests, heads, kv_heads, window, keep_first, ctx, scratch_floats):
    """The argument block of the split-context kernel for `requests` single tokens with a sink."""
    from ctypes import POINTER
    e = _Executor(compiled("executor"))
    P, far = c_void_p, 1 << 24
    e.kernel("window_post", P, c_int, P)
    e.kernel("window_attention_tc/128x128", P, c_int, c_int, P)
    e.kernel("attention_decode/128", P, P)
    e.kernel("attention_portion/128", P, c_int, P)
    e.kernel("attention_decode_scratch/128", c_int, c_int, c_int, result=lambda n, h, s: 0 if s <= 1 else 65536 + n * h * s * 130, restype=c_longlong)
    e.kernel("attention_decode_ext/128", POINTER(_Fast), P, c_int, c_float, P)
    op = e.ex.WindowAttentionOp()
    op.q_in = op.k_in = op.v_in = op.q = op.out = op.cache = op.sink = op.decode_scratch = far
    op.dtype, op.nh, op.nkv, op.dk, op.dv, op.window, op.keep_first, op.scale, op.amplitude = 1, heads, kv_heads, 128, 128, window, keep_first, 0.1, 1.0
    op.decode_scratch_floats, op.cache_pages, op.value_share = scratch_floats, 4096, 1
    step = e.ex.Step()
    step.num_tokens = step.num_requests = step.num_decode = requests
    step.max_decode_ctx, step.num_groups = ctx, 1
    step.groups[0] = e.ex.StepGroup(far, far, 1024, 16, window)
    e.run(e.ex.OP_WINDOW_ATTENTION, op, step)
    return e.given["attention_decode_ext/128"]


def test_kept_first_positions_count_as_keys(compiled):
    """A token sees its window and the kept first positions: as many shares as a window of all of them would get."""
    for requests in (1, 2, 5):
        kept = _window_step(compiled, requests, 16, 4, 128, 4096, 8000, 1 << 30).splits
        assert kept == _window_step(compiled, requests, 16, 4, 4224, 0, 8000, 1 << 30).splits > 3
        assert _window_step(compiled, requests, 16, 4, 128, 1 << 30, 8000, 1 << 30).splits >= kept      # never more keys than there are


def test_shares_are_fewer_where_the_scratch_memory_is_small(compiled):
    """Any scratch memory is enough for one share; more shares only as far as their partial results fit."""
    most = _window_step(compiled, 2, 16, 4, 0, 0, 8000, 1 << 30).splits
    assert most > 3
    assert _window_step(compiled, 2, 16, 4, 0, 0, 8000, 1).splits == 1
    assert _window_step(compiled, 2, 16, 4, 0, 0, 8000, 65536 + 2 * 16 * 3 * 130).splits == 3


@pytest.mark.parametrize("experts,top,n,k,tokens,streams", [
    # the faster of the two kernels as measured, from a quarter to three and a half rows an expert; one whose products are small is
    # streamed, one of many short rows is not
    (8, 2, 2048, 2048, 1, True), (8, 2, 4096, 2048, 14, True), (16, 4, 2048, 1024, 6, True), (32, 4, 2048, 2048, 8, True), (32, 4, 4096, 2048, 8, True),
    (32, 4, 4096, 2048, 20, True), (64, 8, 1024, 2048, 24, True), (128, 8, 1024, 2048, 8, True), (32, 4, 2048, 1024, 24, False), (64, 6, 2048, 1024, 27, False),
    (64, 8, 2048, 512, 16, False), (128, 8, 1024, 2048, 40, False), (128, 8, 2048, 512, 4, False), (128, 8, 2048, 512, 48, False), (128, 8, 1536, 2048, 48, False),
    (64, 4, 2048, 1536, 32, False),
    # from four rows on
    (8, 2, 2048, 2048, 16, False), (32, 4, 4096, 2048, 32, False), (128, 8, 2048, 512, 1000, False)])
def test_grouped_products_of_few_rows(compiled, experts, top, n, k, tokens, streams):
    e = _Executor(compiled("executor"))
    P, far = c_void_p, 1 << 24
    e.kernel("grouped_tcgen05", P, P, c_int, P)
    e.kernel("grouped_tcgen05_supports", P, c_int, result=1)
    e.kernel("grouped_linear_tc", P, c_int, c_int, c_int, P)
    op = e.ex.GroupedLinearOp()
    for name in ("x", "w", "out", "offsets", "order", "mid", "rows"):
        setattr(op, name, far)
    gather = k == 2048 and (experts, n) != (8, 2048)                 # (the gate|up product; the down product's rows lie side by side)
    op.ldx = op.ldw = op.k = k
    op.ldo, op.n, op.w_expert, op.num_experts, op.top_k, op.x_dtype, op.w_dtype, op.gather, op.act = n, n, n * k, experts, top, 1, 1, int(gather), int(gather)
    step = e.ex.Step()
    step.num_tokens = step.num_requests = tokens
    e.run(e.ex.OP_GROUPED_LINEAR, op, step)
    assert list(e.given)[-1] == ("grouped_linear_tc" if streams else "grouped_tcgen05")


@pytest.mark.parametrize("ctx,decode_ctx,short", [(64, 0, True), (2, 0, True), (64, 900, True), (65, 0, False), (3000, 10, False), (0, 0, False)])
def test_short_portions_stay_on_the_warp_level_kernels(compiled, ctx, decode_ctx, short):
    """By the longest context among the requests with several tokens, where the step tells it."""
    P, far = c_void_p, 1 << 24
    e = _Executor(compiled("executor"))
    step = e.ex.Step()
    step.num_tokens, step.num_requests, step.num_portion, step.max_portion_len = 40, 2, 2, 30
    step.max_portion_ctx, step.max_decode_ctx, step.num_decode, step.num_groups = ctx, decode_ctx, 1 if decode_ctx else 0, 1
    step.groups[0] = e.ex.StepGroup(far, far, 1024, 16, 0)
    e.kernel("latent_post", P, c_int, P)
    e.kernel("latent_attention_tc/512", P, P, c_int, c_int, P)
    e.kernel("latent_attention_tc_fits/512", c_int, result=1)
    e.kernel("latent_pair/512", P, c_longlong, c_longlong, P, c_int, c_int, P)
    e.kernel("latent_pair_supports/512", c_int, c_int, result=1)
    op = e.ex.LatentAttentionOp()
    op.kv_in = op.c_gain = op.q = op.out = op.cache = far
    op.dtype, op.nh, op.rank, op.rot, op.scale, op.cache_rows = 1, 16, 512, 64, 0.1, 1 << 16
    e.run(e.ex.OP_LATENT_ATTENTION, op, step)
    assert ("latent_pair/512" in e.given) != short
    step.groups[0].window = 100
    e.kernel("window_post", P, c_int, P)
    e.kernel("window_attention_tc/128x128", P, c_int, c_int, P)
    e.kernel("attention_tc/128", P, c_longlong, c_longlong, P, c_int, P)
    op = e.ex.WindowAttentionOp()
    op.q_in = op.k_in = op.v_in = op.q = op.out = op.cache = op.sink = far
    op.dtype, op.nh, op.nkv, op.dk, op.dv, op.window, op.scale, op.amplitude, op.cache_pages, op.value_share = 1, 16, 4, 128, 128, 100, 0.1, 1.0, 4096, 1
    e.run(e.ex.OP_WINDOW_ATTENTION, op, step)
    assert ("attention_tc/128" in e.given) != short
