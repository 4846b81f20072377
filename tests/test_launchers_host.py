"""Launchers against a stand-in for the CUDA runtime (`fake_cuda_runtime.cpp`): several devices in one process, and the flags that tell
of a wait that gave up."""
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
                            "-Xlinker", "-Bsymbolic", *defines, os.path.join(build.CSRC, build.SOURCES[name]), os.path.join(HERE, "fake_cuda_runtime.cpp"), "-o", at], check=True)
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
