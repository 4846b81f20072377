"""Launchers against a stand-in for the CUDA runtime (`fake_cuda_runtime.cpp`): several devices in one process."""
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
