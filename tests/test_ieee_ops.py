"""The division, reciprocal and square root that the kernels run on the
integer pipe (landslidehysea_gb300/csrc/lsh_ieee.h) round like the IEEE
operations, bit for bit: on the host with the approximation instruction
replaced by values at the edges of its documented error bound, on the GPU
against CUDA's own operations, special values included."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from adj_cases import native_lib

HERE = os.path.dirname(os.path.abspath(__file__))


def operands(n, seed):
    """n pairs: significands of every kind (random, few bits set, nearly all
    set, next to powers of two), near and far exponents, quotients next to 1
    and radicands next to squares."""
    rng = np.random.default_rng(seed)

    def draw():
        m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
        kind = rng.integers(0, 5, n)
        few = m & rng.integers(0, 1 << 52, n, dtype=np.uint64) & rng.integers(0, 1 << 52, n, dtype=np.uint64)
        top = np.uint64((1 << 52) - 1)
        m = np.select([kind == 1, kind == 2, kind == 3, kind == 4],
                      [few, top - few, m % np.uint64(5), top - m % np.uint64(5)], m)
        far = rng.integers(1, 2047, n, dtype=np.uint64)
        e = np.where(rng.random(n) < 0.5, far, 1000 + far % np.uint64(47))
        s = rng.integers(0, 2, n, dtype=np.uint64)
        return ((s << np.uint64(63)) | (e << np.uint64(52)) | m).view(np.float64)

    a, b = draw(), draw()
    near = rng.random(n) < 0.1
    a = np.where(near, (b.view(np.int64) + rng.integers(-3, 4, n)).view(np.float64), a)
    root = np.sqrt(np.abs(b)) if n else b
    with np.errstate(all="ignore"):
        sq = ((root * root).view(np.int64) + rng.integers(-2, 3, n)).view(np.float64)
    a = np.where(rng.random(n) < 0.1, sq, a)
    return np.ascontiguousarray(a), np.ascontiguousarray(b)


@pytest.mark.parametrize("op", [0, 1, 2])
@pytest.mark.parametrize("err", [0.0, 1.0, -1.0])
def test_integer_steps_round_like_the_hosts_operations(op, err):
    lib = native_lib("ieee_check")
    lib.ieeec_check.restype = ctypes.c_longlong
    lib.ieeec_check.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_double]
    a, b = operands(400_000, 7 + op)
    if op == 2:
        b = np.ascontiguousarray(np.abs(np.concatenate([a, b])))
        a = b.copy()
    # on top of its rounding to FP32 (2^-24): 2^-23 in all for rcp, 2^-22.9 for rsqrt
    bound = (2.0 ** -22.9 - 2.0 ** -24) if op == 2 else 2.0 ** -24
    assert lib.ieeec_check(op, a.ctypes.data, b.ctypes.data, b.size, err * bound) == 0


@pytest.mark.gpu
def test_device_forms_round_like_cudas_operations(gpu_lib, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = str(tmp_path / "ieee_check_gpu.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", os.path.join(HERE, "native", "ieee_check_gpu.cu"), "-o", out], check=True)
    lib = ctypes.CDLL(out)
    lib.ieeec_check_gpu.restype = ctypes.c_longlong
    lib.ieeec_check_gpu.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong]
    special = np.array([0.0, 5e-324, 2.2250738585072009e-308, 2.2250738585072014e-308, 1e-300, 1.0, 2.0, 3.0,
                        1.7976931348623157e308, 2.0 ** 1022, 2.0 ** 1023, np.inf, np.nan])
    special = np.concatenate([special, -special])
    grid = np.repeat(special, special.size), np.tile(special, special.size)
    for seed in range(4):
        a, b = operands(4_000_000, 100 + seed)
        a, b = (np.ascontiguousarray(np.concatenate([g, v])) for g, v in zip(grid, (a, b)))
        assert lib.ieeec_check_gpu(a.ctypes.data, b.ctypes.data, a.size) == 0
