"""Blocks that are not whole 64-bit words: 1D budgets around the limits of
the coder's word counts (on the CPU and the GPU), and, on the GPU, CTAs that
stage their run of the stream -- every scalar type and dimensionality, counts
of blocks around a CTA's 128, budgets of both kinds of staging and of none."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DTYPES = [np.float32, np.float64, np.int32, np.int64]


def _values(rng, dt, shape):
    """Walks over twelve decades with flat, zero and noisy stretches."""
    n = int(np.prod(shape))
    a = np.cumsum(rng.standard_normal(n)) * np.exp2(rng.integers(-20, 20, n // 16 + 1).repeat(16)[:n])
    a[rng.random(n) < 0.1] = 0
    a[n // 3: n // 3 + 40] = 7.25
    a = a.reshape(shape)
    return (a * 1000).astype(dt) if np.dtype(dt).kind == "i" else a.astype(dt)


@pytest.fixture(scope="module")
def short(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("sc") / "libshort.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wno-unknown-pragmas",
                    "-I", os.path.join(ROOT, "cuzfp_gb300", "csrc"), "-o", so,
                    os.path.join(ROOT, "tests", "cpp", "short_codes.cpp")], check=True)
    lib = ctypes.CDLL(so)
    V, I, U = ctypes.c_void_p, ctypes.c_int, ctypes.c_uint
    lib.sc_code.argtypes = [I, I, I, U, U, V, V, ctypes.c_size_t]
    return lib


@pytest.mark.parametrize("dt", DTYPES)
def test_short_codes(short, orc, dt):
    """Every 1D budget up to one and two words of code, values and streams as
    the oracle's."""
    a = _values(np.random.default_rng(5), dt, (403,))
    lo = {np.float32: 9, np.float64: 12}.get(dt, 1)
    for bits in range(lo, 129):
        s = np.ascontiguousarray(orc.compress(a, bits / 4.0))
        d = orc.decompress(s, a.shape, dt, bits / 4.0)
        for nw in (0, 1, 2):
            if bits > (64 * nw or 32):
                continue
            w = np.zeros(s.size + 1, np.uint64)
            short.sc_code(0, orc.type_code(dt), nw, a.size, bits, a.ctypes.data, w.ctypes.data, s.size)
            assert np.array_equal(w[: s.size], s), (bits, nw)
            out = np.zeros_like(a)
            short.sc_code(1, orc.type_code(dt), nw, a.size, bits, out.ctypes.data, s.ctypes.data, s.size)
            assert np.array_equal(out.view(np.uint8), d.view(np.uint8)), (bits, nw)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("shape,bits", [
    ((4 * 128 - 1,), (13, 48, 64, 65, 127, 129, 200, 257, 520, 1100)),
    ((4 * 128 + 1,), (12, 16, 20, 21, 32)),
    ((4 * 128 + 5,), (33, 64, 128, 256)), ((2,), (48,)), ((100003,), (48, 100)),
    ((44, 47), (37, 191, 193, 720, 1001, 1100)), ((401, 203), (90,)),
    ((20, 21, 22), (70, 723, 1000, 1023, 1500, 2700, 4100)), ((52, 33, 37), (500,))])
def test_gpu_odd_budgets(gz, orc, cuda, dt, shape, bits):
    import torch
    a = _values(np.random.default_rng(6), dt, shape)
    x = torch.from_numpy(a).to(cuda)
    for b in bits:
        rate = b / 4.0 ** len(shape)
        s = orc.compress(a, rate, 4)
        # what was in the stream buffer before must not show
        w = torch.full((s.size,), -1, dtype=torch.int64, device=cuda)
        gz.compress_tensor(x, rate, out=w)
        assert np.array_equal(w.cpu().numpy().view(np.uint64), s), b
        d = gz.decompress_tensor(w, shape, x.dtype, rate).cpu().numpy()
        assert np.array_equal(d.view(np.uint8), orc.decompress(s, shape, dt, rate, 4).view(np.uint8)), b
