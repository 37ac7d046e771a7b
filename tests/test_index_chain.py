"""The parallel block index of general-mode streams: its kernels' per-thread
code on the CPU (tests/cpp/index_chain.cpp), and the index on the GPU, both
against the oracle compressor's block starts."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DTYPES = [np.float32, np.float64, np.int32, np.int64]


@pytest.fixture(scope="module")
def chain(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("ic") / "libindexchain.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall", "-Wno-unknown-pragmas",
                    "-Wno-maybe-uninitialized", "-I", os.path.join(ROOT, "cuzfp_gb300", "csrc"),
                    "-o", so, os.path.join(ROOT, "tests", "cpp", "index_chain.cpp")], check=True)
    lib = ctypes.CDLL(so)
    U, I, V, L = ctypes.c_uint, ctypes.c_int, ctypes.c_void_p, ctypes.c_ulonglong
    lib.ic_index.argtypes = [I, I, L, U, U, U, I, V, ctypes.c_size_t, L, U, U, U, I, V, V, V]
    return lib


def _field(kind, shape, dt, seed=0):
    """smooth: blocks alike; sparse: mostly zero blocks; cliff: every row
    falls by 2^30 from its first block to its last."""
    rng = np.random.default_rng(seed)
    n = np.indices(shape).astype(np.float64)
    a = sum(np.sin(x / (5.0 + 2 * i)) for i, x in enumerate(n)) + 1e-3 * rng.standard_normal(shape)
    if kind == "sparse":
        a = np.where(rng.random(shape[:1] + (1,) * (len(shape) - 1)) < 0.03, a, 0.0)
    if kind == "cliff":
        a = a * np.exp2(-30.0 * n[-1] / shape[-1])
    return (a * 2.0 ** 20).astype(dt) if np.dtype(dt).kind == "i" else a.astype(dt)


def _modes(orc, dt):
    m = [orc.mode_precision(dt, 14), (40, 900, 20, -1074)]
    if np.dtype(dt).kind == "f":
        m.append(orc.mode_accuracy(dt, 1e-4))
    return m


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("shape", [(5003,), (101, 203), (33, 34, 47)])
@pytest.mark.parametrize("kind", ["smooth", "sparse", "cliff"])
def test_bodies_against_oracle(chain, orc, dt, shape, kind):
    """By walks the index is complete; from headers it is either complete or
    names a field out of its range, and complete with that field in it, try
    by try.  One batch, and batches of two segments; a stream cut short is
    refused."""
    a = _field(kind, shape, dt)
    ints = np.dtype(dt).kind == "i"
    for params in _modes(orc, dt):
        s, offs = orc.compress_params(a, params, with_offsets=True)
        s = np.ascontiguousarray(s)
        bound = 1 + 11 + 64 * 65
        end = ctypes.c_ulonglong(0)

        def index(n, per, heads, field, got):
            return chain.ic_index(orc.type_code(dt), len(shape), offs.size, *params, s.ctypes.data,
                                  n, 0, 8192, bound, per, heads, field, got.ctypes.data,
                                  ctypes.byref(end))

        for heads in (0, 1):
            if heads and (ints or params[0] > 1):
                continue
            for per in (1 << 12, 2):
                got = np.zeros(offs.size, np.uint64)
                seen = (ctypes.c_uint * 2)(2 ** 32 - 1, 0)
                field = (ctypes.c_uint * 2)(*seen)
                for _ in range(40):
                    st = index(s.size, per, heads, field, got)
                    if st != 2:
                        break
                    seen[0], seen[1] = min(seen[0], field[0]), max(seen[1], field[0])
                    field = (ctypes.c_uint * 2)(*seen)
                assert st == 1, (params, heads, per, st)
                assert np.array_equal(got, offs), (params, heads, per)
                assert (end.value + 63) // 64 == s.size
                cut = index(s.size * 9 // 10, per, heads, field, got)
                # (a header cut in two may also read as one out of range)
                assert cut == 0 or (heads and cut == 2) or end.value > s.size * 9 // 10 * 64


@pytest.mark.gpu
@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("shape", [(33,), (517,), (40003,), (16, 36), (301, 203), (16, 12, 12),
                                   (64, 65, 67)])
def test_gpu_index(gz, orc, cuda, dt, shape):
    """Starts from the stream alone, from a handful of blocks up, in each
    mode and kind of field; a stream that ends early is refused; a buffer
    longer than its stream is not."""
    import torch
    for kind in ("smooth", "sparse", "cliff"):
        a = _field(kind, shape, dt, 7)
        for params in _modes(orc, dt) + [(5000, 5000, 20, -1074)]:
            s, offs = orc.compress_params(a, params, with_offsets=True)
            m = gz.Mode(*params)
            x = torch.empty(0, dtype=getattr(torch, np.dtype(dt).name))
            w = torch.from_numpy(np.ascontiguousarray(s).view(np.int64)).to(cuda)
            assert np.array_equal(gz.index_blocks(w, shape, x.dtype, m).cpu().numpy(),
                                  offs.view(np.int64)), (kind, params)
            pad = torch.cat([w, torch.zeros(w.numel() * 3 + 999, dtype=torch.int64, device=cuda)])
            assert np.array_equal(gz.index_blocks(pad, shape, x.dtype, m).cpu().numpy(),
                                  offs.view(np.int64)), (kind, params)
            if w.numel() > 8:
                with pytest.raises(gz.GzfpError):
                    gz.index_blocks(w[: w.numel() // 2].contiguous(), shape, x.dtype, m)


@pytest.mark.gpu
def test_gpu_index_batches(gz, cuda):
    """A stream longer than one batch of the index (2^28 bits)."""
    import torch
    from cuzfp_gb300 import synth
    x = synth.sinusoids_device((320, 300, 308), 16, 32, seed=3, dtype=torch.float64, device=cuda)
    for m in (gz.mode_accuracy(gz.zfp_type.double, 1e-9), gz.mode_precision(gz.zfp_type.double, 44)):
        w, offs = gz.compress_mode(x, m, with_offsets=True)
        assert w.numel() * 64 > 1 << 28
        assert torch.equal(gz.index_blocks(w, x.shape, x.dtype, m), offs)
