"""The parallel block index where a block's budget ends it: what its CTAs read
lies inside the words they stage (on the CPU, tests/cpp/index_bounds.cpp), and
its starts are the oracle compressor's (on the GPU)."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests.test_index_chain import ROOT, _field

FLOATS = [np.float32, np.float64]
# (minbits, maxbits, maxprec, minexp): budgets below a block's longest code
BUDGETS = [(mn, mx, 64, -1074) for mn in (0, 1) for mx in (13, 64, 100, 600, 1000)] + \
          [(0, 100, 20, -1074), (1, 600, 64, -30)]


@pytest.fixture(scope="module")
def bounds(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("ib") / "libindexbounds.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall", "-Wno-unknown-pragmas",
                    "-Wno-maybe-uninitialized", "-I", os.path.join(ROOT, "cuzfp_gb300", "csrc"),
                    "-o", so, os.path.join(ROOT, "tests", "cpp", "index_bounds.cpp")], check=True)
    lib = ctypes.CDLL(so)
    U, I, V, L = ctypes.c_uint, ctypes.c_int, ctypes.c_void_p, ctypes.c_ulonglong
    lib.ib_run.argtypes = [I, I, U, U, U, I, V, ctypes.c_size_t, L, U, U, U, I, V]
    lib.ib_run.restype = None
    return lib


def _bound(dt, dims, params):
    """Bits of the longest block (zfp_stream_maximum_size's bound per block)."""
    P, ebits = (32, 8) if np.dtype(dt).itemsize == 4 else (64, 11)
    values = 4 ** dims
    return min(1 + ebits + values - 1 + values * min(P, params[2]), params[1])


def _check(bounds, orc, dt, dims, params, words, nblocks, fields, sms):
    counts = (ctypes.c_ulonglong * 3)()
    bounds.ib_run(orc.type_code(dt), dims, *params, words.ctypes.data, words.size, nblocks,
                  _bound(dt, dims, params), *fields, sms, counts)
    outside, wrong, parsed = counts
    assert outside == 0 and wrong == 0, (params, sms, outside, wrong, parsed)
    return parsed


@pytest.mark.parametrize("dt", FLOATS)
@pytest.mark.parametrize("shape", [(5003,), (101, 203), (64, 64, 64)])
def test_reads_stay_in_the_staged_words(bounds, orc, dt, shape):
    """Streams of every budget, as few and as many CTAs parse them (sms), from
    a narrow and from the widest range of exponents."""
    a = _field("smooth", shape, dt)
    bias = 127 if dt is np.float32 else 1023
    none = (2 ** 32 - 1, 0)
    for params in BUDGETS + [orc.mode_precision(dt, 28), orc.mode_accuracy(dt, 1e-6)]:
        s, offs = orc.compress_params(a, params, with_offsets=True)
        s = np.ascontiguousarray(s)
        for fields in ((bias - 8, bias + 2), none):
            for sms in (1, 152):
                assert _check(bounds, orc, dt, len(shape), params, s, offs.size, fields, sms)


@pytest.mark.parametrize("dt", FLOATS)
@pytest.mark.parametrize("dims", [1, 2, 3])
def test_reads_on_random_bits(bounds, orc, dt, dims):
    """A stream may hold anything: random words, zeros, ones and sparse ones."""
    rng = np.random.default_rng(dims)
    n = 1000
    kinds = [rng.integers(0, 2 ** 64, n, np.uint64), np.full(n, 2 ** 64 - 1, np.uint64),
             np.uint64(1) << rng.integers(0, 64, n).astype(np.uint64)]
    top, mid = (255, 127) if dt is np.float32 else (2047, 1023)
    parsed = 0
    for words in kinds:
        for params in BUDGETS + [(0, 4171, 64, -1074), (0, 4171, 9, -1074)]:
            for fields in ((0, 30), (mid - 20, mid + 20), (top - 30, top)):
                for nblocks in (40, 4000):
                    parsed += _check(bounds, orc, dt, dims, params, words, nblocks, fields, 152)
    assert parsed > 100000


@pytest.mark.gpu
@pytest.mark.parametrize("dt", FLOATS)
@pytest.mark.parametrize("shape", [(5003,), (101, 203), (64, 64, 64)])
def test_gpu_starts_under_budgets(gz, orc, cuda, dt, shape):
    import torch
    for kind in ("smooth", "sparse"):
        a = _field(kind, shape, dt, 3)
        for params in BUDGETS:
            s, offs = orc.compress_params(a, params, with_offsets=True)
            w = torch.from_numpy(np.ascontiguousarray(s).view(np.int64)).to(cuda)
            t = getattr(torch, np.dtype(dt).name)
            got = gz.index_blocks(w, shape, t, gz.Mode(*params)).cpu().numpy()
            assert np.array_equal(got, offs.view(np.int64)), (kind, params)
