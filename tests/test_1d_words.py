"""1D blocks whose coder finds out how many words and planes it needs: every
budget and precision on the CPU, and the paths that use it (streams behind a
header, listed blocks, batches, general modes) on the GPU."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_odd_budgets import DTYPES, _values

LEAST = {np.float32: 9, np.float64: 12}


def _same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


@pytest.mark.parametrize("dt", DTYPES)
def test_budgets(hostcodec, orc, dt):
    rng = np.random.default_rng(8)
    a = _values(rng, dt, (203,))
    t = orc.type_code(dt)
    for bits in list(range(LEAST.get(dt, 1), 141)) + [191, 192, 193, 255, 257, 300, 319, 321, 400]:
        rate = bits / 4.0
        s = np.ascontiguousarray(orc.compress(a, rate))
        w = np.zeros(s.size, np.uint64)
        hostcodec.hc_compress(t, a.size, 0, 0, rate, a.ctypes.data, w.ctypes.data, s.nbytes)
        assert np.array_equal(w, s), bits
        for words in (s, rng.integers(0, 2 ** 64, s.size, np.uint64)):  # and any stream
            out = np.zeros_like(a)
            hostcodec.hc_decompress(t, a.size, 0, 0, rate, words.ctypes.data, words.nbytes,
                                    out.ctypes.data)
            assert _same(out, orc.decompress(words, a.shape, dt, rate)), bits


@pytest.mark.parametrize("dt", DTYPES)
def test_precisions(hostcodec, orc, dt):
    a = _values(np.random.default_rng(9), dt, (203,))
    t, P = orc.type_code(dt), 8 * np.dtype(dt).itemsize
    modes = [orc.mode_precision(dt, p) for p in range(1, P + 1)]
    modes += [(0, mx, p, -1074) for mx in (13, 40, 64, 65, 100, 150) for p in (5, 33, 64)]
    modes += [(70, 200, 16, -1074)]
    if np.dtype(dt).kind == "f":
        modes += [orc.mode_accuracy(dt, 10.0 ** e) for e in range(-12, 6)]
    for params in modes:
        s = np.ascontiguousarray(orc.compress_params(a, params))
        w = np.zeros(s.size + 1, np.uint64)
        hostcodec.hc_compress_params(t, a.size, 0, 0, *params, a.ctypes.data, w.ctypes.data, w.nbytes)
        assert np.array_equal(w[: s.size], s), params
        out = np.zeros_like(a)
        hostcodec.hc_decompress_params(t, a.size, 0, 0, *params, s.ctypes.data, s.nbytes,
                                       out.ctypes.data)
        assert _same(out, orc.decompress_params(s, a.shape, dt, params)), params


@pytest.mark.gpu
@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("n", [3, 517, 4097])
def test_gpu_paths(gz, orc, cuda, dt, n):
    import torch
    a = _values(np.random.default_rng(n), dt, (n,))
    x = torch.from_numpy(a).to(cuda)
    budgets = (14, 20, 21, 32, 33, 64, 65, 128, 129, 192, 260, 400)
    for bits in budgets:
        rate = bits / 4.0
        s = orc.compress(a, rate)
        d = orc.decompress(s, a.shape, dt, rate)
        w = gz.compress_headed(x, rate)
        assert _same(gz.decompress_headed(w).cpu().numpy(), d), bits
        words = torch.from_numpy(s.view(np.int64)).to(cuda)
        nb = n // 4  # whole blocks
        if nb:
            idx = torch.arange(nb, dtype=torch.int64, device=cuda)
            tiles = gz.decode_blocks(words, x.dtype, 1, bits, idx)
            assert _same(tiles.cpu().numpy().reshape(-1), d[: 4 * nb]), bits
            again = words.clone()
            gz.encode_blocks(x[: 4 * nb].reshape(nb, 4).contiguous(), 1, bits, idx, again)
            assert np.array_equal(again.cpu().numpy().view(np.uint64), s), bits
    rates = [b / 4.0 for b in budgets]
    streams = gz.batch_stream_buffers([x] * len(rates), rates)
    gz.compress_batch([x] * len(rates), rates, streams)
    out = [torch.empty_like(x) for _ in rates]
    gz.decompress_batch(streams, out, rates)
    for r, w, y in zip(rates, streams, out):
        s = orc.compress(a, r)
        assert np.array_equal(w.cpu().numpy().view(np.uint64), s), r
        assert _same(y.cpu().numpy(), orc.decompress(s, a.shape, dt, r)), r
