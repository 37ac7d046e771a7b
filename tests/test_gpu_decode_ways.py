"""4^3 blocks read from the stream in place, by table and by token: streams
behind a header, listed blocks, batches and start bits, at the budgets and
precisions where the way changes, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_index_chain import DTYPES, _field


def _same(t, a):
    return np.array_equal(t.cpu().numpy().view(np.uint8), a.view(np.uint8))


@pytest.mark.gpu
@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("kind", ["smooth", "noise"])
def test_gpu_precisions(gz, orc, cuda, dt, kind):
    import torch
    shape = (13, 20, 30)
    a = _field("smooth", shape, dt, 5)
    if kind == "noise":
        a = (a + np.random.default_rng(1).standard_normal(shape) * a.max()).astype(dt)
    P = 8 * np.dtype(dt).itemsize
    t = getattr(torch, np.dtype(dt).name)
    modes = [orc.mode_precision(dt, p) for p in (1, 11, 12, 13, 15, 16, 17, 31, 32, 33, P - 1, P) if p <= P]
    modes += [(0, 500, 12, -1074), (0, 500, 40, -1074), (0, 1024, 64, -1074), (0, 1025, 64, -1074)]
    for params in modes:
        s, offs = orc.compress_params(a, params, with_offsets=True)
        w = torch.from_numpy(np.ascontiguousarray(s).view(np.int64)).to(cuda)
        o = torch.from_numpy(offs.view(np.int64)).to(cuda)
        y = gz.decompress_mode(w, shape, t, gz.Mode(*params), offsets=o)
        assert _same(y, orc.decompress_params(s, shape, dt, params)), params


@pytest.mark.gpu
@pytest.mark.parametrize("dt", DTYPES)
def test_gpu_many_blocks_of_few_planes(gz, orc, cuda, dt):
    """Above and below the number of blocks from which few planes go by token."""
    import torch
    t = getattr(torch, np.dtype(dt).name)
    for shape in ((108, 108, 107), (104, 108, 107)):
        a = _field("smooth", shape, dt, 2)
        for p in (3, 12, 13, 16, 17):
            params = orc.mode_precision(dt, p)
            s, offs = orc.compress_params(a, params, with_offsets=True)
            w = torch.from_numpy(np.ascontiguousarray(s).view(np.int64)).to(cuda)
            o = torch.from_numpy(offs.view(np.int64)).to(cuda)
            y = gz.decompress_mode(w, shape, t, gz.Mode(*params), offsets=o)
            assert _same(y, orc.decompress_params(s, shape, dt, params)), (shape, p)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", DTYPES)
def test_gpu_budgets(gz, orc, cuda, dt):
    import torch
    rng = np.random.default_rng(4)
    shape = (13, 20, 31)
    nb = 4 * 5 * 8
    a = _field("smooth", shape, dt, 6)
    a = (a + rng.standard_normal(shape) * 1e-3 * a.max()).astype(dt)
    x = torch.from_numpy(a).to(cuda)
    t = x.dtype
    for bits in (70, 511, 640, 1001, 1023, 1024, 1025, 1088, 2047, 2049, 2200):
        rate = bits / 64.0
        s = orc.compress(a, rate)
        w = gz.compress_headed(x, rate)
        assert _same(gz.decompress_headed(w), orc.decompress(s, shape, dt, rate)), bits
        # blocks of any bits, listed; the last ones end with the stream
        junk = rng.integers(0, 2 ** 64, (nb * bits + 63) // 64, np.uint64)
        d = orc.decompress(junk, (16, 20, 32), dt, rate)
        tiles = d.reshape(4, 4, 5, 4, 8, 4).transpose(0, 2, 4, 1, 3, 5).reshape(nb, 64)
        idx = torch.arange(nb, dtype=torch.int64, device=cuda).flip(0)
        got = gz.decode_blocks(torch.from_numpy(junk.view(np.int64)).to(cuda), t, 3, bits, idx)
        assert _same(got.reshape(nb, 64), np.ascontiguousarray(tiles[::-1])), bits
        out = [torch.empty((16, 20, 32), dtype=t, device=cuda)]
        gz.decompress_batch([torch.from_numpy(junk.view(np.int64)).to(cuda)], out, [rate])
        assert _same(out[0], d), bits
