"""The parallel block index of streams of a few dozen to a few thousand blocks
(segments and chunks as short as they come), against the oracle compressor's
block starts."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_index_chain import DTYPES, _field, _modes

SHAPES = [(125,), (129,), (133,), (320,), (325,), (2050,), (20, 28), (36, 36), (90, 91),
          (12, 12, 12), (12, 12, 16), (16, 16, 32), (32, 36, 40)]


@pytest.mark.gpu
@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("shape", SHAPES)
def test_gpu_short_streams(gz, orc, cuda, dt, shape):
    """Both sides of the line between the serial walk and the index; exact
    buffers, longer ones, and streams cut short, which are refused."""
    import torch
    t = getattr(torch, np.dtype(dt).name)
    for kind in ("smooth", "sparse", "cliff"):
        a = _field(kind, shape, dt, 11)
        for params in _modes(orc, dt) + [orc.mode_precision(dt, 3), orc.mode_precision(dt, 30)]:
            s, offs = orc.compress_params(a, params, with_offsets=True)
            m = gz.Mode(*params)
            w = torch.from_numpy(np.ascontiguousarray(s).view(np.int64)).to(cuda)
            pad = torch.cat([w, torch.full((77,), 0x5A5A0FF1, dtype=torch.int64, device=cuda)])
            for words in (w, pad):
                got = gz.index_blocks(words, shape, t, m).cpu().numpy()
                assert np.array_equal(got, offs.view(np.int64)), (kind, params)
            if w.numel() > 8:
                with pytest.raises(gz.GzfpError):
                    gz.index_blocks(w[: w.numel() // 2].contiguous(), shape, t, m)
