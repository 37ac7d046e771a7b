"""General-mode compression over blocks of very different lengths: a few bits
to many words, on average and side by side, against the oracle's streams and
start bits."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_index_chain import DTYPES, _field


@pytest.mark.gpu
@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("shape", [(4,), (1021,), (36, 41), (9, 20, 33)])
def test_gpu_lengths(gz, orc, cuda, dt, shape):
    import torch
    P = 8 * np.dtype(dt).itemsize
    for kind in ("smooth", "sparse", "cliff"):
        a = _field(kind, shape, dt, 5)
        x = torch.from_numpy(a).to(cuda)
        for params in [orc.mode_precision(dt, p) for p in (1, 2, 7, 16, 31, P)] + \
                [(mn, mx, 64, -1074) for mn, mx in ((0, 65), (63, 64), (64, 200), (129, 129))]:
            s, offs = orc.compress_params(a, params, with_offsets=True)
            w, o = gz.compress_mode(x, gz.Mode(*params), with_offsets=True)
            assert np.array_equal(w.cpu().numpy().view(np.uint64), s), (kind, params)
            assert np.array_equal(o.cpu().numpy().view(np.uint64), offs), (kind, params)
            y = gz.decompress_mode(w, shape, x.dtype, gz.Mode(*params), offsets=o)
            z = orc.decompress_params(s, shape, dt, params)
            assert np.array_equal(y.cpu().numpy().view(np.uint8), z.view(np.uint8)), (kind, params)
