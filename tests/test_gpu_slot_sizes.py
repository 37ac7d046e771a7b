"""Listed blocks whose slots lie on both sides of the longest staged one, in
lists on both sides of the length at which long slots of 32-bit values are
read from the stream."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DTYPES = ("float32", "float64", "int32", "int64")


def _field(rng, dt, shape):
    a = np.cumsum(rng.standard_normal(shape), axis=-1)
    return (a * 3000).astype(dt) if np.dtype(dt).kind == "i" else a.astype(dt)


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("words", [1, 15, 16, 17, 31, 32, 33])
def test_listed_slots_of_whole_words(gz, orc, cuda, dt, words):
    import torch
    rng = np.random.default_rng(7)
    a = _field(rng, dt, (18, 21, 15))
    s = orc.compress(a, float(words))
    tiles, codes = orc.field_tiles(a)
    ws = torch.from_numpy(s.view(np.int64)).to(cuda)
    tdt = getattr(torch, dt)
    for count in (1, 33, 700, (1 << 16) + 1):
        idx = rng.integers(0, tiles.shape[0], count)
        exp = orc.decode_blocks(s, dt, 3, words * 64, idx, codes[idx], tiles=np.full((count, 64), 5, dt))
        out = torch.full((count, 64), 5, dtype=tdt, device=cuda)
        gz.decode_blocks(ws, tdt, 3, words * 64, idx.astype(np.int64), codes[idx], out=out)
        assert np.array_equal(out.cpu().numpy().view(np.uint8), exp.view(np.uint8)), count
