"""Batches of one kind of array (dimensions and type) and of all twelve, whose
kernels run side by side."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DTYPES = ("float32", "float64", "int32", "int64")


def _field(rng, dt, shape):
    a = np.cumsum(rng.standard_normal(shape), axis=-1)
    return (a * 3000).astype(dt) if np.dtype(dt).kind == "i" else a.astype(dt)


@pytest.mark.parametrize("kinds", [1, 2, 5, 12])
def test_batch_kinds_side_by_side(gz, orc, cuda, kinds):
    import torch
    rng = np.random.default_rng(8)
    shapes = ((997,), (63, 90), (17, 22, 30))
    pairs = [(dt, sh) for sh in shapes for dt in DTYPES][:kinds]
    arrays = [_field(rng, dt, sh) for dt, sh in pairs for _ in range(2)]
    # staged and unstaged slots of every kind: whole words, and not
    rates = [16.0 if i % 2 == 0 else 13.25 for i in range(len(arrays))]
    fields = [torch.from_numpy(a).to(cuda) for a in arrays]
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            streams = gz.batch_stream_buffers(fields, rates)
            back = [torch.zeros_like(x) for x in fields]
            for _ in range(6):  # more calls than there are work lists
                gz.compress_batch(fields, rates, streams, cuda_stream=stream)
                gz.decompress_batch(streams, back, rates, cuda_stream=stream)
        stream.synchronize()
        for a, r, w, b in zip(arrays, rates, streams, back):
            s = orc.compress(a, r)
            assert np.array_equal(w.cpu().numpy().view(np.uint64)[:s.size], s), (a.shape, a.dtype, r)
            assert np.array_equal(b.cpu().numpy().view(np.uint8),
                                  orc.decompress(s, a.shape, a.dtype, r).view(np.uint8))
