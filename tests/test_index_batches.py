"""The parallel block index of streams in buffers much longer than they are."""
from __future__ import annotations

import time

import pytest


@pytest.mark.gpu
def test_gpu_buffer_longer_than_its_stream(gz, cuda):
    """A buffer of 24 batches whose first holds the stream, with what earlier,
    longer streams left behind it: the same starts, in the time that the
    stream takes (a batch's own work takes about as long as the stream's, so
    that 24 of them are far beyond the limit) and a launch or so per batch."""
    import torch
    from cuzfp_gb300 import synth
    x = synth.sinusoids_device((128, 256, 256), 16, 32, seed=3, dtype=torch.float64, device=cuda)
    m = gz.mode_accuracy(gz.zfp_type.double, 1e-6)
    w, offs = gz.compress_mode(x, m, with_offsets=True)
    long = w.repeat((24 << 28) // 64 // w.numel() + 1)

    def best(words):
        times = []
        for _ in range(6):
            torch.cuda.synchronize()
            t = time.perf_counter()
            got = gz.index_blocks(words, x.shape, x.dtype, m)
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t)
            assert torch.equal(got, offs)
        return min(times[1:])

    assert best(long) < 8 * best(w)
