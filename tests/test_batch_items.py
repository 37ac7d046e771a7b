"""The description of a batch's arrays, made on the host."""
from __future__ import annotations

import numpy as np
import pytest


@pytest.mark.parametrize("rate", [8, 8.0, "8", np.float32(8), np.array(8.0), "tensor"])
def test_rates_of_every_kind(gz, rate):
    """Whatever float() takes is a rate, hashable or not."""
    import torch
    if rate == "tensor":
        rate = torch.tensor(8.0)
    fields = [torch.zeros(5, 6, 7), torch.zeros(5, 6, dtype=torch.float64), torch.zeros(9)]
    words = [torch.zeros(64, dtype=torch.int64) for _ in fields]
    items = gz.batch_items(fields, words, [rate] * 3)
    assert [(i.nx, i.ny, i.nz, i.maxbits) for i in items] == \
        [(7, 6, 5, 512), (6, 5, 0, 128), (9, 0, 0, 32)]
    assert [i.stream_capacity for i in items] == [512] * 3
