"""Output columns that a call allocated itself are the result's alone: dropping
the result gives them back."""
import numpy as np
import pytest

from bats import encoded_col

from ahead_b200.model import GE, LT, RESINT

pytestmark = pytest.mark.gpu


def test_columns_go_back_with_the_result(monkeypatch):
    import gc
    import torch
    import ahead_b200.gpu as mirror
    monkeypatch.setattr(mirror, "_SIZED_BYTES", 0)
    g = mirror.GpuOps(0)
    b = mirror.to_device(encoded_col(RESINT, np.arange(1 << 20)))
    A = b.tail.A
    g.select_an(b, GE, 0, LT, 5 * A)  # (the error vectors' buffer is made)
    gc.collect()
    before = torch.cuda.memory_allocated()
    r, _ = g.select_an(b, GE, 0)
    assert torch.cuda.memory_allocated() >= before + r.count * 8
    del r
    gc.collect()
    assert torch.cuda.memory_allocated() == before
    with pytest.raises(mirror.AheadError):  # (a call that fails lets go of them, too)
        g.select_an(b, 99, 0)
    gc.collect()
    assert torch.cuda.memory_allocated() == before
    g.close()
