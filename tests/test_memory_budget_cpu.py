"""Memory that workspaces may take beyond what they have to, with a fake of the device's counters."""
import pytest
import torch

from arctic_platform_b200.ops.logprob import _bwd_rows
from arctic_platform_b200.utils import memory_budget


@pytest.mark.parametrize("N", [1, 333, 4096, 4097, 16384, 18000, 40000])
@pytest.mark.parametrize("V", [8, 32000, 151936, 1 << 20])
@pytest.mark.parametrize("spare", [0, 1 << 30, 3 << 30, 1 << 40])
def test_rows_of_dlogits(N, V, spare):
    """Chunks cover N, take 4096 rows where nothing is to spare, and never more beyond that than there is or than the budget."""
    rows = _bwd_rows(N, V, spare)
    assert 1 <= rows <= N and -(-N // rows) == -(-N // max(rows, min(N, 4096)))
    units = -(-rows // 4096)
    assert (units - 1) * 4096 * V * 2 <= spare and (units == 1 or units * 4096 * V * 2 <= 5 << 30)
    if spare == 0:
        assert rows <= 4096
    if spare > 5 << 30 and N <= 4096 * ((5 << 30) // (4096 * V * 2)):
        assert rows == N


def test_spare_memory(monkeypatch):
    gb = 1 << 30
    state = {"free": 60 * gb, "capturing": False}
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state["capturing"])
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda i: (state["free"], 100 * gb))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda i: 30 * gb)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda i: 25 * gb)
    monkeypatch.setattr(memory_budget, "_kv_resident", {})
    monkeypatch.setattr(memory_budget, "_kv_awake", {})
    dev = torch.device("cuda", 0)
    assert memory_budget.spare_bytes(dev) == 65 * gb - 12 * gb
    memory_budget.set_kv_resident(dev, 40 * gb)               # counted by the driver while it is there ...
    state["free"] = 20 * gb
    assert memory_budget.spare_bytes(dev) == 25 * gb - 12 * gb
    memory_budget.set_kv_resident(dev, 0)                     # ... and asleep its place stays its own
    state["free"] = 60 * gb
    assert memory_budget.spare_bytes(dev) == 25 * gb - 12 * gb
    state["free"] = 1 * gb
    assert memory_budget.spare_bytes(dev) == 0
    state.update(free=60 * gb, capturing=True)
    assert memory_budget.spare_bytes(dev) == 0
