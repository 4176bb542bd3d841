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
    state = {"free": 60 * gb, "unused": 5 * gb, "capturing": False, "asked": 0}

    def ask(i):
        state["asked"] += 1
        return state["free"], 100 * gb

    current = lambda n: {"all": {"current": n}}
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state["capturing"])
    monkeypatch.setattr(torch.cuda, "mem_get_info", ask)
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict",
                        lambda i: {"reserved_bytes": current(25 * gb + state["unused"]), "allocated_bytes": current(25 * gb)})
    monkeypatch.setattr(memory_budget, "_kv_resident", {})
    monkeypatch.setattr(memory_budget, "_kv_awake", {})
    dev, most = torch.device("cuda", 0), 1000 * gb
    assert memory_budget.spare_bytes(dev, most) == 65 * gb - 12 * gb
    assert memory_budget.spare_bytes(dev, 3 * gb) == 3 * gb
    memory_budget.set_kv_resident(dev, 40 * gb)               # counted by the driver while it is there ...
    state["free"] = 20 * gb
    assert memory_budget.spare_bytes(dev, most) == 25 * gb - 12 * gb
    memory_budget.set_kv_resident(dev, 0)                     # ... and asleep its place stays its own, given back to the driver
    state["free"] = 60 * gb
    assert memory_budget.spare_bytes(dev, most) == 25 * gb - 12 * gb
    state.update(free=20 * gb, unused=45 * gb)                # or kept by the caching allocator
    assert memory_budget.spare_bytes(dev, most) == 25 * gb - 12 * gb
    state["asked"] = 0
    assert memory_budget.spare_bytes(dev, 5 * gb) == 5 * gb and state["asked"] == 0
    state.update(free=1 * gb, unused=5 * gb)
    assert memory_budget.spare_bytes(dev, most) == 0
    state.update(free=60 * gb, capturing=True)
    assert memory_budget.spare_bytes(dev, most) == 0
