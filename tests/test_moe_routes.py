"""Which kernels routed experts go to, by size and by the switches that override it."""
import pytest

from tiny_inference_server_b200.kernels import ops


def _route(monkeypatch, pairs, rows, d, hidden, experts, **switches):
    for name, value in switches.items():
        monkeypatch.setattr(ops, name, value)
    return ops._experts_route(pairs, rows, d, hidden, experts)


@pytest.mark.parametrize("pairs,rows,d,hidden,experts,route", [
    (24, 8, 1536, 1024, 16, "few"), (96, 32, 1536, 1024, 16, "few"), (99, 33, 1536, 1024, 16, "tc"), (6144, 2048, 1536, 1024, 16, "tc"),
    (24, 4, 1024, 512, 64, "dots"), (6, 1, 1024, 512, 128, "few"), (96, 12, 1024, 512, 128, "grouped"), (1024, 128, 1024, 512, 128, "tc"),
    (120, 40, 256, 128, 16, "grouped"), (24, 8, 1544, 1024, 16, "dots"), (24, 8, 4096, 2048, 8, "few"), (16, 8, 4096, 2048, 8, "dots")])
def test_sizes(pairs, rows, d, hidden, experts, route, monkeypatch):
    assert _route(monkeypatch, pairs, rows, d, hidden, experts) == route


def test_switches(monkeypatch):
    wide = (200, 66, 1536, 1024, 16)
    assert _route(monkeypatch, *wide) == "tc"
    assert _route(monkeypatch, *wide, MOE_TC_WIDE_MIN_PAIRS=0) == "grouped"            # never: as any width
    assert _route(monkeypatch, *wide, MOE_TC_WIDE_MIN_PAIRS=96, MOE_TC_MIN_PAIRS=0) == "grouped"
    assert _route(monkeypatch, 24, 8, 1536, 1024, 16, MOE_FEW_MAX_PAIRS=0) == "dots"
    # the streaming kernel's own limit holds whatever the switch says
    assert _route(monkeypatch, 384, 128, 1536, 1024, 16, MOE_FEW_MAX_PAIRS=10 ** 6) == "few"
    assert _route(monkeypatch, 387, 129, 1536, 1024, 16, MOE_FEW_MAX_PAIRS=10 ** 6) == "grouped"
    assert _route(monkeypatch, *wide, MOE_FEW_MAX_PAIRS=96, MOE_GROUPED_MIN_PAIRS=0) == "dots"
