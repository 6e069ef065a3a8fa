"""The adjoint smoother's room is a convenience: without memory for it, or inside a
capture, the sweeps form their systems as they go (host checks on a stand-in)."""
from types import SimpleNamespace

import pytest
import torch

from glide_b200 import grid as G


@pytest.fixture(autouse=True)
def no_capture(monkeypatch):
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)


def _level():
    return SimpleNamespace(_adj_factors=None, nb=1, nh=6, dtype=torch.float32, device=torch.device("cpu"))


def test_room_is_made_once():
    g = _level()
    a = G.Grid.adjoint_factors(g)
    assert a.numel() == 18 * 6 and G.Grid.adjoint_factors(g) is a


def test_no_memory_is_no_room(monkeypatch):
    def empty(*a, **k):
        raise torch.OutOfMemoryError("CUDA out of memory")
    g = _level()
    with monkeypatch.context() as m:
        m.setattr(torch, "empty", empty)
        assert G.Grid.adjoint_factors(g) is None
    assert G.Grid.adjoint_factors(g) is not None   # asked again when there is memory


def test_capture_makes_no_room(monkeypatch):
    g = _level()
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert G.Grid.adjoint_factors(g) is None


class _Sweeps(SimpleNamespace):
    def __getattr__(self, name):   # every field of the level
        return torch.zeros(1)


@pytest.mark.parametrize("n,given", [(3, 3), (0, 0), (-2, 0), (True, 1)])
def test_sweep_counts_are_those_of_a_range(monkeypatch, n, given):
    calls = []
    lib = SimpleNamespace(glide_vanka_adjoint_sweeps=lambda *a: calls.append(a[10]) or 0)
    g = _Sweeps(_lib=lib, _s=lambda: None, level_args=lambda: G.N.LevelArgs(), adjoint_factors=lambda: None)
    G.Grid.vanka_sweep_adjoint(g, n)
    assert calls == [given]


@pytest.mark.parametrize("n", [2.0, "2", None])
def test_sweep_counts_are_whole_numbers(n):
    g = _Sweeps(_lib=SimpleNamespace(), _s=lambda: None, level_args=lambda: G.N.LevelArgs(), adjoint_factors=lambda: None)
    with pytest.raises(TypeError):
        G.Grid.vanka_sweep_adjoint(g, n)
