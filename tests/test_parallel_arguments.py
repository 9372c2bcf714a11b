"""Argument checks of the expert-parallel steps in front of the native calls (no GPU needed)."""
import types

import pytest
import torch

from oneccl_b200.parallel import ep


class _Native:
    def __init__(self):
        self.calls = []

    def moe_dispatch(self, *a):
        self.calls.append(a)

    moe_combine = moe_dispatch


@pytest.fixture
def native(monkeypatch):
    n = _Native()
    monkeypatch.setattr(ep, "native", lambda: n)
    return n


def _group(world, emulated):
    return types.SimpleNamespace(world=world, emulated_mode=emulated, n_entries=world if emulated else 1,
                                 handle=types.SimpleNamespace(value=0))


def _args(W, T=6, H=8):
    t = {"x": torch.zeros(W, T, H), "order": torch.zeros(W, T), "counts": torch.zeros(W, W), "meta": torch.zeros(W, 2 * W + 2)}
    return t, [torch.zeros(T * W, H) for _ in range(W)], [torch.zeros(W * W) for _ in range(W)]


@pytest.mark.parametrize("form", [list, tuple, lambda t: t])  # lists, tuples, one stacked tensor
@pytest.mark.parametrize("W", [1, 3])
def test_every_rank_has_its_tensor(native, W, form):
    t, recv, table = _args(W)
    g = _group(W, True)
    ep.fused_dispatch(g, form(t["x"]), form(t["order"]), form(t["counts"]), form(t["meta"]), recv, table, 1)
    ep.fused_combine(g, form(t["order"]), form(t["order"]), form(t["order"]), form(t["x"]), form(t["meta"]), recv, 1)
    for call in native.calls:
        lists = [a for a in call if isinstance(a, (list, tuple))]
        assert len(lists) >= 4 and all(len(x) == W for x in lists)
        assert [v.data_ptr() for v in lists[-1]] == [v.data_ptr() for v in t["meta"]]
        assert any(isinstance(a, torch.Tensor) and a.data_ptr() == recv[0].data_ptr() for a in call)


def test_a_bare_tensor_stands_for_one_rank(native):
    t, recv, table = _args(1)
    ep.fused_dispatch(_group(1, True), t["x"][0], t["order"][0], t["counts"][0], t["meta"][0], recv, table, 1)
    ep.fused_dispatch(_group(4, False), t["x"][0], t["order"][0], t["counts"][0], t["meta"][0], recv[0], table[0], 1)
    assert all(len(a) == 1 for call in native.calls for a in call if isinstance(a, list))


@pytest.mark.parametrize("world,emulated,given", [(3, True, 2), (3, True, 1), (3, True, 4), (3, False, 3)])
def test_other_numbers_of_tensors_are_refused(native, world, emulated, given):
    t, recv, table = _args(given)
    with pytest.raises(ValueError, match="ranks"):
        ep.fused_dispatch(_group(world, emulated), list(t["x"]), list(t["order"]), list(t["counts"]), list(t["meta"]), recv, table, 1)
    t, recv, table = _args(world)
    lists = {k: list(v) for k, v in t.items()}
    lists["x"] = lists["x"] + lists["x"][:1]
    with pytest.raises(ValueError, match="ranks"):
        ep.fused_combine(_group(world, True), lists["order"], lists["order"], lists["order"], lists["x"], lists["meta"], recv, 1)
    assert native.calls == []
