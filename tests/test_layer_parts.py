"""CPU test of MoeLayer.forward's choice between one library call and its launchers (the calls themselves are recorded, not made)."""
import pytest
import torch

from strixite_b200 import kernels as K
from strixite_b200.layer import MoeBuffers, MoeLayer, MoeWeights


def view(n, k):
    return K.QDeviceView(torch.empty((n, k // 2), dtype=torch.uint8), torch.empty((n, k // 128), dtype=torch.int16),
                         torch.empty((n, k // 128), dtype=torch.int16), n, k, 128, 4)


def calls_of(monkeypatch, cls, prepare=lambda layer: None, ctx=lambda mp: None):
    E, k, d, I, T = 4, 2, 256, 128, 3
    made = []
    for name in ("moe_layer", "moe_route_small", "moe_router", "moe_group_routes", "linear_qw_experts_gather_grouped_swiglu",
                 "linear_qw_experts_combine_grouped"):
        monkeypatch.setattr(K, name, lambda *a, _n=name, **kw: made.append(_n))
    ctx(monkeypatch)
    layer = cls(MoeWeights(view(E * 2 * I, d), view(E * d, I)), E, k, MoeBuffers(T, d, I, E, k, torch.device("cpu"), False))
    prepare(layer)
    layer.forward(torch.empty((T, d), dtype=torch.bfloat16), torch.empty((T, E)), torch.empty((T, d)), math=K.MoeMath.F32)
    return made


LAUNCHERS = ["linear_qw_experts_gather_grouped_swiglu", "linear_qw_experts_combine_grouped"]


def test_forward_is_one_call(monkeypatch):
    assert calls_of(monkeypatch, MoeLayer) == ["moe_layer"]


@pytest.mark.parametrize("part", ["route", "experts", "run_experts", "shared_expert"])
@pytest.mark.parametrize("where", ["subclass", "instance", "class"])
def test_an_overridden_part_is_called(monkeypatch, part, where):
    seen = []
    own = getattr(MoeLayer, part)

    def mine(self, *a, **kw):
        seen.append(part)
        return own(self, *a, **kw)

    if where == "subclass":
        made = calls_of(monkeypatch, type("Mine", (MoeLayer,), {part: mine}))
    elif where == "instance":
        made = calls_of(monkeypatch, MoeLayer, lambda layer: setattr(layer, part, mine.__get__(layer)))
    else:
        made = calls_of(monkeypatch, MoeLayer, ctx=lambda mp: mp.setattr(MoeLayer, part, mine))
    assert made == ["moe_route_small"] + LAUNCHERS
    assert seen == ([] if part == "shared_expert" else [part])  # this layer has no shared expert


def test_small_slots_is_heeded(monkeypatch):
    made = calls_of(monkeypatch, MoeLayer, lambda layer: setattr(layer, "small_slots", 0))
    assert made == ["moe_router", "moe_group_routes"] + LAUNCHERS
