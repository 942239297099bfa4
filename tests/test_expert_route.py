"""What a gate launch sorted on the way reaches the expert products through the route they share, never through the ids or weights themselves."""
import types

import pytest
import torch

from jittorinfer_b200.ops import ExpertRoute, native

E, K, D, F = 8, 2, 64, 32


@pytest.fixture
def launches(monkeypatch):
    """Names of the launches; nothing is computed."""
    names = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: names.append(name) or 0
    monkeypatch.setattr(native, "load", lambda: Lib())
    monkeypatch.setattr(native, "_stream", lambda: 0)
    monkeypatch.setattr(native, "workspace", lambda dev: types.SimpleNamespace(
        scratch=torch.zeros(4), counters=torch.zeros(4, dtype=torch.int32), status=torch.zeros(4, dtype=torch.int32),
        route_counter=torch.zeros(1, dtype=torch.int32), sm_count=148, SCRATCH_BYTES=16, N_COUNTERS=4))
    return names


def gate(route, T=4):
    return native.moe_gate(torch.zeros(T, D).bfloat16(), torch.zeros(E, D), None, K, 1, 1, 1.0, False, False, route=route)


def experts(ids, wts, gated=True, route=None):
    w, wd = torch.zeros(E, F, D).bfloat16(), torch.zeros(E, D, F).bfloat16()
    return native.moe_routed(torch.zeros(ids.shape[0], D).bfloat16(), ids, wts, w if gated else None, w, wd, route=route)


@pytest.mark.parametrize("gated", [True, False])
def test_a_route_saves_the_sort(launches, gated):
    route = ExpertRoute(0, E)
    ids, wts = gate(route)
    _, dest = experts(ids, wts, gated, route)
    assert dest is route.pairs[2] and "jib_moe_gate_sort" in launches and "jib_moe_permute" not in launches


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("route", [None, (0, E)])
def test_without_one_ids_are_sorted_as_they_are_now(launches, gated, route):
    """Raw pointers and ``.data`` change ids without a trace; so nothing hangs on the tensors."""
    ids, wts = gate(route)
    ids.data[0, 0] += 1
    experts(ids, wts, gated)
    assert launches.count("jib_moe_permute") == 1
    assert native.moe_permute(ids, 0, E)[1] is not None and launches.count("jib_moe_permute") == 2


def test_weights_of_another_call_are_sorted_with_these_ids(launches):
    """Ids of a later gate may lie where earlier ones did: the address says nothing."""
    first = gate(ExpertRoute(0, E))
    second = gate(ExpertRoute(0, E))
    second[0].set_(first[0])
    experts(second[0], first[1], gated=False)
    assert launches.count("jib_moe_permute") == 1


def test_each_gate_call_refills_its_route(launches):
    route = ExpertRoute(0, E)
    gate(route)
    old = route.pairs
    ids, wts = gate(route, T=native.GATE_SORT_MAX_T + 1)
    assert old is not None and route.pairs is None
    experts(ids, wts, route=route)
    assert launches.count("jib_moe_permute") == 1


@pytest.mark.parametrize("base,T", [(1, 4), (0, 3)])
def test_a_route_of_other_experts_or_tokens_is_refused(launches, base, T):
    route = ExpertRoute(base, E)
    gate(route)
    with pytest.raises(ValueError, match="route of"):
        experts(torch.zeros(T, K, dtype=torch.int32), torch.zeros(T, K), route=route)
