"""Gate and expert sort of up to 64 tokens as one launch, and the sort by matching: against the separate launches and a stable sort."""
import pytest
import torch

from jittorinfer_b200.ops import ExpertRoute

pytestmark = pytest.mark.gpu
DEV = "cuda"


def check_sort(ids, base, E_local, seg, src, dest):
    T, k = ids.shape
    flat = ids.flatten().long().cpu() - base
    ok = (flat >= 0) & (flat < E_local)
    order = torch.sort(torch.where(ok, flat, torch.full_like(flat, E_local)), stable=True).indices
    n = int(ok.sum())
    want = torch.full_like(flat, -1)
    want[order[:n]] = torch.arange(n)
    assert torch.equal(dest.flatten().cpu().long(), want)
    assert torch.equal(src.cpu().long()[:n], order[:n] // k) and bool((src[n:] == -1).all())
    counts = torch.bincount(flat[ok], minlength=E_local)
    assert torch.equal(seg.cpu().long(), torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)]))
    active = torch.full((E_local,), -1)
    hit = torch.nonzero(counts).flatten()
    active[:len(hit)] = hit
    room = torch.as_strided(seg, (E_local,), (1,), seg.storage_offset() + E_local + 1)
    assert torch.equal(room.cpu().long(), active)
    return order[:n]


# warps with no, one and two tokens; runs of 32 pairs that end within, at and past a warp; experts below, at and past a lane's registers
@pytest.mark.parametrize("T", [1, 3, 4, 5, 31, 32, 33, 64, 65])
@pytest.mark.parametrize("E,k,n_shared,n_group,topk_group,top2,sigmoid,norm,base,E_local",
                         [(64, 6, 2, 1, 1, False, False, False, 0, 66), (160, 6, 0, 8, 3, False, False, False, 40, 20),
                          (256, 8, 0, 8, 4, True, True, True, 0, 256), (7, 7, 1, 1, 1, False, True, True, 0, 8), (33, 31, 1, 1, 1, False, False, True, 3, 5)])
def test_one_launch(nat, T, E, k, n_shared, n_group, topk_group, top2, sigmoid, norm, base, E_local):
    gen = torch.Generator(device=DEV).manual_seed(T + E)
    x = torch.randn(T, 512, generator=gen, device=DEV).bfloat16()
    w = torch.randn(E, 512, generator=gen, device=DEV) * 0.05
    if n_group == 1:
        w[E // 2:] = w[:E - E // 2].clone()                                   # choices between experts of equal score
    bias = torch.rand(E, generator=gen, device=DEV) * 0.01 if sigmoid and n_group > 1 else None
    lb = torch.randn(E, generator=gen, device=DEV) if n_group == 1 and E != 64 else None
    args = (x, w, bias, k, n_group, topk_group, 2.5, norm, sigmoid, n_shared, top2)
    ids0, wts0 = nat.moe_gate(*args, logit_bias=lb)
    route = ExpertRoute(base, E_local)
    for _ in range(2):
        ids, wts = nat.moe_gate(*args, route=route, logit_bias=lb)
    assert torch.equal(ids, ids0) and torch.equal(wts, wts0)
    assert (route.pairs is None) == (T > nat.GATE_SORT_MAX_T)
    if route.pairs is not None:
        seg, src, dest, rows = route.pairs
        order = check_sort(ids, base, E_local, seg, src, dest)
        assert torch.equal(rows[:len(order)].cpu(), wts.flatten().cpu()[order])
    check_sort(ids, base, E_local, *nat.moe_permute(ids, base, E_local))
    with torch.inference_mode():
        ids, wts = nat.moe_gate(*args, route=route, logit_bias=lb)
        assert torch.equal(ids, ids0) and (route.pairs is None or torch.equal(route.pairs[2], dest))
    # a pair instead of a route: gate and sort stay apart
    assert torch.equal(nat.moe_gate(*args, route=(base, E_local), logit_bias=lb)[0], ids0)


def test_no_numbers_and_infinities(nat):
    """Scores that are all NaN pick expert 0; logits of minus infinity are probabilities of 0, taken in order of their ids."""
    E, k = 40, 4
    logits = torch.zeros(3, E, device=DEV)
    logits[0] = float("nan")
    logits[1] = float("-inf")
    logits[1, 7] = 1.0
    logits[2, 33] = logits[2, 5] = 3.0
    ids = torch.empty(3, k, dtype=torch.int32, device=DEV)
    wts = torch.empty(3, k, device=DEV)
    nat._ck(nat.load().jib_moe_gate(None, None, None, None, logits.data_ptr(), ids.data_ptr(), wts.data_ptr(), 3, 8, E, k, 1, 1, 1.0, 0, 0, 0, 0, 0,
                                    nat._stream()), "moe_gate")
    assert ids[0].tolist() == [0, 0, 0, 0]
    assert ids[1].tolist() == [7, 0, 1, 2] and wts[1].tolist() == [1.0, 0.0, 0.0, 0.0]
    assert ids[2].tolist() == [5, 33, 0, 1]


@pytest.mark.parametrize("E,n_group,k", [(32, 8, 6), (64, 16, 8), (256, 32, 31), (40, 20, 4)])
@pytest.mark.parametrize("top2", [False, True])
def test_fewer_eligible_experts_than_choices(nat, E, n_group, k, top2):
    """One group of E / n_group experts is left; the choices past them re-pick the lowest masked id, 0, with its own weight."""
    T, gs = 5, E // n_group
    logits = torch.randn(T, E, generator=torch.Generator().manual_seed(E)) * 2
    p = torch.softmax(logits.double(), -1)
    want = torch.zeros(T, k, dtype=torch.long)
    for t in range(T):
        score = p[t].view(n_group, gs)
        best = int((score.topk(2, -1).values.sum(-1) if top2 else score.max(-1).values).argmax())
        mine = sorted(range(best * gs, best * gs + gs), key=lambda e: (-float(p[t, e]), e))
        want[t, :gs] = torch.tensor(mine)
    dev = logits.to(DEV)
    ids, wts = torch.empty(T, k, dtype=torch.int32, device=DEV), torch.empty(T, k, device=DEV)
    nat._ck(nat.load().jib_moe_gate(None, None, None, None, dev.data_ptr(), ids.data_ptr(), wts.data_ptr(), T, 8, E, k, n_group, 1, 1.0, 0, 0, 0, int(top2), 0,
                                    nat._stream()), "moe_gate")
    assert torch.equal(ids.long().cpu(), want)
    assert bool(((wts.double().cpu() - p.gather(1, want)).abs() <= 1e-6 * p.gather(1, want)).all())
    both, rows = torch.empty_like(ids), torch.empty_like(wts)
    seg, src, dest = (torch.empty(n, dtype=torch.int32, device=DEV) for n in (2 * E + 1, T * k, T * k))
    nat._ck(nat.load().jib_moe_gate_sort(None, None, None, None, dev.data_ptr(), both.data_ptr(), rows.data_ptr(), T, 8, E, k, n_group, 1, 1.0, 0, 0, 0,
                                         int(top2), 0, 0, E, seg.data_ptr(), src.data_ptr(), dest.data_ptr(), None, nat._stream()), "moe_gate_sort")
    assert torch.equal(both, ids) and torch.equal(rows, wts)
    check_sort(ids, 0, E, seg[:E + 1], src, dest.view(T, k))


@pytest.mark.parametrize("T,k,E,base", [(77, 8, 66, 0), (128, 8, 66, 0), (129, 31, 256, 100), (511, 8, 256, 0), (1, 1, 1, 0)])
def test_sort_by_matching(nat, T, k, E, base):
    ids = torch.randint(0, E + base, (T, k), device=DEV, dtype=torch.int32)
    ids[::3] = ids[0, 0].clone()                                              # long runs of one expert
    wts = torch.rand(T, k, device=DEV)
    rows = torch.full((T * k,), -7.0, device=DEV)
    seg, src, dest = nat.moe_permute(ids, base, E, wts, rows)
    order = check_sort(ids, base, E, seg, src, dest)
    assert torch.equal(rows[:len(order)].cpu(), wts.flatten().cpu()[order])
