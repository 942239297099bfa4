"""Grouped expert products of 17 to 80 tokens in tiles of 16 rows: grid and list form, foreign experts and skewed routing against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 16 and 81: the other paths; one row past tiles of 16; an expert with every token (five tiles) beside experts with none; the last sizes: the list
@pytest.mark.parametrize("T,E,k,F,d,base", [(16, 20, 6, 192, 256, 0), (17, 20, 6, 192, 256, 0), (23, 20, 6, 192, 256, 0), (24, 20, 6, 192, 256, 0), (33, 66, 8, 136, 200, 0), (80, 66, 8, 192, 256, 0),
                                            (81, 66, 8, 192, 256, 0), (64, 24, 6, 192, 256, 40), (80, 160, 6, 1024, 3072, 0), (24, 256, 6, 128, 128, 0)])
@pytest.mark.parametrize("gated", [True, False])
def test_against_float64(nat, T, E, k, F, d, base, gated):
    gen = torch.Generator(device=DEV).manual_seed(T + E)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=gen, device=DEV) * scale).bfloat16()      # noqa: E731
    wg, wu, wd = rnd(E, F, d, scale=d ** -0.5), rnd(E, F, d, scale=d ** -0.5), rnd(E, d, F, scale=F ** -0.5)
    x = rnd(T, d)
    # the first column always the same expert, the others at random; with a base some belong to other ranks
    ids = torch.stack([torch.randperm(E + 2 * base - 1, generator=gen, device=DEV)[:k] for _ in range(T)]).int()
    ids[:, 0] = E + 2 * base - 1 if base == 0 else base + 3
    if base:
        ids[:, 1:] = torch.where(ids[:, 1:] == base + 3, torch.full_like(ids[:, 1:], 0), ids[:, 1:])
    wts = torch.rand(T, k, generator=gen, device=DEV)
    y, dest = nat.moe_routed(x, ids, wts, wg if gated else None, wu, wd, base)
    for t in [*range(0, T, 7), T - 1]:
        for j in range(k):
            e, row = int(ids[t, j]) - base, int(dest[t, j])
            if e < 0 or e >= E:
                assert row == -1
                continue
            xt = x[t].double()
            u = wu[e].double() @ xt
            h = torch.nn.functional.silu(wg[e].double() @ xt) * u if gated else torch.nn.functional.gelu(wts[t, j].double() * u)
            want = wd[e].double() @ h
            # h and the result are rounded to bf16 (2^-9 each), sums to fp32
            lim = 2.0 ** -8 * want.abs() + 2.0 ** -8 * (wd[e].double().abs() @ h.abs()) + 1e-5
            assert bool(((y[row].double() - want).abs() <= lim).all())
