"""Decode attention over grouped heads: key splits without a tile, partial tiles and batches with and without a dry round, against float64."""
import types

import pytest
import torch

from jittorinfer_b200.ops import reference as ref
from jittorinfer_b200.ops.specs import Gqa

pytestmark = pytest.mark.gpu
DEV = "cuda"


def mixer(H, G, window=0):
    return types.SimpleNamespace(heads=H, kv_heads=G, dim=128, vdim=128, rot=128, window=window, chunk=0, sink=False, scale=0.09, softcap=0.0, eps=1e-6,
                                 out_scale=1.0, sink_w=None, neighbours=False, unit=False, gate_each=False, pool=0)


# more CTAs per row than tiles of 64 keys (the table is wide), one key, tile edges; 300 sequences: past the batches that take a dry round
@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("H,G", [(16, 4), (8, 8), (48, 2)])
@pytest.mark.parametrize("lens", [[1], [64, 65, 1], [63, 200, 513, 128], [0, 9], [5 + i % 90 for i in range(300)]])
def test_decode(nat, H, G, window, lens):
    B, D = len(lens), 128
    width = 16
    gen = torch.Generator(device=DEV).manual_seed(B + H)
    nb = [(n + 63) // 64 for n in lens]
    cache = torch.randn((sum(nb) + 1) * 64, 2 * G * D, generator=gen, device=DEV).bfloat16()
    bt = torch.zeros(B, width, dtype=torch.int32)
    at = 1
    for i, n in enumerate(nb):
        bt[i, :n] = torch.arange(at, at + n)
        at += n
    q = torch.randn(B, H, D, generator=gen, device=DEV).bfloat16()
    out = torch.full((B, H * D), 7.0, device=DEV).bfloat16()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)      # noqa: E731
    m = mixer(H, G, window)
    for _ in range(2):
        nat.gqa_attention(m, q, cache, None, bt.to(DEV), i32(lens), i32(list(range(B + 1))), 64, 1, None, out)
    for i in [*range(min(B, 4)), B - 1]:
        n = lens[i]
        if n == 0:
            assert not bool(out[i].any())
            continue
        lo = max(0, n - window) if window else 0
        rows = cache[torch.cat([bt[i, j].long() * 64 + torch.arange(64) for j in range(nb[i])])[lo:n].to(DEV)].double()
        k, v = (x.view(n - lo, G, D).repeat_interleave(H // G, 1) for x in rows.split(G * D, 1))
        p = torch.softmax(torch.einsum("hd,nhd->hn", q[i].double(), k) * m.scale, -1)
        want = torch.einsum("hn,nhd->hd", p, v)
        got = out[i].view(H, D).double()
        # probabilities and the result are rounded to bf16 (half of 2^-8 each), sums and exponentials to fp32
        lim = 2.0 ** -8 * torch.einsum("hn,nhd->hd", p, v.abs()) + 2.0 ** -8 * want.abs() + 1e-5
        assert bool(((got - want).abs() <= lim).all()), float(((got - want).abs() / lim).max())


# the loop's branches, each in batches with a dry round (3 sequences) and without one (300)
@pytest.mark.parametrize("n", [3, 300])
@pytest.mark.parametrize("option", [dict(chunk=96), dict(softcap=2.5), dict(sink=True), dict(sink=True, softcap=2.5, window=70), dict(gate=1), dict(gate=2, chunk=64),
                                    dict(window=70, pool=16), dict(window=33, pool=7, sink=True, gate=2)])
def test_options(nat, option, n):
    H, G, D = 8, 2, 128
    option = dict(option)
    gate = option.pop("gate", 0)
    gen = torch.Generator(device=DEV).manual_seed(n)
    m = Gqa(H, G, D, D, D, 0.09, gate_each=gate == 2, **option)
    if m.sink:
        m.sink_w = torch.randn(H, generator=gen, device=DEV)
    lens = [(200, 1, 97)[i] if i < 3 else 5 + i % 190 for i in range(n)]
    nb = [(s + 63) // 64 for s in lens]
    bt = torch.zeros(n, 6, dtype=torch.int32)
    at = 1
    for i, k in enumerate(nb):
        bt[i, :k] = torch.arange(at, at + k)
        at += k
    bt = bt.to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)      # noqa: E731
    rows = lambda k: torch.randn(k, m.kv_row, generator=gen, device=DEV).bfloat16()      # noqa: E731
    cache, pool = rows(at * 64), rows(at * m.pool_rows(64)) if m.pool else None
    q = torch.randn(n, H, D, generator=gen, device=DEV).bfloat16()
    g = torch.randn(n, H * (D if gate == 2 else 1), generator=gen, device=DEV).bfloat16() if gate else None
    out, want, size = (torch.zeros(n, H * D, dtype=t, device=DEV) for t in (torch.bfloat16, torch.float32, torch.float32))
    args = (bt, i32(lens), i32(list(range(n + 1))), 64, 1, None)
    for _ in range(2):
        nat.gqa_attention(m, q, cache, g, *args, out, pool)
    ref.gqa_attention(m, q, cache, g, *args, want, pool)
    # |v| in the values' place bounds the sums that the rounded probabilities go into
    both = [t.float() for t in (cache, pool) if t is not None]
    for t in both:
        t[:, G * D:] = t[:, G * D:].abs()
    ref.gqa_attention(m, q, both[0], g, *args, size, both[1] if m.pool else None)
    # probabilities and the result are rounded to bf16 (half of 2^-8 each); gates and the softcap's tanh by fast functions (2^-20 of a score)
    lim = 2.0 ** -8 * size + 2.0 ** -8 * want.abs() + 1e-4
    assert bool(((out.float() - want).abs() <= lim).all()), float(((out.float() - want).abs() / lim).max())
