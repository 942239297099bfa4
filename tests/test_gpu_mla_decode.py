"""Latent attention of decode steps: tile edges and table widths (they bound the splits) against the reference."""
import pytest
import torch

from jittorinfer_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, seed, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).bfloat16()


def tables(lens, spare=2, width=None):
    """Shuffled blocks of 64 rows; the cache rows that no sequence owns hold large values."""
    nb = [(n + 63) // 64 for n in lens]
    perm = torch.randperm(sum(nb) + spare, generator=torch.Generator().manual_seed(3))
    bt = torch.zeros(len(lens), width or max(max(nb), 1), dtype=torch.int32)
    at = 0
    for i, n in enumerate(nb):
        bt[i, :n] = perm[at:at + n].int()
        at += n
    return bt.to(DEV), (sum(nb) + spare) * 64


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def close(a, b):
    """bf16 probabilities and results: 2^-8 of a row's size, four times over."""
    assert float((a.float() - b.float()).norm() / b.float().norm()) < 0.012
    assert float((a.float() - b.float()).abs().max()) < 0.05 * float(b.float().abs().max())


# one row, around the 16-row steps of the value product, a block of 64 and a tile of 128; table rows of exactly the needed width (fewest
# splits) and much wider ones (most splits); a window that ends inside a step, a block and a tile; more CTAs than SMs: past those with a dry pass
@pytest.mark.parametrize("H", [16, 24, 128])
@pytest.mark.parametrize("width", [None, 40])
@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("lens", [[1], [15, 16, 17], [63, 64, 65], [127, 128, 129, 193], [0, 40], [2000], [1 + i * 7 % 200 for i in range(160)]])
def test_decode(nat, H, width, window, lens):
    bt, rows = tables(lens, width=width)
    cache, q = rnd(rows, 576, seed=1), rnd(len(lens), H, 576, seed=2, scale=0.3)
    qs = i32(list(range(len(lens) + 1)))
    for _ in range(2):
        o = nat.mla_attention(q, cache, bt, i32(lens), qs, 0.11, 512, 64, 1, None, window)
    want = ref.mla_attention(q, cache, bt, i32(lens), qs, 0.11, 512, 64, window)
    close(o[[i for i, n in enumerate(lens) if n]], want[[i for i, n in enumerate(lens) if n]])
    assert all(not bool(o[i].any()) for i, n in enumerate(lens) if n == 0)


def test_rows_past_the_end_are_not_used(nat):
    """A block's rows behind a sequence's last 16-row step may hold anything."""
    bt, rows = tables([70], width=4)
    cache, q = rnd(rows, 576, seed=4), rnd(1, 16, 576, seed=5, scale=0.3)
    want = nat.mla_attention(q, cache, bt, i32([70]), i32([0, 1]), 0.11, 512, 64, 1).clone()
    cache.view(-1, 64, 576)[int(bt[0, 1]), 16:] = float("nan")
    assert torch.equal(nat.mla_attention(q, cache, bt, i32([70]), i32([0, 1]), 0.11, 512, 64, 1), want)
