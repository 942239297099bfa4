"""A mixed step in two attention forms against the absorbed form for every row."""
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


@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("rot_half,shared", [(False, False), (True, True)])
@pytest.mark.parametrize("qlens,lens", [([1, 1, 150, 70], [900, 300, 150, 200]), ([1, 64], [70, 64]), ([1, 1, 1, 129, 1], [65, 1, 640, 129, 1])])
def test_mixed(nat, qlens, lens, window, rot_half, shared):
    """``shared``: a layer that reads another layer's rows (queries only)."""
    from jittorinfer_b200 import ops
    H, dn, dr, dv, r, T = 16, 128, 64, 128, 512, sum(qlens)
    bt, rows = tables(lens)
    # rows of this step that a window hides from the decoding sequences stay in the cache all the same
    cache, c2 = rnd(rows, 576, seed=6, scale=0.5), None
    c2 = cache.clone()
    qkv = rnd(T, H * (dn + dr) + 576, seed=7, scale=0.5)
    q, ckv = qkv[:, :H * (dn + dr)], None if shared else qkv[:, H * (dn + dr):]
    w_kv_b = rnd(H * (dn + dv), r, seed=8, scale=0.05)
    w = w_kv_b.view(H, dn + dv, r)
    w_uk, w_uv = w[:, :dn].transpose(1, 2).contiguous(), w[:, dn:].contiguous()
    norm_w = torch.rand(r, device=DEV) + 0.5
    rope = ref.yarn_table(1024, dr, 10000.0, 1.0, 0.0, 1.0, 0, dr, device=torch.device(DEV))
    pos = i32([s - n + j for n, s in zip(qlens, lens) for j in range(n)])
    seq = [i for i, n in enumerate(qlens) for _ in range(n)]
    slots = i32([int(bt[i, int(p) // 64]) * 64 + int(p) % 64 for i, p in zip(seq, pos.tolist())])
    qs = i32([0] + torch.tensor(qlens).cumsum(0).tolist())
    meta = {"q_lens": qlens, "s_lens": lens, "total_kv": sum(lens), "n_q_tiles": sum((n + 127) // 128 for n in qlens),
            "kv_decode": sum(s for n, s in zip(qlens, lens) if n <= 1)}
    parts = ops.mla_mixed_split(T, dn, dr, dv, r, 64, meta, window)
    assert parts is not None and parts[0] == next(i for i, n in enumerate(qlens) if n != 1)
    args = (norm_w, 1e-6, rope, pos, slots)
    # the general path: absorbed form for every row
    q_full = torch.empty(T, H, r + dr, dtype=q.dtype, device=DEV)
    q_nope = ops.mla_qkv_post(q, ckv, *args, c2, q_full, H, dn, dr, r, rot_half)
    ops.q_absorb(q_nope, w_uk, q_full, r)
    want = ops.v_up(ops.mla_attention(q_full, c2, bt, i32(lens), qs, 0.07, r, 64, max(qlens), meta, window), w_uv)
    got = ops.mla_mixed(q, ckv, *args, cache, w_uk, w_uv, w_kv_b, bt, i32(lens), qs, 0.07, H, dn, dr, r, 64, parts, window, rot_half)
    assert torch.equal(cache, c2)                         # the same rows written
    close(got, want)
