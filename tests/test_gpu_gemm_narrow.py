"""Products of up to 8 tokens that one wave of CTAs holds in flight: row tiles, runs of K, heads, functions and residuals against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, seed, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).bfloat16()


def bounded(y, ref, sums, K, more=0.0):
    """Rounding of the result (half of 2^-8 for bf16) plus fp32 sums of K products of total size ``sums``."""
    eps = 2.0 ** -8 if y.dtype == torch.bfloat16 else 2.0 ** -22
    lim = eps * ref.abs() + K * 2.0 ** -24 * sums + more + 1e-30
    assert bool(((y.double() - ref).abs() <= lim).all()), float(((y.double() - ref).abs() / lim).max())


# 9: the other kernel; rows below, at and past a warp's 16 and a CTA's 16 .. 128; one block of 32 along K, uneven shares of it, several rounds
@pytest.mark.parametrize("T", [1, 3, 8, 9])
@pytest.mark.parametrize("N,K", [(1, 32), (15, 64), (130, 96), (1024, 1024), (200, 1024 - 32), (4096, 256), (17, 40)])
def test_single(nat, T, N, K):
    x, w = rnd(T, K + 8, seed=T)[:, 8:], rnd(N, K, seed=N, scale=K ** -0.5)       # rows that start 16 bytes in
    ref, sums = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    bias, res, res32 = torch.randn(N, device=DEV), rnd(T, N, seed=3), torch.randn(T, N, device=DEV)
    bounded(nat.gemm(x, w), ref, sums, K)
    bounded(nat.gemm(x, w, out_dtype=torch.float32), ref, sums, K)
    bounded(nat.gemm(x, w, residual=res), ref + res.double(), sums, K, 2.0 ** -23 * (ref.abs() + res.double().abs()))
    bounded(nat.gemm(x, w, residual=res32, out_dtype=torch.float32), ref + res32.double(), sums, K, 2.0 ** -23 * (ref.abs() + res32.double().abs()))
    bounded(nat.gemm(x, w, residual=bias.expand(T, -1), out_dtype=torch.float32), ref + bias.double(), sums, K, 2.0 ** -23 * (ref.abs() + bias.double().abs()))
    out = torch.full((T + 1, N + 3), 7.0, device=DEV).bfloat16()
    bounded(nat.gemm(x, w, out=out[:T, :N]), ref, sums, K)
    assert bool((out[T] == 7.0).all()) and bool((out[:, N:] == 7.0).all())
    y = nat.gemm(x, w, out_dtype=torch.float32, unary=("relu2",))
    bounded(y, ref.clamp_min(0) ** 2, 2 * ref.abs() * sums + sums ** 2 * K * 2.0 ** -24, K, 2.0 ** -22 * ref ** 2)
    y = nat.gemm(x, w, out_dtype=torch.float32, unary=("cap", 0.5, 3.0))
    bounded(y, 3.0 * torch.tanh(ref * 0.5 / 3.0), sums, K, 3.0 * 2.0 ** -20)
    y = nat.gemm(x, w, out_dtype=torch.float32, unary=("gelu",))
    bounded(y, torch.nn.functional.gelu(ref), 1.2 * sums, K, 3e-7 * (1 + ref.abs()))


@pytest.mark.parametrize("T", [1, 5, 8])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
@pytest.mark.parametrize("N,K", [(16, 32), (130, 2048), (1408, 1536), (40, 2080)])
def test_gated(nat, T, act, N, K):
    x, wg, wu = rnd(T, K, seed=T), rnd(N, K, seed=1, scale=K ** -0.5), rnd(N, K, seed=2, scale=K ** -0.5)
    a, b = x.double() @ wg.double().T, x.double() @ wu.double().T
    f = torch.nn.functional.silu(a) if act == "silu" else torch.nn.functional.gelu(a, approximate="tanh")
    sa, sb = x.double().abs() @ wg.double().abs().T, x.double().abs() @ wu.double().abs().T
    # both functions' slopes stay below 1.2; __expf and the division add a few 2^-22
    bounded(nat.gemm(x, wg, wu, act=act), f * b, 1.2 * sa * b.abs() + sb * f.abs(), K, 2.0 ** -20 * (f * b).abs())


@pytest.mark.parametrize("T", [1, 7])
@pytest.mark.parametrize("B,N,K", [(16, 512, 128), (16, 128, 512), (3, 20, 64), (128, 512, 128)])
def test_heads(nat, T, B, N, K):
    """Strided token rows per head, results into a wider tensor, as the absorbed projections use it."""
    w = rnd(B, N, K, seed=B, scale=K ** -0.5)
    x = rnd(T, B, K + 64, seed=T)[..., :K]
    out = torch.full((T, B, N + 8), 7.0, device=DEV).bfloat16()
    nat.gemm_batched(x.data_ptr(), x.stride(0), x.stride(1), w, out.data_ptr(), out.stride(0), out.stride(1), T, x.device)
    ref = torch.einsum("tbk,bnk->tbn", x.double(), w.double())
    bounded(out[..., :N], ref, torch.einsum("tbk,bnk->tbn", x.double().abs(), w.double().abs()), K)
    assert bool((out[..., N:] == 7.0).all())


def test_rows_past_the_matrix_do_not_count(nat):
    """Infinities next to the matrix and next to the token rows stay out of the sums."""
    w, x = rnd(24, 64, seed=1), rnd(4, 64, seed=2)
    w[20:] = float("inf")
    x[2:] = float("nan")
    y = nat.gemm(x[:2], w[:20])
    assert bool(torch.isfinite(y).all())
