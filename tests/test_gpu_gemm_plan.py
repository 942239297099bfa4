"""Products of more than 32 tokens take the tile width and split count of a cost model: every kind of choice against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def bounded(y, ref, x, w, K):
    """Rounding of the result (bf16: half of 2^-8; twice that, for the activation's own rounding) plus fp32 sums of K products."""
    eps = 2.0 ** -8 if y.dtype == torch.bfloat16 else 2.0 ** -22
    lim = eps * ref.abs() + K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 1e-30
    assert bool(((y.double() - ref).abs() <= lim).all()), float(((y.double() - ref).abs() / lim).max())


# one token past and below the tile edges; few feature tiles (splits in a cluster), one full wave, several (persistent rounds), a ragged one
@pytest.mark.parametrize("T", [33, 48, 64, 65, 77, 129, 333, 777])
@pytest.mark.parametrize("N,K", [(2048, 2048), (2112, 5120), (200, 5632), (4096, 512), (3648, 2040)])
def test_planned_products(nat, T, N, K):
    g = torch.Generator(device=DEV).manual_seed(T * 31 + N)
    x = torch.randn(T, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    bias = torch.randn(N, generator=g, device=DEV)
    ref = x.double() @ w.double().T
    for _ in range(2):                                   # the second launch finds counters and scratch as the first left them
        bounded(nat.gemm(x, w), ref, x, w, K)
    bounded(nat.gemm(x, w, out_dtype=torch.float32), ref, x, w, K)
    y = nat.gemm(x, w, residual=bias.expand(T, -1), out_dtype=torch.float32)
    bounded(y, ref + bias.double(), x, w, K)
    nat.check_status()


@pytest.mark.parametrize("T", [33, 64, 100, 200, 600])
def test_planned_gated_pairs(nat, T):
    K, N = 2048, 1408
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn(T, K, generator=g, device=DEV).bfloat16()
    wg, wu = ((torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).bfloat16() for _ in range(2))
    a, b = x.double() @ wg.double().T, x.double() @ wu.double().T
    ref = a * torch.sigmoid(a) * b
    # an error of d in either product moves the result by at most 1.1 d |other| (the slope of x sigmoid(x) stays below 1.1)
    d = K * 2.0 ** -24
    lim = 2.0 ** -8 * ref.abs() + 1.1 * d * ((x.double().abs() @ wg.double().abs().T) * b.abs() + (x.double().abs() @ wu.double().abs().T) * (a.abs() + 1))
    assert bool(((nat.gemm(x, wg, wu).double() - ref).abs() <= lim).all())
    nat.check_status()


@pytest.mark.parametrize("T,tile", [(33, 64), (100, 128), (333, 256)])
@pytest.mark.parametrize("N,K", [(2048, 2048), (2112, 5120), (1024, 1024)])
def test_results_of_32_bits_are_those_of_the_covering_tile(nat, T, tile, N, K):
    """Fewer splits mean longer sums in the tensor cores: only results that are rounded to 16 bits take the cost model's choice."""
    g = torch.Generator(device=DEV).manual_seed(T + N)
    x = torch.randn(T, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    y = nat.gemm(x, w, out_dtype=torch.float32)
    assert torch.equal(y, nat.gemm(x, w, out_dtype=torch.float32, bn=tile))
