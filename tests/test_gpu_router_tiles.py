"""Router logits of more than 16 tokens come from tiles that split the model width: tile edges and remainders against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 16: the other kernel; one past a tile of 16 tokens, several tiles, more tiles than CTA slots; experts below, at and past a tile of 64;
# widths of less than one chunk of 64, a ragged one, one run of many chunks
@pytest.mark.parametrize("T", [1, 16, 17, 33, 77, 2049])
@pytest.mark.parametrize("E,d,shared_gate", [(64, 2048, False), (7, 40, False), (160, 5120, False), (65, 1000, False), (32, 1536, True)])
def test_logits(nat, T, E, d, shared_gate):
    gen = torch.Generator(device=DEV).manual_seed(T * 131 + E)
    x = torch.randn(T, d, generator=gen, device=DEV).bfloat16()
    w = torch.randn(E + shared_gate, d, generator=gen, device=DEV) * d ** -0.5
    logits = torch.full((T + 1, E + shared_gate), 7.0, device=DEV)
    ids = torch.empty(T, 5, dtype=torch.int32, device=DEV)
    wts = torch.empty(T, 5, device=DEV)
    nat._ck(nat.load().jib_moe_gate(x.data_ptr(), w.data_ptr(), None, None, logits.data_ptr(), ids.data_ptr(), wts.data_ptr(), T, d, E, 4, 1, 1,
                                    1.0, 0, 0, 1, 0, int(shared_gate), nat._stream()), "moe_gate")
    ref = x.double() @ w.double().T
    # fp32 sums of d products: at most d roundings of half a unit each
    lim = d * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 1e-30
    assert bool(((logits[:T].double() - ref).abs() <= lim).all())
    assert bool((logits[T] == 7.0).all())                # nothing past the last token
    assert bool((ids[:, 4] == E).all())                  # the shared expert rides along
    # the chosen experts are the largest of the logits that the kernel wrote (no ties among random values)
    want = logits[:T, :E].topk(4, -1).indices
    assert torch.equal(ids[:, :4].long(), want)


def logits_of(nat, x, w):
    T, d = x.shape
    E = w.shape[0]
    logits, ids, wts = torch.empty(T, E, device=DEV), torch.empty(T, 2, dtype=torch.int32, device=DEV), torch.empty(T, 2, device=DEV)
    nat._ck(nat.load().jib_moe_gate(x.data_ptr(), w.data_ptr(), None, None, logits.data_ptr(), ids.data_ptr(), wts.data_ptr(), T, d, E, 2, 1, 1, 1.0,
                                    0, 0, 0, 0, 0, nat._stream()), "moe_gate")
    return logits


# spans of 256 elements: one, a part of one, fewer than 8, each number of CTAs of a cluster; turns of 2048: one, a part of the second, all four
@pytest.mark.parametrize("T", [17, 40, 333, 2500])
@pytest.mark.parametrize("E,d", [(64, 2048), (7, 8), (65, 264), (130, 776), (160, 5120), (64, 1544), (32, 2056), (66, 8192)])
def test_a_token_has_the_same_logits_in_any_batch(nat, T, E, d):
    gen = torch.Generator(device=DEV).manual_seed(T + d)
    x = torch.randn(T, d, generator=gen, device=DEV).bfloat16()
    w = torch.randn(E, d, generator=gen, device=DEV) * d ** -0.5
    w[2, d // 2] = float("inf")
    some = torch.cat([logits_of(nat, x[t:t + 16].contiguous(), w) for t in range(0, T, 16)])
    assert bool((x[:, d // 2] != 0).all()) and bool(torch.isinf(some[:, 2]).all())
    assert torch.equal(logits_of(nat, x, w), some)


def test_rows_past_the_last_expert_are_not_read(nat):
    """An infinity in a neighbouring allocation's row must not reach the sums: 65 experts of a matrix of 66 rows, the last one infinite."""
    gen = torch.Generator(device=DEV).manual_seed(5)
    x = torch.randn(40, 64, generator=gen, device=DEV).bfloat16()
    w = torch.randn(66, 64, generator=gen, device=DEV)
    w[65] = float("inf")
    ids, wts = nat.moe_gate(x, w[:65], None, 4, 1, 1, 1.0, False, False)
    assert bool(torch.isfinite(wts).all())
