"""Which kernel and which tiles a product gets (host code of the CUDA library, no GPU): both sides of every line, as measured."""
import ctypes as C
import os

import pytest

from jittorinfer_b200 import build
from jittorinfer_b200.ops import native

pytestmark = pytest.mark.skipif(not os.path.exists(build.KERNELS_SO), reason="the CUDA library is not built")
RULES, PLANNED, NARROW = 0, 1, 2


def form(T, N, K, heads=1, gated=False, **more):
    lib = native.load()
    lib.jib_gemm_form.restype, lib.jib_gemm_form.argtypes = C.c_int, [C.POINTER(native.GemmDesc), C.POINTER(C.c_int), C.POINTER(C.c_int)]
    d = native.GemmDesc()
    d.x = d.w = d.out = d.scratch = 4096
    if gated:
        d.w2 = 4096
    d.T, d.N, d.K, d.batch, d.x_row_stride, d.w_row_stride, d.ldo = T, N, K, heads, K * heads, K, N * heads
    d.x_batch_stride, d.w_batch_stride, d.out_batch_stride = K, N * K, N
    for k, v in more.items():
        setattr(d, k, v)
    bn, splits = C.c_int(), C.c_int()
    return lib.jib_gemm_form(C.byref(d), bn, splits), bn.value, splits.value


@pytest.mark.parametrize("N,K,heads,gated,narrow", [
    (8192, 256, 1, False, True), (12288, 256, 1, False, False), (512, 128, 32, False, True), (128, 512, 16, False, True), (128, 512, 128, False, False),
    (8192, 512, 1, False, True), (10240, 512, 1, False, False), (4096, 1024, 1, False, True), (6144, 1024, 1, False, False),
    (40960, 128, 1, False, True), (32768, 128, 1, False, False), (512, 128, 128, False, True), (49152, 256, 1, False, False), (2048, 2048, 1, False, False),
    (3072, 2048, 1, True, True), (4096, 2048, 1, True, True), (10752, 1024, 1, True, False), (7680, 1024, 1, True, True), (2048, 2080, 1, True, False),
    (5632, 2048, 1, True, True), (7168, 2048, 1, True, True), (7168, 1536, 1, True, True), (9216, 1024, 1, True, True), (7840, 1536, 1, True, False),
    (8192, 2048, 1, True, False)])
def test_up_to_8_tokens(N, K, heads, gated, narrow):
    for T in (1, 8):
        assert form(T, N, K, heads, gated)[0] == (NARROW if narrow else RULES)
    assert form(9, N, K, heads, gated)[0] == RULES
    assert form(8, N, K, heads, gated, bn=16)[0] == form(8, N, K, heads, gated, splits=2)[0] == RULES


def test_operands_that_16_byte_reads_do_not_fit():
    for more in ({"x": 4104}, {"w": 4104}, {"x_row_stride": 260}, {"w_row_stride": 260}, {"seg": 4096}):
        assert form(4, 1024, 256, **more)[0] == RULES, more
    assert form(4, 1024, 264)[0] == RULES and form(4, 1024, 256)[0] == NARROW


def test_weights_that_l2_does_not_hold_are_read_once():
    """CTAs run through the features before they come to the next token tile."""
    for N, K, gated in ((24576, 5120, False), (10944, 5120, True), (12288, 5120, True), (24576, 2560, False)):
        for T in (33, 64, 77, 128):
            f, bn, splits = form(T, N, K, 1, gated)
            assert f == PLANNED and bn >= T and splits == 1, (N, K, T, bn)
    # others fill the SMs with small tiles
    for T, N, K, gated, bn in ((64, 2048, 2048, False, 16), (777, 2048, 2048, False, 128), (48, 1408, 2048, True, 16)):
        assert form(T, N, K, 1, gated)[:2] == (PLANNED, bn)


def test_what_is_not_planned():
    assert form(33, 2048, 2048)[0] == PLANNED and form(32, 2048, 2048)[0] == RULES
    for more in ({"out_f32": 1}, {"splits": 2}, {"bn": 64}, {"seg": 4096}, {"ag_flags": 4096}):
        assert form(100, 2048, 2048, **more)[0] == RULES, more
    assert form(100, 2048, 2048, 2)[0] == RULES
    assert form(100, 128 * 2 * 148, 512)[0] == PLANNED and form(100, 128 * 2 * 148 + 1, 512)[0] == RULES
