"""CPU: which kernels a prompt pass takes, by its sizes (the rules are functions of sizes and addresses alone)."""
import ctypes as C

import pytest


@pytest.fixture(scope="module")
def conv_takes(ops):
    f = C.CDLL(ops.LIB_PATH)["_ZN4b20018gemm_la_conv_takesEPKvS1_xi"]
    f.restype, f.argtypes = C.c_bool, [C.c_void_p, C.c_void_p, C.c_longlong, C.c_int]
    return f


@pytest.mark.parametrize("rows,seqs,fused", [
    (1, 1, True), (253, 1, True), (2, 2, False), (371, 2, False), (372, 2, True), (999, 3, True), (65536, 64, True),
    (64, 64, False), (128, 8, False), (480, 8, False), (800, 8, True), (2560, 128, False), (3072, 128, True), (8192, 128, True),
    (3000, 1024, False), (4096, 256, False), (8192, 256, True), (8192, 512, False), (16384, 1024, False), (1 << 31, 1024, True),
])
def test_fused_deltanet_projection_where_it_is_the_faster_one(conv_takes, rows, seqs, fused):
    assert conv_takes(16, 32, rows, seqs) == fused


def test_fused_deltanet_projection_wants_whole_vectors(conv_takes):
    assert not conv_takes(8, 32, 4096, 1) and not conv_takes(16, 34, 4096, 1)


@pytest.mark.parametrize("kind,rows,ff,width,pair", [
    (0, 128, 3584, 1024, False), (0, 129, 3584, 1024, True), (1, 129, 64, 1024, True), (1, 4096, 5632, 2048, True), (1, 4096, 11008, 4096, False),
    (1, 256, 8, 2304, False), (1, 256, 12, 1024, False), (1, 256, 64, 1028, False), (2, 256, 64, 1024, False),
])
def test_paired_feed_forward_where_it_is_the_faster_one(ops, kind, rows, ff, width, pair):
    """kind: fp16, bf16, fp32."""
    f = C.CDLL(ops.LIB_PATH)["_ZN4b20014gemm_glu_takesENS_8ElemTypeEPKvS2_S2_iii"]
    f.restype, f.argtypes = C.c_bool, [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_int]
    assert f(kind, 16, 32, 48, rows, ff, width) == pair
