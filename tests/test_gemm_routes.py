"""Which kernel takes a quantised layer, by its sizes (csrc/gemm_w4.cu, csrc/gemm_w4_dec.cu).  The rules are host code and need no
GPU."""
import pytest

from zse_b200.ops import native

F16, SWIGLU, PLANES, ROPE = 0, 1, 2, 3
SMALL, WIDE, NARROW, PAIR = -1, 0, 1, 2


@pytest.mark.parametrize("M", [1, 2, 5, 8])
@pytest.mark.parametrize("N,K,epilogue,small", [
    (3584, 14336, F16, False), (1024, 8192, F16, False), (2048, 16384, F16, False),       # narrow and deep: a cluster along K
    (3584, 4096, F16, True), (2048, 2048, F16, True), (5120, 13824, F16, True), (8192, 28672, F16, True),
    (3584, 14336, PLANES, True), (37888, 3584, SWIGLU, True), (2 * 448, 8192, SWIGLU, False)])
def test_up_to_8_tokens(M, N, K, epilogue, small):
    tiles, splits, cluster, kind = native.gemm_w4_plan(M, N, K, epilogue)
    assert (kind == SMALL) == small
    if not small:
        assert cluster > 1 and cluster == splits
    assert native.gemm_w4_plan(9, N, K, epilogue)[3] == NARROW or native.gemm_w4_plan(9, N, K, epilogue)[3] == WIDE


@pytest.mark.parametrize("M", [1, 8])
@pytest.mark.parametrize("N,K,epilogue,small", [
    (4608, 3584, ROPE, True), (7168, 5120, ROPE, True), (896, 5120, ROPE, True), (1280, 8192, ROPE, False),
    (3584, 18944, F16, False), (3584, 14336, F16, True), (1024, 8192, F16, False), (37888, 3584, SWIGLU, True),
    (3584, 14336, PLANES, True), (3584, 3584, 4, False)])
def test_up_to_8_tokens_of_the_decode_entry(M, N, K, epilogue, small):
    assert native.gemm_w4_dec_small(M, N, K, epilogue) == small
    assert not native.gemm_w4_dec_small(9, N, K, epilogue)


@pytest.mark.parametrize("M,N,K,epilogue,kind", [
    (65, 37888, 3584, SWIGLU, PAIR), (96, 4608, 3584, F16, PAIR), (128, 3584, 14336, F16, WIDE), (320, 3584, 14336, F16, PAIR),
    (65, 3584, 18944, PLANES, PAIR), (2048, 27648, 5120, SWIGLU, PAIR), (65, 256, 128, F16, WIDE), (64, 37888, 3584, SWIGLU, NARROW)])
def test_more_than_64_tokens(M, N, K, epilogue, kind):
    assert native.gemm_w4_plan(M, N, K, epilogue)[3] == kind


@pytest.mark.parametrize("M,N,epilogue", [(96, 4608, F16), (512, 2048, F16), (512, 4096, SWIGLU), (2048, 27648, SWIGLU)])
def test_a_cluster_that_was_asked_for(M, N, epilogue):
    """k_split on an epilogue that needs the whole sum is a cluster along K, which the paired kernel does not have."""
    for ks in (2, 4):
        assert native.gemm_w4_plan(M, N, 5120, epilogue, ks)[1:] == (ks, ks, WIDE)
    assert native.gemm_w4_plan(M, N, 5120, epilogue, 1)[3] == PAIR
    assert native.gemm_w4_plan(M, N, 5120, PLANES, 2)[1::2] == (2, PAIR)
