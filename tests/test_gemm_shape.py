"""The rule that gives a GEMM its tile width, K split and stages
(csrc/gemm_shape.h), on the host alone."""
import numpy as np
import pytest

# CTAs that 148 SMs hold at once at one a SM, clusters losing what a processing
# cluster of SMs leaves over; widths 64, 128, 256 x splits 1, 2, 4, 8
CTAS = np.array([[148, 148, 144, 128]] * 3)
SHAPES = [(128, 256, 5248), (128, 1024, 5248), (128, 5248, 1024), (512, 5248, 1024),
          (4096, 1024, 5248), (2176, 1408, 704), (128, 128, 64), (65536, 128, 1024)]


def waves(shape, M, N, ctas, sms):
    bn, split, stages = shape
    slots = ctas[{64: 0, 128: 1, 256: 2}[bn], {1: 0, 2: 1, 4: 2, 8: 3}[split]] if split > 1 \
        else sms * (2 if stages == 3 else 1)
    return -(-(M // 128) * (N // bn) * split // slots)


@pytest.mark.parametrize("none", [(), (2,), (8,), (2, 4), (2, 4, 8)])
def test_no_split_the_gpu_cannot_hold(xamg, none):
    """A cluster size of which the GPU holds none is never chosen."""
    ctas = CTAS.copy()
    for s in none:
        ctas[:, {2: 1, 4: 2, 8: 3}[s]] = 0
    splits = set()
    for M, N, K in SHAPES:
        bn, split, stages = xamg.gemm_shape(M, N, K, True, 148, ctas)
        assert N % bn == 0 and split not in none and K // 64 >= (4 * split if split > 1 else 1)
        assert 3 <= stages <= 8 and stages * (128 + bn) * 128 <= 192 * 1024
        assert waves((bn, split, stages), M, N, ctas, 148) >= 1
        splits.add(split)
    assert (max(splits) > 1) == (len(none) < 3)


def test_training_products_never_split(xamg):
    for M, N, K in SHAPES:
        assert xamg.gemm_shape(M, N, K, False, 148, CTAS)[1] == 1


@pytest.mark.parametrize("M,N,K", [(512, 5248, 5248), (4096, 640, 5248), (4096, 5248, 5248),
                                   (1280, 5248, 2560), (1280, 5248, 1024)])
def test_more_tiles_than_sms_take_two_ctas_an_sm(xamg, M, N, K):
    """One CTA an SM would take these sizes in twice the waves, at the same time a
    k-block."""
    assert xamg.gemm_shape(M, N, K, True, 148, CTAS) == (128, 1, 3)
