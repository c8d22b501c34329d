"""The rule that gives a GEMM its tile width, K split and stages
(csrc/gemm_shape.h), on the host alone."""
import numpy as np
import pytest

# CTAs that 148 SMs hold at once at one a SM, clusters losing what a processing
# cluster of SMs leaves over; widths 64, 128, 256 x splits 1, 2, 4, 8
CTAS = np.array([[148, 148, 144, 128]] * 3)
SHAPES = [(128, 256, 5248), (128, 1024, 5248), (128, 5248, 1024), (512, 5248, 1024),
          (4096, 1024, 5248), (2176, 1408, 704), (128, 128, 64), (65536, 128, 1024)]


def test_training_products_never_split(xamg):
    for M, N, K in SHAPES:
        assert xamg.gemm_shape(M, N, K, False, 148, CTAS)[1] == 1


@pytest.mark.parametrize("M,N,K", [(512, 5248, 5248), (4096, 640, 5248), (4096, 5248, 5248),
                                   (1280, 5248, 2560), (1280, 5248, 1024)])
def test_more_tiles_than_sms_take_two_ctas_an_sm(xamg, M, N, K):
    """One CTA an SM would take these sizes in twice the waves, at the same time a
    k-block."""
    assert xamg.gemm_shape(M, N, K, True, 148, CTAS) == (128, 1, 3)
