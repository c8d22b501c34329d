"""The tcgen05 BF16 GEMM (XAMG_b200_gemm_bf16) against a float64 product of the
same BF16-rounded operands. FP32 accumulation differs from the exact sum by at
most K * 2^-24 * (|A| |B|^T) per element (plus one BF16 rounding of the
output for the BF16 modes); the tests allow twice that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(gpu, M, N, K, mode, seed, bias=True):
    import torch
    g = torch.Generator().manual_seed(seed)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16)
    B = torch.randn(N, K, generator=g).to(torch.bfloat16)
    bv = torch.randn(N, generator=g) if bias else None
    aux = torch.randn(M, N, generator=g).to(torch.bfloat16)
    out_dt = torch.float32 if mode == 0 else torch.bfloat16
    Ad, Bd = A.cuda(), B.cuda()
    Cd = torch.full((M, N), float("nan"), dtype=out_dt, device="cuda")
    bd = bv.cuda() if bias else None
    auxd = aux.cuda()
    gpu.call("XAMG_b200_gemm_bf16", M, N, K, Ad.data_ptr(), Bd.data_ptr(), Cd.data_ptr(), N, mode,
             bd.data_ptr() if bias else None, auxd.data_ptr(), N,
             torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    a = A.double().numpy()
    b = B.double().numpy()
    ref = a @ b.T
    bound = 2.0 * K * 2.0 ** -24 * (np.abs(a) @ np.abs(b).T) + 1e-30
    if bias and mode != 3:
        ref = ref + bv.double().numpy()[None, :]
        bound = bound + 2.0 ** -23 * np.abs(ref)
    if mode == 2:
        ref = np.maximum(ref, 0.0)
    if mode == 3:
        ref = np.where(aux.double().numpy() > 0, ref, 0.0)
    got = Cd.double().cpu().numpy()
    if mode != 0:
        bound = bound + 2.0 ** -8 * np.abs(ref)
    return got, ref, bound


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (256, 384, 640), (384, 256, 1024),
                                   (1024, 1024, 4096)])
def test_gemm_f32_bias(gpu, M, N, K):
    got, ref, bound = run(gpu, M, N, K, 0, seed=M + N + K)
    assert np.all(np.abs(got - ref) <= bound), np.abs(got - ref).max()


@pytest.mark.parametrize("mode", [1, 2, 3])
def test_gemm_bf16_modes(gpu, mode):
    got, ref, bound = run(gpu, 256, 256, 512, mode, seed=mode)
    assert np.all(np.abs(got - ref) <= bound), np.abs(got - ref).max()


def test_gemm_rejects_bad_shapes(gpu):
    import torch
    A = torch.zeros(128, 64, dtype=torch.bfloat16, device="cuda")
    C = torch.zeros(128, 128, dtype=torch.float32, device="cuda")
    rc = gpu.lib().XAMG_b200_gemm_bf16(100, 128, 64, A.data_ptr(), A.data_ptr(), C.data_ptr(),
                                       128, 0, None, None, 0, None)
    assert rc == -2


@pytest.mark.parametrize("M,N,K,mode", [(128, 256, 2368, 0),    # K split over a cluster, unevenly
                                        (128, 1024, 1088, 2), (256, 384, 2048, 3),
                                        (1280, 2048, 64, 1),    # one k-block, 256-wide tiles
                                        (2176, 2304, 704, 0)])  # more tiles than SMs
def test_gemm_tile_shapes(gpu, M, N, K, mode):
    """The tile widths and K splits the launcher chooses between."""
    got, ref, bound = run(gpu, M, N, K, mode, seed=M + K)
    assert np.all(np.abs(got - ref) <= bound), np.abs(got - ref).max()


def test_gemm_unaligned_bias_and_padded_rows(gpu):
    """A bias that starts off a 16-byte boundary and rows of C wider than N."""
    import torch
    M, N, K, ldc = 128, 128, 1024, 136
    g = torch.Generator().manual_seed(9)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16)
    B = torch.randn(N, K, generator=g).to(torch.bfloat16)
    bias = torch.randn(N + 1, generator=g)
    Ad, Bd, bd = A.cuda(), B.cuda(), bias.cuda()
    C = torch.full((M, ldc), 7.0, device="cuda")
    gpu.call("XAMG_b200_gemm_bf16", M, N, K, Ad.data_ptr(), Bd.data_ptr(), C.data_ptr(), ldc, 0,
             bd.data_ptr() + 4, None, 0, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    ref = (A.double() @ B.double().T + bias[1:].double()).numpy()
    bound = 2.0 * K * 2.0 ** -24 * (A.double().abs() @ B.double().abs().T).numpy() \
        + 2.0 ** -23 * np.abs(ref)
    got = C.cpu().double().numpy()
    assert np.all(np.abs(got[:, :N] - ref) <= bound)
    assert np.all(got[:, N:] == 7.0)


@pytest.mark.parametrize("M,N,K,mode,shape", [
    (128, 128, 64, 0, (64, 1, 8)), (512, 1024, 704, 2, (64, 1, 8)),
    (384, 384, 1024, 3, (64, 4, 8)), (128, 256, 2368, 1, (64, 8, 8)),
    (1280, 1024, 704, 0, (128, 1, 6)), (1280, 1024, 704, 3, (128, 1, 6)),
    (1280, 640, 2368, 2, (128, 2, 6)), (256, 1152, 2368, 0, (128, 4, 6)),
    (2176, 1408, 704, 0, (128, 1, 3)), (2176, 2304, 704, 2, (128, 1, 3)),
    (2176, 1408, 704, 3, (128, 1, 3)), (1280, 2304, 1088, 0, (256, 1, 4)),
    (1280, 2304, 1088, 3, (256, 1, 4)), (1280, 1024, 2368, 2, (256, 2, 4))])
def test_gemm_shapes(gpu, M, N, K, mode, shape):
    """Every tile width with and without a K split, one CTA an SM and two, fewer
    tiles than SMs and more, k-blocks that the split does not divide."""
    assert gpu.gemm_shape(M, N, K) == shape
    got, ref, bound = run(gpu, M, N, K, mode, seed=M + K)
    assert np.all(np.abs(got - ref) <= bound), np.abs(got - ref).max()
