"""The learned-guess MLP on the GPU (forward and backward on the tcgen05 GEMM)
against its CPU restatement (oracle/mlp_oracle.py): the same BF16 rounding
points, FP32 instead of float64 accumulation. Gradients must agree to 1 % of
each block's largest entry; a few steps of Adam must reduce the loss of a
learnable map tenfold."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "oracle"))
import mlp_oracle as MO  # noqa: E402

pytestmark = pytest.mark.gpu


def blocks(g, n_in, h, n_out):
    sizes = [h * n_in, h, h * h, h, n_out * h, n_out]
    out, off = [], 0
    for s in sizes:
        out.append(g[off:off + s])
        off += s
    return out


@pytest.mark.parametrize("n_in,h,n_out,B", [(256, 128, 128, 128), (128, 256, 384, 256)])
def test_gradients_against_oracle(gpu, n_in, h, n_out, B):
    import torch
    m = gpu.Mlp(n_in, h, n_out, seed=3)
    p = m.params()
    rng = np.random.default_rng(4)
    X = rng.standard_normal((B, n_in)).astype(np.float32)
    T = rng.standard_normal((B, n_out)).astype(np.float32)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    Yd = torch.empty(B, n_out, dtype=torch.float32, device="cuda")
    m.predict(Xd.data_ptr(), Yd.data_ptr(), B)
    g, loss = m.gradients(Xd.data_ptr(), Td.data_ptr(), B)
    _, _, _, Yr = MO.forward(p.astype(np.float64), X.astype(np.float64), n_in, h, n_out)
    gr, lr_ = MO.gradients(p.astype(np.float64), X.astype(np.float64), T.astype(np.float64),
                           n_in, h, n_out)
    Y = Yd.cpu().numpy()
    assert np.abs(Y - Yr).max() <= 1e-2 * np.abs(Yr).max()
    assert abs(loss - lr_) <= 1e-3 * lr_
    for gb, rb in zip(blocks(g, n_in, h, n_out), blocks(gr, n_in, h, n_out)):
        assert np.abs(gb - rb).max() <= 1e-2 * np.abs(rb).max() + 1e-12


@pytest.mark.parametrize("n_in,h,n_out,B,widths",
                         [(640, 384, 1152, 384, {64}), (256, 1024, 128, 640, {64}),
                          (1408, 1280, 2176, 1280, {128})])
def test_gradients_of_several_tiles(gpu, n_in, h, n_out, B, widths):
    """Several tiles in every product, transposed operands included, in tiles of 64
    columns and of 128 (one CTA an SM and two); training products never split K.
    With B x h activations a pre-activation within the FP32 accumulation's error
    of zero can fall on the other side of the ReLU than in the oracle: that
    moves one sample's share of one row of a weight gradient, about
    1 / sqrt(B h) of the block's norm (0.3 % here), so blocks are compared in
    the 2-norm, 1 % allowing some ten of them."""
    import torch
    shapes = [gpu.gemm_shape(*mnk, False, transposed=True)
              for mnk in ((n_out, h, B), (h, h, B), (h, n_in, B))]
    assert {s[0] for s in shapes} == widths and {s[1] for s in shapes} == {1}
    assert widths == {64} or {s[2] for s in shapes} == {3, 6}
    m = gpu.Mlp(n_in, h, n_out, seed=3)
    p = m.params()
    rng = np.random.default_rng(4)
    X = rng.standard_normal((B, n_in)).astype(np.float32)
    T = rng.standard_normal((B, n_out)).astype(np.float32)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    g, loss = m.gradients(Xd.data_ptr(), Td.data_ptr(), B)
    gr, lr_ = MO.gradients(p.astype(np.float64), X.astype(np.float64), T.astype(np.float64),
                           n_in, h, n_out)
    assert abs(loss - lr_) <= 1e-3 * lr_
    for gb, rb in zip(blocks(g, n_in, h, n_out), blocks(gr, n_in, h, n_out)):
        assert np.linalg.norm(gb - rb) <= 1e-2 * np.linalg.norm(rb)


def test_targets_off_a_16_byte_boundary(gpu):
    """The loss gradient reads the targets in the last layer's epilogue: the
    same loss and gradients for targets that start 4 bytes further."""
    import torch
    n_in, h, n_out, B = 256, 128, 256, 128
    rng = np.random.default_rng(8)
    X = torch.from_numpy(rng.standard_normal((B, n_in)).astype(np.float32)).cuda()
    T = torch.from_numpy(rng.standard_normal(B * n_out).astype(np.float32)).cuda()
    T1 = torch.empty(B * n_out + 1, dtype=torch.float32, device="cuda")
    T1[1:] = T
    torch.cuda.synchronize()
    m = gpu.Mlp(n_in, h, n_out, seed=2)
    g0, l0 = m.gradients(X.data_ptr(), T.data_ptr(), B)
    g1, l1 = m.gradients(X.data_ptr(), T1.data_ptr() + 4, B)
    assert l0 == l1 and g0.tobytes() == g1.tobytes()


def test_training_reduces_the_loss(gpu):
    import torch
    n_in, h, n_out, B = 128, 256, 128, 512
    rng = np.random.default_rng(5)
    M = rng.standard_normal((n_in, n_out)) / np.sqrt(n_in)
    X = rng.standard_normal((B, n_in)).astype(np.float32)
    T = (X @ M).astype(np.float32)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    m = gpu.Mlp(n_in, h, n_out, seed=6)
    first = m.train_step(Xd.data_ptr(), Td.data_ptr(), B, 1e-3)
    for _ in range(300):
        last = m.train_step(Xd.data_ptr(), Td.data_ptr(), B, 1e-3)
    assert last < first / 10, (first, last)


def test_a_batch_that_does_not_fit_leaves_the_network_usable(gpu):
    """A batch whose activations exceed the device's memory (274 GB for the inputs
    alone) is refused every time it is asked for, not only the first, and the
    network then works as before."""
    import torch
    n_in, h, n_out, B = 128, 128, 128, 128
    X = torch.randn(B, n_in, device="cuda")
    T = torch.randn(B, n_out, device="cuda")
    Y = torch.empty(B, n_out, device="cuda")
    torch.cuda.synchronize()
    m = gpu.Mlp(n_in, h, n_out, seed=1)
    g0, l0 = m.gradients(X.data_ptr(), T.data_ptr(), B)
    for _ in range(2):
        with pytest.raises(gpu.XamgError) as e:
            m.predict(X.data_ptr(), Y.data_ptr(), 1 << 30)
        assert e.value.code == -9
    g1, l1 = m.gradients(X.data_ptr(), T.data_ptr(), B)
    assert l0 == l1 and g0.tobytes() == g1.tobytes()
