"""The bracket network's GEMM tiles: every way an operand is read (element by element, 16-byte
pieces along k or along C's side), sizes off the 64 x 64 x 32 tile, and the split weight gradients
at row counts around their blocks."""
import numpy as np
import pytest

from oracle import mlp_oracle

pytestmark = pytest.mark.gpu

# BF16 products are exact in FP32; K terms are summed in FP32, so the error is at most K 2^-24 of
# the sum of the terms' sizes.


@pytest.mark.parametrize("M,N,K", [(64, 64, 32), (1, 2, 4), (65, 68, 36), (63, 260, 400), (7, 5, 3),
                                   (128, 4, 1028)])
@pytest.mark.parametrize("ta,tb,shift", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0), (0, 0, 1)])
def test_gemm_reads(built, M, N, K, ta, tb, shift):
    import torch
    g = torch.Generator().manual_seed(M * 7 + N + K)
    a, b = torch.randn(M, K, generator=g), torch.randn(K, N, generator=g)
    ab, bb = a.bfloat16().double(), b.bfloat16().double()
    want, size = ab @ bb, ab.abs() @ bb.abs()

    def place(x, t):  # (device tensor to keep, pointer, stride of rows, stride of columns)
        y = (x.t() if t else x).contiguous().flatten()
        d = torch.zeros(y.numel() + 4, device="cuda")
        d[shift:shift + y.numel()] = y.cuda()  # shift: a pointer that is not 16-byte aligned
        r, c = (1, x.shape[0]) if t else (x.shape[1], 1)
        return d, d.data_ptr() + 4 * shift, r, c
    da, pa, ar, ac = place(a, ta)
    db, pb, br, bc = place(b, tb)
    c = torch.empty(M, N, device="cuda")
    torch.cuda.synchronize()
    built.gemm_bf16(M, N, K, pa, ar, ac, pb, br, bc, c.data_ptr())
    err = (c.cpu().double() - want).abs()
    assert bool((err <= K * 2.0 ** -24 * size + 1e-30).all())


@pytest.mark.parametrize("B", [1, 63, 64, 65, 2047, 2049])
def test_split_gradients(built, B):
    import torch
    model = built.Model(0, seed=5)
    rng = np.random.default_rng(B)
    X = rng.normal(size=(B, 400)).astype(np.float32)
    X[:, 386:] = 0
    T = rng.normal(size=B).astype(np.float32)
    dX, dT = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    torch.cuda.synchronize()
    g, loss = model.gradients(dX.data_ptr(), dT.data_ptr(), B)
    g2, _ = model.gradients(dX.data_ptr(), dT.data_ptr(), B)
    assert np.array_equal(g, g2)  # partial sums are added in a fixed order
    want_loss, want = mlp_oracle.loss_and_grads(model.get_params(), X, T.astype(np.float64))
    assert abs(loss - want_loss) <= 1e-2 * abs(want_loss)
    o = 0
    for n, k in mlp_oracle.SIZES:  # the tolerance of test_gpu_bracket.py's gradients
        for size in (n * k, n):
            d = g[o:o + size] - want[o:o + size]
            assert np.linalg.norm(d) <= 2e-3 * max(np.linalg.norm(want[o:o + size]), 1e-30)
            o += size
