"""The classifier's forward and backward kernels at the edges of their tiles
(64 samples), of the grid, and on a large odd batch, against the same sums in
64 bits.  Tolerances are the rounding bounds of 32-bit sums: a sum of m terms
in any order is within (m - 1) u of the sum of the terms' magnitudes, u = 2^-24,
with m the longest chain of additions, plus the terms' own relative errors."""
import numpy as np
import pytest

from tracklooper_b200 import lst, t5dnn

pytestmark = pytest.mark.gpu

U = 2.0 ** -24
SIZES = [1, 2, 63, 64, 65, 127, 129, 4097, 37889, 300001]


def weights64(w):
    w = w.astype(np.float64)
    return (w[:t5dnn.B0].reshape(38, 32), w[t5dnn.B0:t5dnn.W2], w[t5dnn.W2:t5dnn.B2].reshape(32, 32),
            w[t5dnn.B2:t5dnn.W4], w[t5dnn.W4:t5dnn.B4], w[t5dnn.B4])


@pytest.mark.parametrize("n", SIZES)
def test_forward(n):
    import torch

    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 38), dtype=np.float32)
    w = t5dnn.random_weights(n)
    w[t5dnn.B0:t5dnn.W2] = rng.standard_normal(32) * 0.1
    w[t5dnn.B4] = 0.3
    lib = lst.library()
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    h1, h2, z = (torch.full(s, 7.0, device="cuda") for s in ((n, 32), (n, 32), (n,)))
    assert lib.lst_t5dnn_forward(wd.data_ptr(), xd.data_ptr(), n, h1.data_ptr(), h2.data_ptr(), z.data_ptr(),
                                 torch.cuda.current_stream().cuda_stream) == 0
    w0, b0, w2, b2, w4, b4 = weights64(w)
    x64 = x.astype(np.float64)
    p1 = x64 @ w0 + b0
    e1 = 39 * U * (np.abs(x64) @ np.abs(w0) + np.abs(b0))
    a1 = np.maximum(p1, 0)
    p2 = a1 @ w2 + b2
    e2 = e1 @ np.abs(w2) + 33 * U * ((a1 + e1) @ np.abs(w2) + np.abs(b2))
    a2 = np.maximum(p2, 0)
    p3 = a2 @ w4 + b4
    e3 = e2 @ np.abs(w4) + 33 * U * ((a2 + e2) @ np.abs(w4) + np.abs(b4))
    for got, want, err in ((h1, a1, e1), (h2, a2, e2), (z, p3, e3)):
        assert (np.abs(got.cpu().numpy() - want) <= 1.01 * err + 1e-30).all()


@pytest.mark.parametrize("n", SIZES)
def test_backward(n):
    import torch

    rng = np.random.default_rng(n + 1)
    x = rng.standard_normal((n, 38), dtype=np.float32)
    h1, h2 = (np.maximum(rng.standard_normal((n, 32), dtype=np.float32), 0) for _ in range(2))
    dz = rng.standard_normal(n, dtype=np.float32)
    w = t5dnn.random_weights(n)
    lib = lst.library()
    dev = [torch.from_numpy(a).cuda() for a in (w, x, h1, h2, dz)]
    grad = torch.full((t5dnn.N_PARAMS,), 7.0, device="cuda")
    scratch = torch.full((int(lib.lst_t5dnn_scratch_floats(n)),), 7.0, device="cuda")
    assert lib.lst_t5dnn_backward(*[t.data_ptr() for t in dev], n, grad.data_ptr(), scratch.data_ptr(),
                                  torch.cuda.current_stream().cuda_stream) == 0
    _, _, w2, _, w4, _ = weights64(w)
    x64, h164, h264, dz64 = (a.astype(np.float64) for a in (x, h1, h2, dz))
    g2 = np.where(h2 > 0, dz64[:, None] * w4, 0)
    d1 = np.where(h1 > 0, g2 @ w2.T, 0)
    m1 = np.where(h1 > 0, np.abs(g2) @ np.abs(w2).T, 0)
    want = np.concatenate([(x64.T @ d1).ravel(), d1.sum(0), (h164.T @ g2).ravel(), g2.sum(0), h264.T @ dz64,
                           [dz64.sum()]])
    size = np.concatenate([(np.abs(x64).T @ m1).ravel(), m1.sum(0), (h164.T @ np.abs(g2)).ravel(), np.abs(g2).sum(0),
                           h264.T @ np.abs(dz64), [np.abs(dz64).sum()]])
    # a block's sum runs over its tiles (64 samples each), the blocks' sums are
    # added 32 apart and folded; a term carries its product's and dh1's rounding
    chain = 64 * (-(-n // 64) // 592 + 1) + 592 // 32 + 1 + 6 + 34 + 2
    assert (np.abs(grad.cpu().numpy() - want) <= 1.01 * chain * U * size + 1e-30).all()


@pytest.mark.parametrize("n", [1, 65, 70001])
def test_forward_sums_in_order(n):
    """Unfused 32-bit sums in the order of the inputs, the bias last: every gate as in the plain loop."""
    import torch

    rng = np.random.default_rng(n + 2)
    x = rng.standard_normal((n, 38), dtype=np.float32)
    w = t5dnn.random_weights(n).astype(np.float32)
    w[t5dnn.B0:t5dnn.W2] = rng.standard_normal(32) * 0.1

    def layer(a, m, b):
        acc = np.zeros((n, m.shape[1]), np.float32)
        for k in range(m.shape[0]):
            acc = acc + a[:, k:k + 1] * m[k]
        return acc + b

    a1 = np.maximum(layer(x, w[:t5dnn.B0].reshape(38, 32), w[t5dnn.B0:t5dnn.W2]), np.float32(0))
    a2 = np.maximum(layer(a1, w[t5dnn.W2:t5dnn.B2].reshape(32, 32), w[t5dnn.B2:t5dnn.W4]), np.float32(0))
    z = layer(a2, w[t5dnn.W4:t5dnn.B4].reshape(32, 1), w[t5dnn.B4])[:, 0]
    lib = lst.library()
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    got = [torch.empty(s, device="cuda") for s in ((n, 32), (n, 32), (n,))]
    assert lib.lst_t5dnn_forward(wd.data_ptr(), xd.data_ptr(), n, got[0].data_ptr(), got[1].data_ptr(),
                                 got[2].data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    for a, b in zip(got, (a1, a2, z)):
        assert np.array_equal(a.cpu().numpy(), b)
