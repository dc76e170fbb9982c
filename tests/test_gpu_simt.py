"""The CUDA-core contraction at the edges of its tile shapes, copy modes and K ranges, against 64-bit products.

The bound is the a-priori one of a length-K sum of rounded products: |error| <= (K + 4) * 2^-24 * sum|a||b| per output
element, whatever the order of the additions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


# around the 16, 32, 64 and 128 row tiles; K below, at and off the 16-column block; long K with few tiles (cluster of
# CTAs over K); N across a tile
GEMM = [(1, 1, 1), (1, 1191, 39), (15, 17, 16), (16, 128, 4096), (17, 129, 515), (33, 65, 2050), (64, 64, 4100),
        (127, 130, 31), (129, 300, 64), (300, 1000, 20), (2048, 1500, 48), (5, 40, 1030)]


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("shape", GEMM, ids=lambda s: "x".join(map(str, s)))
def test_gemm_operator_edges(handle, shape, ta, tb):
    M, N, K = shape
    rng = np.random.default_rng(M * 7 + N * 3 + K)
    for pad in (0, 1):                  # a padded leading dimension takes the 16-byte copies away
        A = rng.standard_normal((K, M + pad) if ta else (M, K + pad)).astype(np.float32)
        B = rng.standard_normal((N, K + pad) if tb else (K, N + pad)).astype(np.float32)
        Cm = rng.standard_normal((M, N + pad)).astype(np.float32)
        a64 = (A[:, :M].T if ta else A[:, :K]).astype(np.float64)
        b64 = (B[:, :K].T if tb else B[:, :N]).astype(np.float64)
        got = handle.gemm(ta, tb, M, N, K, 0.5, _t(A), A.shape[1], _t(B), B.shape[1], 2.0, _t(Cm), Cm.shape[1]).cpu().numpy()
        want = 0.5 * (a64 @ b64) + 2.0 * Cm[:, :N]
        bound = EPS * ((K + 4) * 0.5 * (np.abs(a64) @ np.abs(b64)) + 4 * np.abs(Cm[:, :N]) + 4 * np.abs(want))
        assert (np.abs(got[:, :N] - want) <= bound).all(), float((np.abs(got[:, :N] - want) / bound).max())
        assert np.array_equal(got[:, N:], Cm[:, N:])


# (B, C, H, W, F, k, stride, pad, layout): row windows, per-channel planes, pixel-major with and without whole quads
CONV = [(2, 3, 23, 19, 33, 5, 2, 2, 0), (3, 1, 9, 9, 8, 3, 1, 1, 0), (2, 7, 13, 11, 70, 3, 1, 1, 0), (2, 6, 13, 11, 20, 3, 2, 0, 1),
        (1, 20, 9, 14, 130, 3, 1, 1, 1), (4, 144, 6, 6, 40, 3, 1, 1, 1), (2, 64, 17, 5, 64, 1, 1, 0, 1), (1, 4, 31, 33, 16, 11, 4, 0, 1)]


@pytest.mark.parametrize("case", CONV, ids=lambda c: "x".join(map(str, c)))
def test_conv_fp32_edges(handle, case):
    """Also: image i of a batch equals image i alone, bit for bit."""
    import torch
    from nebula_b200 import api
    B, C, H, W, F, k, s, p, layout = case
    g = torch.Generator(device="cuda").manual_seed(C * 100 + k)
    x = torch.randn((B, C, H, W), device="cuda", generator=g)
    w = torch.randn((F, C, k, k), device="cuda", generator=g)
    b = torch.randn(F, device="cuda", generator=g)
    handle.set_math("fp32")
    outs = []
    for n in (B, 1):
        plan = api.Conv2d(handle, n, C, H, W, F, k, s, p, False, "linear", layout)
        plan.set_weights(w, b)
        xin = x[B - n:]
        y = plan.forward((xin.permute(0, 2, 3, 1) if layout else xin).contiguous())
        outs.append((y.permute(0, 3, 1, 2) if layout else y).clone())
        handle.synchronize()
        plan.close()
    conv = torch.nn.functional.conv2d
    want = conv(x.double(), w.double(), b.double(), s, p)
    bound = EPS * (C * k * k + 4) * conv(x.double().abs(), w.double().abs(), b.double().abs(), s, p)
    assert bool(((outs[0].double() - want).abs() <= bound).all())
    assert torch.equal(outs[0][B - 1:], outs[1])
