"""Products of at most eight rows on the CUDA cores: rows around the kernel's 1, 2, 4 and 8, columns around its 64, K around its
blocks of 64 and in several ranges, against 64-bit products; and the rows of a larger product bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


@pytest.mark.parametrize("N,K", [(1, 132), (63, 300), (65, 516), (1000, 4096), (128, 9216), (250, 1028), (64, 260)])
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8])
def test_few_rows(handle, M, N, K):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    a, b = torch.randn(9, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g)
    c = torch.randn(M, N + 3, device="cuda", generator=g)
    got = c.clone()
    handle.gemm(False, True, M, N, K, 0.5, a, K, b, K, 2.0, got, N + 3)
    a64, b64, c64 = a[:M].double(), b.double(), c[:, :N].double()
    want = 0.5 * (a64 @ b64.T) + 2.0 * c64
    bound = EPS * ((K + 4) * 0.5 * (a64.abs() @ b64.abs().T) + 4 * c64.abs() + 4 * want.abs())
    assert bool(((got[:, :N].double() - want).abs() <= bound).all())
    assert torch.equal(got[:, N:], c[:, N:])


@pytest.mark.parametrize("K,N", [(4096, 1000), (520, 200), (36, 64)])
def test_connected_rows_alone_and_in_a_batch(handle, K, N):
    import torch
    from nebula_b200 import api
    g = torch.Generator(device="cuda").manual_seed(K)
    w, bias, x = torch.randn(N, K, device="cuda", generator=g), torch.randn(N, device="cuda", generator=g), torch.randn(20, K, device="cuda", generator=g)
    handle.set_math("fp32")
    outs = []
    for m in (20, 8, 3, 1):
        plan = api.Connected(handle, m, K, N, False, "leaky")
        plan.set_weights(w, bias)
        outs.append(plan.forward(x[:m].contiguous()))
        handle.synchronize()
        plan.close()
    for y in outs[1:]:
        assert torch.equal(y.reshape(-1, N), outs[0].reshape(-1, N)[:y.numel() // N])
