"""The CUDA-core contraction launched ahead of the kernel in front: a few CTAs with short ranges of K read what a tensor-core layer
writes just before, queued without a wait between them; longer ranges and more CTAs, which are launched in order, too."""
import pytest

pytestmark = pytest.mark.gpu

# rows, K (beyond the small-product kernel's), columns: tiles with whole quads and without, the kernel of few rows; ahead, and in order
PRODUCTS = [(32, 132, 62), (20, 131, 5), (3, 260, 62), (8, 132, 64), (1, 400, 200), (64, 512, 30), (65, 256, 30), (65, 260, 30), (300, 264, 100), (8, 2000, 64)]


def _queued(handle, rows, K, call, N):
    """A layer of K outputs, then `call(mid, out)` on what it wrote: five pairs queued, each against the pair with a wait behind each call."""
    import torch
    from nebula_b200 import api
    g = torch.Generator(device="cuda").manual_seed(K)
    front = api.Connected(handle, rows, 4096, K, False, "linear")
    front.set_weights(torch.randn(K, 4096, device="cuda", generator=g), torch.zeros(K, device="cuda"))
    xs = [torch.randn(rows, 4096, device="cuda", generator=g) for _ in range(5)]
    mid, out, want = torch.empty(rows, K, device="cuda"), torch.empty(5, rows, N, device="cuda"), torch.empty(5, rows, N, device="cuda")
    for dst, wait in ((want, True), (out, False)):
        torch.cuda.synchronize()
        for i, x in enumerate(xs):
            handle.check(handle.lib.nb_fc_forward(front.p, x.data_ptr(), mid.data_ptr()))
            if wait:
                handle.synchronize()
            call(mid, dst[i])
            if wait:
                handle.synchronize()
        handle.synchronize()
    front.close()
    assert bool(want.abs().amax() > 0) and torch.equal(out, want)


@pytest.mark.parametrize("rows,K,N", PRODUCTS)
def test_product_behind_a_layer(handle, rows, K, N):
    import torch
    w = torch.randn(N, K, device="cuda")
    handle.set_math("tf32")
    _queued(handle, rows, K, lambda mid, y: handle.gemm(False, True, rows, N, K, 1.0, mid, K, w, K, 0.0, y, N), N)


@pytest.mark.parametrize("rows,inputs,N", [(8, 28, 62), (3, 30, 62), (40, 30, 7), (700, 20, 200)])
def test_connected_layer_behind_a_layer(handle, rows, inputs, N):
    """(fewer inputs than the tensor cores take)"""
    import torch
    from nebula_b200 import api
    handle.set_math("tf32")
    back = api.Connected(handle, rows, inputs, N, False, "relu")
    back.set_weights(torch.randn(N, inputs, device="cuda"), torch.randn(N, device="cuda"))
    _queued(handle, rows, inputs, lambda mid, y: handle.check(handle.lib.nb_fc_forward(back.p, mid.data_ptr(), y.data_ptr())), N)
    back.close()
