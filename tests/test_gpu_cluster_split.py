"""Contractions whose K is cut over a cluster, at the edges: boxes of few and ragged rows, columns off the tile width, a last
slice that is shorter, shares that leave CTAs without rows, NCHW and NHWC rows, the shortcut and the pool folded in.  NCHW
layers on their own, networks for what only they fold, against the CPU oracle."""
import numpy as np
import pytest

from tests.util import assert_close, logit_err, NET_TOL

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


# (B, C, H, W, F, k, stride, pad)
CONVS = [(1, 512, 7, 7, 512, 3, 1, 1), (1, 256, 1, 1, 64, 1, 1, 0), (2, 132, 9, 7, 36, 3, 1, 1), (3, 96, 13, 5, 68, 5, 2, 2),
         (1, 128, 28, 28, 128, 3, 1, 1), (5, 2048, 3, 3, 60, 1, 1, 0), (7, 64, 11, 11, 260, 3, 2, 0), (40, 256, 2, 2, 132, 2, 1, 0)]


@pytest.mark.parametrize("mode", ["tf32", "tf32x3"])
@pytest.mark.parametrize("case", CONVS, ids=lambda c: "x".join(map(str, c)))
def test_nchw_convolution(handle, mode, case):
    from nebula_b200 import api
    from oracle import oracle as O
    B, C, H, W, F, k, s, p = case
    rng = np.random.default_rng(C + F)
    x = rng.standard_normal((B, C, H, W), dtype=np.float32)
    w = (rng.standard_normal((F, C, k, k)) * np.sqrt(2.0 / (C * k * k))).astype(np.float32)
    b = (0.1 * rng.standard_normal(F)).astype(np.float32)
    bn = ((rng.random(F) + 0.5).astype(np.float32), (0.1 * rng.standard_normal(F)).astype(np.float32), (rng.random(F) + 0.5).astype(np.float32))
    handle.set_math(mode)
    plan = api.Conv2d(handle, B, C, H, W, F, k, s, p, True, "leaky")
    plan.set_weights(w, b, bn)
    xd = _t(x)
    y = plan.forward(xd)
    again = plan.forward(xd)            # (queued behind it)
    handle.synchronize()
    plan.close()
    assert_close(y.cpu().numpy(), O.conv_forward(x, w, b, k, s, p, "leaky", bn), mode, f"{case}")
    assert (y == again).all()


@pytest.mark.parametrize("mode", ["tf32", "tf32x3"])
@pytest.mark.parametrize("batch", [1, 3])
@pytest.mark.parametrize("size", [20, 14])
def test_network_of_small_layers(handle, mode, batch, size):
    """Pool and shortcut folded in, connected layers of several depths behind."""
    import torch
    from nebula_b200 import api
    from nebula_b200.workloads import NetBuilder
    from oracle import oracle as O
    b = NetBuilder("n", batch, channels=64, height=size, width=size, bias_init="bias_n01")
    b.conv(128, 3, 1, 1, "relu", bn=True)
    b.conv(128, 3, 1, 1, "relu")
    b.maxpool(2, 2, 0)
    b.conv(256, 1, 1, 0, "leaky")
    b.conv(256, 3, 1, 1, "linear", bn=True)
    b.shortcut(2, "relu")
    b.connected(300, "tanh")
    b.connected(100, "logistic")
    b.connected(12, "linear")
    wl = b.build("normal")
    w, x = wl.make_weights(3), wl.make_input(4)
    ref = O.forward_network(wl.cfg, w, x, keep_all=True)
    handle.set_math(mode)
    net = api.Network(handle, wl.cfg)
    net.load_weights(w)
    net.forward(torch.from_numpy(x).cuda())
    handle.synchronize()
    got = net.logits()
    net.close()
    # TF32: six layers of 2^-12 per operand, few samples: the limit of the suite's small networks (tests/util.py)
    assert logit_err(got, ref[-1], batch) <= (2.6e-3 if mode == "tf32" else NET_TOL[mode])


@pytest.mark.parametrize("mode", ["tf32", "tf32x3"])
@pytest.mark.parametrize("rows,inputs,outputs", [(32, 500, 30), (1, 1000, 1), (5, 516, 62), (130, 2052, 67), (33, 4096, 5), (64, 300, 129)])
def test_connected_with_ragged_outputs(handle, mode, rows, inputs, outputs):
    import torch
    from nebula_b200 import api
    g = torch.Generator(device="cuda").manual_seed(inputs + outputs)
    w, bias = torch.randn(outputs, inputs, device="cuda", generator=g) * inputs ** -0.5, torch.randn(outputs, device="cuda", generator=g)
    x = torch.randn(rows, inputs, device="cuda", generator=g)
    handle.set_math(mode)
    plan = api.Connected(handle, rows, inputs, outputs, False, "logistic")
    plan.set_weights(w, bias)
    y = torch.full((rows * outputs + 64,), 7.0, device="cuda")
    handle.check(handle.lib.nb_fc_forward(plan.p, x.data_ptr(), y.data_ptr()))
    handle.synchronize()
    plan.close()
    z = x.double() @ w.double().T + bias.double()
    # TF32 rounds each operand by 2^-11 at most; 3xTF32 drops products of 2^-22 and adds in fp32, as TF32 does; the logistic's
    # slope is 1/4 at most and its own rounding a few ulp
    unit = 2.0 ** -10 if mode == "tf32" else 2.0 ** -21
    bound = 0.25 * ((unit + inputs * 2.0 ** -24) * (x.double().abs() @ w.double().abs().T) + 2.0 ** -23 * z.abs()) + 2.0 ** -22
    assert bool(((y[:rows * outputs].view(rows, outputs).double() - torch.sigmoid(z)).abs() <= bound).all())
    assert bool((y[rows * outputs:] == 7.0).all())


@pytest.mark.parametrize("rows,K,N", [(32, 30, 62), (3, 30, 62), (20, 7, 5), (8, 64, 64)])
def test_few_cuda_core_ctas_behind_a_tensor_core_layer(handle, rows, K, N):
    """Launched ahead of the layer in front, the product must still read what that layer wrote."""
    import torch
    from nebula_b200 import api
    g = torch.Generator(device="cuda").manual_seed(K)
    handle.set_math("tf32")
    front = api.Connected(handle, rows, 4096, K, False, "linear")
    front.set_weights(torch.randn(K, 4096, device="cuda", generator=g), torch.zeros(K, device="cuda"))
    w = torch.randn(N, K, device="cuda", generator=g)
    xs = [torch.randn(rows, 4096, device="cuda", generator=g) for _ in range(5)]
    mid, out = torch.empty(rows, K, device="cuda"), torch.empty(5, rows, N, device="cuda")
    torch.cuda.synchronize()
    for i, x in enumerate(xs):
        handle.check(handle.lib.nb_fc_forward(front.p, x.data_ptr(), mid.data_ptr()))
        handle.gemm(False, True, rows, N, K, 1.0, mid, K, w, K, 0.0, out[i], N)
    handle.synchronize()
    for i, x in enumerate(xs):
        m = front.forward(x)
        handle.synchronize()
        z = torch.empty(rows, N, device="cuda")
        handle.gemm(False, True, rows, N, K, 1.0, m.reshape(rows, K), K, w, K, 0.0, z, N)
        handle.synchronize()
        assert torch.equal(z, out[i])
    front.close()


@pytest.mark.parametrize("C,F,size", [(128, 64, 5), (192, 128, 7), (256, 64, 7), (384, 96, 5), (512, 512, 7), (768, 64, 9)])
def test_short_slices_keep_the_cross_terms_apart(handle, C, F, size):
    """3xTF32 on positive operands, where the tensor core's truncation of the running sum shows as a shrink: a part of at most three
    K blocks adds twelve products to a chain that grows linearly and loses at most an ulp (2^-23) at each: 12 / 2 ulp.  With the
    cross terms in the same chain a slice of two or three blocks has 24 or 36 (384 channels: 8.3e-7, 2.1e-7 with them apart)."""
    import torch
    from nebula_b200 import api
    g = torch.Generator(device="cuda").manual_seed(C)
    w, x = torch.rand(F, C, 1, 1, device="cuda", generator=g), torch.rand(1, C, size, size, device="cuda", generator=g)
    handle.set_math("tf32x3")
    plan = api.Conv2d(handle, 1, C, size, size, F, 1, 1, 0, False, "linear")
    plan.set_weights(w, torch.zeros(F, device="cuda"))
    y = plan.forward(x)
    handle.synchronize()
    plan.close()
    want = torch.einsum("fc,chw->fhw", w.double().reshape(F, C), x.double()[0])
    shrink = ((y.double().reshape(want.shape) - want) / want).mean().item()
    assert abs(shrink) <= 6 * 2.0 ** -23
