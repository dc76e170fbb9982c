"""Calls at the edges of what the routes accept, against the CPU oracle."""
import numpy as np
import pytest

from tests.util import assert_close

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


# (OH, OW, stride, k): planes one to three pixels thin whose pixel box, grown to whole 8-row groups, would traverse more than
# the 256 elements a TMA box may (85 -> 88 at stride 3, 51 -> 56 at stride 5, 36 -> 40 at stride 7 ...)
@pytest.mark.parametrize("case", [(1, 85, 3, 1), (51, 1, 5, 1), (52, 2, 5, 1), (1, 42, 6, 1), (1, 36, 7, 1), (36, 3, 7, 1), (36, 3, 7, 3)], ids=str)
def test_thin_strided_planes(handle, case):
    from nebula_b200 import api
    from oracle import oracle as O
    OH, OW, s, k = case
    C, F, H, W = 64, 48, (OH - 1) * s + k, (OW - 1) * s + k
    rng = np.random.default_rng(OH * OW)
    x = rng.standard_normal((1, C, H, W), dtype=np.float32)
    w = (rng.standard_normal((F, C, k, k)) * np.sqrt(2.0 / (C * k * k))).astype(np.float32)
    b = (0.1 * rng.standard_normal(F)).astype(np.float32)
    handle.set_math("tf32")
    plan = api.Conv2d(handle, 1, C, H, W, F, k, s, 0, False, "relu", api.LAYOUT_NHWC)
    plan.set_weights(w, b)
    y = plan.forward(_t(x.transpose(0, 2, 3, 1))).cpu().numpy().transpose(0, 3, 1, 2)
    handle.synchronize()
    plan.close()
    assert_close(y, O.conv_forward(x, w, b, k, s, 0, "relu"), "tf32", f"{case}")


@pytest.mark.parametrize("mode", ["tf32", "tf32x3"])
def test_folded_shortcut_of_a_split_layer_to_any_address(handle, mode):
    """Few tiles and a long contraction (cut along K where the output allows), the output 4 bytes off a 16-byte boundary."""
    import ctypes
    import torch
    from nebula_b200 import api
    from oracle import oracle as O
    rng = np.random.default_rng(2)
    x = rng.standard_normal((1, 256, 7, 7), dtype=np.float32)
    w = (rng.standard_normal((96, 256, 3, 3)) * np.sqrt(2.0 / (256 * 9))).astype(np.float32)
    b = (0.1 * rng.standard_normal(96)).astype(np.float32)
    r = rng.standard_normal((1, 96, 7, 7), dtype=np.float32)
    handle.set_math(mode)
    plan = api.Conv2d(handle, 1, 256, 7, 7, 96, 3, 1, 1, False, "linear", api.LAYOUT_NHWC)
    plan.set_weights(w, b)
    xd, rd = _t(x.transpose(0, 2, 3, 1)), _t(r.transpose(0, 2, 3, 1))
    f = api.ConvFusion(rd.data_ptr(), 96, 7, 7, api.ACT["relu"], None)
    outs = []
    for off in (0, 1):
        y = torch.empty(7 * 7 * 96 + 4, device="cuda")[off:off + 7 * 7 * 96]
        handle.check(handle.lib.nb_conv2d_forward_fused(plan.p, xd.data_ptr(), y.data_ptr(), ctypes.byref(f)))
        outs.append(y.cpu().numpy().reshape(7, 7, 96).transpose(2, 0, 1)[None])
    handle.synchronize()
    plan.close()
    ref = np.maximum(O.conv_forward(x, w, b, 3, 1, 1, "linear") + r, 0)
    for y in outs:
        assert_close(y, ref, mode)


@pytest.mark.parametrize("mode", ["tf32", "tf32x3", "fp32"])
@pytest.mark.parametrize("case", [(16, 32, 1024), (5, 32, 1024), (1, 3, 900), (3, 130, 1000)], ids=str)
def test_rnn_wider_than_a_cluster(handle, mode, case):
    """One launch per step: the output gate sees the rows of step 0 and those of the other steps; a prepared plan has the
    scratch of both."""
    import torch
    from nebula_b200 import api
    from oracle import oracle as O
    T, B, H = case
    rng = np.random.default_rng(H)
    blobs = [{"bias": (0.1 * rng.standard_normal(H)).astype(np.float32), "w": (rng.uniform(-1, 1, (H, n)) / np.sqrt(n)).astype(np.float32)}
             for n in (64, H, H)]
    x = rng.standard_normal((T, B, 64), dtype=np.float32)
    handle.set_math(mode)
    plan = api.Rnn(handle, T, B, 64, H, False, "tanh")
    plan.set_weights(np.concatenate([a.ravel() for b in blobs for a in (b["bias"], b["w"])]))
    prepared = plan.prepare()
    y = plan.forward(_t(x))
    assert plan.workspace_size() == prepared
    handle.synchronize()
    plan.close()
    assert_close(y.cpu().numpy(), O.rnn_forward(x, blobs, H, "tanh"), mode, f"rnn {case}", factor=3.0)


# (rows, inputs, outputs, launches): a quarter of the SMs filled or not, half of them from 8192 inputs on
@pytest.mark.parametrize("case", [(600, 2048, 512, 3), (1300, 2048, 512, 2), (130, 8192, 2100, 3), (400, 8192, 3000, 2)], ids=str)
def test_split_connected_by_rows(handle, case):
    from nebula_b200 import api
    from oracle import oracle as O
    B, inp, out, launches = case
    rng = np.random.default_rng(inp)
    x = rng.standard_normal((B, inp), dtype=np.float32)
    w = (rng.standard_normal((out, inp), dtype=np.float32) / np.sqrt(inp)).astype(np.float32)
    b = (0.1 * rng.standard_normal(out)).astype(np.float32)
    handle.set_math("tf32x3")
    plan = api.Connected(handle, B, inp, out, False, "relu")
    plan.set_weights(w, b)
    prepared = plan.prepare()
    n0 = handle.launch_count()
    y = plan.forward(_t(x))
    assert handle.launch_count() - n0 == launches - 1 and plan.workspace_size() == prepared
    handle.synchronize()
    plan.close()
    rows = np.r_[0:40, B - 40:B]
    assert_close(y.cpu().numpy()[rows], O.connected_forward(x[rows], w, b, "relu"), "tf32x3", f"{case}")


# (kind, T, B, hidden, activation, mode, all steps in one launch): batches that go through a cluster in waves
RECURRENT_CASES = [("lstm", 6, 20, 300, "linear", "tf32", True), ("lstm", 6, 512, 300, "linear", "tf32", False), ("lstm", 5, 400, 420, "linear", "tf32x3", False),
                   ("lstm", 6, 300, 100, "linear", "tf32", True), ("lstm", 4, 1024, 416, "tanh", "tf32", False), ("lstm", 3, 900, 300, "linear", "fp32", False),
                   ("lstm", 3, 700, 301, "linear", "tf32", False), ("lstm", 1, 5, 40, "linear", "tf32", False), ("rnn", 6, 32, 256, "tanh", "tf32", True),
                   ("rnn", 5, 300, 800, "tanh", "tf32", False), ("rnn", 4, 260, 800, "relu", "tf32x3", False), ("rnn", 3, 600, 864, "tanh", "fp32", False)]


@pytest.mark.parametrize("case", RECURRENT_CASES, ids=lambda c: "-".join(map(str, c)))
def test_recurrence_of_large_batches(handle, case):
    from nebula_b200 import api
    from nebula_b200.workloads import NetBuilder
    from oracle import oracle as O
    kind, T, B, H, act, mode, one_launch = case
    nb = NetBuilder("r", B, input_size=32, time_steps=T, bias_init="bias_n01")
    getattr(nb, kind)(H, act, bound=1.0 / np.sqrt(H))
    wl = nb.build("normal")
    w, x = wl.make_weights(H), wl.make_input(B)
    handle.set_math(mode)
    plan = (api.Lstm if kind == "lstm" else api.Rnn)(handle, T, B, 32, H, False, act)
    plan.set_weights(w)
    prepared = plan.prepare()
    n0 = handle.launch_count()
    y = plan.forward(_t(x))
    n = handle.launch_count() - n0
    # per step: a launch per step, behind the input side's; an LSTM's single step of linear gates is one cell update
    assert (n <= 5) == (one_launch or T == 1), n
    assert plan.workspace_size() == prepared
    handle.synchronize()
    plan.close()
    assert_close(y.cpu().numpy(), O.forward_network(wl.cfg, w, x)[0], mode, f"{case}", factor=1.0 if act in ("linear", "relu") else 3.0)


@pytest.mark.parametrize("H", [64, 416])
def test_tf32_lstm_of_any_batch_equals_its_slices(handle, H):
    """Widths that are multiples of 32: TF32 products in one kernel up to 128 rows, launched per step beyond, bit for bit alike."""
    import torch
    from nebula_b200 import api
    T, B = 4, 200
    g = torch.Generator(device="cuda").manual_seed(1)
    w = torch.randn(8 * (H + H * H), device="cuda", generator=g) / H ** 0.5
    x = torch.randn(T, B, H, device="cuda", generator=g)
    handle.set_math("tf32")
    outs = []
    for lo, hi in ((0, 200), (0, 100), (100, 129), (129, 200)):
        plan = api.Lstm(handle, T, hi - lo, H, H, False, "linear")
        plan.set_weights(w)
        outs.append(plan.forward(x[:, lo:hi].contiguous()))
        handle.synchronize()
        plan.close()
    assert torch.equal(outs[0], torch.cat(outs[1:], 1))


# around the products that _gemm_ runs in 16 x 16 tiles: the last and the first K of either kernel, many tiles, one element
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("shape", [(70, 90, 32), (70, 90, 33), (33, 17, 128), (33, 17, 129), (70, 90, 256), (70, 90, 257), (800, 810, 32), (530, 900, 33), (1, 1, 3)], ids=str)
def test_small_products(handle, shape, ta, tb):
    """Bound: (K + 4) * 2^-24 * sum|a||b| per element, whatever the order of the additions."""
    M, N, K = shape
    rng = np.random.default_rng(K)
    A = rng.standard_normal((K, M + 1) if ta else (M, K)).astype(np.float32)
    B = rng.standard_normal((N, K) if tb else (K, N + 1)).astype(np.float32)
    Cm = rng.standard_normal((M, N + 1)).astype(np.float32)
    a64 = (A[:, :M].T if ta else A).astype(np.float64)
    b64 = (B.T if tb else B[:, :N]).astype(np.float64)
    got = handle.gemm(ta, tb, M, N, K, -0.5, _t(A), A.shape[1], _t(B), B.shape[1], 1.5, _t(Cm), N + 1).cpu().numpy()
    want = -0.5 * (a64 @ b64) + 1.5 * Cm[:, :N]
    bound = 2.0 ** -24 * ((K + 4) * 0.5 * (np.abs(a64) @ np.abs(b64)) + 4 * np.abs(Cm[:, :N]) + 4 * np.abs(want))
    assert (np.abs(got[:, :N] - want) <= bound).all()
    assert np.array_equal(got[:, N:], Cm[:, N:])


@pytest.mark.parametrize("which", ["out", "cell", "x"])
@pytest.mark.parametrize("H", [64, 40])
def test_lstm_to_any_address(handle, H, which):
    """A caller's tensors 4 bytes off a 16-byte boundary: the same results as on one (x: on the CUDA cores, so only close)."""
    import torch
    from nebula_b200 import api
    T, B = 3, 5
    g = torch.Generator(device="cuda").manual_seed(H)
    handle.set_math("tf32")
    plan = api.Lstm(handle, T, B, H, H, False, "linear")
    plan.set_weights(torch.randn(8 * (H + H * H), device="cuda", generator=g) / H ** 0.5)
    x = torch.randn(T * B * H, device="cuda", generator=g)
    def run(off):
        t = {k: torch.zeros(T * B * H + 4, device="cuda")[off.get(k, 0):][:T * B * H] for k in ("x", "out", "cell")}
        t["x"].copy_(x)
        handle.check(handle.lib.nb_lstm_forward(plan.p, t["x"].data_ptr(), t["out"].data_ptr(), t["cell"].data_ptr()))
        handle.synchronize()
        return t["out"].clone(), t["cell"].clone()
    want, got = run({}), run({which: 1})
    plan.close()
    for a, b in zip(want, got):
        assert torch.equal(a, b) if which != "x" else float((a - b).abs().max()) <= 1e-3 * float(a.abs().max())


# (images, of them alone, C, H, F, k): a convolution cut along K for the few images and not, or otherwise, for the many
@pytest.mark.parametrize("mode", ["tf32", "tf32x3"])
@pytest.mark.parametrize("case", [(64, 1, 256, 7, 96, 3), (40, 4, 512, 7, 512, 3), (30, 2, 1024, 7, 64, 1), (9, 3, 128, 14, 256, 3)], ids=str)
def test_few_images_of_a_batch(handle, mode, case):
    """Small batches are cut along K where large ones are not, so an image alone and in its batch add in different orders.  Both
    are sums of the same products: they differ by at most the truncations of their accumulations, 2^-23 of sum|a||b| for each of
    the K / 8 steps and the slices on either side (3xTF32: promoted every 12 steps, and the rounding of two operands' low terms)."""
    from nebula_b200 import api
    B, n, C, H, F, k = case
    rng = np.random.default_rng(C)
    x = rng.standard_normal((B, H, H, C), dtype=np.float32)
    w = (rng.standard_normal((F, C, k, k)) * np.sqrt(2.0 / (C * k * k))).astype(np.float32)
    handle.set_math(mode)
    ys = []
    for images in (x, x[B - n:]):
        plan = api.Conv2d(handle, len(images), C, H, H, F, k, 1, k // 2, False, "linear", api.LAYOUT_NHWC)
        plan.set_weights(w, np.zeros(F, np.float32))
        ys.append(plan.forward(_t(images)).cpu().numpy().astype(np.float64)[-n:])
        handle.synchronize()
        plan.close()
    xp = np.pad(np.abs(x[B - n:]).astype(np.float64), ((0, 0), (k // 2,) * 2, (k // 2,) * 2, (0, 0)))
    size = sum(xp[:, i:i + H, j:j + H] @ np.abs(w[:, :, i, j]).T.astype(np.float64) for i in range(k) for j in range(k))
    steps = 2 * (C * k * k / 8 + 16) if mode == "tf32" else 2 * (12 + C * k * k / 96 + 16) + 4
    assert (np.abs(ys[0] - ys[1]) <= steps * 2.0 ** -23 * size).all()


def test_small_products_in_the_order_of_large_ones(handle):
    """The first rows of a product that runs in 16 x 16 tiles and of one of more rows that does not, bit for bit."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(0)
    for K in (40, 100):
        a, b = torch.randn(2048, K, device="cuda", generator=g), torch.randn(1000, K, device="cuda", generator=g)
        outs = []
        for M in (64, 2048):
            c = torch.empty(M, 1000, device="cuda")
            handle.gemm(False, True, M, 1000, K, 1.0, a, K, b, K, 0.0, c, 1000)
            outs.append(c[:64])
        assert torch.equal(*outs)
