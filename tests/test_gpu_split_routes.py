"""TF32 connected layers below 512 and from 2048 inputs on, at any number of rows: clusters, slabs or whole tiles add the same slices of K in the same order, so a
batch and its slices give the same bits; and convolutions of the caller's NCHW tensors whose K is cut into slabs, not over clusters.
Against 64-bit products."""
import pytest

pytestmark = pytest.mark.gpu

# inputs, outputs, activation: clusters at few rows, off the 32-wide K blocks and the tile widths; rows that need slabs and whole tiles
LAYERS = [(500, 30, "logistic"), (300, 62, "relu"), (480, 1000, "tanh"), (352, 500, "leaky"), (508, 2280, "relu"), (5916, 408, "leaky"),
          (4844, 1264, "logistic"), (12456, 16, "linear"), (2468, 130, "tanh"), (42568, 28, "linear"), (2052, 67, "logistic")]
ROWS = [1, 5, 127, 128, 129, 300, 610, 1100, 2500]


@pytest.mark.parametrize("layer", LAYERS, ids=lambda c: "x".join(map(str, c)))
def test_rows_do_not_change_a_row(handle, layer):
    import torch
    from nebula_b200 import api
    inputs, outputs, act = layer
    g = torch.Generator(device="cuda").manual_seed(inputs)
    w, b = torch.randn(outputs, inputs, device="cuda", generator=g) * inputs ** -0.5, torch.randn(outputs, device="cuda", generator=g)
    x = torch.randn(max(ROWS), inputs, device="cuda", generator=g)
    handle.set_math("tf32")
    got = []
    for rows in ROWS:
        plan = api.Connected(handle, rows, inputs, outputs, False, act)
        plan.set_weights(w, b)
        prepared = plan.prepare()
        got.append(plan.forward(x[:rows]))
        handle.synchronize()
        assert plan.workspace_size() == prepared
        plan.close()
    got = [y.reshape(-1, outputs) for y in got]
    for rows, y in zip(ROWS, got):
        assert torch.equal(y, got[-1][:rows]), f"{rows} rows"
    z = x[:300].double() @ w.double().T
    f = {"linear": lambda v: v, "relu": lambda v: v.clamp(min=0), "leaky": lambda v: torch.where(v > 0, v, 0.1 * v), "tanh": torch.tanh,
         "logistic": torch.sigmoid}[act]
    # TF32 rounds each operand by 2^-11 at most, and sums round in fp32; no activation here is steeper than 1
    bound = (2.0 ** -10 + inputs * 2.0 ** -24) * (x[:300].double().abs() @ w.double().abs().T) + 2.0 ** -22 * (z + b).abs() + 2.0 ** -22
    assert bool(((got[5].double() - f(z + b.double())).abs() <= bound).all())


# (mode, B, C, H, W, F, k, stride, pad, launches): long K on a third of the SMs' tiles and more: a layout pass, the product, the addition of
# its slabs, a layout pass; shorter, or on fewer tiles: clusters, which write NCHW
@pytest.mark.parametrize("case", [("tf32x3", 5, 176, 34, 34, 32, 7, 1, 3, 4), ("tf32", 7, 384, 65, 19, 44, 7, 1, 0, 4), ("tf32x3", 1, 96, 20, 20, 64, 3, 1, 1, 2)],
                         ids=lambda c: "x".join(map(str, c)))
def test_slabs_or_clusters(handle, case):
    import torch
    from nebula_b200 import api
    mode, B, C, H, W, F, k, s, p, launches = case
    g = torch.Generator(device="cuda").manual_seed(C)
    x, w = torch.randn(B, C, H, W, device="cuda", generator=g), torch.randn(F, C, k, k, device="cuda", generator=g)
    b = torch.randn(F, device="cuda", generator=g)
    handle.set_math(mode)
    plan = api.Conv2d(handle, B, C, H, W, F, k, s, p, False, "leaky")
    plan.set_weights(w, b)
    prepared = plan.prepare()
    n0 = handle.launch_count()
    y = plan.forward(x)
    assert handle.launch_count() - n0 == launches and plan.workspace_size() == prepared
    again = plan.forward(x)
    handle.synchronize()
    plan.close()

    def conv(x, w):
        return torch.cat([torch.matmul(w.double().reshape(F, -1), torch.nn.functional.unfold(i[None].double(), k, padding=p, stride=s)) for i in x]).reshape(y.shape)
    z, size = conv(x, w) + b.double().reshape(1, -1, 1, 1), conv(x.abs(), w.abs()) + b.double().abs().reshape(1, -1, 1, 1)
    # TF32 rounds each operand by 2^-11 at most; 3xTF32 drops products of 2^-22; sums round in fp32
    unit = (2.0 ** -10 if mode == "tf32" else 2.0 ** -21) + C * k * k * 2.0 ** -24
    assert torch.equal(y, again) and bool(((y.double() - torch.where(z > 0, z, 0.1 * z)).abs() <= unit * size).all())
