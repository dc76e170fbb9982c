"""logistic, loggy and tanh against the reference's double formulas: each value is that formula's, rounded to fp32, but for the
rounding of its last double operations, which moves a result by one ulp now and then."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ref(x, act):
    z = x.astype(np.float64)
    with np.errstate(all="ignore"):
        if act == "tanh":
            e = np.exp(2.0 * z)
            return ((e - 1.0) / (e + 1.0)).astype(np.float32)
        e = np.exp(-z)
        return (1.0 / (1.0 + e) if act == "logistic" else 2.0 / (1.0 + e) - 1.0).astype(np.float32)


@pytest.mark.parametrize("act", ["logistic", "loggy", "tanh"])
@pytest.mark.parametrize("n", [3, 4, 1 << 20])          # one by one, and four at a time
def test_double_activations(handle, act, n):
    import torch
    rng = np.random.default_rng(n)
    x = np.concatenate([rng.standard_normal(n // 2) * 3, rng.uniform(-1000, 1000, n - n // 2 - n // 4),
                        np.exp(rng.uniform(-60, 0, n // 4)) * rng.choice([-1, 1], n // 4)]).astype(np.float32)
    edges = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 354.0, 354.8914, 354.89136, 354.9, -354.9, 709.0, 709.9, -709.9, 3e38, -3e38,
                      1e-45, -1e-38, 88.0, -88.0, -103.9, -104.5], np.float32)
    if n > 4:
        x[:len(edges)] = edges
    got = handle.activation(torch.from_numpy(x).cuda(), act).cpu().numpy()
    want = _ref(x, act)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    # near zero the formulas subtract numbers next to 1: what is left of either side is exact to some 2^-52 in all
    diff = np.abs(got[ok].astype(np.float64) - want[ok])
    ulp = np.spacing(np.abs(want[ok])).astype(np.float64)
    assert (diff <= np.maximum(ulp, 2.0 ** -50)).all()
    assert ((diff > 0) & (np.abs(want[ok]) > 1e-6)).mean() <= 1e-5
