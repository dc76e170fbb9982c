"""NHWC pooling at the edges of what is fetched ahead: windows of one value to a hundred, padding and strides that cut them on every
side, few outputs and many, in the reference's order of additions: bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["max", "avg"])
@pytest.mark.parametrize("case", [(1, 4, 5, 7, 1, 1, 0), (2, 8, 9, 6, 2, 2, 1), (1, 2048, 7, 7, 7, 7, 0), (3, 12, 11, 13, 3, 2, 1), (2, 64, 17, 9, 4, 3, 2),
                                  (1, 16, 20, 23, 5, 1, 4), (5, 36, 12, 12, 6, 5, 3), (2, 20, 16, 16, 10, 3, 0), (40, 96, 30, 30, 3, 1, 1)], ids=str)
def test_windows(handle, mode, case):
    import torch
    from nebula_b200 import api
    from oracle import oracle as O
    B, C, H, W, k, s, p = case
    x = np.random.default_rng(C + k).standard_normal((B, C, H, W), dtype=np.float32)
    y = handle.pool(torch.from_numpy(np.ascontiguousarray(x.transpose(0, 2, 3, 1))).cuda(), k, s, p, mode, layout=api.LAYOUT_NHWC)
    assert np.array_equal(y.cpu().numpy().transpose(0, 3, 1, 2), O.pool_forward(x, k, s, p, mode == "max"))
