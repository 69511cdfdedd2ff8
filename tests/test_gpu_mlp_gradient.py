"""The network's gradient at the edges of its tiles and slices (csrc/bte_mlp.cuh:
16 rows per warp, 64 per column slice, 256 per weight slice), against the oracle."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# The oracle rounds to BF16 where the kernels do and sums in FP64.  An FP32 sum that falls on
# the other side of a rounding moves a value by one BF16 step, 2^-8 of it, in each of the six
# roundings between the input and the first layer's gradient.
STEP = 2.0 ** -8


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 63, 64, 65, 255, 256, 257, 513, 3000])
def test_gradient_at_slice_edges(sbte, rows):
    from oracle import mlp
    from staticbtesolver_gb300 import learned
    L, _ = sbte._load()
    rng = np.random.default_rng(rows)
    X = rng.normal(0, 1, (rows, 8)).astype(np.float32)
    Y = (X[:, 0] * 2.0 - X[:, 1] + 3.0).astype(np.float32)
    p = learned.init_params(7)
    p[mlp.OFF_B1:mlp.OFF_W2] = 0.05
    p[mlp.OFF_B2:mlp.OFF_W3] = -0.03
    p[mlp.OFF_B3:mlp.OFF_W4] = 0.02
    g = np.full(mlp.NPARAM, np.nan, np.float32)
    loss = C.c_double(0)
    ptr = lambda v: v.ctypes.data_as(C.c_void_p)
    assert L.bte_mlp_gradient(ptr(X), ptr(Y), rows, ptr(p), ptr(g), C.byref(loss)) == 0
    lo, go = mlp.loss_grad(p, X, Y)
    yo, _ = mlp.forward(p, X)
    dev = 3 * STEP * np.abs(yo).max()
    assert abs(loss.value - lo) <= dev * np.abs(yo - Y).mean() + dev ** 2
    cuts = [mlp.OFF_W1, mlp.OFF_B1, mlp.OFF_W2, mlp.OFF_B2, mlp.OFF_W3, mlp.OFF_B3, mlp.OFF_W4, mlp.OFF_B4, mlp.NPARAM]
    for a, b in zip(cuts[:-1], cuts[1:]):
        assert np.linalg.norm(g[a:b] - go[a:b]) <= 6 * STEP * np.linalg.norm(go[a:b]), (a, b)
