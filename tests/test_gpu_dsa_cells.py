"""The low-order solve (k_dsa_pcg) where a thread has no, one, two or more cells and a cell few or
many faces (the first two cells' operands are loaded ahead for up to four faces), against Jacobi's
iteration to rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize("n,links", [(1, 2), (33, 2), (700, 4), (3000, 2), (30000, 4), (100001, 3), (160000, 2),
                                     (160001, 4)])
def test_cells_per_thread_and_faces(sbte, n, links):
    """Cells coupled to `links` others along a ring (distances 1, 2) with weights of at most 1, and
    one wall of weight 1 each."""
    rng = np.random.default_rng(n)
    c = np.arange(n)
    nb, W = np.full((links + 1, n), -1, np.int32), np.zeros((links + 1, n))
    W[links] = 1.0
    for k in range(links // 2 if n > 4 else 0):
        w = rng.uniform(0.2, 1.0, n)  # of the link c -> c + k + 1
        nb[2 * k], W[2 * k] = (c + k + 1) % n, w
        nb[2 * k + 1], W[2 * k + 1] = (c - k - 1) % n, np.roll(w, k + 1)
    b = rng.uniform(-1, 1, n)
    x = sbte.dsa_solve(nb, W, b, tol=TOL)[0]
    D = W.sum(0)
    exact = np.zeros(n)
    for _ in range(250):  # contracts by links / (links + 1) at least
        exact = (b + sum(W[f] * exact[nb[f]] for f in range(links) if nb[f, 0] >= 0)) / D
    # scaled operator >= 1 / (links + 1): the preconditioned residual bounds the plain one up to
    # sqrt(links + 2), and that the error by links + 1; FP32 vectors: 1e-5 more
    error, size = np.linalg.norm(np.sqrt(D) * (x - exact)), np.linalg.norm(b / np.sqrt(D))
    assert error <= (links + 1) * (np.sqrt(links + 2) * TOL + 1e-5) * size
