"""One CSR system by a thread-block cluster (csrc/bte_krylov.cuh) at the edges of its rule: sizes
around full warps, CTAs and clusters, rows of 3, 4, 8 and more entries, repeated entries, rows
without any; against Jacobi's iteration to rounding, as the phase kernels that take the rest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _system(n, entries, seed, repeat=False, hole=False):
    """Diagonal in [1, 2], the other entries of a row together at most half of it: the inverse's
    row sums are at most 2."""
    rng = np.random.default_rng(seed)
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [rng.uniform(1, 2, n)]
    diag = vals[0].copy()
    if repeat:  # the diagonal in two halves
        vals[0] = vals[0] / 2
        rows.append(rows[0]), cols.append(cols[0]), vals.append(vals[0])
    for _ in range(entries - len(rows) if n > 1 else 0):  # (never a second diagonal entry: the last one counts)
        rows.append(np.arange(n))
        cols.append((rows[-1] + rng.integers(1, n, n)) % n)
        vals.append(-diag * rng.uniform(0.2, 0.5, n) / (entries - 1))
    rows, cols, vals = (np.concatenate(v) for v in (rows, cols, vals))
    b = rng.uniform(-1, 1, n)
    if hole:  # an unknown without equation, decoupled
        keep = (rows != n // 2) & (cols != n // 2)
        rows, cols, vals = rows[keep], cols[keep], vals[keep]
        b[n // 2] = 0.0
    o = np.lexsort((cols, rows))
    ptr = np.searchsorted(rows[o], np.arange(n + 1)).astype(np.int32)
    return ptr, cols[o].astype(np.int32), vals[o], b


@pytest.mark.parametrize("kernel", ["cluster", "phase"])
@pytest.mark.parametrize("n,entries", [(1, 3), (31, 3), (33, 4), (256, 3), (257, 8), (511, 3), (512, 5), (513, 4),
                                       (4095, 3), (4097, 9), (24577, 8), (28672, 8), (28673, 8), (28673, 4),
                                       (32768, 3), (32769, 3)])
def test_sizes_and_row_lengths(sbte, monkeypatch, kernel, n, entries):
    _check(sbte, monkeypatch, kernel, _system(n, entries, n + entries))


@pytest.mark.parametrize("kernel", ["cluster", "phase"])
@pytest.mark.parametrize("n", [40, 1000])
@pytest.mark.parametrize("form", [dict(repeat=True), dict(hole=True)])
def test_repeated_and_missing_entries(sbte, monkeypatch, kernel, n, form):
    _check(sbte, monkeypatch, kernel, _system(n, 4, n, **form))


def _check(sbte, monkeypatch, kernel, system):
    import scipy.sparse as sp
    if kernel == "phase":
        monkeypatch.setenv("BTE_KRYLOV", "phase")
    else:
        monkeypatch.delenv("BTE_KRYLOV", raising=False)
    ptr, col, val, b = system
    n = len(b)
    x, _, converged = sbte.bicgstab_csr(ptr, col, val, b, maxit=500, tol=TOL)
    assert converged
    A = sp.csr_matrix((val, col, ptr), shape=(n, n)) + sp.diags((np.diff(ptr) == 0).astype(float))
    d, exact = A.diagonal(), np.zeros(n)
    for _ in range(60):  # Jacobi steps, each halves the error
        exact = exact + (b - A @ exact) / d
    # |x - exact|_inf <= |A^-1|_inf |r|_2, the true residual within 1 % of its recursion's at these
    # conditions (500 steps move it by 500 x 10 eps at most)
    assert np.abs(x - exact).max() <= 2 * 1.01 * TOL * np.linalg.norm(b)
