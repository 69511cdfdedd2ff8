"""How k_bicg_cluster leaves and restarts an iteration: exact breakdowns (r_hat . q = 0 and r_hat . r = 0),
the iteration limit, and the best iterate of an extended limit; cluster against the phase kernels
(BTE_KRYLOV=phase) or against the residuals of what is returned."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, entries):
    r, c, v = (np.array(x) for x in zip(*entries))
    o = np.lexsort((c, r))
    return np.searchsorted(r[o], np.arange(n + 1)).astype(np.int32), c[o].astype(np.int32), v[o].astype(float)


def _copies(block, b, m, zeros):
    """m copies of a small system, unknown i of copy k at i m + k (so that its neighbours lie m unknowns, often
    CTAs, away); `zeros` further stored entries of value 0 per row."""
    s = len(b)
    n = s * m
    entries = [(i * m + k, j * m + k, block[i][j]) for i in range(s) for j in range(s) for k in range(m)
               if block[i][j] or i == j]
    if n > zeros + 1:
        entries += [(r, (r + 1 + z) % n, 0.0) for r in range(n) for z in range(zeros)]
    return _csr(n, entries) + (np.repeat(np.asarray(b, float), m),)


def _both(sbte, monkeypatch, system, **kw):
    monkeypatch.delenv("BTE_KRYLOV", raising=False)
    cluster = sbte.bicgstab_csr(*system, **kw)
    monkeypatch.setenv("BTE_KRYLOV", "phase")
    return cluster, sbte.bicgstab_csr(*system, **kw)


# Diagonals are 1 (no preconditioning) and every value before the restart is a small integer or a
# power of two, so the sums that vanish do so exactly in any order.  After the restart (x = 0,
# r_hat = 6.8 b + 0.6) a block of s unknowns ends within s steps.
BREAKDOWNS = {
    # b . A b = 0 in the first step; r_hat . A b = -1.2 a copy after the restart
    "rwq": ([[1, -2.5], [0, 1]], [1, 2], [1, 3, 130, 511, 600, 1500], 1 + 2),
    # A b = (1, -1, -2): s = (0, 1, 2), s . A s = 0, so omega = 0 and r_hat . r = 0 with r = s in the
    # second (alpha is a power of two for copies of one less than one)
    "rwr": ([[1, 0.25, 0.5], [-1, 1, -2.5], [-2, 0, 1]], [1, 0, 0], [1, 3, 127, 511, 1023], 2 + 3),
}


@pytest.mark.parametrize("zeros", [0, 1, 4])
@pytest.mark.parametrize("kind,m", [(k, m) for k, v in BREAKDOWNS.items() for m in v[2]])
def test_exact_breakdowns(sbte, monkeypatch, kind, m, zeros):
    block, b, _, steps = BREAKDOWNS[kind]
    (x, its, conv), (xp, itp, convp) = _both(sbte, monkeypatch, _copies(block, b, m, zeros), tol=1e-8)
    exact = np.repeat(np.linalg.solve(np.asarray(block, float), b), m)
    assert conv and convp and its == itp == steps  # (a solve without breakdown takes len(b) at most)
    # the blocks' inverses have norms below 3; the last step's residual is of the order of 1e-12
    for v in (x, xp):
        assert np.linalg.norm(v - exact) <= 3e-8 * np.sqrt(m) * np.linalg.norm(b)


def test_breakdown_of_every_restart(sbte, monkeypatch):
    """r_hat = 7.4 where b = 1, 0.6 where it is 0 and so is A b: every step breaks down again, and x = 0 at
    the limit, from both.  (One copy with a right-hand side, its unknowns in two CTAs: -7.4 + 7.4.)"""
    ptr, col, val, b = _copies([[1, -2], [0, 1]], [1, 1], 700, 0)
    b[:] = 0
    b[[0, 700]] = 1
    (x, its, conv), (xp, itp, convp) = _both(sbte, monkeypatch, (ptr, col, val, b), maxit=9)
    assert its == itp == 9 and not conv and not convp and not x.any() and not xp.any()


@pytest.mark.parametrize("n,entries", [(33, 3), (300, 4), (1000, 8), (5000, 3), (32768, 3)])
@pytest.mark.parametrize("maxit", [1, 2])
def test_iterate_at_the_limit(sbte, monkeypatch, n, entries, maxit):
    """The first iterates follow from sums of n terms whose terms have few signs: alpha and omega carry
    the rounding of those, n eps at worst, a hundredfold through the differences of a step."""
    from test_gpu_csr_cluster import _system

    system = _system(n, entries, n)
    (x, its, conv), (xp, itp, convp) = _both(sbte, monkeypatch, system, maxit=maxit, tol=1e-30)
    assert its == itp == maxit and not conv and not convp
    assert xp.any() and np.linalg.norm(x - xp) <= 200 * n * np.finfo(float).eps * np.linalg.norm(xp)


@pytest.fixture(scope="module")
def oracle_systems(oracle_mod, get_case):
    """Every system of the first outer iteration (no intensities, T = T_ref)."""
    import scipy.sparse as sp

    o = oracle_mod.Oracle(*get_case("square16_b8").args())
    zero = np.zeros((o.n_band, o.n_dir, o.n_cell)), np.zeros((o.n_cell, o.n_band))
    out = {}
    for b in range(o.n_band):
        for d in range(o.n_dir):
            ptr, col, val, rhs = o.assemble(b, d, *zero)
            if rhs.any():
                out[b, d] = sp.csr_matrix((val, col, ptr), shape=(o.n_cell, o.n_cell)), rhs
    return out


def test_best_iterate_of_an_extended_limit(sbte, get_case, oracle_systems):
    """plain_cycles = k keeps the iterate with the smallest residual up to k x inner_maxit steps: what is
    returned is never worse than x = 0, and never worse than with a lower k (the same steps, more of
    them).  The residual the choice is made by is the recursion's; 1e-6 of ||b|| covers its distance
    from the true one over 44 steps."""
    ctx = sbte.Context(0).load(sbte.Problem(*get_case("square16_b8").args()))

    def residuals(**kw):
        ctx.solve(max_iter=1, tol=0.0, form=sbte.FORM_PLAIN, **kw)
        e = ctx.energy()
        return np.array([np.linalg.norm(rhs - A @ e[bd]) / np.linalg.norm(rhs) for bd, (A, rhs) in
                         oracle_systems.items()])

    assert residuals().max() <= 2e-9  # (converged: the systems are these)
    last = np.ones(len(oracle_systems))
    for k in (2, 3, 4):
        res = residuals(plain_cycles=k, inner_maxit=11)
        assert np.all(res <= last + 1e-6)
        last = res
    assert np.mean(last < 0.5) > 0.5  # (and not x = 0 throughout)
    ctx.close()
