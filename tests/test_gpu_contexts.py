"""Contexts of different sizes alive at once, and calls of different sizes from several host threads:
what a kernel may be launched with is no one problem's, and contexts are independent, so each solve
gives what it gives alone, to the bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh(sbte, tmp_path_factory):
    """The first `cells` of 5,202 triangles; a face cut open joins the wall of entity 0."""
    from staticbtesolver_gb300 import synth

    p = synth.make_problem("nondelaunay51_b3", str(tmp_path_factory.mktemp("contexts")))
    a = sbte.Problem(p.geo, p.bc_file, p.band_file, p.DM, p.num_theta, p.num_phi, p.T_ref, p.L_x, p.L_y, p.L_z).arrays()

    def cut(cells):
        c = dict(a, n_cell=cells)
        for k in ("nbr", "area", "normal", "volume", "centroid"):
            c[k] = a[k][:cells]
        c["nbr"] = np.where(c["nbr"] >= cells, -1, c["nbr"])
        return c

    return cut


def _fields(ctx, **kw):
    ctx.solve(max_iter=3, tol=0.0, **kw)
    return ctx.energy(), ctx.temperature()


@pytest.mark.parametrize("kw", [dict(form="PLAIN"), dict(form="MIXED"), dict(form="SWEEP"), dict(form="SWEEP", dsa=True),
                                dict(form="MIXED", dsa=True)], ids=str)
def test_a_smaller_context_between_two_solves(sbte, mesh, kw):
    kw = dict(kw, form=getattr(sbte, "FORM_" + kw["form"]))
    sizes = (4000, 578, 1500, 130)
    ctxs = [sbte.Context(0) for _ in sizes]
    for ctx, n in zip(ctxs, sizes):
        ctx.set_arrays(mesh(n))
    first = [_fields(ctx, **kw) for ctx in ctxs]  # each smaller than the one before it
    for ctx, (e, T) in zip(ctxs, first):
        e1, T1 = _fields(ctx, **kw)
        assert np.array_equal(e, e1) and np.array_equal(T, T1)
    for ctx in ctxs:
        ctx.close()


def _in_threads(jobs):
    """Every job in a thread of its own, all started together; their errors, in order."""
    errors, start = [None] * len(jobs), threading.Barrier(len(jobs))

    def go(k):
        try:
            start.wait()
            jobs[k]()
        except BaseException as e:
            errors[k] = e

    threads = [threading.Thread(target=go, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def _bidiagonal(n, seed):
    rng = np.random.default_rng(seed)
    ptr = np.concatenate([[0], 1 + 2 * np.arange(n)]).astype(np.int32)
    col = np.zeros(2 * n - 1, np.int32)
    col[0::2], col[1::2] = np.arange(n), np.arange(n - 1)
    val = np.empty(2 * n - 1)
    val[0::2], val[1::2] = rng.uniform(1, 2, n), rng.uniform(-0.5, -0.2, n - 1)
    return ptr, col, val, rng.uniform(-1, 1, n)


def test_csr_systems_of_several_sizes_in_threads(sbte):
    systems = [_bidiagonal(n, n) for n in (300, 2500, 9000, 30000)]
    alone = [sbte.bicgstab_csr(*s) for s in systems]

    def job(s, want):
        def go():
            for _ in range(150):
                x, its, conv = sbte.bicgstab_csr(*s)
                assert its == want[1] and conv == want[2] and np.array_equal(x, want[0])
        return go

    assert _in_threads([job(s, w) for s, w in zip(systems, alone)]) == [None] * len(systems)


def test_set_up_and_solves_of_several_sizes_in_threads(sbte, mesh):
    problems = [mesh(n) for n in (60, 700, 2049, 5000)]

    def solve(a, kw):
        ctx = sbte.Context(0)
        ctx.set_arrays(a)
        out = _fields(ctx, **kw)
        ctx.close()
        return out

    for kw in (dict(form=sbte.FORM_SWEEP, dsa=True), dict(form=sbte.FORM_PLAIN), dict(form=sbte.FORM_MIXED)):
        alone = [solve(a, kw) for a in problems]

        def job(a, want):
            def go():
                for _ in range(8):
                    e, T = solve(a, kw)
                    assert np.array_equal(e, want[0]) and np.array_equal(T, want[1])
            return go

        assert _in_threads([job(a, w) for a, w in zip(problems, alone)]) == [None] * len(problems)
