"""The stream form of the upwind sweep (k_sweep_stream) against the
level-synchronous kernel (k_sweep): per cell the same operations in the same
order, so temperatures, intensities, fluxes and iteration counts are the same
to the bit (tolerance zero; a wall without faces has no flux in either; the margins are summed by another kernel in
another order: 1e-12 relative).  Meshes at the edges: one cell, rows and chunks
of 32 and 128 positions exactly full and one over, levels of a single cell (1D),
levels wider than a chunk (3D), cyclic graphs (lagged upstream values and
repeated sweeps), specular, diffuse and isothermal walls, band batches."""
import numpy as np
import pytest

from test_gpu_sweep import _odd_slab, _rewired

pytestmark = pytest.mark.gpu

CELLS = [1, 2, 31, 32, 33, 127, 128, 129, 2047, 2048, 2049, 5000]


def _both(sbte, monkeypatch, problem, expect=3, **kw):
    out = {}
    for kernel in ("level", "stream", None):
        if kernel:
            monkeypatch.setenv("BTE_SWEEP_KERNEL", kernel)
        else:
            monkeypatch.delenv("BTE_SWEEP_KERNEL")
        if kernel == "stream" and expect != 3:
            continue
        ctx = sbte.Context(0)
        ctx.set_arrays(problem) if isinstance(problem, dict) else ctx.load(problem)
        st, rep = ctx.solve(form=sbte.FORM_SWEEP, **kw)
        out[kernel] = (st, ctx.temperature(), ctx.energy(), ctx.heat_flux()[0], ctx.margins(), rep.as_dict())
        ctx.close()
    st, T, e, q, m, r = out["level"]
    assert r["sweep_kernel"] == 0 and out[None][5]["sweep_kernel"] == expect
    for kernel in out:
        s1, T1, e1, q1, m1, r1 = out[kernel]
        assert s1 == st and r1["n_iter"] == r["n_iter"] and r1["inner_iterations"] == r["inner_iterations"]
        assert np.array_equal(T, T1) and np.array_equal(e, e1) and np.array_equal(q, q1, equal_nan=True), kernel
        np.testing.assert_allclose(m, m1, rtol=1e-12)


@pytest.mark.parametrize("name", ["square16_b8", "square10_b40", "2DM2DG", "3DM2DG", "cube4_b2", "2Dcase5",
                                  "square16_b8/cycles", "slab1d/odd", "cube9_b3", "nondelaunay40_b11"])
def test_stream_equals_level_kernel(sbte, get_case, monkeypatch, tmp_path, name):
    from staticbtesolver_gb300 import synth

    base = name.split("/")[0]
    if base in ("cube9_b3", "nondelaunay40_b11"):
        p = synth.make_problem(base, str(tmp_path))
        problem = sbte.Problem(p.geo, p.bc_file, p.band_file, p.DM, p.num_theta, p.num_phi, p.T_ref, p.L_x, p.L_y, p.L_z)
    else:
        c = get_case(base)
        problem = (_rewired(sbte, c, n_swaps=10) if name.endswith("/cycles")
                   else sbte.Problem(*(_odd_slab(c) if name.endswith("/odd") else c.args())))
    _both(sbte, monkeypatch, problem, max_iter=6, tol=0.0)


@pytest.mark.parametrize("cells", CELLS)
def test_stream_cell_counts(sbte, monkeypatch, tmp_path, cells):
    """The first `cells` triangles of a mesh; a face cut open joins the wall of entity 0."""
    from staticbtesolver_gb300 import synth

    p = synth.make_problem("nondelaunay51_b3", str(tmp_path))
    a = sbte.Problem(p.geo, p.bc_file, p.band_file, p.DM, p.num_theta, p.num_phi, p.T_ref, p.L_x, p.L_y, p.L_z).arrays()
    a["n_cell"] = cells
    for k in ("nbr", "area", "normal", "volume", "centroid"):
        a[k] = a[k][:cells]
    a["nbr"] = np.where(a["nbr"] >= cells, -1, a["nbr"])
    _both(sbte, monkeypatch, a, max_iter=4, tol=0.0)


def test_stream_batches_and_accelerators(sbte, get_case, monkeypatch):
    problem = sbte.Problem(*get_case("square10_b40").args())
    _both(sbte, monkeypatch, problem, max_iter=5, tol=0.0, batch_systems=7 * 32)
    for kw in (dict(accel=3, accel_every=4), dict(accel=2, accel_every=4), dict(dsa=True)):
        _both(sbte, monkeypatch, problem, max_iter=14, tol=0.0, **kw)


def test_narrow_levels_keep_the_level_kernel(sbte, get_case, monkeypatch):
    """A 1D slab has one cell per level: padded to rows of 32 the coefficients of
    a long one would be many times the state, so k_sweep stays; a short one's
    are small."""
    args = list(get_case("slab1d").args())
    for cells, expect in (("700", 3), ("80000", 0)):
        args[0] = cells
        _both(sbte, monkeypatch, sbte.Problem(*args), expect=expect, max_iter=2, tol=0.0)
