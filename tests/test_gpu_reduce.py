"""The reductions that close an outer iteration (k_reduce_cells; k_reduce and k_recover beyond its
sizes): cells beside full warps, bands and cells on both sides of the rule, against the same sums over the intensities in numpy.  The
bounds are the rounding of sums of that many terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


CASES = [(1, 1), (31, 2), (32, 3), (33, 4), (100, 8), (64, 9), (65, 64), (95, 65), (2049, 5), (5000, 1), (10240, 8),
         (10241, 8), (10240, 3), (10241, 3)]


@pytest.mark.parametrize("form,cells,bands", [("sweep", *c) for c in CASES] + [("plain", *c) for c in CASES[:10]])
def test_sums_of_an_iteration(sbte, tmp_path, form, cells, bands):
    from staticbtesolver_gb300 import synth

    p = synth.make_problem("nondelaunay51_b3" if cells <= 5202 else "nondelaunay72_b3", str(tmp_path))
    a = sbte.Problem(p.geo, p.bc_file, p.band_file, p.DM, p.num_theta, p.num_phi, p.T_ref, p.L_x, p.L_y, p.L_z).arrays()
    a["n_cell"] = cells
    for k in ("nbr", "area", "normal", "volume", "centroid"):
        a[k] = a[k][:cells]
    a["nbr"] = np.where(a["nbr"] >= cells, -1, a["nbr"])
    a["bands"] = b = synth.debye_bands(bands)
    kw = dict(tol=0.0, form=sbte.FORM_SWEEP if form == "sweep" else sbte.FORM_PLAIN)
    e = []
    for its in (1, 2):
        ctx = sbte.Context(0)
        ctx.set_arrays(a)
        ctx.solve(max_iter=its, **kw)
        e.append(ctx.energy())
    T, Tb, margin = ctx.temperature(), ctx.band_temperature(), ctx.margins()
    ND, T_ref = a["n_dir"], a["T_ref"]
    terms = e[1] * np.asarray(a["omega"])[None, :, None] / b["C"][:, None, None]
    ref = terms.sum(1).T + T_ref
    assert np.all(np.abs(Tb - ref) <= (ND + 8) * EPS * (np.abs(terms).sum(1).T + T_ref))
    mean = (b["Lr"] * Tb).sum(1) / b["Lr"].sum()
    assert np.all(np.abs(T - mean) <= (2 * bands + 8) * EPS * np.abs(Tb).max(1))
    for k, d in enumerate((e[0], e[1] - e[0])):
        np.testing.assert_allclose(margin[k], (d ** 2).sum() / (bands * cells), rtol=(bands * ND + cells + 64) * EPS)
