"""The wall heat flux (k_heat_face, k_heat_final) at faces beside full warps, several bands and
directions that eight warps do not share evenly, against the same sums in numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("name,bands", [("square10_b40", 40), ("square10_b40", 1), ("2DM2DG", 9), ("cube4_b2", 2),
                                        ("cube4_b2", 17), ("3DM2DG", 3)])
def test_wall_flux(sbte, get_case, name, bands):
    from staticbtesolver_gb300 import synth

    a = sbte.Problem(*get_case(name).args()).arrays()
    a["bands"] = b = synth.debye_bands(bands)
    ctx = sbte.Context(0)
    ctx.set_arrays(a)
    ctx.solve(max_iter=3, tol=0.0, form=sbte.FORM_SWEEP)
    e, (q, q_band) = ctx.energy(), ctx.heat_flux()
    # outgoing flux of a face: sum_d e_d w_d, w = (s . n) A Omega (DM 3 on a 3D mesh), (S . n) A otherwise
    s, S, omega = (np.asarray(a[k]) for k in ("s", "S", "omega"))
    D = s.reshape(-1, 3) * omega[:, None] if a["DM"] == 3 and a["dim"] == 3 else S.reshape(-1, 3)
    for i, index in enumerate(a["bcs"]["index"]):
        c, f = np.nonzero(a["nbr"] == index)  # (walls are negative neighbours)
        w = (a["normal"][c, f] @ D.T) * a["area"][c, f][:, None]
        terms = np.einsum("bdk,kd->bdk", e[:, :, c], w)
        scale = b["vg"] / a["area"][c, f].sum()
        exact, size = terms.sum((1, 2)) * scale, np.abs(terms).sum((1, 2)) * scale
        tol = (terms[0].size + 16) * EPS * size  # rounding of a sum of that many terms
        assert len(c) and np.all(np.abs(q_band[i] - exact) <= tol)
        assert abs(q[i] - exact.sum()) <= tol.sum() + (bands + 4) * EPS * np.abs(exact).sum()
