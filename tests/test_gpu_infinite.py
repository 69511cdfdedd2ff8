"""A state that overflows: the solve says so (a non-finite margin), and the temperatures are infinite where
the sums over the intensities are, in both closing reductions (one launch for few rows, k_reduce beyond),
as a division gives it, not NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bands", [1, 4, 8, 9])  # (32 directions: one launch up to 8 bands)
def test_infinite_sums_give_infinite_temperatures(sbte, get_case, bands):
    from staticbtesolver_gb300 import synth

    a = sbte.Problem(*get_case("square10_b40").args()).arrays()
    a["bands"] = b = synth.debye_bands(bands)
    bcs = {k: np.array(v) for k, v in a["bcs"].items()}
    wall = int(np.flatnonzero(bcs["type"] == 1)[0])
    bcs["T"][wall] = 1e308 / b["C"].min() * 100  # C_b (T - T_ref) / Omega_tot overflows
    ctx = sbte.Context(0)
    ctx.set_arrays(dict(a, bcs=bcs))
    with pytest.raises(sbte.BteError) as e:
        ctx.solve(max_iter=3, tol=0.0, form=sbte.FORM_SWEEP)
    assert e.value.status == 7
    I, Tb, T = ctx.energy(), ctx.band_temperature(), ctx.temperature()
    with np.errstate(invalid="ignore", over="ignore"):
        ref = ((I * np.asarray(a["omega"])[None, :, None]).sum(1) / b["C"][:, None]).T + a["T_ref"]
        mean = (b["Lr"] * Tb).sum(1) / b["Lr"].sum()
    assert np.isposinf(ref).any()
    for got, want in ((Tb, ref), (T, mean)):
        assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isnan(got), np.isnan(want))
    ctx.close()
