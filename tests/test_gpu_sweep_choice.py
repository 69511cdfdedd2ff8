"""Which sweep kernel and shape a plan gets (sweep_choose, csrc/bte_api.cu).  The stream kernel leaves the
margin to the closing reduction, which costs a small state with many directions or bands more than it
saves: there k_sweep, which sums the margin, stays.  Either way the same temperatures, intensities and
fluxes to the bit, margins to 1e-12 (summed in another order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (case, angular divisions, bands, kernel): 4 x divisions directions on triangles, 8 x their square on tetrahedra;
# the kernels measured to be the faster one, by 15 % or more
CHOICES = [("square16_b8", 8, 8, 3), ("square10_b40", 8, 24, 3), ("square10_b40", 8, 1, 3), ("square10_b40", 32, 24, 0),
           ("square10_b40", 128, 4, 0), ("square16_b8", 128, 8, 0), ("cube4_b2", 4, 2, 3), ("cube4_b2", 4, 20, 0),
           ("cube4_b2", 8, 8, 0), ("cube4_b2", 2, 8, 3)]


@pytest.mark.parametrize("name,div,bands,kernel", CHOICES)
def test_kernel_of_a_plan(sbte, get_case, monkeypatch, name, div, bands, kernel):
    from staticbtesolver_gb300 import synth

    args = list(get_case(name).args())
    args[4] = args[5] = div
    a = sbte.Problem(*args).arrays()
    a["bands"] = synth.debye_bands(bands)
    out = []
    for env in (None, "level", "stream"):
        monkeypatch.delenv("BTE_SWEEP_KERNEL", raising=False)
        if env:
            monkeypatch.setenv("BTE_SWEEP_KERNEL", env)
        ctx = sbte.Context(0)
        ctx.set_arrays(a)
        _, rep = ctx.solve(max_iter=4, tol=0.0, form=sbte.FORM_SWEEP)
        out.append((rep.sweep_kernel, ctx.temperature(), ctx.energy(), ctx.heat_flux()[0], ctx.margins()))
        assert env or ctx.sweep_tuning() == []  # (no trial sweeps)
        ctx.close()
    assert [o[0] for o in out] == [kernel, 0, 3]
    for o in out[1:]:
        assert all(np.array_equal(p, q, equal_nan=True) for p, q in zip(o[1:4], out[0][1:4]))
        np.testing.assert_allclose(o[4], out[0][4], rtol=1e-12)


@pytest.mark.parametrize("bands", [12, 20, 24, 32, 40])
def test_blocks_of_narrow_levels_are_resident_together(sbte, get_case, bands):
    """Levels of one row gain nothing from more warps: a shape whose blocks need a second wave takes
    twice as long (24 bands on 200 to 2,450 triangles did)."""
    import torch

    from staticbtesolver_gb300 import synth

    a = sbte.Problem(*get_case("square10_b40").args()).arrays()
    a["bands"] = synth.debye_bands(bands)
    ctx = sbte.Context(0)
    ctx.set_arrays(a)
    _, rep = ctx.solve(max_iter=2, tol=0.0, form=sbte.FORM_SWEEP)
    assert rep.sweep_kernel == 3
    blocks = -(-bands // rep.sweep_group) * a["n_dir"]
    resident = min(65536 // (80 * rep.sweep_threads), 2048 // rep.sweep_threads)  # (80 registers a thread)
    assert blocks <= torch.cuda.get_device_properties(0).multi_processor_count * resident
    ctx.close()
