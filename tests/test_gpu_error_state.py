"""A call that failed leaves nothing behind: the next call on the same thread, of another context or the same
one, does not report its error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_out_of_memory_does_not_reach_the_next_call(sbte, get_case):
    import torch

    from staticbtesolver_gb300 import synth

    a = sbte.Problem(*get_case("square16_b8").args()).arrays()
    big = dict(a, bands=synth.debye_bands(2000))  # 2,000 bands x 32 directions x 2,048 cells: 1 GB an array
    rng = np.random.default_rng(1)
    csr = (np.arange(101, dtype=np.int32), np.arange(100, dtype=np.int32), rng.uniform(1, 2, 100), rng.uniform(0, 1, 100))
    good = sbte.Context(0)
    good.set_arrays(a)
    _, rep = good.solve(max_iter=2, tol=0.0, form=sbte.FORM_SWEEP)
    T = good.temperature()
    bad = sbte.Context(0)
    bad.set_arrays(big)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (600 << 20), dtype=torch.uint8, device="cuda")
    try:
        for follow in range(3):
            with pytest.raises(sbte.BteError) as e:
                bad.solve(max_iter=2, tol=0.0, form=sbte.FORM_SWEEP)
            assert e.value.status == 4
            if follow == 0:
                good.solve(max_iter=2, tol=0.0, form=sbte.FORM_SWEEP)
                assert np.array_equal(good.temperature(), T)
            elif follow == 1:
                x, _, converged = sbte.bicgstab_csr(*csr)
                assert converged and np.allclose(x, csr[3] / csr[2], rtol=1e-8)
            else:
                fresh = sbte.Context(0)
                fresh.set_arrays(a)
                fresh.solve(max_iter=2, tol=0.0, form=sbte.FORM_SWEEP)
                assert np.array_equal(fresh.temperature(), T)
                fresh.close()
    finally:
        del hold
        torch.cuda.empty_cache()
    bad.solve(max_iter=1, tol=0.0, form=sbte.FORM_SWEEP)  # (with the memory back)
    bad.close()
    good.close()
