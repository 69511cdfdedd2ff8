"""Device memory that the stream kernel's padded plan does not fit in, but k_sweep's does: the solve goes
on with k_sweep, as it did without the stream kernel, and gives the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_falls_back_when_the_padded_plan_does_not_fit(sbte, get_case, monkeypatch):
    import torch

    # one cell per level: rows of 32 positions, 31 of them padding
    args = list(get_case("slab1d").args())
    args[0] = "1000"
    a = sbte.Problem(*args).arrays()
    lanes = len(a["bands"]["vg"]) * a["n_dir"]
    args[0] = str(min(30000, (200 << 20) // (16 * 32 * lanes)))  # the padded coefficients take 200 MB at most
    a = sbte.Problem(*args).arrays()

    def solve(kernel=None):
        monkeypatch.delenv("BTE_SWEEP_KERNEL", raising=False)
        if kernel:
            monkeypatch.setenv("BTE_SWEEP_KERNEL", kernel)
        before = torch.cuda.mem_get_info()[0]
        ctx = sbte.Context(0)
        ctx.set_arrays(a)
        _, rep = ctx.solve(max_iter=3, tol=0.0, form=sbte.FORM_SWEEP)
        out = rep.sweep_kernel, ctx.temperature(), ctx.energy(), before - torch.cuda.mem_get_info()[0]
        ctx.close()
        return out

    solve(), solve("level")  # (kernels loaded)
    (ks, Ts, es, stream), (kl, Tl, el, level) = solve(), solve("level")
    assert (ks, kl) == (3, 0) and stream > level + (64 << 20)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (stream + level) // 2, dtype=torch.uint8, device="cuda")
    try:
        k, T, e, _ = solve()
        assert k != 3 and np.array_equal(T, Ts) and np.array_equal(e, es) and np.array_equal(T, Tl)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert solve()[0] == 3  # (and with the memory back, the stream kernel)
