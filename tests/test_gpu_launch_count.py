"""bte_report.kernel_launches counts launches: the last reduction of the wall heat flux has one where the
problem has walls, and none where it has not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_no_wall_no_launch(sbte, get_case):
    a = sbte.Problem(*get_case("square10_b40").args()).arrays()
    one = {k: np.array(v)[:1] for k, v in a["bcs"].items()}
    one["index"] = np.array([-1000], np.int32)  # (an entity without faces: a row of the result, no face)
    none = {k: v[:0] for k, v in one.items()}
    launches = []
    for bcs in (one, none):
        ctx = sbte.Context(0)
        ctx.set_arrays(dict(a, bcs=bcs))
        _, rep = ctx.solve(max_iter=2, tol=0.0, form=sbte.FORM_SWEEP)
        launches.append(rep.kernel_launches)
        ctx.close()
    assert launches[0] == launches[1] + 1
