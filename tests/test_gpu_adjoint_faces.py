"""The face derivatives' elevation terms, formed from the depths' terms, on
grids whose rows leave partial warps: the gradient against forward-mode dual
numbers, to the same 1e-6 relative as test_gpu_adjoint.py."""
import numpy as np
import pytest

import synth
from test_gpu_adjoint import EVERY, N, dual_check, dual_lib, warm_model  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 33, 50])
def test_gradient_matches_dual_numbers(gpu_lib, dual_lib, n):  # noqa: F811
    case = synth.catchment_case(n=n, DX=20.0, hours=72, relief=60.0, hydro_only=True,
                                lateral=False, storm_start_h=0.2, seed=n)
    rng = np.random.default_rng(n)
    case.elev = np.ascontiguousarray(case.elev + rng.uniform(0.0, 1e-3, case.elev.shape))
    rec, q = warm_model(case).adj_forward(N)
    target = np.ascontiguousarray(0.9 * q)
    m = warm_model(case)
    loss, gn, gr, info, ge = m.adj_gradient(N, EVERY, target, elev=True)
    m = warm_model(case)
    for grad, name in ((gn, "dman"), (ge, "delev")):
        v = np.zeros_like(grad)
        v[1:-1, 1:-1] = rng.standard_normal((n, n))
        f, (lo, dlo), args, keep = dual_check(case, rec, target, m, **{name: v})
        dual_lib.hco_dual_run(*args)
        assert lo.value == pytest.approx(loss, rel=1e-8)
        assert abs(dlo.value) > 0
        assert float(np.sum(grad * v)) == pytest.approx(dlo.value, rel=1e-6)
