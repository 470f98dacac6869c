"""gb_profile_iteration on a system whose solves' waits run out, and after it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import lap_gb300 as gb  # noqa: E402
from lap_gb300 import gen  # noqa: E402


def budget(s, ns):
    gb.check(gb.lib().gb_debug_set_spin_budget(s.h, ns), "set budget")


@pytest.mark.parametrize("precision", [0, 2])
def test_waits_that_run_out(precision):
    """A chain of 150 rows a tile apart, as test_gpu_flow_solve.py's: with a
    spin budget of 1 ns its far rows give up.  A profile says so, as a solve
    does, and neither leaves anything behind for the next."""
    at = 1024 * np.arange(150)
    ei, ej = (np.concatenate(v) for v in zip(*((at[:-j], at[j:]) for j in range(1, 6))))
    A = gen.laplacian_from_edges(150 * 1024, ei, ej, np.ones(len(ei)), shift=1.0)
    b = torch.from_numpy(np.random.default_rng(8).uniform(-1.0, 1.0, A.n)).cuda()
    s = gb.System.from_csr(A, "ichol")
    kw = dict(tol=1e-10, maxit=1000, precision=precision)
    x, _ = s.solve(b, **kw)
    names = [k["name"] for k in s.profile(b, precision=precision, iters=2)]
    budget(s, 1)
    assert s.solve(b, **kw)[1]["status"] == 4
    with pytest.raises(gb.GbError):
        s.profile(b, precision=precision, iters=2)
    budget(s, 0)
    assert [k["name"] for k in s.profile(b, precision=precision, iters=2)] == names
    again, r = s.solve(b, **kw)
    assert r["status"] == 0 and torch.equal(again, x)
    s.close()
