"""gb_profile_iteration: what it reports is what solves run, also where the
recurrence is one launch, and on a system whose waits run out."""
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


@pytest.mark.parametrize("prec", ["line_jacobi", "none"])
def test_one_launch_recurrence(prec):
    """256 x 256 runs whole in one launch: one entry, whose time is that of a
    solve's iteration (two timings of the same loop, the least of three each,
    within a quarter; the loop's own kernels took twice as long).  700 x 700
    does not fit the device and runs them."""
    A, b = gen.grid2d_unit(256, seed=1001)
    b = torch.from_numpy(b).cuda()
    s = gb.System.from_csr(A, prec)
    for precision in (0, 1):
        runs = [s.profile(b, precision=precision, iters=500) for _ in range(3)]
        assert [[k["name"] for k in r] for r in runs] == [["team"]] * 3
    ms = min(s.profile(b, precision=0, iters=500)[0]["ms"] for _ in range(3))
    run = min(r["device_ms"] / r["iters"] for _, r in (s.solve(b, tol=0.0, maxit=500) for _ in range(3)))
    assert 0.75 < ms / run < 1.25
    x, r = s.solve(b, tol=1e-10, maxit=5000)
    assert r["status"] == 0 and r["flag"] == 0
    s.close()
    A, b = gen.grid2d_unit(700, seed=1001)
    s = gb.System.from_csr(A, prec)
    assert [k["name"] for k in s.profile(torch.from_numpy(b).cuda(), iters=4)] == ["spmv_pq", "update"]
    s.close()
