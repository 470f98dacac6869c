"""One-launch recurrences (team.cu) whose waits run out: a block leaves before
it sends its team anything, the others give up after the spin budget (2 ms
here), and the launch ends; the solve returns the status and the next one is
whole again.  That block is the one that writes the state, one among others, or
the last."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import lap_gb300 as gb  # noqa: E402
from test_gpu_team import box, path, weighted  # noqa: E402

BUDGET = 2_000_000  # ns


@pytest.mark.parametrize("block", [0, 5, 117])
@pytest.mark.parametrize("precision", [0, 1])
def test_system(precision, block):
    A = weighted(box(300, 200, 1), 3)  # 118 blocks of two rows a thread
    b = torch.from_numpy(np.random.default_rng(4).uniform(-1.0, 1.0, A.n)).cuda()
    s = gb.System.from_csr(A, "line_jacobi")
    kw = dict(tol=1e-10, maxit=5000, precision=precision)
    x, r = s.solve(b, **kw)
    L = gb.lib()
    gb.check(L.gb_debug_set_spin_budget(s.h, BUDGET), "budget")
    gb.check(L.gb_debug_set_team_silent(s.h, None, block), "silent")
    _, q = s.solve(b, **kw)
    gb.check(L.gb_debug_set_team_silent(s.h, None, -1), "silent")
    gb.check(L.gb_debug_set_spin_budget(s.h, 0), "budget")
    again, p = s.solve(b, **kw)
    assert r["status"] == p["status"] == 0 and q["status"] == 4 and torch.equal(again, x)
    s.close()


@pytest.mark.parametrize("block", [0, 12, 16])
@pytest.mark.parametrize("precision", [0, 2])
def test_batch(precision, block):
    mats = [weighted(box(100, 30, 1), 1), weighted(path(300), 2), weighted(box(50, 20, 1), 3)]  # 12 + 2 + 4 blocks
    b = torch.from_numpy(np.random.default_rng(4).uniform(-1.0, 1.0, sum(A.n for A in mats))).cuda()
    B = gb.Batch(mats)
    kw = dict(tol=1e-10, maxit=5000, precision=precision)
    x, it, fl, r = B.solve(b, **kw)
    L = gb.lib()
    gb.check(L.gb_debug_set_batch_spin_budget(B.h, BUDGET), "budget")
    gb.check(L.gb_debug_set_team_silent(None, B.h, block), "silent")
    with pytest.raises(gb.GbError):
        B.solve(b, **kw)
    gb.check(L.gb_debug_set_team_silent(None, B.h, -1), "silent")
    gb.check(L.gb_debug_set_batch_spin_budget(B.h, 0), "budget")
    again, jt, gl, p = B.solve(b, **kw)
    assert r["status"] == p["status"] == 0 and torch.equal(again, x) and (it == jt).all() and not gl.any()
    B.close()
