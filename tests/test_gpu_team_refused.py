"""A one-launch recurrence (team.cu) that the device refuses to hold whole:
the solve runs the captured loop and says nothing of it.  Asking for 200 KB of
shared memory a block leaves one block an SM, fewer than these systems have.

Bounds as between the two loops elsewhere: at tol 1e-10 x within 1e-8,
FP64 iterations within one.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import lap_gb300 as gb  # noqa: E402
from test_gpu_team import box, weighted  # noqa: E402

REFUSED = 200 * 1024


def team_smem(bytes, system=None, batch=None):
    gb.check(gb.lib().gb_debug_set_team_smem(system and system.h, batch and batch.h, bytes), "team smem")


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("prec", ["line_jacobi", "none"])
def test_system(prec, precision):
    A = weighted(box(600, 500, 1), 3)  # 293 blocks
    b = torch.from_numpy(np.random.default_rng(4).uniform(-1.0, 1.0, A.n)).cuda()
    s = gb.System.from_csr(A, prec)
    kw = dict(tol=1e-10, maxit=20000, precision=precision)
    x, r = s.solve(b, **kw)
    team_smem(REFUSED, system=s)
    for graph in (True, False):
        y, q = s.solve(b, use_graph=graph, **kw)
        assert q["flag"] == q["status"] == 0 and q["rel_true_res"] < 1.01e-10
        assert float(torch.linalg.norm(x - y) / torch.linalg.norm(x)) < 1e-8
        if precision == 0:
            assert abs(q["iters"] - r["iters"]) <= 1
    _, q = s.solve(b, tol=1e-10, maxit=4)
    assert (q["flag"], q["iters"]) == (1, 5)
    team_smem(0, system=s)
    again, _ = s.solve(b, **kw)
    assert torch.equal(again, x)
    s.close()


@pytest.mark.parametrize("precision", [0, 2])
def test_batch(precision):
    mats = [weighted(box(60, 50 - k % 3, 1), k) for k in range(60)]  # 240 blocks
    b = torch.from_numpy(np.random.default_rng(4).uniform(-1.0, 1.0, sum(A.n for A in mats))).cuda()
    B = gb.Batch(mats)
    kw = dict(tol=1e-10, maxit=20000, precision=precision)
    x, it, _, _ = B.solve(b, **kw)
    team_smem(REFUSED, batch=B)
    for graph in (True, False):
        y, its, fl, r = B.solve(b, use_graph=graph, **kw)
        assert r["status"] == 0 and not fl.any() and r["rel_true_res"] < 1.01e-10
        for u, v in zip(B.split(x), B.split(y)):
            assert float(torch.linalg.norm(u - v) / torch.linalg.norm(u)) < 1e-8
        if precision == 0:
            assert np.abs(its - it).max() <= 1
    team_smem(0, batch=B)
    assert torch.equal(B.solve(b, **kw)[0], x)
    B.close()
