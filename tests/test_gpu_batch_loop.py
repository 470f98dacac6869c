"""Batches that the one-launch recurrences (team.cu) do not take, so that their
captured loop of row-bundle kernels runs: a system with a row of 66 entries
among the others.  Against the CPU oracle and the same batch run eagerly, in
FP64 and split precision, with default and with tuned sizes.

Bounds as in test_gpu_team.py: at tol 1e-10 x within 1e-8 of the oracle's
1e-13 solution, FP64 iterations within one.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import lap_gb300 as gb  # noqa: E402
import oracle  # noqa: E402
from test_gpu_team import box, path, star, weighted  # noqa: E402


def systems():
    mats = [path(1), path(33), path(257), box(40, 30, 1), star(900, 64), box(17, 13, 11), box(300, 70, 1)]
    return [weighted(A, k) for k, A in enumerate(mats)]


def solve_both_ways(B, b, **kw):
    x, it, fl, r = B.solve(b, **kw)
    y, jt, gl, q = B.solve(b, use_graph=False, **kw)
    assert torch.equal(x, y) and (it == jt).all() and (fl == gl).all()
    return x, it, fl, r


@pytest.mark.parametrize("prec", ["line_jacobi", "none"])
def test_matches_oracle(prec):
    mats = systems()
    rhs = [np.random.default_rng(k).uniform(-1.0, 1.0, A.n) for k, A in enumerate(mats)]
    b = torch.from_numpy(np.concatenate(rhs)).cuda()
    refs = [oracle.solve(A.n, A.ia, A.ja, A.a, f, prec, 1e-13, 20000)["x"] for A, f in zip(mats, rhs)]
    its = [oracle.solve(A.n, A.ia, A.ja, A.a, f, prec, 1e-10, 20000)["iters"] for A, f in zip(mats, rhs)]
    B = gb.Batch(mats, prec)
    for tuned in (False, True):
        if tuned:
            t = B.autotune(b, iters=8)
            assert t["ms_best"] <= t["ms_default"]
        for precision in (0, 2):
            x, it, fl, r = solve_both_ways(B, b, tol=1e-10, maxit=20000, precision=precision)
            assert r["status"] == 0 and not fl.any() and r["rel_true_res"] < 1.01e-10
            for u, ref in zip(B.split(x), refs):
                assert np.linalg.norm(u.cpu().numpy() - ref) / np.linalg.norm(ref) < 1e-8
            if precision == 0:
                assert np.abs(it - its).max() <= 1
    B.close()


def test_iteration_cap():
    """cg.c's flag 1 after maxit + 1 iterations, for the systems still at work."""
    mats = systems()
    b = torch.from_numpy(np.random.default_rng(1).uniform(-1.0, 1.0, sum(A.n for A in mats))).cuda()
    B = gb.Batch(mats)
    _, it, fl, r = solve_both_ways(B, b, tol=1e-12, maxit=5)
    assert (it[1:] == 6).all() and (fl[1:] == 1).all() and r["flag"] == 1
    assert it[0] == 1 and fl[0] == 0  # one row: exact after one
    B.close()
