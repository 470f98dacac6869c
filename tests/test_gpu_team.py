"""Recurrences run whole in one launch (team.cu: line_jacobi and no
preconditioner, systems whose blocks fit the device at once), at the sizes
where blocks, rows of a thread and the mail can go wrong, against the CPU
oracle -- and just past the limits, where the captured loop runs.

Bounds as for the captured loop: at tol 1e-10 x within 1e-8 of the oracle's
1e-13 solution, iterations within one (FP64).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import lap_gb300 as gb  # noqa: E402
import oracle  # noqa: E402
from lap_gb300 import gen  # noqa: E402
from test_step_plan import box, path  # noqa: E402


def star(n, leaves):
    """A path whose first row has `leaves` neighbours besides."""
    ei = np.concatenate([np.arange(n - 1), np.zeros(leaves, int)])
    ej = np.concatenate([np.arange(1, n), np.arange(2, 2 + leaves)])
    return gen.laplacian_from_edges(n, ei, ej, np.ones(len(ei)), shift=0.5)


def weighted(A, seed):
    rng = np.random.default_rng(seed)
    row = np.repeat(np.arange(A.n), np.diff(A.ia))
    up = row < A.ja
    return gen.laplacian_from_edges(A.n, row[up], A.ja[up], rng.lognormal(0.0, 0.3, int(up.sum())), shift=0.3)


GRAPHS = {
    "one_row": lambda: box(1, 1, 1),
    "rows_255": lambda: path(255),
    "rows_257": lambda: path(257),
    "rows_38913": lambda: path(152 * 256 + 1),  # two rows of a thread, or two blocks an SM
    "box_300x200": lambda: box(300, 200, 1),
    "box_61x70x43": lambda: box(61, 70, 43),  # three rows of a thread and more
    "box_700x700": lambda: box(700, 700, 1),  # past the device's blocks: the captured loop
    "row_of_63": lambda: star(900, 61),
    "row_of_66": lambda: star(900, 64),  # past a thread's row: the captured loop
}


@pytest.mark.parametrize("prec", ["line_jacobi", "none"])
@pytest.mark.parametrize("name", GRAPHS)
def test_matches_oracle(name, prec):
    A = weighted(GRAPHS[name](), 3)
    b = np.random.default_rng(4).uniform(-1.0, 1.0, A.n)
    ref = oracle.solve(A.n, A.ia, A.ja, A.a, b, prec, 1e-13, 20000)
    it = oracle.solve(A.n, A.ia, A.ja, A.a, b, prec, 1e-10, 20000)["iters"]
    s = gb.System.from_csr(A, prec)
    # one row: the FP32 recurrence is exact after a step, and resuming it from
    # rho = 0 is a breakdown, as in the captured loop
    for p in (0, 1) if A.n > 1 else (0,):
        x, r, hist = s.solve(torch.from_numpy(b).cuda(), tol=1e-10, maxit=20000, precision=p, hist_len=64)
        assert r["flag"] == 0 and r["status"] == 0 and r["rel_true_res"] < 1.01e-10, (p, r)
        assert np.linalg.norm(x.cpu().numpy() - ref["x"]) / np.linalg.norm(ref["x"]) < 1e-8, p
        if p == 0:
            assert abs(r["iters"] - it) <= 1
            # one row is solved exactly: its last residual is 0
            assert hist[0] == pytest.approx(r["res0"], rel=1e-12) and len(hist) == min(64, r["iters"] + 1)
        again, _ = s.solve(torch.from_numpy(b).cuda(), tol=1e-10, maxit=20000, precision=p, use_graph=False)
        assert torch.equal(again, x)
    # an iteration cap: cg.c's flag 1 after maxit + 1 iterations
    if it > 6:
        _, r = s.solve(torch.from_numpy(b).cuda(), tol=1e-10, maxit=4)
        assert (r["flag"], r["iters"]) == (1, 5)
    s.close()


@pytest.mark.parametrize("precision", [0, 2])
def test_batch_of_uneven_systems(precision):
    sizes = [1, 2, 255, 256, 257, 1023, 4000, 30011]
    mats = [weighted(path(n) if n < 300 else box(n // 7, 7, 1), n) for n in sizes]
    rhs = [np.random.default_rng(n).uniform(-1.0, 1.0, A.n) for n, A in zip(sizes, mats)]
    B = gb.Batch(mats)
    b = torch.from_numpy(np.concatenate(rhs)).cuda()
    x, it, fl, r = B.solve(b, tol=1e-10, maxit=5000, precision=precision)
    assert r["status"] == 0 and not fl.any()
    again, _, _, _ = B.solve(b, tol=1e-10, maxit=5000, precision=precision, use_graph=False)
    assert torch.equal(again, x)
    for A, f, xs, its in zip(mats, rhs, B.split(x), it):
        ref = oracle.solve(A.n, A.ia, A.ja, A.a, f, "line_jacobi", 1e-13, 20000)
        assert np.linalg.norm(xs.cpu().numpy() - ref["x"]) / np.linalg.norm(ref["x"]) < 1e-8
        if precision == 0:
            want = oracle.solve(A.n, A.ia, A.ja, A.a, f, "line_jacobi", 1e-10, 20000)["iters"]
            assert abs(int(its) - want) <= 1
    B.close()
