"""The PCG on factors that take the value-polling triangular solves
(tri_flow.h), against the same solve on the records and the CPU oracle: rows
of 31 to 33 and 63 to 97 dependencies, hubs of thousands, a row on every
other, power-law graphs, random labellings.

Bounds as for the record form: at tol 1e-10 x within 1e-8 of the oracle's
1e-13 solution in each precision, FP64 iterations within 2% (or one).
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
from test_flow_plan import hub, shuffled  # noqa: E402

def band(n, k):
    """Row i on the k rows before it."""
    ei, ej = (np.concatenate(v) for v in zip(*((np.arange(n - j), np.arange(j, n)) for j in range(1, k + 1))))
    return gen.laplacian_from_edges(n, ei, ej, np.random.default_rng(1).uniform(0.5, 1.5, len(ei)), shift=0.1)


GRAPHS = {
    "edges_of_32": lambda: shuffled(hub(4000, [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 34, 63, 64, 65, 95, 96, 97]), 1),
    "hubs": lambda: shuffled(hub(6000, [1024, 1055, 2000, 5900]), 2),
    "star": lambda: shuffled(hub(5000, [4999]), 3),
    "chung_lu": lambda: gen.chung_lu(9000, seed=5)[0],
    "one_tile": lambda: gen.chung_lu(700, seed=6)[0],
    "band_of_7": lambda: band(500, 7),
    "shuffled_grid": lambda: shuffled(gen.grid3d(29), 4),
}


@pytest.mark.parametrize("prec", ["ichol", "GS_std"])
@pytest.mark.parametrize("name", GRAPHS)
def test_matches_records_and_oracle(name, prec, monkeypatch):
    A = GRAPHS[name]()
    b = np.random.default_rng(8).uniform(-1.0, 1.0, A.n)
    ref = oracle.solve(A.n, A.ia, A.ja, A.a, b, prec, 1e-13, 20000)
    it = oracle.solve(A.n, A.ia, A.ja, A.a, b, prec, 1e-10, 20000)["iters"]
    s = gb.System.from_csr(A, prec)
    monkeypatch.setenv("GBLAP_TRI_FORM", "levels")
    rec = gb.System.from_csr(A, prec)
    monkeypatch.delenv("GBLAP_TRI_FORM")
    bt = torch.from_numpy(b).cuda()
    for p in (0, 1, 2):
        x, r = s.solve(bt, tol=1e-10, maxit=20000, precision=p)
        y, q = rec.solve(bt, tol=1e-10, maxit=20000, precision=p)
        assert r["flag"] == q["flag"] == 0 and r["status"] == q["status"] == 0 and r["rel_true_res"] < 1.01e-10, (p, r)
        assert np.linalg.norm(x.cpu().numpy() - ref["x"]) / np.linalg.norm(ref["x"]) < 1e-8, p
        if p == 0:
            assert abs(r["iters"] - it) <= max(1, int(np.ceil(0.02 * it)))
            assert abs(r["iters"] - q["iters"]) <= max(1, int(np.ceil(0.02 * it)))
        again, _ = s.solve(bt, tol=1e-10, maxit=20000, precision=p, use_graph=False)
        assert torch.equal(again, x)  # reproducible, captured or not
    s.close()
    rec.close()


@pytest.mark.parametrize("precision", [0, 2])
def test_wide_levels(precision, monkeypatch):
    """A level of thousands of records (two blocks an SM), against the records
    and reproducible; the bounds above."""
    A = gen.knn_graph(100000, 8, seed=4)
    b = torch.from_numpy(np.random.default_rng(8).uniform(-1.0, 1.0, A.n)).cuda()
    s = gb.System.from_csr(A, "ichol")
    monkeypatch.setenv("GBLAP_TRI_FORM", "levels")
    rec = gb.System.from_csr(A, "ichol")
    x, r = s.solve(b, tol=1e-12, maxit=20000, precision=precision)
    y, q = rec.solve(b, tol=1e-12, maxit=20000, precision=precision)
    assert r["flag"] == q["flag"] == 0 and r["status"] == q["status"] == 0
    assert abs(r["iters"] - q["iters"]) <= max(1, int(np.ceil(0.02 * q["iters"])))
    assert float(torch.linalg.norm(x - y) / torch.linalg.norm(y)) < 1e-8
    again, _ = s.solve(b, tol=1e-12, maxit=20000, precision=precision)
    assert torch.equal(again, x)
    s.close()
    rec.close()


def test_a_wait_that_runs_out():
    """A chain of 150 rows a tile apart, each on the five before it, among
    rows of their own: the far ones wait for more than two clock checks.  With
    a spin budget of 1 ns they give up, the solve returns the status, and the
    next one is whole again."""
    at = 1024 * np.arange(150)
    ei, ej = (np.concatenate(v) for v in zip(*((at[:-j], at[j:]) for j in range(1, 6))))
    A = gen.laplacian_from_edges(150 * 1024, ei, ej, np.ones(len(ei)), shift=1.0)
    b = torch.from_numpy(np.random.default_rng(8).uniform(-1.0, 1.0, A.n)).cuda()
    s = gb.System.from_csr(A, "ichol")
    for p in (0, 2):
        x, r = s.solve(b, tol=1e-10, maxit=1000, precision=p)
        gb.check(gb.lib().gb_debug_set_spin_budget(s.h, 1), "set budget")
        _, q = s.solve(b, tol=1e-10, maxit=1000, precision=p)
        gb.check(gb.lib().gb_debug_set_spin_budget(s.h, 0), "reset budget")
        again, r2 = s.solve(b, tol=1e-10, maxit=1000, precision=p)
        assert r["status"] == r2["status"] == 0 and q["status"] == 4 and torch.equal(again, x)
    s.close()
