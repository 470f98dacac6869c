"""The PCG's fused products on matrices most of whose rows have a little more
than 32 entries, alone and with a few much longer ones: which rows of a bundle
the whole warp sums depends on the others.  Against the CPU oracle, and the
time of such a product against that of a matrix just short of the limit.

Bounds: at tol 1e-10 x within 1e-8 of the oracle's 1e-13 solution in each
precision, FP64 iterations within 2% (or one).
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


def band(n, k, extra=()):
    """Row i on the k rows before it and the k after; extra: (row, degree)s of
    further random neighbours."""
    rng = np.random.default_rng(3)
    ei = np.concatenate([np.arange(n - j) for j in range(1, k + 1)] + [np.full(d, i) for i, d in extra])
    ej = np.concatenate([np.arange(j, n) for j in range(1, k + 1)] +
                        [rng.choice(np.delete(np.arange(n), np.arange(max(0, i - k), min(n, i + k + 1))), d, replace=False)
                         for i, d in extra])
    return gen.laplacian_from_edges(n, ei, ej, rng.uniform(0.5, 1.5, len(ei)), shift=0.5)


GRAPHS = {
    "33": lambda: band(3000, 16),
    "61": lambda: band(3000, 30),
    "101": lambda: band(2000, 50),
    "31_and_longer": lambda: band(3000, 15, [(100, 20), (101, 90), (1500, 300), (2500, 470)]),
    "33_and_longer": lambda: band(3000, 16, [(100, 20), (101, 90), (1500, 300), (2500, 900)]),
}


@pytest.mark.parametrize("prec", ["none", "ichol"])
@pytest.mark.parametrize("name", GRAPHS)
def test_matches_oracle(name, prec):
    A = GRAPHS[name]()
    b = np.random.default_rng(8).uniform(-1.0, 1.0, A.n)
    ref = oracle.solve(A.n, A.ia, A.ja, A.a, b, prec, 1e-13, 20000)
    it = oracle.solve(A.n, A.ia, A.ja, A.a, b, prec, 1e-10, 20000)["iters"]
    s = gb.System.from_csr(A, prec)
    for p in (0, 1, 2) if prec == "ichol" else (0, 1):
        x, r = s.solve(torch.from_numpy(b).cuda(), tol=1e-10, maxit=20000, precision=p)
        assert r["flag"] == 0 and r["status"] == 0 and r["rel_true_res"] < 1.01e-10, (p, r)
        assert np.linalg.norm(x.cpu().numpy() - ref["x"]) / np.linalg.norm(ref["x"]) < 1e-8, p
        if p == 0:
            assert abs(r["iters"] - it) <= max(1, int(np.ceil(0.02 * it)))
        again, _ = s.solve(torch.from_numpy(b).cuda(), tol=1e-10, maxit=20000, precision=p, use_graph=False)
        assert torch.equal(again, x)
    s.close()


def test_33_entries_take_about_as_long_as_31():
    """200k rows, GS_std: 6% more entries; a quarter more time at most."""
    ms = {}
    for k in (15, 16):
        A = band(200000, k)
        s = gb.System.from_csr(A, "GS_std")
        b = torch.from_numpy(np.random.default_rng(8).uniform(-1.0, 1.0, A.n)).cuda()
        for p in (0, 1, 2):
            runs = [s.profile(b, precision=p, iters=8) for _ in range(3)]
            ms[k, p] = min(q["ms"] for r in runs for q in r if q["name"].startswith("spmv_pq"))
        s.close()
    for p in (0, 1, 2):
        assert ms[16, p] < 1.25 * ms[15, p], ms
