"""The PCG's fused products on matrices with long rows, at the edges of the
kernels that sum them by the whole warp: rows of 32 and 33 entries, of 512 and
513 (staged or not), of a whole batch of gathers and one more, a full row.

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
from test_flow_plan import hub  # noqa: E402

# off-diagonal entries of the last rows; the diagonal is one more
DEGREES = {"32": [30, 31, 32], "512": [510, 511, 512, 513], "batch": [766, 767, 768, 1023, 1024], "full": [4999]}


@pytest.mark.parametrize("prec", ["line_jacobi", "ichol"])
@pytest.mark.parametrize("name", DEGREES)
def test_matches_oracle(name, prec):
    A = hub(5000, DEGREES[name], seed=4)
    b = np.random.default_rng(8).uniform(-1.0, 1.0, A.n)
    ref = oracle.solve(A.n, A.ia, A.ja, A.a, b, prec, 1e-13, 20000)
    it = oracle.solve(A.n, A.ia, A.ja, A.a, b, prec, 1e-10, 20000)["iters"]
    s = gb.System.from_csr(A, prec)
    for p in (0, 1) if prec == "line_jacobi" else (0, 1, 2):  # the split form is for the triangular ones
        x, r = s.solve(torch.from_numpy(b).cuda(), tol=1e-10, maxit=20000, precision=p)
        assert r["flag"] == 0 and r["status"] == 0 and r["rel_true_res"] < 1.01e-10, (p, r)
        assert np.linalg.norm(x.cpu().numpy() - ref["x"]) / np.linalg.norm(ref["x"]) < 1e-8, p
        if p == 0:
            assert abs(r["iters"] - it) <= max(1, int(np.ceil(0.02 * it)))
        again, _ = s.solve(torch.from_numpy(b).cuda(), tol=1e-10, maxit=20000, precision=p, use_graph=False)
        assert torch.equal(again, x)
    s.close()
