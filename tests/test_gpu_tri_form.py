"""The PCG in each form its triangular factors are solved in, and with the two
halves in different forms (lock step and records, lock step and value polling,
either way round), against the CPU oracle.

Bounds as for one form: at tol 1e-10 x within 1e-8 of the oracle's 1e-13
solution in each precision, FP64 iterations within 2% (or one).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import lap_gb300 as gb  # noqa: E402
import oracle  # noqa: E402
from test_gpu_team import weighted  # noqa: E402
from test_tri_form import CASES, forms  # noqa: E402

NAMES = ["20000x6", "45000x3", "hub_first", "hub_last", "hubs_first", "hubs_last", "shuffled_64x64", "red_black_30x30",
         "blocks_30x30", "diagonal"]


@pytest.mark.parametrize("prec", ["ichol", "GS_std"])
@pytest.mark.parametrize("name", NAMES)
def test_matches_oracle(name, prec):
    make, want = CASES[name]
    A = weighted(make(), 7) if name != "diagonal" else make()
    assert forms(A) == want
    b = np.random.default_rng(8).uniform(-1.0, 1.0, A.n)
    ref = oracle.solve(A.n, A.ia, A.ja, A.a, b, prec, 1e-13, 20000)
    it = oracle.solve(A.n, A.ia, A.ja, A.a, b, prec, 1e-10, 20000)["iters"]
    s = gb.System.from_csr(A, prec)
    for p in (0, 1, 2):
        x, r = s.solve(torch.from_numpy(b).cuda(), tol=1e-10, maxit=20000, precision=p)
        assert r["flag"] == 0 and r["status"] == 0 and r["rel_true_res"] < 1.01e-10, (p, r)
        assert np.linalg.norm(x.cpu().numpy() - ref["x"]) / np.linalg.norm(ref["x"]) < 1e-8, p
        if p == 0:
            assert abs(r["iters"] - it) <= max(1, int(np.ceil(0.02 * it)))
        again, _ = s.solve(torch.from_numpy(b).cuda(), tol=1e-10, maxit=20000, precision=p, use_graph=False)
        assert torch.equal(again, x)  # reproducible, captured or not
    s.close()
