"""Systems with so many entries that the captured loop is faster run it, in the
precisions where it is: by the entry names of gb_profile_iteration, and the
solves against a float64 residual."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import lap_gb300 as gb  # noqa: E402
from test_gpu_rows_past_32 import band  # noqa: E402

ONE, LOOP = ["team"], ["spmv_pq", "update"]


@pytest.mark.parametrize("n,k,want", [
    (200000, 4, (ONE, ONE)),    # 1.8M entries
    (200000, 16, (ONE, LOOP)),  # 6.6M: FP32 46 us an iteration as a loop, 53 in one launch
    (400000, 12, (LOOP, LOOP)),  # 10.0M: FP64 89 and 97 us
])
def test_form(n, k, want):
    A = band(n, k)
    b = torch.from_numpy(np.random.default_rng(8).uniform(-1.0, 1.0, A.n)).cuda()
    s = gb.System.from_csr(A, "line_jacobi")
    for p in (0, 1):
        assert [q["name"] for q in s.profile(b, precision=p, iters=4)] == want[p]
        _, r = s.solve(b, tol=1e-9, maxit=5000, precision=p)
        assert r["flag"] == r["status"] == 0 and r["rel_true_res"] < 1.01e-9
    s.close()
    B = gb.Batch([A])
    for p in (0, 2):
        _, _, fl, r = B.solve(b, tol=1e-9, maxit=5000, precision=p)
        assert not fl.any() and r["status"] == 0 and r["rel_true_res"] < 1.01e-9
    B.close()
