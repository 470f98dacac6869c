"""A chain of 9M levels: a triangular solve on it takes longer than the second
after which a wait gives up, so no tile may start waiting at its beginning for
what its end brings.  One iteration of the GS_std PCG against the oracle's, whose
two serial sums of 9M terms round to about sqrt(n) 2^-53 = 3e-13 each; the
bound is thirty times that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import lap_gb300 as gb  # noqa: E402
import oracle  # noqa: E402


def test_no_wait_gives_up():
    n = 9_000_000
    ia = np.clip(3 * np.arange(n + 1) - 1, 0, 3 * n - 2).astype(np.int32)
    cols = np.arange(n)[:, None] + np.array([-1, 0, 1])
    inside = (cols >= 0) & (cols < n)
    ja = cols[inside].astype(np.int32)
    a = np.broadcast_to(np.array([-1.0, 4.0, -1.0]), (n, 3))[inside]
    b = np.random.default_rng(1).uniform(-1.0, 1.0, n)
    ref = oracle.solve(n, ia, ja, a, b, "GS_std", 1e-10, 0)
    s = gb.System(torch.from_numpy(ia).cuda(), torch.from_numpy(ja).cuda(), torch.from_numpy(a).cuda(), "GS_std")
    x, r = s.solve(torch.from_numpy(b).cuda(), tol=1e-10, maxit=0)
    s.close()
    assert r["status"] != 4 and r["iters"] == ref["iters"] == 1
    assert np.linalg.norm(x.cpu().numpy() - ref["x"]) / np.linalg.norm(ref["x"]) < 1e-11
