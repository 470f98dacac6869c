"""gb_batch_autotune times the loop a batch's solves run: one launch for all
systems where they fit the device (team.cu), the row-bundle loop otherwise.

The two loops' times differ by well over a quarter on small systems; two
timings of one loop, the smaller of three each, do not.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import lap_gb300 as gb  # noqa: E402
from test_gpu_team import box, path, weighted  # noqa: E402

ITERS = 400


def rhs(mats):
    return torch.from_numpy(np.random.default_rng(4).uniform(-1.0, 1.0, sum(A.n for A in mats))).cuda()


def test_one_launch_batch_is_timed_as_it_runs():
    t = []
    for k in range(3):  # classes of their own: each is timed, none taken from the cache
        mats = [weighted(box(40, 30 + k, 1), s) for s in range(8)]
        b = rhs(mats)
        B = gb.Batch(mats)
        x = B.solve(b, tol=1e-10, maxit=5000)[0]
        t.append(B.autotune(b, iters=ITERS))
        assert (t[-1]["rows_per_bundle"], t[-1]["chunk_rows"]) == (32, 2048)
        assert torch.equal(B.solve(b, tol=1e-10, maxit=5000)[0], x)
        t[-1]["run"] = min(B.solve(b, tol=0.0, maxit=ITERS)[3]["device_ms"] for _ in range(3))
        B.close()
    assert all(v["ms_best"] == v["ms_default"] for v in t)
    assert min(v["ms_default"] / v["run"] for v in t) < 1.25


def test_one_launch_choice_is_not_taken_for_the_bundle_loop():
    """The same count, rows, entries and longest row: 450 systems of 800 rows
    are 450 blocks, which fit; 225 of 1,030 and 225 of 570 are 675."""
    even = [path(800) for _ in range(450)]
    uneven = [path(n) for n in (1030, 570) for _ in range(225)]
    B = gb.Batch(even)
    assert B.autotune(rhs(even), iters=4)["ms_best"] > 0.0
    B.close()
    B = gb.Batch(uneven)
    t = B.autotune(rhs(uneven), iters=4)
    assert 0.0 < t["ms_best"] <= t["ms_default"]
    B.close()
