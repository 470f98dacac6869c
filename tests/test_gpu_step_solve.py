"""The PCG on factors that take the lock-step triangular solves (tri_step.h),
at the shapes where their plan or kernel can go wrong, against the CPU
oracle: one row, rows short of and past a page, one and several solver warps,
levels of several steps, an odd step count, dependencies at the far end of the
previous tile, several clusters, groups that are not all resident.

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
from test_step_plan import box, local_random, path, plan  # noqa: E402


def weighted(A, seed):
    """A's pattern with lognormal weights and a shift of 0.1."""
    rng = np.random.default_rng(seed)
    row = np.repeat(np.arange(A.n), np.diff(A.ia))
    up = row < A.ja
    return gen.laplacian_from_edges(A.n, row[up], A.ja[up], rng.lognormal(0.0, 0.5, int(up.sum())), shift=0.1)


GRAPHS = {
    "one_row": lambda: box(1, 1, 1),
    "path_127": lambda: path(127),
    "path_129": lambda: path(129),
    "path_4097": lambda: path(4097),
    "two_wide_levels": lambda: path(4000, 2000),
    "box_33x31x17": lambda: box(33, 31, 17),
    "box_5x3x301": lambda: box(5, 3, 301),
    "box_257x65": lambda: box(257, 65, 1),
    "box_70x70x40": lambda: box(70, 70, 40),
    "local_random": lambda: local_random(20000, 300, 5),
}


@pytest.mark.parametrize("prec", ["ichol", "GS_std"])
@pytest.mark.parametrize("name", GRAPHS)
def test_matches_oracle(name, prec):
    A = weighted(GRAPHS[name](), 7)
    assert not isinstance(plan(A, True, 4), int) and not isinstance(plan(A, False, 8), int)
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


def test_groups_not_all_resident():
    """200 x 200 planes leave room for one plane a tile: 300 tiles, more than
    the device holds, so clusters take groups one after another."""
    nx, ny, nz = 200, 200, 300
    n = nx * ny * nz
    i = torch.arange(n, device="cuda")
    x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
    keep = torch.stack([z > 0, y > 0, x > 0, x >= 0, x < nx - 1, y < ny - 1, z < nz - 1], 1)
    step = torch.tensor([-nx * ny, -nx, -1, 0, 1, nx, nx * ny], device="cuda")
    ja = (i[:, None] + step)[keep].to(torch.int32)
    ia = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ia[1:] = keep.sum(1).cumsum(0)
    a = torch.where(step == 0, 6.5, -1.0).to(torch.float64).expand(n, 7)[keep]
    s = gb.System(ia.to(torch.int32), ja, a, "ichol")
    b = torch.randn(n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    xs = []
    for p in (0, 2, 2):
        v, r = s.solve(b, tol=1e-10, maxit=500, precision=p)
        assert r["flag"] == 0 and r["status"] == 0 and r["rel_true_res"] < 1.01e-10, (p, r)
        xs.append(v)
    assert float((xs[0] - xs[1]).norm() / xs[0].norm()) < 1e-8 and torch.equal(xs[1], xs[2])
    s.close()
