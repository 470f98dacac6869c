"""y = alpha A x + beta y bit for bit against the reference's order (separate
multiplies and adds), where the kernel reads rows per lane (bundles of at most
eight entries a row, alpha 1) and just past it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import lap_gb300 as gb  # noqa: E402
from lap_gb300 import gen  # noqa: E402


def rows_of(lengths, seed):
    """A square CSR whose row i has lengths[i] entries at random columns."""
    rng = np.random.default_rng(seed)
    n = len(lengths)
    ia = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    ja = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lengths]).astype(np.int32)
    a = rng.standard_normal(len(ja))
    a[rng.random(len(ja)) < 0.05] = -0.0
    return gen.CSR(n, ia, ja, a)


@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (1.0, 1.0), (1.0, -0.5), (0.5, 0.0), (-1.0, 1.0)])
@pytest.mark.parametrize("lengths", ["1..8", "9 in one bundle", "8", "empty rows"])
def test_bit_exact(lengths, alpha, beta):
    rng = np.random.default_rng(2)
    n = 1000  # a last bundle of eight rows
    k = {"1..8": rng.integers(1, 9, n), "9 in one bundle": np.where(np.arange(n) == 500, 9, 5),
         "8": np.full(n, 8), "empty rows": rng.integers(0, 3, n)}[lengths]
    A = rows_of(k, 3)
    x, y = rng.standard_normal(n), rng.standard_normal(n)
    dia, dja, da, dx, dy = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (A.ia, A.ja, A.a, x, y))
    al, be = C.c_double(alpha), C.c_double(beta)
    torch.cuda.synchronize()
    gb.lib().cuda_csr_matvec(n, A.nnz, gb.ptr(dia), gb.ptr(dja), gb.ptr(da), gb.ptr(dx), gb.ptr(dy), C.byref(al),
                             C.byref(be))
    want = np.where(beta == 0.0, 0.0, y * beta)
    for i in range(n):
        s = want[i]
        for e in range(A.ia[i], A.ia[i + 1]):
            s = s + (alpha * A.a[e]) * x[A.ja[e]]
        want[i] = s
    torch.cuda.synchronize()
    got = dy.cpu().numpy()
    assert np.array_equal(got, want) and np.array_equal(np.signbit(got), np.signbit(want))
