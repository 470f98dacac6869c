"""The value-polling triangular solves' plan (tri_flow.h), replayed on the CPU
against the substitution it stands for.

The replay walks the records in ticket order, as one warp alone would: every
value a lane reads must have been written by an earlier record, every row and
part is written once, every part is read once, and the solution is that of
plain substitution.
"""
import numpy as np
import pytest

import lap_gb300 as gb
from lap_gb300 import gen


def plan(A, lower):
    ia, ja = np.ascontiguousarray(A.ia, np.int32), np.ascontiguousarray(A.ja, np.int32)
    info = np.zeros(3, np.int32)
    head = (A.n, ia.ctypes.data, ja.ctypes.data, int(lower), info.ctypes.data)
    assert gb.lib().gb_debug_flow_plan(*head, *[None] * 5) == 0
    lanes = [np.zeros(info[0] * 32, np.int32) for _ in range(4)]
    g = np.zeros(info[0], np.int32)
    assert gb.lib().gb_debug_flow_plan(*head, *(v.ctypes.data for v in lanes), g.ctypes.data) == 0
    return info, *(v.reshape(-1, 32) for v in lanes), g


def hub(n, degrees, seed=1):
    """Rows of the given numbers of random lower neighbours, at the far end,
    and a path through the rest."""
    rng = np.random.default_rng(seed)
    r, c = list(range(1, n - len(degrees))), list(range(n - len(degrees) - 1))
    for k, deg in enumerate(degrees):
        i = n - len(degrees) + k
        r += [i] * deg
        c += list(rng.choice(i, deg, replace=False))
    return gen.laplacian_from_edges(n, np.array(c), np.array(r), rng.uniform(0.5, 1.5, len(r)), shift=0.5)


def shuffled(A, seed):
    """A with its rows in random order."""
    p = np.random.default_rng(seed).permutation(A.n)
    row = np.repeat(np.arange(A.n), np.diff(A.ia))
    up = row < A.ja
    return gen.laplacian_from_edges(A.n, p[row[up]], p[A.ja[up]], -A.a[up], shift=0.1)


GRAPHS = {
    "edges_of_32": lambda: hub(400, [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 34, 63, 64, 65, 95, 96, 97]),
    "hubs": lambda: hub(3000, [1024, 1055, 2000, 2900]),
    "star": lambda: hub(2500, [2499]),
    "one_row": lambda: gen.laplacian_from_edges(1, np.zeros(0, int), np.zeros(0, int), np.zeros(0), shift=1.0),
    "diagonal": lambda: gen.laplacian_from_edges(70, np.zeros(0, int), np.zeros(0, int), np.zeros(0), shift=1.0),
    "chung_lu": lambda: gen.chung_lu(3000, seed=5)[0],
    "shuffled_grid": lambda: shuffled(gen.grid3d(11), 3),
}


@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("name", GRAPHS)
def test_replay(name, lower):
    A = GRAPHS[name]()
    (nrec, nparts, nlev), col, out, vsrc, dsrc, g = plan(A, lower)
    n = A.n
    diag = A.a[[A.ia[i] + int(np.searchsorted(A.ja[A.ia[i]:A.ia[i + 1]], i)) for i in range(n)]]
    rhs = np.random.default_rng(9).standard_normal(n)
    val = np.full(n + nparts, np.nan)
    reads = np.zeros(n + nparts, int)
    used = np.zeros(A.nnz, int)
    for q in range(nrec):
        assert g[q] in (1, 2, 4, 8, 16, 32)
        new = {}
        for k in range(0, 32, g[q]):
            lane = slice(k, k + g[q])
            i = out[q, k]
            assert (out[q, lane] == i).all()
            if i < 0:
                assert (col[q, lane] < 0).all()
                continue
            owner = dsrc[q, k]
            assert (dsrc[q, lane] == owner).all() and (i == owner if i < n else i < n + nparts)
            s = 0.0
            for c, v in zip(col[q, lane], vsrc[q, lane]):
                if c < 0:
                    assert v == -1
                    continue
                assert not np.isnan(val[c])  # an earlier record wrote it
                reads[c] += 1
                if v >= 0:
                    assert A.ja[v] == c and A.ia[owner] <= v < A.ia[owner + 1]
                    used[v] += 1
                    s += A.a[v] / diag[owner] * val[c]
                else:
                    assert v == -2 and c >= n
                    s += val[c]
            new[i] = rhs[i] / diag[i] - s if i < n else s
        for i, v in new.items():
            assert np.isnan(val[i])
            val[i] = v
    row = np.repeat(np.arange(n), np.diff(A.ia))
    one_sided = (A.ja < row) if lower else (A.ja > row)
    assert (used == one_sided).all() and (reads[n:] == 1).all() and not np.isnan(val).any()
    want = np.zeros(n)
    for i in range(n) if lower else range(n - 1, -1, -1):
        e = np.arange(A.ia[i], A.ia[i + 1])[one_sided[A.ia[i]:A.ia[i + 1]]]
        want[i] = (rhs[i] - A.a[e] @ want[A.ja[e]]) / diag[i]
    assert np.allclose(val[:n], want, rtol=1e-10, atol=1e-12 * np.abs(want).max())
