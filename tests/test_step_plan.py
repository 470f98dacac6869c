"""The lock-step triangular solves' plan (tri_step.h), replayed on the CPU.

The plan resolves every dependency to a place in shared memory: a window of
the tile's own values, reused in step order, or an inbox the previous tile
fills.  The replay walks it as the kernel does -- each step reads all its
places before it writes -- and checks that every place read holds exactly the
row the matrix names, that indices stay inside their arrays, and that each
row is solved once with each of its entries.
"""
import ctypes as C

import numpy as np
import pytest

import lap_gb300 as gb
from lap_gb300 import gen

PAGE, CHUNK = 128, 192


def plan(A, lower, elem, tile_rows=0):
    L = gb.lib()
    ia, ja = np.ascontiguousarray(A.ia, np.int32), np.ascontiguousarray(A.ja, np.int32)
    info = np.zeros(12, np.int32)
    head = (A.n, ia.ctypes.data, ja.ctypes.data, int(lower), elem, tile_rows, info.ctypes.data)
    rc = L.gb_debug_step_plan(*head, *[None] * 6)
    if rc:
        return rc
    tiles = np.zeros((info[0], 8), np.int32)
    ends = np.zeros(info[8], np.uint16)
    meta = np.zeros((info[7] * PAGE, 4), np.uint32)
    src = np.zeros((info[7] * PAGE, 4), np.int32)
    needs, thr = np.zeros(info[7], np.uint16), np.zeros(info[11], np.uint16)
    out = (tiles, ends, meta, src, needs, thr)
    assert L.gb_debug_step_plan(*head, *(v.ctypes.data for v in out)) == 0
    keys = ("tiles", "rows", "nw", "np", "window", "inbox", "max_steps", "pages", "steps", "smem", "nat", "chunks")
    return dict(zip(keys, (int(v) for v in info))), *out


def replay(A, lower, elem, tile_rows=0):
    info, tiles, ends, meta, src, needs, thr = plan(A, lower, elem, tile_rows)
    window, inbox, nat = info["window"], info["inbox"], info["nat"]
    assert (nat or window & (window - 1) == 0) and window + inbox + 1 <= 65535
    assert info["smem"] <= 231168 and info["np"] in (8, 16, 32) and info["max_steps"] == tiles[:, 5].max()
    rows_of = np.repeat(np.arange(A.n), np.diff(A.ia))
    solved = np.zeros(A.n, int)
    used = np.zeros(A.nnz, int)
    before = np.full(inbox, -1)  # what the previous tile pushed: row by inbox place
    for q in range(info["tiles"]):
        row0, npos, page0, npages, step0, nsteps, nexp, thr0 = tiles[q]
        assert 0 < npos <= npages * PAGE and nexp <= inbox
        held = np.concatenate([np.full(window, -1), before, [-2]])
        pushed = np.full(inbox, -1)
        # natural order: where a row lies, which chunk it is loaded and stored in
        i = np.arange(npos)
        place_of = (i & ~31) | ((i + 3 * (i >> 5)) & 31)
        chunk_of = (i if lower else npos - 1 - i) // CHUNK
        if nat:
            assert len(np.unique(place_of)) == npos and place_of.max() < window
        at = np.zeros(npos, int)  # position of each row
        a = 0
        for s in range(step0, step0 + nsteps):
            b = int(ends[s])
            assert a < b <= min(npos, a + 32 * info["nw"])
            P = page0 * PAGE + np.arange(a, b)
            place = np.stack([meta[P, 0] & 0xffff, meta[P, 0] >> 16, meta[P, 1] & 0xffff, meta[P, 1] >> 16], 1)
            own = (meta[P, 2] & 0xffff).astype(int)
            row = row0 + (np.argsort(place_of)[np.searchsorted(np.sort(place_of), own)] if nat else own)
            at[row - row0] = np.arange(a, b)
            if nat:
                assert (place_of[row - row0] == own).all()
                assert (needs[page0 + np.arange(a, b) // PAGE] > chunk_of[row - row0]).all()
            assert place.max() <= window + inbox
            got = held[place]
            for k in range(4):
                there = src[P, k] >= 0
                np.testing.assert_array_equal(got[there, k], A.ja[src[P, k][there]])
                np.testing.assert_array_equal(row[there], rows_of[src[P, k][there]])
                assert (got[~there, k] == -2).all()  # no entry: the zero place
                used[src[P, k][there]] += 1
            # no place read in a step is written in it: its warps are not ordered
            written = own if nat else np.arange(a, b) & (window - 1)
            assert not np.isin(written, place[place < window]).any()
            held[written] = row
            ex = (meta[P, 2] >> 16).astype(int)
            out = ex != 0xffff
            assert (ex[out] < nexp).all()
            pushed[ex[out]] = row[out]
            solved[row] += 1
            a = b
        assert a == npos and (pushed[:nexp] >= 0).all()
        for c in range(chunk_of.max() + 1 if nat else 0):
            assert thr[thr0 + c] == at[chunk_of == c].max() + 1
        before = pushed
    assert (solved == 1).all()
    want = A.ja < rows_of if lower else A.ja > rows_of
    np.testing.assert_array_equal(used, want.astype(int))
    return info


def box(nx, ny, nz):
    idx = np.arange(nx * ny * nz).reshape(nz, ny, nx)
    e = [(idx[:, :, :-1], idx[:, :, 1:]), (idx[:, :-1], idx[:, 1:]), (idx[:-1], idx[1:])]
    ei, ej = (np.concatenate([p[k].ravel() for p in e]) for k in (0, 1))
    return gen.laplacian_from_edges(nx * ny * nz, ei, ej, np.ones(len(ei)), shift=1.0)


def path(n, step=1):
    return gen.laplacian_from_edges(n, np.arange(n - step), np.arange(step, n), np.ones(n - step), shift=1.0)


def local_random(n, near, seed):
    """Up to four dependencies a row on either side, at random distances <= near."""
    rng = np.random.default_rng(seed)
    i = np.arange(n - 1)
    j = np.minimum(i + rng.integers(1, near + 1, n - 1), n - 1)
    k = np.concatenate([i * n + j, (i * n + i + 1)])
    k = np.unique(k)
    up = k // n, k % n
    deg = np.bincount(up[1], minlength=n)
    keep = deg[up[1]] <= 4
    return gen.laplacian_from_edges(n, up[0][keep], up[1][keep], np.ones(int(keep.sum())), shift=1.0)


@pytest.mark.parametrize("elem", [4, 8])
@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 1), (33, 1, 1), (7, 5, 1), (40, 37, 1), (20, 20, 20), (31, 9, 23),
                                   (5, 3, 61)])
def test_grids(shape, lower, elem):
    replay(box(*shape), lower, elem)


@pytest.mark.parametrize("rows", [35, 64, 127, 128, 129, 700])
@pytest.mark.parametrize("lower", [True, False])
def test_tile_heights(rows, lower):
    """Heights that cut planes anywhere, down to the band itself."""
    A = box(7, 5, 40)
    info = replay(A, lower, 4, rows)
    assert info["rows"] == rows


@pytest.mark.parametrize("lower", [True, False])
def test_other_local_graphs(lower):
    for A in (path(1), path(300), path(3000, 3), local_random(2000, 40, 1), local_random(5000, 700, 2)):
        replay(A, lower, 8)


def test_wide_levels_take_several_steps():
    A = path(4000, 2000)  # two levels of 2000 rows
    info = replay(A, True, 4, 4000)
    assert info["nw"] == 8 and info["steps"] == 2 * -(-2000 // 256)


def test_factors_that_keep_their_records():
    rng = np.random.default_rng(3)
    far = gen.laplacian_from_edges(200000, np.arange(100000), np.arange(100000, 200000), np.ones(100000), shift=1.0)
    assert plan(far, True, 4) == 8  # the previous tile's exports would not fit beside it
    assert plan(gen.knn_graph(300, rng=rng), True, 4) == 8  # rows of more than four dependencies
