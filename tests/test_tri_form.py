"""Which form the PCG solves a triangular factor in (tri_plan.cu): lock step,
value polling or the records, by what each is estimated to take.  The forms
named here are those measured fastest."""
import numpy as np
import pytest

import lap_gb300 as gb
from lap_gb300 import gen
from test_flow_plan import hub, shuffled
from test_step_plan import box, path

RECORDS, STEP, FLOW = range(3)


def forms(A):
    """(FP64 lower, FP64 upper, FP32 lower, FP32 upper)"""
    ia, ja = np.ascontiguousarray(A.ia, np.int32), np.ascontiguousarray(A.ja, np.int32)
    out = np.full(4, -1, np.int32)
    for k, (elem, lower) in enumerate(((8, 1), (8, 0), (4, 1), (4, 0))):
        assert gb.lib().gb_debug_tri_form(A.n, ia.ctypes.data, ja.ctypes.data, lower, elem, out[k:].ctypes.data) == 0
    return tuple(int(v) for v in out)


def reordered(A, p):
    """Row i of A becomes row p[i]."""
    row = np.repeat(np.arange(A.n), np.diff(A.ia))
    up = row < A.ja
    return gen.laplacian_from_edges(A.n, p[row[up]], p[A.ja[up]], -A.a[up], shift=0.1)


def red_black(nx, ny):
    A, i = box(nx, ny, 1), np.arange(nx * ny)
    p = np.empty(A.n, int)
    p[np.argsort((i % nx + i // nx) & 1, kind="stable")] = i
    return reordered(A, p)


def hubs(n_hubs, first, side=(50, 100), deg=500):
    """A grid with hubs of deg further neighbours each, as its first or last rows."""
    A = box(*side, 1)
    row = np.repeat(np.arange(A.n), np.diff(A.ia))
    up = row < A.ja
    rng = np.random.default_rng(2)
    at = rng.choice(np.arange(n_hubs + side[0] + 1, A.n), (n_hubs, deg), replace=False)
    ei = np.concatenate([row[up], np.repeat(np.arange(n_hubs), deg)])
    ej = np.concatenate([A.ja[up], at.ravel()])
    if not first:
        ei, ej = A.n - 1 - ei, A.n - 1 - ej
    return gen.laplacian_from_edges(A.n, ei, ej, rng.uniform(0.5, 1.5, len(ei)), shift=0.5)


def stencil27(nx, ny, nz):
    i = np.arange(nx * ny * nz)
    c = np.stack([i % nx, i // nx % ny, i // (nx * ny)])
    ei, ej = [], []
    for o in [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1) if (c, b, a) > (0, 0, 0)]:
        t = c + np.array(o)[:, None]
        ok = ((t >= 0) & (t < np.array([nx, ny, nz])[:, None])).all(0)
        ei.append(i[ok])
        ej.append((t[0] + nx * t[1] + nx * ny * t[2])[ok])
    ei, ej = np.concatenate(ei), np.concatenate(ej)
    return gen.laplacian_from_edges(len(i), ei, ej, np.ones(len(ei)), shift=0.5)


def blocks(count, k):
    """Separate k x k grids, one after another."""
    A = box(k, k, 1)
    row = np.repeat(np.arange(A.n), np.diff(A.ia))
    up = row < A.ja
    off = A.n * np.arange(count)[:, None]
    ei, ej = (row[up] + off).ravel(), (A.ja[up] + off).ravel()
    return gen.laplacian_from_edges(A.n * count, ei, ej, np.ones(len(ei)), shift=0.5)


CASES = {
    "20^3": (lambda: box(20, 20, 20), (STEP,) * 4),
    "64^3": (lambda: box(64, 64, 64), (STEP,) * 4),
    "97x61x83": (lambda: box(97, 61, 83), (STEP,) * 4),
    "100x100": (lambda: box(100, 100, 1), (STEP,) * 4),
    "1000x700": (lambda: box(1000, 700, 1), (STEP,) * 4),
    "path": (lambda: path(20000), (STEP,) * 4),
    "blocks_30x30": (lambda: blocks(110, 30), (STEP,) * 4),
    "shuffled_64x64": (lambda: shuffled(box(64, 64, 1), 1), (FLOW,) * 4),
    "shuffled_140x140": (lambda: shuffled(box(140, 140, 1), 1), (FLOW,) * 4),
    "shuffled_200x200": (lambda: shuffled(box(200, 200, 1), 1), (FLOW,) * 4),
    "shuffled_path": (lambda: shuffled(path(20000), 1), (FLOW,) * 4),
    "red_black_30x30": (lambda: red_black(30, 30), (FLOW,) * 4),
    "red_black_200x200": (lambda: red_black(200, 200), (FLOW,) * 4),
    "diagonal": (lambda: blocks(20000, 1), (FLOW,) * 4),
    "chung_lu": (lambda: gen.chung_lu(20000, seed=5)[0], (FLOW,) * 4),
    "27_point": (lambda: stencil27(30, 30, 30), (FLOW,) * 4),
    "all_hubs": (lambda: shuffled(hub(6000, [1024, 1055, 2000, 5900]), 2), (FLOW,) * 4),
    "20000x6": (lambda: box(20000, 6, 1), (RECORDS, RECORDS, STEP, STEP)),
    "45000x3": (lambda: box(45000, 3, 1), (RECORDS,) * 4),
    "148x148x20": (lambda: box(148, 148, 20), (RECORDS, RECORDS, STEP, STEP)),
    "300x300x4": (lambda: box(300, 300, 4), (RECORDS,) * 4),
    "hub_first": (lambda: hubs(1, True), (STEP, RECORDS) * 2),
    "hub_last": (lambda: hubs(1, False), (RECORDS, STEP) * 2),
    "hubs_first": (lambda: hubs(8, True), (STEP, FLOW) * 2),
    "hubs_last": (lambda: hubs(8, False), (FLOW, STEP) * 2),
}


@pytest.mark.parametrize("name", CASES)
def test_form(name):
    make, want = CASES[name]
    assert forms(make()) == want


@pytest.mark.parametrize("name,want", [
    ("GBLAP_TRI_FORM", (RECORDS,) * 4),
    ("GBLAP_TRI_TILE_ROWS", (RECORDS,) * 4),  # the FP32 tile follows it
    ("GBLAP_TRI_TILE_ROWS32", (STEP, STEP, RECORDS, RECORDS)),
    ("GBLAP_TRI_FIXED", (STEP, STEP, RECORDS, RECORDS)),
    ("GBLAP_TRI_FP64_CLUSTER", (RECORDS, RECORDS, STEP, STEP)),
])
def test_a_setting_keeps_the_records_it_speaks_of(name, want, monkeypatch):
    monkeypatch.setenv(name, "1024")
    assert forms(box(20, 20, 20)) == want


def test_bad_input():
    A = path(4)
    f = np.zeros(1, np.int32)
    ia, ja = A.ia.astype(np.int32), A.ja.astype(np.int32)
    args = (A.n, ia.ctypes.data, ja.ctypes.data, 1, 8, f.ctypes.data)
    for k, bad in ((0, 0), (1, None), (2, None), (4, 5), (5, None)):
        assert gb.lib().gb_debug_tri_form(*args[:k], bad, *args[k + 1:]) == 5  # GB_BAD_INPUT
