"""The LU's interchanges as gathers, restated in NumPy: positions instead of moved rows, and the moves of a sub-panel."""
import numpy as np
import pytest


def swaps(n, r0, w, piv):
    """Row at every position after the interchanges k <-> piv[k], one by one (LAPACK's laswp)."""
    rows = np.arange(n)
    for k in range(w):
        p = piv[k]
        rows[[r0 + k, p]] = rows[[p, r0 + k]]
    return rows


def moves_by_position(n, r0, w, piv):
    """Every row's thread tracks its position (panel_reg_kernel)."""
    pos = np.arange(n)
    for k in range(w):
        at_piv, at_k = pos == piv[k], pos == r0 + k
        pos[at_k & ~at_piv] = piv[k]
        pos[at_piv] = r0 + k
    src, dst = np.empty(w, int), np.empty(w, int)
    for row in range(r0, n):
        if pos[row] < r0 + w:
            src[pos[row] - r0] = row
        if row < r0 + w:
            dst[row - r0] = pos[row]
    return src, dst


def moves_from_pivots(r0, w, piv):
    """From the pivots alone (moves_kernel)."""
    top, out_row, out_of = list(range(r0, r0 + w)), [], []
    for k in range(w):
        p = piv[k]
        if p < r0 + w:
            top[k], top[p - r0] = top[p - r0], top[k]
            continue
        if p not in out_row:
            out_row.append(p)
            out_of.append(p)
        e = out_row.index(p)
        top[k], out_of[e] = out_of[e], top[k]
    src, dst = np.array(top), np.full(w, -1)
    for k in range(w):
        if top[k] < r0 + w:
            dst[top[k] - r0] = r0 + k
    for row, of in zip(out_row, out_of):
        if of < r0 + w:
            dst[of - r0] = row
    return src, dst


@pytest.mark.parametrize("n,r0,w", [(40, 0, 16), (40, 8, 16), (16, 0, 16), (17, 1, 16), (64, 32, 32), (9, 4, 5), (1, 0, 1)])
def test_moves_equal_the_interchanges(n, r0, w):
    rng = np.random.default_rng(n + w)
    for _ in range(200):
        few = rng.random() < 0.5  # the same few rows again and again
        piv = [int(rng.integers(r0 + k, n if not few else min(n, r0 + k + 3))) for k in range(w)]
        want = swaps(n, r0, w, piv)
        src, dst = moves_by_position(n, r0, w, piv)
        src2, dst2 = moves_from_pivots(r0, w, piv)
        assert np.array_equal(src, src2) and np.array_equal(dst, dst2)
        rows = np.arange(n)
        got = rows.copy()
        for k in range(w):  # all loads before any store
            if dst[k] >= r0 + w:
                got[dst[k]] = rows[r0 + k]
            got[r0 + k] = rows[src[k]]
        assert np.array_equal(got, want)
