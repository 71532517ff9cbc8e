"""The drainage network read back from caller-chosen receivers: levels, the
depth-first order, counts and donors against a walk in numpy, at the edges of
the blocks that scan the roots, on forests of single cells, long chains and
cycles."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = np.array([-1, -1, 0, 1, 1, 1, 0, -1])
DY = np.array([0, -1, -1, -1, 0, 1, 1, 1])


def forest(W, H, kind, seed):
    """Receiver codes (-1 none) of a forest: each interior cell drains towards
    a neighbour of smaller random key, or along a serpentine."""
    rec = np.full(W * H, -1, np.int32)
    rng = np.random.default_rng(seed)
    key = rng.permutation(W * H)
    for y in range(2, H - 2):
        for x in range(2, W - 2):
            c = y * W + x
            if kind == "serpentine":
                east = (y - 2) % 2 == 0
                end = W - 3 if east else 2
                rec[c] = 6 if x == end else (4 if east else 0)
            elif kind == "random":
                nb = c + DY * W + DX
                down = np.flatnonzero(key[nb] < key[c])
                if len(down) and rng.random() < 0.97:
                    rec[c] = down[rng.integers(len(down))]
    return rec


def walk(rec, W):
    """Levels, the Braun-Willett order and the starts of its trees."""
    n = rec.size
    to = np.where(rec < 0, -1, np.arange(n) + DY[rec] * W + DX[rec])
    kids = [[] for _ in range(n)]
    for c in range(n):
        if to[c] >= 0:
            kids[to[c]].append(c)
    level = np.zeros(n, np.int32)
    stack, starts = [], []
    for root in np.flatnonzero(to < 0):
        starts.append(len(stack))
        todo = [int(root)]
        while todo:
            c = todo.pop()
            if to[c] >= 0:
                level[c] = level[to[c]] + 1
            stack.append(c)
            todo.extend(reversed(kids[c]))
    return level, np.array(stack, np.int32), np.array(starts + [n], np.int32)


def inject(pkg, m, rec):
    return pkg.library().fs_test_order_from_receivers(
        m.handle, rec.ctypes.data_as(C.POINTER(C.c_int32)))


@pytest.mark.parametrize("W,H,kind", [
    (3, 3, "random"), (5, 5, "random"), (31, 33, "random"), (32, 32, "random"),
    (41, 25, "random"), (64, 31, "none"), (66, 70, "serpentine"), (257, 129, "random"),
    (200, 100, "serpentine")])
def test_network_of_given_receivers(pkg, W, H, kind):
    rec = forest(W, H, kind, W * H)
    level, stack, starts = walk(rec, W)
    with pkg.FastScape_RBP(W, H, params=pkg.workload_params()) as m:
        pkg.check(inject(pkg, m, rec))
        lv, nl = m.levels()
        st, ss = m.stack_dfs()
        np.testing.assert_array_equal(lv, level)
        assert nl == level.max() + 1
        np.testing.assert_array_equal(st, stack)
        np.testing.assert_array_equal(ss, starts)
        np.testing.assert_array_equal(m.receivers(), rec)
        cells = np.arange(W * H)
        np.testing.assert_array_equal(m.receiver_index(),
                                      np.where(rec < 0, cells, cells + DY[rec] * W + DX[rec]))
        count = np.ones(W * H)
        for c in stack[::-1]:
            if rec[c] >= 0:
                count[c + DY[rec[c]] * W + DX[rec[c]]] += count[c]
        np.testing.assert_array_equal(m.accumulation(), count * m.params.cell_area)


@pytest.mark.parametrize("loop", [[4, 0], [4, 6, 1], [4, 6, 0, 2]])
def test_cycles_are_reported(pkg, loop):
    W = H = 12
    rec = np.full(W * H, -1, np.int32)
    x = y = 5
    for k in loop:
        rec[y * W + x] = k
        x, y = x + DX[k], y + DY[k]
    assert (x, y) == (5, 5)
    rec[4 * W + 5] = 6  # and a path that runs into it
    with pkg.FastScape_RBP(W, H, params=pkg.workload_params()) as m:
        assert inject(pkg, m, rec) == -6
        assert pkg.library().fs_get_levels(m.handle, None, None) == -6
        m.step(2)
        assert np.all(np.isfinite(m.getH()))
