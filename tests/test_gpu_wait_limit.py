"""The limit on waits between blocks counts from the last progress of any tile:
a timestep that takes many times the limit is no reason to stop while tiles get
further. Paths that cross hundreds of tiles, few levels in each, and one long
path inside a tile that all other blocks of the queue wait for."""
import numpy as np
import pytest

from oracle.pyoracle import Params

pytestmark = pytest.mark.gpu


def channel(W, H):
    """A channel along the middle row, 1 cm a cell, between walls, to x = 1: one
    path of W cells."""
    h = np.full((H, W), 1e6)
    h[H // 2] = 0.01 * np.arange(W)
    return ring(h)


def snake(W, H):
    """Level ground but for a channel that snakes through the tile at x = 64,
    y = 32 and leaves it westward: a path of 870 cells, all in that tile."""
    h = np.zeros((H, W))
    h[31:66, 62:130] = 1000.0
    p, x, y = 1, 65, 34
    step = 1
    while y < 63:
        for x in range(65, 127)[::step]:
            h[y, x] = 1 + 0.01 * p
            p += 1
        h[y + 1, x] = 1 + 0.01 * p
        p += 1
        y += 2
        step = -step
    h[34, 62:65] = 0.5, 0.7, 0.9
    return ring(h)


def ring(h):
    h[:2] = h[-2:] = 0
    h[:, :2] = h[:, -2:] = 0
    return np.ascontiguousarray(h).reshape(-1)


@pytest.mark.parametrize("W,H,n,limit_ms,build", [
    (20000, 9, 1.0, 4.0, channel),   # 313 tiles, all on the GPU at once
    (192, 9824, 1.5, 2.0, snake)])   # 921 tiles: the queue
def test_a_long_path_is_progress(pkg, oracle, W, H, n, limit_ms, build):
    h = build(W, H)
    p = pkg.workload_params(neq=n)
    ref = oracle.phases(h.copy(), W, H, Params(*p.as_tuple()))
    assert len(ref["levels"]) > (15000 if build is channel else 800)
    with pkg.FastScape_RBP(W, H, params=p, init=pkg.INIT_ZERO) as m:
        m.setH(h)
        m.set_timing(pkg.TIMING_CALL)
        m.step(1)
        took = m.phase_times(reset=True)[3]
        m.setH(h)
        m.set_barrier_timeout(limit_ms)
        m.step(1)
        assert took > 2 * limit_ms  # or the limit tests nothing
        if n == 1.0:
            assert np.array_equal(m.getH(), ref["h"])
        else:
            np.testing.assert_allclose(m.getH(), ref["h"], rtol=1e-12, atol=0)
