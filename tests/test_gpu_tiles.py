"""The tile walk at the sizes where it can go wrong: grids that end at, one cell
short of and one cell past a 64 x 32 tile, grids a few cells wide, a grid of
more tiles than fit the GPU at once (trees rooted in their tile, then the
others, pulled or from the queue of tiles) and subsets of a batch of such
grids -- receivers, level ids, drainage and elevation against the oracle's
timestep. n = 1 bit for bit; n = 2 within 1e-12 relative per timestep, as in
test_gpu_parity.py."""
import numpy as np
import pytest

from oracle.pyoracle import Params

pytestmark = pytest.mark.gpu


def field(W, H, kind, seed=5):
    """"young": noise, paths of a dozen cells. "deep": a cone with noise, paths
    of half the grid's width that cross many tiles."""
    rng = np.random.default_rng(seed)
    yy, xx = np.divmod(np.arange(W * H), W)
    h = rng.uniform(0, 1 if kind == "young" else 3, W * H)
    if kind == "deep":
        h += 5.0 * np.minimum.reduce([xx, yy, W - 1 - xx, H - 1 - yy])
    h[(xx <= 1) | (yy <= 1) | (xx >= W - 2) | (yy >= H - 2)] = 0
    return h


@pytest.mark.parametrize("kind", ["young", "deep"])
@pytest.mark.parametrize("W,H,n", [(64, 32, 1), (63, 31, 1), (65, 33, 1), (128, 64, 2),
                                   (191, 97, 1), (5, 300, 1), (700, 5, 1), (1601, 1483, 1)])
def test_timesteps_equal_the_oracle(pkg, oracle, W, H, n, kind):
    p = pkg.workload_params() if n == 1 else pkg.reference_params()
    op = Params(*p.as_tuple())
    h = field(W, H, kind)
    with pkg.FastScape_RBP(W, H, params=p, init=pkg.INIT_ZERO) as m:
        m.setH(h)
        for s in range(2):
            if n != 1:
                m.setH(h)
            m.step(1)
            ref = oracle.phases(h, W, H, op)
            assert np.array_equal(m.receivers(), ref["rec"]), s
            assert np.array_equal(m.levels()[0], ref["level_id"]), s
            assert np.array_equal(m.accumulation(), ref["accum"]), s
            if n == 1:
                assert np.array_equal(m.getH(), ref["h"]), s
            else:
                np.testing.assert_allclose(m.getH(), ref["h"], rtol=1e-12, atol=0)
            h = ref["h"]


@pytest.mark.parametrize("W,H", [(1024, 608), (320, 1952), (1216, 1024), (1344, 928),
                                 (1536, 1216), (704, 2656)])
def test_block_widths(pkg, oracle, W, H):
    """The most tiles that blocks of each width hold on 152 SMs (two, four and
    six to an SM), and one more: wide levels and narrow ones in one grid."""
    p = pkg.workload_params()
    op = Params(*p.as_tuple())
    h = field(W, H, "young")
    h.reshape(H, W)[:, W // 2:] += field(W, H, "deep").reshape(H, W)[:, W // 2:]
    with pkg.FastScape_RBP(W, H, params=p, init=pkg.INIT_ZERO) as m:
        m.setH(h)
        m.step(1)
        ref = oracle.phases(h, W, H, op)
        assert np.array_equal(m.receivers(), ref["rec"])
        assert np.array_equal(m.accumulation(), ref["accum"])
        assert np.array_equal(m.getH(), ref["h"])


def test_subset_of_large_grids(pkg):
    """A subset of a batch, its tiles in a list: the others keep their fields."""
    sides = [(900, 800), (1000, 700), (1100, 900), (70, 90)]
    p = pkg.workload_params()
    kinds = ["young", "deep", "deep", "young"]
    with pkg.FastScapeBatch([w for w, _ in sides], [h for _, h in sides], [p] * 4) as b:
        singles = []
        for r, (w, h) in enumerate(sides):
            f = field(w, h, kinds[r], seed=r)
            b.setH(r, f)
            m = pkg.FastScape_RBP(w, h, params=p, init=pkg.INIT_ZERO)
            m.setH(f)
            singles.append(m)
        for subset in ([2, 0, 3], [1], [3, 1, 0, 2]):
            b.set_active(subset)
            b.step(2)
            for r in subset:
                singles[r].step(2)
            for r in range(4):
                assert np.array_equal(b.getH(r), singles[r].getH()), (subset, r)
            for r in subset:
                assert np.array_equal(b.accumulation(r), singles[r].accumulation()), (subset, r)
        for m in singles:
            m.close()


@pytest.mark.parametrize("W,H", [(5, 5), (8, 7), (100, 100), (156, 260), (157, 260), (400, 300)])
@pytest.mark.parametrize("ground", ["flat", "terraces", "tiny"])
def test_queued_receivers(pkg, oracle, W, H, ground):
    """Ground that the FP32 filter leaves open, cell by cell: eight threads a
    cell up to 38912 of them (156 x 260 flat), one above; several timesteps, so
    that a queue left over from the one before would show."""
    rng = np.random.default_rng(W * H)
    h = {"flat": np.zeros(W * H), "terraces": rng.integers(0, 3, W * H).astype(float),
         "tiny": 1 + rng.integers(0, 4, W * H) * 2.0**-52}[ground]
    hh = h.reshape(H, W)
    hh[:2] = hh[-2:] = 0
    hh[:, :2] = hh[:, -2:] = 0
    p = pkg.workload_params()
    op = Params(*p.as_tuple())
    with pkg.FastScape_RBP(W, H, params=p, init=pkg.INIT_ZERO) as m:
        m.setH(h)
        for s in range(3):
            m.step(1)
            ref = oracle.phases(h, W, H, op)
            assert np.array_equal(m.receivers(), ref["rec"]), s
            assert np.array_equal(m.getH(), ref["h"]), s
            h = ref["h"]
        m.setH(h)
        m.step(3)
        for s in range(3):
            h = oracle.phases(h, W, H, op)["h"]
        assert np.array_equal(m.getH(), h)


@pytest.mark.parametrize("W,H", [(36, 36), (37, 37), (420, 1060), (420, 1064), (612, 772),
                                 (612, 773)])
def test_receiver_tile_rows(pkg, oracle, W, H):
    """Receiver tiles of 32 rows up to 151 of 96 rows, and of 96 beyond: grids
    at the edge of a tile and around the line between the two."""
    p = pkg.workload_params()
    op = Params(*p.as_tuple())
    h = field(W, H, "young")
    with pkg.FastScape_RBP(W, H, params=p, init=pkg.INIT_ZERO) as m:
        for tma in (False, True) if W % 2 == 0 else (False,):  # rows of whole 16 bytes
            m.setH(h)
            pkg.check(pkg.library().fs_use_tma_staging(m.handle, int(tma)))
            m.step(1)
            ref = oracle.phases(h, W, H, op)
            assert np.array_equal(m.receivers(), ref["rec"]), tma
            assert np.array_equal(m.getH(), ref["h"]), tma
