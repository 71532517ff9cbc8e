"""The per-realization walk, which a caller asks for or the autotuner chooses:
blocks of every width (by the realizations an SM has to hold), every n, both
subtractions, more levels than a block keeps in shared memory, growing tables
and subsets, bit for bit against the tile walk of the same batch, and n = 1
against the oracle. walk_mode says which of the two runs."""
import numpy as np
import pytest

from oracle.pyoracle import Params
from test_gpu_parity import serpentine, valley

pytestmark = pytest.mark.gpu

SIZES = [(40, 33), (3, 9), (64, 32), (5, 5), (70, 45), (12, 50), (97, 20)]


def pair(pkg, sides, n, seed=0):
    """Two equal batches, the second asked for the per-realization walk."""
    rng = np.random.default_rng(seed)
    ps = [pkg.workload_params(keq=10 ** rng.uniform(-6, -5), meq=rng.uniform(0.3, 0.6),
                              ueq=10 ** rng.uniform(-4, -2.3), neq=n) for _ in sides]
    two = [pkg.FastScapeBatch([w for w, _ in sides], [h for _, h in sides], ps,
                              init=pkg.INIT_PHILOX, seeds=list(range(len(sides))))
           for _ in range(2)]
    two[1].use_cta_walk(True)
    return two[0], two[1], ps


def same(a, c, rs):
    for r in rs:
        assert np.array_equal(a.receivers(r), c.receivers(r)), r
        assert np.array_equal(a.accumulation(r), c.accumulation(r)), r
        assert np.array_equal(a.levels(r)[0], c.levels(r)[0]), r
        assert np.array_equal(a.getH(r), c.getH(r)), r


@pytest.mark.parametrize("reals", [3, 310, 620])
@pytest.mark.parametrize("n,int_sub", [(1.0, False), (1.0, True), (2.0, False), (2.0, True),
                                       (1.5, False)])
def test_widths(pkg, oracle, reals, n, int_sub):
    sides = [SIZES[r % len(SIZES)] for r in range(reals)]
    a, c, ps = pair(pkg, sides, n, seed=reals)
    with a, c:
        c.use_int_sub(int_sub)
        assert c.launch_config()["cta_walk"] and not a.launch_config()["cta_walk"]
        start = [c.getH(r) for r in range(3)]
        for k in (1, 3):
            a.step(k)
            c.step(k)
            same(a, c, range(0, reals, max(1, reals // 40)))
        if n == 1.0:
            for r in range(3):
                ref = oracle.steps(start[r], *sides[r], Params(*ps[r].as_tuple()), 4)
                assert np.array_equal(c.getH(r), ref), r
        subset = list(range(reals - 1, 0, -2))
        a.set_active(subset)
        c.set_active(subset)
        assert c.launch_config()["cta_walk"]
        a.step(2)
        c.step(2)
        same(a, c, range(0, reals, max(1, reals // 40)))


@pytest.mark.parametrize("reals", [2, 320, 640])
@pytest.mark.parametrize("n", [1.0, 2.0])
def test_many_levels_and_growing_tables(pkg, reals, n):
    """One realization of 2489 levels, one whose counts outgrow its table, with
    subsets that number them anew."""
    sides = [(120, 50), (420, 400)] + [SIZES[r % len(SIZES)] for r in range(reals - 2)]
    sides[0], sides[-1] = sides[-1], sides[0]
    v = sides.index((420, 400))
    s = sides.index((120, 50))
    a, c, ps = pair(pkg, sides, n, seed=reals)
    with a, c:
        for b in (a, c):
            b.setH(s, serpentine(120, 50))
            b.setH(v, valley(420, 400))
            b.set_active([v, s])
        a.step(1)
        c.step(1)
        same(a, c, [s, v])
        assert c.levels(s)[1] > 2048
        assert c.accumulation(v).max() / ps[v].cell_area > 65536
        for b in (a, c):
            b.set_active(None)
            b.step(2)
        same(a, c, [0, s, v, reals - 1])


def test_the_autotuners_choice(pkg):
    """Chosen by size, used where the tiles do not fit the GPU at once, asked
    for it is used all the same."""
    torch = pytest.importorskip("torch")
    room = 6 * torch.cuda.get_device_properties(0).multi_processor_count
    few, many = 4, room // 64 + 2  # 256^2: 32 tiles; 500^2: 128
    p = pkg.workload_params()
    with pkg.FastScapeBatch([500] * many, [500] * many, [p] * many,
                            seeds=list(range(many))) as b:
        b.autotune(1)
        assert many * 128 > room and b.launch_config()["cta_walk"]
        b.set_active(list(range(few)))
        assert few * 128 < room and not b.launch_config()["cta_walk"]
        b.use_cta_walk(True)
        assert b.launch_config()["cta_walk"]
    with pkg.FastScapeBatch([256] * few, [256] * few, [p] * few, seeds=list(range(few))) as b:
        b.autotune(1)
        assert not b.launch_config()["cta_walk"]


@pytest.mark.parametrize("w,n,cta", [(122, 1.0, False), (122, 2.0, True), (122, 1.5, True),
                                     (300, 2.0, False)])
def test_the_autotuners_line_for_small_realizations(pkg, w, n, cta):
    """Tiles that fit the GPU in blocks of 128 threads only, five to an SM: for
    n != 1 the per-realization walk if none has more than eight tiles."""
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per = (w + 63) // 64 * 4
    reals = 5 * sms // per
    p = pkg.workload_params(neq=n)
    with pkg.FastScapeBatch([w] * reals, [98] * reals, [p] * reals, init=pkg.INIT_PHILOX,
                            seeds=list(range(reals))) as b, \
            pkg.FastScape_RBP(w, 98, params=p, init=pkg.INIT_PHILOX, seed=1) as m:
        b.autotune(1)
        assert b.launch_config()["cta_walk"] == cta
        b.step(3)
        m.step(3)
        assert np.array_equal(b.getH(1), m.getH())
