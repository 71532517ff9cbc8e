"""Launches of more tiles than the GPU holds at once, whose trees are rooted in
their tile, pulled, or eroded from the queue of tiles, in the forms that the
smaller grids of the other files never take there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def field(W, H, kind, seed):
    """As test_gpu_tiles.py's: noise, or a cone with noise."""
    rng = np.random.default_rng(seed)
    yy, xx = np.divmod(np.arange(W * H), W)
    h = rng.uniform(0, 1 if kind == "young" else 3, W * H)
    if kind == "deep":
        h += 5.0 * np.minimum.reduce([xx, yy, W - 1 - xx, H - 1 - yy])
    h[(xx <= 1) | (yy <= 1) | (xx >= W - 2) | (yy >= H - 2)] = 0
    return h


def tiles(sides):
    return sum((w + 63) // 64 * ((h + 31) // 32) for w, h in sides)


def most_resident():
    """Tiles that the GPU holds at once: six blocks on an SM."""
    torch = pytest.importorskip("torch")
    return 6 * torch.cuda.get_device_properties(0).multi_processor_count


SIDES = [(300, 200), (1400, 1100), (1000, 700)]


@pytest.mark.parametrize("before", ["nothing", "another batch", "a failed timestep"])
@pytest.mark.parametrize("kinds", [("young", "deep", "young"), ("deep", "young", "young")])
def test_strict_subset_from_the_queue(pkg, before, kinds):
    """The first timesteps of a subset that leaves realization 0 out, in memory
    just allocated, in memory that another batch's tiles and queue lay in, and
    after a timestep that an error of realization 0 stopped while tiles of the
    others were queued. The others must evolve as models of their own, and
    realization 0 must not change."""
    assert tiles(SIDES[1:]) > most_resident()
    p = pkg.workload_params()
    ps = [p, p, p]
    if before == "a failed timestep":
        ps[0] = pkg.workload_params(ueq=1e306)  # uplifted to infinity
    if before == "another batch":
        with pkg.FastScape_RBP(1700, 1500, params=p, init=pkg.INIT_ZERO) as m:
            m.setH(field(1700, 1500, "deep", 9))
            m.step(2)
    fields = [field(w, h, k, 20 + r) for r, ((w, h), k) in enumerate(zip(SIDES, kinds))]
    with pkg.FastScapeBatch([w for w, _ in SIDES], [h for _, h in SIDES], ps,
                            init=pkg.INIT_ZERO) as b:
        for r in range(3):
            b.setH(r, fields[r])
        if before == "a failed timestep":
            with pytest.raises(pkg.FastScapeError) as e:
                b.step(1)
            assert e.value.status == -5
            for r in range(3):
                b.setH(r, fields[r])
        b.set_active([1, 2])
        b.step(2)
        assert np.array_equal(b.getH(0), fields[0])
        for r in (1, 2):
            with pkg.FastScape_RBP(*SIDES[r], params=p, init=pkg.INIT_ZERO) as m:
                m.setH(fields[r])
                m.step(2)
                assert np.array_equal(b.getH(r), m.getH()), r
                assert np.array_equal(b.receivers(r), m.receivers()), r
                assert np.array_equal(b.accumulation(r), m.accumulation()), r


@pytest.mark.parametrize("kind", ["young", "deep"])
@pytest.mark.parametrize("n", [1.0, 2.0])
def test_erosion_paths_agree(pkg, n, kind):
    """Every arithmetic of the erosion on more tiles than fit the GPU: the
    integer subtractions and the FP64 ones against the reference's Newton loop
    taken literally, bit for bit."""
    W, H = 1601, 1483
    assert tiles([(W, H)]) > most_resident()
    p = pkg.workload_params() if n == 1.0 else pkg.reference_params()
    h = field(W, H, kind, 31)
    out = []
    for int_sub, literal in ((0, 0), (1, 0), (0, 1)):
        with pkg.FastScape_RBP(W, H, params=p, init=pkg.INIT_ZERO) as m:
            pkg.check(pkg.library().fs_use_int_sub(m.handle, int_sub))
            pkg.check(pkg.library().fs_test_set_erosion_path(m.handle, literal))
            m.setH(h)
            m.step(3)
            out.append((m.getH(), m.accumulation()))
    for g, acc in out[:2]:
        assert np.array_equal(g, out[2][0])
        assert np.array_equal(acc, out[2][1])


@pytest.mark.parametrize("kind", ["young", "deep"])
@pytest.mark.parametrize("n", [2.0, 1.5])
def test_steeper_exponents_against_the_oracle(pkg, oracle, n, kind):
    """n = 2 and a general n there, each timestep from the oracle's ground,
    within test_gpu_parity.py's 1e-12 for n != 1."""
    from oracle.pyoracle import Params
    W, H = 1601, 1483
    p = pkg.reference_params() if n == 2.0 else pkg.workload_params(neq=n)
    h = field(W, H, kind, 32)
    with pkg.FastScape_RBP(W, H, params=p, init=pkg.INIT_ZERO) as m:
        for s in range(2):
            m.setH(h)
            m.step(1)
            ref = oracle.phases(h.copy(), W, H, Params(*p.as_tuple()))
            assert np.array_equal(m.receivers(), ref["rec"]), s
            assert np.array_equal(m.accumulation(), ref["accum"]), s
            np.testing.assert_allclose(m.getH(), ref["h"], rtol=1e-12, atol=0)
            h = ref["h"]


def test_general_exponent_on_many_tiles(pkg, oracle):
    """From 4096 tiles on, a general n's wide levels are eroded in their tiles."""
    from oracle.pyoracle import Params
    W, H = 2100, 4100
    assert tiles([(W, H)]) > 4096
    p = pkg.workload_params(neq=1.5)
    h = field(W, H, "young", 33)
    ref = oracle.phases(h.copy(), W, H, Params(*p.as_tuple()))
    with pkg.FastScape_RBP(W, H, params=p, init=pkg.INIT_ZERO) as m:
        m.setH(h)
        m.step(1)
        assert np.array_equal(m.accumulation(), ref["accum"])
        np.testing.assert_allclose(m.getH(), ref["h"], rtol=1e-12, atol=0)


@pytest.mark.parametrize("int_sub", [0, 1])
def test_rounds_of_the_whole_gpu(pkg, oracle, int_sub):
    """n = 1 with more than 8.4e6 cells in trees that leave their tile: nearly
    all of the deep part's 13e6, beside young ground whose cells are pulled. A
    batch's subset and the oracle."""
    from oracle.pyoracle import Params
    W, H = 4500, 3600
    p = pkg.workload_params()
    h = field(W, H, "young", 41)
    hh = h.reshape(H, W)
    hh[:, :3700] = field(3700, H, "deep", 42).reshape(H, 3700)
    ref = h.copy()
    for _ in range(2):
        ref = oracle.phases(ref, W, H, Params(*p.as_tuple()))["h"]
    small = field(70, 90, "deep", 43)
    with pkg.FastScapeBatch([70, W], [90, H], [p, p], init=pkg.INIT_ZERO) as b:
        b.use_int_sub(int_sub)
        b.setH(0, small)
        b.setH(1, h)
        b.set_active([1])
        b.step(2)
        assert np.array_equal(b.getH(0), small)
        assert np.array_equal(b.getH(1), ref)
        b.setH(1, h)
        b.set_active(None)
        b.step(2)
        assert np.array_equal(b.getH(1), ref)


@pytest.mark.parametrize("W,H", [(8, 32000), (5, 52000)])
@pytest.mark.parametrize("n", [1.0, 2.0])
def test_narrow_grids_on_the_callers_buffer(pkg, W, H, n):
    """The static scratch at its most tiles: as an allocating model."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    assert tiles([(W, H)]) > most_resident()
    p = pkg.workload_params(neq=n)
    h = field(W, H, "deep", 51)
    d = torch.from_numpy(h.copy()).cuda()
    f = pkg.library().fs_step_noalloc
    f.argtypes = [C.c_void_p, C.c_int, C.c_int, C.POINTER(pkg.Params), C.c_int, C.c_void_p]
    assert f(C.c_void_p(d.data_ptr()), W, H, C.byref(p), 3, None) == 0, pkg.last_error()
    with pkg.FastScape_RBP(W, H, params=p, init=pkg.INIT_ZERO) as m:
        m.setH(h)
        m.step(3)
        assert np.array_equal(d.cpu().numpy(), m.getH())
