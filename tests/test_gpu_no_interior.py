"""Grids without an interior (fewer than five cells one way) have no receivers:
a timestep changes nothing, every cell drains itself. Alone, beside others in a
batch, on the caller's own buffer, and the tallest that the limit on the cell
count admits."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def field(W, H, seed=1):
    h = np.random.default_rng(seed).uniform(0, 1, (H, W))
    h[:2] = h[-2:] = 0
    h[:, :2] = h[:, -2:] = 0
    return h.reshape(-1)


def check(pkg, b, r, W, H, h):
    n = W * H
    assert np.array_equal(b.getH(r), h)
    assert np.array_equal(b.receivers(r), np.full(n, -1, np.int32))
    assert np.array_equal(b.accumulation(r), np.full(n, pkg.workload_params().cell_area))
    assert np.array_equal(b.levels(r)[0], np.zeros(n, np.int32)) and b.levels(r)[1] == 1


@pytest.mark.parametrize("W,H", [(3, 3), (4, 4), (3, 1000), (4, 999), (1000, 3), (700, 4), (5, 4)])
def test_alone(pkg, W, H):
    p = pkg.workload_params()
    h = np.random.default_rng(2).uniform(0, 5, W * H)
    with pkg.FastScape_RBP(W, H, params=p, init=pkg.INIT_ZERO) as m:
        m.setH(h)
        m.step(3)
        assert m.steps_executed() == 3
        m.autotune(1)
        m.set_timing(pkg.TIMING_KERNELS)
        m.step(1)
        m.set_timing(pkg.TIMING_CALL)
        m.step(1)
        assert m.steps_executed() == 5
        assert np.array_equal(m.getH(), h)
        assert np.array_equal(m.receivers(), np.full(W * H, -1))
        assert np.array_equal(m.receiver_index(), np.arange(W * H))
        assert np.array_equal(m.accumulation(), np.full(W * H, p.cell_area))
        assert np.array_equal(m.donor_mask(), np.zeros(W * H))
        assert m.levels()[1] == 1
        stack, starts = m.stack_dfs()
        assert np.array_equal(stack, np.arange(W * H))
        assert np.array_equal(starts, np.arange(W * H + 1))


@pytest.mark.parametrize("cta", [False, True])
@pytest.mark.parametrize("sides", [[(3, 500), (90, 70), (4, 4)], [(120, 40), (50, 3), (64, 64)],
                                   [(3, 9), (4, 80)]])
def test_beside_others(pkg, sides, cta):
    p = pkg.workload_params()
    hs = [field(w, h, r) for r, (w, h) in enumerate(sides)]
    with pkg.FastScapeBatch([w for w, _ in sides], [h for _, h in sides], [p] * len(sides),
                            init=pkg.INIT_ZERO) as b:
        b.use_cta_walk(cta)
        for r, h in enumerate(hs):
            b.setH(r, h)
        flat = [r for r, s in enumerate(sides) if min(s) < 5]
        b.step(2)
        b.set_active(flat)
        b.step(1)
        b.analyze()
        for r in flat:
            check(pkg, b, r, *sides[r], hs[r])
        b.set_active(None)
        b.step(1)
        b.analyze()
        for r, (w, h) in enumerate(sides):
            if r in flat:
                check(pkg, b, r, w, h, hs[r])
                continue
            with pkg.FastScape_RBP(w, h, params=p, init=pkg.INIT_ZERO) as m:
                m.setH(hs[r])
                m.step(3)
                assert np.array_equal(b.getH(r), m.getH()), r


@pytest.mark.parametrize("W,H", [(3, 87381), (4, 65536), (65536, 4)])
def test_on_the_callers_buffer(pkg, W, H):
    torch = pytest.importorskip("torch")
    p = pkg.workload_params()
    h = torch.rand(W * H, dtype=torch.float64, device="cuda")
    want = h.clone()
    f = pkg.library().fs_step_noalloc
    f.argtypes = [C.c_void_p, C.c_int, C.c_int, C.POINTER(pkg.Params), C.c_int, C.c_void_p]
    assert f(C.c_void_p(h.data_ptr()), W, H, C.byref(p), 2, None) == 0, pkg.last_error()
    assert torch.equal(h, want)


def test_the_tallest(pkg):
    """1.6e9 cells, three to a row."""
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[0] < 70 << 30:
        pytest.skip("needs 70 GB of device memory")
    with pkg.FastScape_RBP(3, 2**29, params=pkg.workload_params(), init=pkg.INIT_ZERO) as m:
        m.step(1)
        assert m.steps_executed() == 1
