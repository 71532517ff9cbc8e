"""What a batch holds on the device: 26 bytes a cell (elevation 8, receiver 1,
donor mask 1, roots 4, filter queues 8, count 4), 12812 a tile of 64 x 32 cells
and at first 65536 records of 64 bytes for each realization's table; nothing
more for the per-realization walk."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reals", [1, 4])
def test_bytes_per_cell(pkg, reals):
    torch = pytest.importorskip("torch")
    w, h = 1600, 1504  # whole tiles
    p = pkg.workload_params()
    with pkg.FastScapeBatch([9, 9], [9, 9], [p, p], init=pkg.INIT_ZERO) as b:
        b.use_cta_walk(True)
        b.step(1)  # the context's own memory
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    with pkg.FastScapeBatch([w] * reals, [h] * reals, [p] * reals, init=pkg.INIT_ZERO) as b:
        b.use_cta_walk(True)
        b.step(1)
        held = free0 - torch.cuda.mem_get_info()[0]
        cells = b.cells()
    # allocations come in blocks of 2 MB, some 16 of them; a graph takes a few
    assert held <= 26 * cells + 12812 * cells // 2048 + reals * 65536 * 64 + 24 * 2**21
