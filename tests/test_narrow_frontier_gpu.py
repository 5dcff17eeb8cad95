"""Searches whose frontier fits one batch for their whole length (chains,
strips, corridors): one block passes the keys round by round while the others
wait, far longer than the heap's time limit.  The limits here are a hundredth
of the default one, so that some ten thousand rounds outlast them; a round
takes 10 to 30 us.  Results equal the CPU oracles."""
import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpuheap_gb300 import batch as gb  # noqa: E402
from gpuheap_gb300 import sssp as gsssp  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda(ghlib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.set_device(0)
    yield


def strip(length, width, seed):
    """A grid graph of length x width vertices, edges both ways, weights 1..1000."""
    rng = np.random.default_rng(seed)
    v = np.arange(length * width).reshape(length, width)
    a = np.concatenate([v[:-1].ravel(), v[:, :-1].ravel()])
    b = np.concatenate([v[1:].ravel(), v[:, 1:].ravel()])
    w = rng.integers(1, 1001, a.size)
    src, dst, wt = np.concatenate([a, b]), np.concatenate([b, a]), np.concatenate([w, w])
    order = np.argsort(src, kind="stable")
    rowptr = np.zeros(v.size + 1, np.int64)
    rowptr[1:] = np.cumsum(np.bincount(src, minlength=v.size))
    return rowptr, dst[order].astype(np.int32), wt[order].astype(np.uint32)


@pytest.mark.parametrize("variant", ["bottomup", "topdown"])
@pytest.mark.parametrize("length,width,B", [(20000, 1, 256), (6000, 100, 2048), (400, 400, 256)])
def test_sssp_on_chains_strips_and_grids(variant, length, width, B):
    rowptr, col, w = strip(length, width, length)
    g = gsssp.Graph(rowptr.size - 1, torch.from_numpy(rowptr).cuda(), torch.from_numpy(col).cuda(),
                    torch.from_numpy(w.view(np.int32)).cuda())
    want = pyoracle.dijkstra(rowptr, col, w, np.array([0], np.int64), threads=1)[0]
    heap = gsssp.make_heap(g, batch_size=B, variant=variant)
    heap.set_timeout(0.02)
    dist, _ = gsssp.sssp(heap, g, 0)
    assert np.array_equal(dist.cpu().numpy().view(np.uint32), want)
    heap.close()


@pytest.mark.parametrize("variant", ["bottomup", "topdown"])
def test_astar_through_a_long_corridor(variant):
    """Four blocks on a serpentine: one cell wide, some 45000 cells long."""
    side = 301
    grid = gb.gen_grid(side, 11, obstacle_per_mille=0)
    for y in range(1, side, 2):
        grid[y, :] = 0
        grid[y, side - 1 if y % 4 == 1 else 0] = 5
    want = pyoracle.astar_grid(grid)
    assert want < 0xFFFFFFFF
    b = gb.Batch([("astar", grid)], batch_size=64, variant=variant, astar_cells_per_block=1 << 14, astar_max_blocks=4,
                 timeout=0.02)
    try:
        assert b.info()["tasks"] == 4
        b.run("persistent")
        res, st, _ = b.results()
        assert not st.any() and int(res[0]) == int(want)
    finally:
        b.close()
