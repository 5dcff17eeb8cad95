"""The bulk inserts and deletes that whole heaps no longer take by
themselves, at scale: the owner mode with one, two and seven workers, the
owner mode and the ticketed delete loops on 2^24 keys with the default wait
limit, and bulk inserts into reserved targets by many blocks.  They are still
what a chosen owner depth, limited deletes without a count and few batches
into a large heap run.  Outputs equal std::sort."""
import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import gpuheap_gb300 as gh  # noqa: E402

VIEW = {"u32": np.int32, "u64": np.int64}
NP_KEY = {"u32": np.uint32, "u64": np.uint64}


@pytest.fixture(scope="module", autouse=True)
def _cuda(ghlib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.set_device(0)
    yield


def to_dev(a, key):
    return torch.from_numpy(np.ascontiguousarray(a).view(VIEW[key])).cuda()


def filled(h, key, n, seed):
    keys = pyoracle.gen(key, seed, "uniform", n)
    dev = to_dev(keys, key)
    h.insert(dev)
    return np.sort(keys), torch.zeros_like(dev)


@pytest.mark.parametrize("variant", ["topdown", "bottomup"])
@pytest.mark.parametrize("grid", [2, 3, 8])
@pytest.mark.parametrize("depth", [2, 3])
def test_owner_with_few_workers(variant, grid, depth):
    """Lends wait for a free worker and lent nodes come back."""
    B, n = 1024, 1 << 19
    with gh.Heap(n // B, B, key="u32", variant=variant) as h:
        h.set_grid(grid)
        h.set_owner_depth(depth)
        want, out = filled(h, "u32", n, grid)
        assert h.delete(out) == n
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
        st = h.owner_stats()
        assert st["deletes"] > n // B // 2 and st["lends"] > 0


@pytest.mark.parametrize("variant", ["topdown", "bottomup"])
@pytest.mark.parametrize("key,B,pb,depth", [("u32", 256, True, 0), ("u32", 512, True, 0), ("u32", 512, False, 0),
                                            ("u64", 1024, True, 0), ("u32", 512, True, 2), ("u32", 1024, False, 3),
                                            ("u64", 1024, True, 2)])
def test_delete_loops_at_scale(variant, key, B, pb, depth):
    n = 1 << 24
    with gh.Heap(n // B + 1, B, key=key, variant=variant, partial_buffer=pb) as h:
        h.set_owner_depth(depth)
        want, out = filled(h, key, n + (B // 3 if pb else 0), B + depth)
        assert h.delete(out) == want.size
        assert np.array_equal(out.cpu().numpy().view(NP_KEY[key]), want)
        assert (h.owner_stats()["deletes"] > n // B // 2) == (depth > 0)


@pytest.mark.parametrize("variant", ["topdown", "bottomup"])
@pytest.mark.parametrize("key,B,nodes,batches", [("u32", 1024, 8192, 100), ("u32", 2048, 8192, 160), ("u64", 512, 20000, 152),
                                                 ("u32", 16, 4000, 80)])
def test_reserved_inserts_by_many_blocks(variant, key, B, nodes, batches):
    """Too few batches for a heap build: they meet in the heap's top."""
    n, m = nodes * B, batches * B
    keys = pyoracle.gen(key, nodes, "uniform", n + m)
    keys[n:] >>= NP_KEY[key](3)  # most of them bubble to the top
    with gh.Heap(nodes + batches, B, key=key, variant=variant) as h:
        h.insert(to_dev(keys[:n], key))
        h.insert(to_dev(keys[n:], key))
        ok, msg = h.check_insert_heap()
        assert ok, msg
        assert h.node_count() == nodes + batches
        out = to_dev(keys, key)
        assert h.delete(out) == n + m
        assert np.array_equal(out.cpu().numpy().view(NP_KEY[key]), np.sort(keys))
