"""GPU tests of the bulk insert's heap build (k_build): the new batches and
their ancestors are sifted from the bottom up instead of one insert after
another.

Bar: bit-exact.  After every bulk insert checkInsertHeap holds and the
counters are right; everything comes out as std::sort orders it.  Sizes lie
around the edges of levels, of the rule that chooses the build (the heap at
most 48 times the new batches) and of a ragged last batch."""
import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import gpuheap_gb300 as gh  # noqa: E402

VIEW = {"u32": np.int32, "i32": np.int32, "u64": np.int64}
NP_KEY = {"u32": np.uint32, "i32": np.int32, "u64": np.uint64}


@pytest.fixture(scope="module", autouse=True)
def _cuda(ghlib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.set_device(0)
    yield


def to_dev(a, key):
    return torch.from_numpy(np.ascontiguousarray(a).view(VIEW[key])).cuda()


# batches of the bulk inserts, one after another into the same heap
SEQUENCES = [(1,), (2, 1), (3, 4), (7, 1, 9), (47, 1, 1), (94, 2, 2), (64, 1, 2, 3), (200, 6, 7, 100), (1, 1, 1, 1, 1),
             (1023, 21, 22, 1200)]


@pytest.mark.parametrize("variant", ["topdown", "bottomup"])
@pytest.mark.parametrize("pb", [True, False])
@pytest.mark.parametrize("key,B", [("u32", 16), ("i32", 128), ("u32", 1024), ("u64", 64), ("u64", 2048), ("u32", 4096)])
def test_bulk_inserts_into_used_heaps(variant, pb, key, B):
    for seq in SEQUENCES:
        if sum(seq) * B > 1 << 20:
            continue
        tail = B // 3 if pb else 0
        n = sum(seq) * B + tail
        for dist in ("uniform", "reverse"):
            keys = pyoracle.gen(key, 7 * B + len(seq), dist, n)
            dev = to_dev(keys, key)
            with gh.Heap(sum(seq) + 1, B, key=key, variant=variant, partial_buffer=pb) as h:
                pos = 0
                for i, m in enumerate(seq):
                    size = m * B + (tail if i == len(seq) - 1 else 0)
                    h.insert(dev[pos:pos + size])
                    h.sync()
                    pos += size
                    ok, msg = h.check_insert_heap()
                    assert ok, (seq, i, msg)
                    assert h.item_count() == pos and h.node_count() == pos // B
                out = torch.zeros(n, dtype=dev.dtype, device="cuda")
                assert h.delete(out) == n
                assert np.array_equal(out.cpu().numpy().view(NP_KEY[key]), np.sort(keys)), (seq, dist)


@pytest.mark.parametrize("variant", ["topdown", "bottomup"])
def test_build_between_deletes(variant):
    """Bulk inserts into a heap that deletes have emptied in part, with one
    block, a few and more than the GPU holds, at an odd key address."""
    B, n = 256, 150 * 256
    keys = pyoracle.gen("u32", 5, "uniform", 2 * n + 1)
    dev = to_dev(keys, "u32")[1:]
    for grid in (1, 3, 2000):
        with gh.Heap(512, B, key="u32", variant=variant) as h:
            h.set_grid(grid)
            out = torch.zeros(2 * n, dtype=torch.int32, device="cuda")
            h.insert(dev[:n])
            a = h.delete(out, max_keys=n // 2)
            h.insert(dev[n:2 * n])
            ok, msg = h.check_insert_heap()
            assert ok, msg
            b = h.delete(out[a:])
            assert a + b == 2 * n
            got = out.cpu().numpy().view(np.uint32)
            first = np.sort(keys[1:n + 1])
            assert np.array_equal(got[:a], first[:a])
            assert np.array_equal(got[a:], np.sort(np.concatenate([first[a:], keys[n + 1:]])))
