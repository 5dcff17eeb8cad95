"""GPU tests of the bulk deletes that are one radix sort (k_drain), of a whole
heap and of its smallest keys.

Bar: bit-exact.  The output is the sorted keys, and the heap is empty
afterwards as the delete loops leave it: counters, lock words and every node
at init_limits (the loops leave the last root's keys in node 1).  Sizes lie around a tile (8192 four-byte or 4096 eight-byte
keys), the fewest nodes the drain takes on and a ragged partial buffer; keys
include equal ones, few distinct ones and digits that all keys share."""
import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import gpuheap_gb300 as gh  # noqa: E402

VIEW = {"u32": np.int32, "i32": np.int32, "u64": np.int64}
NP_KEY = {"u32": np.uint32, "i32": np.int32, "u64": np.uint64}
INIT = {"u32": 0xFFFFFFFF, "i32": 0x7FFFFFFF, "u64": 0xFFFFFFFFFFFFFFFF}


@pytest.fixture(scope="module", autouse=True)
def _cuda(ghlib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.set_device(0)
    yield


def make_keys(key, n, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "equal":
        return np.full(n, 7 if key != "i32" else -7, NP_KEY[key])
    if kind == "two":
        return np.where(rng.random(n) < 0.3, 3, 1 << 20).astype(NP_KEY[key])
    if kind == "middle":  # only the second byte varies
        return (rng.integers(0, 256, n) * 256 + 5).astype(NP_KEY[key])
    if kind == "signed":
        return rng.integers(-1000, 1000, n).astype(np.int64).astype(NP_KEY[key])
    return pyoracle.gen(key, seed, kind, n)


def to_dev(a, key):
    return torch.from_numpy(np.ascontiguousarray(a).view(VIEW[key])).cuda()


def drained_ok(h, key, n, B):
    items, status, counters = h.snapshot()
    if n // B < 4:  # the delete loops leave the last root's keys in node 1
        items[B:2 * B] = NP_KEY[key](INIT[key])
    assert np.all(items == NP_KEY[key](INIT[key])) and not status.any()
    assert list(counters[:4]) == [0, 0, n, 0]


@pytest.mark.parametrize("variant", ["topdown", "bottomup"])
@pytest.mark.parametrize("pb", [True, False])
@pytest.mark.parametrize("key,B,ns", [("u32", 16, (3 * 16, 4 * 16, 8192 - 16, 8192, 8192 + 16)),
                                      ("i32", 256, (1024, 8192, 3 * 8192 + 256, 1 << 20)),
                                      ("u64", 64, (256, 4096 - 64, 4096, 4096 + 64, 1 << 17)),
                                      ("u32", 1024, (3 * 1024, 4 * 1024, 17 * 1024, 300 * 1024)),
                                      ("u64", 2048, (4 * 2048, 256 * 2048))])
def test_whole_heap(variant, pb, key, B, ns):
    for n in ns:
        n += (B - 1 if n % 3 else 1) if pb else 0
        with gh.Heap(n // B + 1, B, key=key, variant=variant, partial_buffer=pb) as h:
            for kind in ("uniform", "zipf", "equal", "two", "middle", "signed", "reverse"):
                if kind == "signed" and key != "i32":
                    continue
                keys = make_keys(key, n, kind, n + len(kind))
                h.reset()
                h.insert(to_dev(keys, key))
                out = torch.zeros(n + 5, dtype=torch.int64 if key == "u64" else torch.int32, device="cuda")
                assert h.delete(out[1:], max_keys=n) == n, (n, kind)
                got = out.cpu().numpy().view(NP_KEY[key])
                assert np.array_equal(got[1:n + 1], np.sort(keys)), (n, kind)
                assert got[0] == 0 and not got[n + 1:].any()
                drained_ok(h, key, n, B)


def taken_by(want, B, pb, limit=None, threshold=None):
    """Keys a bulk delete takes: whole batches, then the partial buffer."""
    n = len(want)
    limit = n if limit is None else limit
    got = 0
    while n - got > 0:
        size = B if n - got >= B else n - got
        if got + size > limit or (threshold is not None and not int(want[got]) < threshold):
            break
        got += size
    return got


@pytest.mark.parametrize("variant", ["topdown", "bottomup"])
@pytest.mark.parametrize("pb", [True, False])
@pytest.mark.parametrize("key,B,n", [("u32", 128, 300 * 128), ("i32", 64, 8192 + 64 * 64), ("u64", 512, 400 * 512),
                                     ("u32", 2048, 130 * 2048)])
def test_part_of_the_heap(variant, pb, key, B, n):
    """Limits and thresholds that leave keys behind: the smallest come out in
    order, the rest is a valid heap of the right counts, which takes inserts
    and gives up the rest in order."""
    n += B // 2 + 1 if pb else 0
    for kind in ("uniform", "two", "middle", "signed", "equal"):
        if kind == "signed" and key != "i32":
            continue
        keys = make_keys(key, n, kind, n + len(kind))
        want = np.sort(keys)
        more = make_keys(key, 3 * B, "uniform", 1)
        dt = torch.int64 if key == "u64" else torch.int32
        for share in (0.4, 0.97, 1.0):
            for how in ("limit", "threshold"):
                limit = int(share * n) - (1 if share == 1.0 else 0)
                thr = int(want[min(n - 1, int(share * n))])
                exp = taken_by(want, B, pb, limit=limit) if how == "limit" else taken_by(want, B, pb, threshold=thr)
                with gh.Heap(n // B + 4, B, key=key, variant=variant, partial_buffer=pb) as h:
                    h.insert(to_dev(keys, key))
                    out = torch.zeros(n + 1, dtype=dt, device="cuda")
                    got = h.delete(out[1:], max_keys=limit) if how == "limit" else h.delete_below(out[1:], thr)
                    assert got == exp, (kind, share, how)
                    res = out.cpu().numpy().view(NP_KEY[key])
                    assert np.array_equal(res[1:got + 1], want[:got]) and res[0] == 0 and not res[got + 1:].any()
                    items, status, counters = h.snapshot()
                    assert not status.any() and list(counters[:4]) == [(n - got) // B, (n - got) % B, got, 0]
                    used = items[:(n - got) // B * B + B]
                    assert np.all(items[len(used):] == NP_KEY[key](INIT[key])) or got in (0, n)  # or the loops' last root
                    ok, msg = h.check_insert_heap()
                    assert ok, msg
                    h.insert(to_dev(more, key))
                    ok, msg = h.check_insert_heap()
                    assert ok, msg
                    out = torch.zeros(n - got + 3 * B, dtype=dt, device="cuda")
                    assert h.delete(out) == out.numel()
                    assert np.array_equal(out.cpu().numpy().view(NP_KEY[key]), np.sort(np.concatenate([want[got:], more])))


@pytest.mark.parametrize("grid", [1, 2, 7, 5000])
def test_grids_and_reuse(grid):
    """Any number of blocks, the heap used again after a drain, and a limit
    one key short of the whole heap, which leaves the last keys in it."""
    B, n = 256, 200 * 256 + 100
    keys = pyoracle.gen("u32", grid, "uniform", n)
    dev, want = to_dev(keys, "u32"), np.sort(keys)
    with gh.Heap(512, B, key="u32") as h:
        h.set_grid(grid)
        out = torch.zeros(n, dtype=torch.int32, device="cuda")
        for _ in range(2):
            h.insert(dev)
            assert h.delete(out) == n
            assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
        h.insert(dev)
        assert h.delete(out, max_keys=n - 1) == n - 100
        assert h.item_count() == 100
        assert h.delete(out) == 100
        assert np.array_equal(out.cpu().numpy().view(np.uint32)[:100], want[-100:])


def test_taken_lock_word_is_waited_for():
    """A lock word that nothing releases: the drain leaves the heap to the
    delete loops, whose wait runs out; the heap works after a reset."""
    B, n = 256, 40 * 256
    keys = to_dev(pyoracle.gen("u32", 3, "uniform", n), "u32")
    with gh.Heap(64, B, key="u32") as h:
        out = torch.zeros(n, dtype=torch.int32, device="cuda")
        for node in (0, 3, 40):
            h.set_timeout(2.0)
            h.insert(keys)
            h.sync()
            h.set_timeout(0.05)
            h.inject_lock(node, 1 << 30)
            with pytest.raises(gh.HeapError) as e:
                h.delete(out)
            assert e.value.status == gh.GH_ERR_TIMEOUT
            h.reset()
        h.insert(keys)
        assert h.delete(out) == n


def test_captured_in_a_graph():
    """A bulk insert and a whole-heap delete captured once and replayed."""
    B, n = 1024, 300 * 1024 + 77
    src = to_dev(pyoracle.gen("u32", 1, "uniform", n), "u32")
    out = torch.zeros_like(src)
    with gh.Heap(512, B, key="u32") as h:
        s = torch.cuda.Stream()

        def step():
            h.reset_async(s)
            h.insert(src, stream=s)
            h.delete(out, stream=s, sync=False)

        step()
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            step()
        for seed in (2, 3):
            keys = pyoracle.gen("u32", seed, "uniform", n)
            src.copy_(to_dev(keys, "u32"))
            torch.cuda.synchronize()
            g.replay()
            torch.cuda.synchronize()
            h.sync()
            assert np.array_equal(out.cpu().numpy().view(np.uint32), np.sort(keys))


@pytest.mark.parametrize("nodes,owner", [(200, True), (256, False)])
def test_a_small_restored_heap_is_replayed_by_the_owner(nodes, owner):
    """gh_heap_restore: below 256 nodes the deletes go one by one (owner mode,
    its counters), until the next reset."""
    B, n = 1024, nodes * 1024
    keys = pyoracle.gen("u32", nodes, "uniform", n)
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    with gh.Heap(512, B, key="u32") as h:
        h.insert(to_dev(keys, "u32"))
        h.sync()
        items, _, counters = h.snapshot()
        assert h.delete(out) == n and h.owner_stats()["deletes"] == 0
        h.restore(items, counters[:3])
        assert h.delete(out) == n
        assert (h.owner_stats()["deletes"] > 0) == owner
        assert np.array_equal(out.cpu().numpy().view(np.uint32), np.sort(keys))
        before = h.owner_stats()["deletes"]
        h.sort(to_dev(keys, "u32"), out)
        assert h.owner_stats()["deletes"] == before
        assert np.array_equal(out.cpu().numpy().view(np.uint32), np.sort(keys))


def test_a_chosen_owner_depth_keeps_the_owner_mode():
    B, n = 1024, 400 * 1024
    keys = pyoracle.gen("u32", 8, "uniform", n)
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    with gh.Heap(512, B, key="u32") as h:
        h.sort(to_dev(keys, "u32"), out)
        assert h.owner_stats()["deletes"] == 0
        h.set_owner_depth(3)
        h.sort(to_dev(keys, "u32"), out)
        assert h.owner_stats()["deletes"] > 300
        assert np.array_equal(out.cpu().numpy().view(np.uint32), np.sort(keys))
