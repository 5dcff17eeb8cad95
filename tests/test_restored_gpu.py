"""A heap that gh_heap_restore filled: only the first bulk operation on it
goes delete by delete below 256 nodes (for the owner mode's counters); after
any bulk insert, delete or collection the heap is emptied by one sort."""
from collections import Counter

import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import gpuheap_gb300 as gh  # noqa: E402


def to_dev(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


@pytest.mark.parametrize("first", ["insert", "delete", "collect", "concurrent"])
def test_the_replay_ends_with_the_first_bulk_operation(ghlib, first):
    B, n = 1024, 150 * 1024
    keys = pyoracle.gen("u32", 31, "uniform", n)
    more = pyoracle.gen("u32", 32, "uniform", 40 * B)
    with gh.Heap(512, B, key="u32") as h:
        h.insert(to_dev(keys))
        h.sync()
        items, _, counters = h.snapshot()
        h.reset()
        h.restore(items, counters[:3])
        out = torch.zeros(n + 40 * B, dtype=torch.int32, device="cuda")
        left = np.sort(keys)
        if first == "insert":
            h.insert(to_dev(more))
            left = np.sort(np.concatenate([keys, more]))
        elif first == "delete":
            assert h.delete(out, max_keys=B) == B
            left = left[B:]
        elif first == "collect":
            assert h.gc() == n
        else:
            got = h.concurrent(to_dev(more), out)
            left = Counter(np.concatenate([keys, more]).tolist()) - Counter(out.cpu().numpy().view(np.uint32)[:got].tolist())
            left = np.sort(np.array(list(left.elements()), np.uint32))
        before = h.owner_stats()
        assert h.delete(out) == left.size
        assert np.array_equal(out.cpu().numpy().view(np.uint32)[:left.size], left)
        assert h.owner_stats() == before  # no owner ran
