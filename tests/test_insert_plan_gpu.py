"""Bulk inserts into used heaps on either side of the line between a heap
build and single inserts (gpuheap_gb300/csrc/insert_plan.h): after both the
heap is valid and gives everything up in order."""
import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import gpuheap_gb300 as gh  # noqa: E402

NP_KEY = {"u32": np.uint32, "u64": np.uint64}


def most_nodes(top, node_bytes, m):
    """The largest heap that m batches still build into."""
    cube = m**3 // (4 if top else 32 if node_bytes < 512 else 16) if m < 64 else 1 << 40
    times = 48 if top else min(48, (6 if node_bytes < 128 else 12 if node_bytes < 512 else 24 if node_bytes < 1024 else 48) *
                               max(m, 128) // 128)
    return min(cube, (times - 1) * m)


@pytest.mark.parametrize("variant", ["topdown", "bottomup"])
@pytest.mark.parametrize("key,B", [("u32", 16), ("u64", 32), ("u32", 128), ("u64", 512)])
@pytest.mark.parametrize("pb", [True, False])
def test_either_side_of_the_line(ghlib, variant, key, B, pb):
    node_bytes = B * (8 if key == "u64" else 4)
    for m in (1, 2, 3, 4, 8, 13, 24, 64):
        edge = most_nodes(variant == "topdown", node_bytes, m)
        for n in (edge, edge + 1):
            if (n + m) * B > 1 << 20:
                continue
            tail = B // 2 if pb else 0
            keys = pyoracle.gen(key, n + m + B, "uniform", (n + m) * B + tail)
            dev = torch.from_numpy(keys.view(np.int64 if key == "u64" else np.int32)).cuda()
            with gh.Heap(n + m + 1, B, key=key, variant=variant, partial_buffer=pb) as h:
                if n:
                    h.insert(dev[:n * B])
                h.insert(dev[n * B:])
                h.sync()
                ok, msg = h.check_insert_heap()
                assert ok, (m, n, msg)
                assert h.node_count() == n + m and h.item_count() == keys.size
                out = torch.zeros_like(dev)
                assert h.delete(out) == keys.size
                assert np.array_equal(out.cpu().numpy().view(NP_KEY[key]), np.sort(keys)), (m, n)
