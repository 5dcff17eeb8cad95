"""The output cursor near its limit of 2^31 - 1 keys: a delete whose batch
would take it past writes nothing.  The cursor is set by gh_heap_restore and
the output pointer moved back by it, so that the keys land in a small buffer."""
import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import gpuheap_gb300 as gh  # noqa: E402


@pytest.mark.parametrize("variant", ["topdown", "bottomup"])
@pytest.mark.parametrize("below,takes", [(3 * 256, 3), (2 * 256 + 1, 2), (256, 1), (255, 0), (0, 0)])
def test_deletes_stop_at_the_cursors_limit(ghlib, variant, below, takes):
    B, n = 256, 8 * 256
    cursor = 2**31 - 1 - below
    keys = pyoracle.gen("u32", 9, "uniform", n)
    with gh.Heap(16, B, key="u32", variant=variant) as h:
        h.insert(torch.from_numpy(keys.view(np.int32)).cuda())
        h.sync()
        items, _, counters = h.snapshot()
        h.restore(items, [counters[0], counters[1], cursor])
        out = torch.zeros(n, dtype=torch.int32, device="cuda")
        for i in range(takes + 2):
            assert h.delete_root(out.data_ptr() - 4 * cursor) == (B if i < takes else 0)
        assert h.item_count() == n - takes * B
        assert np.array_equal(out.cpu().numpy().view(np.uint32)[:takes * B], np.sort(keys)[:takes * B])
        assert h.snapshot()[2][2] == cursor + takes * B
        rest = torch.zeros(n, dtype=torch.int32, device="cuda")
        assert h.delete(rest) == n - takes * B  # a bulk delete starts from its own output's beginning
        assert np.array_equal(rest.cpu().numpy().view(np.uint32)[:n - takes * B], np.sort(keys)[takes * B:])
