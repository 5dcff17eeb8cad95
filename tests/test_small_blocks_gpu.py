"""Batched searches on blocks of half a warp: batch size 32 takes 16 threads
(block_threads may be half the batch size), where an insert batch cannot be
sorted in the registers of whole warps."""
import numpy as np
import pytest

from test_batch_gpu import oracle_results, small_mix

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpuheap_gb300 import batch as gb  # noqa: E402


@pytest.mark.parametrize("variant", ["bottomup", "topdown"])
@pytest.mark.parametrize("bs,threads", [(32, 16), (32, 32), (64, 32)])
def test_searches_on_small_blocks(ghlib, variant, bs, threads):
    inst = small_mix(seed=bs + threads)
    b = gb.Batch(inst, batch_size=bs, variant=variant, block_threads=threads, astar_cells_per_block=1 << 12)
    try:
        assert b.info()["block_threads"] == threads
        for mode in ("persistent", "plain"):
            b.run(mode)
            res, st, _ = b.results()
            assert not st.any()
            assert np.array_equal(res, oracle_results(inst)), mode
    finally:
        b.close()
