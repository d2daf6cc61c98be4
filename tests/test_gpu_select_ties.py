"""Ties of the select over whole chunks of its widest kernel (1024 threads, 32768 positions a chunk), against the oracle."""
import numpy as np
import pytest
import torch

from oracle import pikv_oracle as O

pytestmark = pytest.mark.gpu


# few segments and n > 32768 take the 1024-thread kernel; every position, exactly one chunk, or one short of a chunk shares
# the timestamp at the cut
@pytest.mark.parametrize("n", [40000, 70000])
@pytest.mark.parametrize("tied", ["timestamps", "scores", "both"])
@pytest.mark.parametrize("run", [None, (0, 32768), (0, 32767), (32768, 65536)])
def test_select_ties_over_a_whole_chunk(n, tied, run):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import ops
    rng = np.random.default_rng(n)
    heavy, recent = 900, 700

    def values(is_tied):
        x = rng.random(n).astype(np.float32)
        if is_tied and run is None:
            x[:] = 0.0
        elif is_tied:                                # the run and its neighbours above the rest: the cut falls among equals
            x[run[0]:run[1]] = 2.0
            x[run[1]: run[1] + 100] = 2.0
        return x

    acc, ts = values(tied != "timestamps"), values(tied != "scores")
    if tied != "scores" and run is not None and run[0]:
        ts[:run[0]][rng.permutation(run[0])[: recent // 2]] = 3.0      # half of what is kept lies above the tie, in the first chunk
    mask, keep, count = ops.h2o_select(torch.from_numpy(acc)[None].cuda(), torch.from_numpy(ts)[None].cuda(), heavy, recent)
    evict, kept = O.h2o_select(acc, ts, heavy, recent)
    assert int(count[0]) == len(kept)
    np.testing.assert_array_equal(mask[0].cpu().numpy(), evict)
    np.testing.assert_array_equal(keep[0, : len(kept)].cpu().numpy(), kept)
