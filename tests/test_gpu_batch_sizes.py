"""Batches either side of the sizes at which the batched form changes its launches: every read's result
is the one that it has in a batch of other sizes."""
import numpy as np
import pytest

import mirage_b200 as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 1023, 1024, 1025, 2047, 2048, 2049, 3073, 49151, 49152, 49153])
def test_batches_of_every_launch_size(golden, n):
    g = golden("uneven_small")
    ix = M.Index(g.image)
    lens = g.reads.lengths()
    one = ix.classify(g.reads.data, g.reads.offs)
    m = len(lens)
    reps = n // m + 1
    offs = np.zeros(n + 1, np.uint64)
    offs[1:] = np.cumsum(np.tile(lens, reps)[:n])
    data = np.tile(g.reads.data[: int(g.reads.offs[-1])], reps)[: int(offs[-1])]
    got = ix.classify(data, offs)
    src = np.arange(n) % m
    count = (one.reads["n_fwd"] + one.reads["n_rc"]).astype(np.int64)
    for f in one.reads.dtype.names:
        if f != "cand_off":
            assert np.array_equal(got.reads[f], one.reads[f][src]), f
    assert np.array_equal(got.reads["cand_off"].astype(np.int64), np.cumsum(count[src]) - count[src])
    at = np.repeat(one.reads["cand_off"].astype(np.int64)[src] - (np.cumsum(count[src]) - count[src]), count[src])
    assert np.array_equal(got.cands.view(np.uint8), one.cands[at + np.arange(len(at))].view(np.uint8))
    ix.close()
