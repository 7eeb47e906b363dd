"""Heavy shots of a code without guided tables, from host memory: the per-shot path reads each
record's bits from the cache that the chunk step filled, as soon as it sees the shot's queue
entry.  Every batch has other records in the same launch slots, so a shot that read the cache too
early has an earlier batch's record and result."""
import numpy as np
import pytest

import oracle as O
from library_s_grand_gb300 import capi

pytestmark = pytest.mark.gpu


def test_records_are_in_the_cache_before_their_queue_entries(gpulib, port):
    rng = np.random.default_rng(5)
    h = np.zeros((256, 1024), np.int32)
    for c in range(1024):
        h[rng.choice(256, 3, replace=False), c] = 1
    cfg = (2, 256, 0, 64, 10, -1)
    few = (rng.random((251, 256)) < 0.5).astype(np.int32)
    prc, want, _ = port.css(O.UNIFORM, h, h, None, few[:20], O.Config(*cfg), "x")
    rc, one = capi.run_grand_shots_cc(gpulib, h, h, None, few, capi.GrandDecoderConfig(*cfg), b"x")
    one = capi.results_array(one)
    assert prc == 0 and rc == 0 and len(O.fields_equal(one[:20], want)) == 0
    assert len({(int(r["tam"]), int(r["total_tested_combinations"])) for r in one}) > 240
    for rep in range(200):  # about 10^6 shots
        which = (np.arange(5000) + 7 * rep) % 251
        rc, res = capi.run_grand_shots_cc(gpulib, h, h, None, few[which], capi.GrandDecoderConfig(*cfg), b"x")
        bad = O.fields_equal(capi.results_array(res), one[which])
        assert rc == 0 and len(bad) == 0, (rep, bad[:5])
