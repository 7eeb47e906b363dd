"""A batch that fills the search arena more than a hundred times over: every shot is searched,
in as many rounds as that takes."""
import numpy as np
import pytest

import oracle as O
from library_s_grand_gb300 import capi

pytestmark = pytest.mark.gpu


def test_many_rounds_leave_no_shot(gpulib, port):
    # 256 rows: no guided search; random syndromes have up to 900 active positions, about 23000
    # words of the 32 M word arena a shot
    rng = np.random.default_rng(5)
    h = np.zeros((256, 1024), np.int32)
    for c in range(1024):
        h[rng.choice(256, 3, replace=False), c] = 1
    cfg = (2, 256, 0, 64, 10, -1)
    few = (rng.random((250, 256)) < 0.5).astype(np.int32)
    prc, want, _ = port.css(O.UNIFORM, h, h, None, few[:40], O.Config(*cfg), "x")
    assert prc == 0 and int(want["total_tested_combinations"].min()) > 1 << 17
    rc, one = capi.run_grand_shots_cc(gpulib, h, h, None, few, capi.GrandDecoderConfig(*cfg), b"x")
    one = capi.results_array(one)
    assert rc == 0 and len(O.fields_equal(one[:40], want)) == 0
    rc, res = capi.run_grand_shots_cc(gpulib, h, h, None, np.tile(few, (600, 1)),
                                      capi.GrandDecoderConfig(*cfg), b"x")
    res = capi.results_array(res)
    assert rc == 0
    assert len(O.fields_equal(res, np.tile(one, 600))) == 0
