"""The sampler at the largest shot count an int holds: its blocks' counters go past the last shot
without wrapping round, and the shots are those of the same numbers drawn alone."""
import numpy as np
import pytest

from library_s_grand_gb300 import capi
from library_s_grand_gb300.engine import Engine

pytestmark = pytest.mark.gpu


def test_largest_shot_count(gpulib):
    import torch
    shots = 2**31 - 1
    if torch.cuda.mem_get_info()[0] < 6 * shots:
        pytest.skip("needs 9 GB")
    h = np.ones((1, 3), np.int32)
    eng = Engine(gpulib)
    eng.add_css(h, h, "x", False, capi.GrandDecoderConfig(2, 256, 0, 64, 10, -1))
    p = torch.full((3,), 0.2, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    rec = torch.full((shots,), 7, dtype=torch.int32, device="cuda")
    assert eng.sample(0, p.data_ptr(), 11, 5, shots, rec.data_ptr(), s) == 0
    few = torch.full((5000,), 7, dtype=torch.int32, device="cuda")
    for at in (0, 2**30 - 2500, shots - 5000):
        assert eng.sample(0, p.data_ptr(), 11, 5 + at, 5000, few.data_ptr(), s) == 0
        assert torch.equal(rec[at:at + 5000], few) and 0 < int(few.sum()) < 5000
    assert int(rec.max()) == 1
    eng.close()
