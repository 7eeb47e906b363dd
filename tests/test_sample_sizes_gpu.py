"""Device sampler against its host restatement, bit for bit, where the kernel's division of the
work can go wrong: positions around a group of 128 and at the largest code, fewer shots than
blocks, as many, and one more, shot numbers on both sides of 2^32, and a seed of two words."""
import numpy as np
import pytest

from library_s_grand_gb300 import capi, synth
from library_s_grand_gb300 import sample as SM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,shots,first", [
    (127, 1, 0), (128, 151, 5), (129, 153, (1 << 32) - 70), (720, 700, (3 << 32) - 350),
    (4000, 152, (1 << 40) + 1), (1, 33, 0),
])
def test_records_equal_host_restatement(gpulib, m, shots, first):
    import torch
    from library_s_grand_gb300.engine import Engine
    dem = synth.random_dem(m, detectors=41, mechanisms=m, logicals=33)
    p = dem.p.astype(np.float32)
    p[:: 7] = 0.03
    p[0] = 1.0
    p[-1:] = 0.0 if m > 1 else 0.5
    eng = Engine(gpulib)
    eng.add_dem(dem.h, dem.l, capi.GrandDecoderConfig(3, 256, 0, 48, 10, -1), 0, None)
    seed = 0xFEDC_BA98_7654_3210
    L = eng.rec_lens[0]
    d_p = torch.from_numpy(p).cuda()
    d_rec = torch.full((shots * L,), -7, dtype=torch.int32, device="cuda")
    assert eng.sample(0, d_p.data_ptr(), seed, first, shots, d_rec.data_ptr()) == 0
    torch.cuda.synchronize()
    want = SM.dem_records(dem.h, dem.l, p, seed, first, shots)
    assert np.array_equal(d_rec.cpu().numpy().reshape(shots, L), want)
