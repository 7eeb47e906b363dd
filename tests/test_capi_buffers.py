"""The wrappers' output buffers are not zeroed before a call that fills them; a call that
did not decode returns zeros all the same, and inputs the buffer protocol does not take
(read-only, empty) still pass."""
import numpy as np
import pytest

from library_s_grand_gb300 import build, capi, synth


@pytest.mark.parametrize("shots", [0, 1, 63, 64, 1000])
@pytest.mark.parametrize("wrapper", ["plain", "ex", "packed", "dem_ex"])
def test_refused_calls_return_zeros(shots, wrapper):
    build.build()
    lib = capi.load_library()
    code, dem = synth.BB_CODES[72](), synth.random_dem(0, detectors=20, mechanisms=40, logicals=3)
    cfg = capi.GrandDecoderConfig(0, 256, 0, 64, 10, -1)  # max_error_weight 0: refused before any GPU call
    syn = np.ones((shots, code.n), np.int32)
    syn.setflags(write=False)
    extra = []
    if wrapper == "plain":
        rc, res = capi.run_grand_shots_cc(lib, code.hx, code.hz, None, syn, cfg, b"x")
        res = capi.results_array(res) if shots else np.zeros(0, capi.RESULT_DTYPE)
    elif wrapper == "ex":
        rc, res, dec = capi.decode_css_ex(lib, "uniform", code.hx, code.hz, None, syn, cfg, "x")
        extra = [dec]
    elif wrapper == "packed":
        rc, res = capi.decode_css_packed(lib, code.hx, code.hz, capi.pack_bits(syn),
                                         capi.PACKED_SYNDROMES, cfg, "x")
    else:
        det, log = np.ones((shots, 20), np.int32), np.zeros((shots, 3), np.int32)
        rc, res, dec, dlog, cost = capi.decode_dem_ex(lib, "uniform", dem.h, dem.l, det, log, cfg)
        extra = [dec, dlog, cost]
    assert rc == -1 and len(res) == shots
    assert not np.asarray(res).view(np.uint8).any()
    assert not any(a.any() for a in extra)
