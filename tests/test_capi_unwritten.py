"""What the wrappers return when the library does not write: zeros, whichever error it gives
and whatever the sizes; results that it did write stay, also beside an error code."""
import ctypes

import numpy as np
import pytest

from library_s_grand_gb300 import capi, synth


class _Lib:
    """A library whose calls return rc, having written every result (found = 7) or none."""

    def __init__(self, rc, writes):
        def call(*args):
            results = next(a for a in args if isinstance(a, ctypes.Array)
                           and a._type_ is capi.GrandDecoderResult)
            for i in range(len(results) if writes else 0):
                results[i].found = 7
            return rc
        self.grand_decode_cc = self.grand_decode_cc_ex = self.grand_decode_cc_packed = call
        self.grand_decode_cln_ex = call


@pytest.mark.parametrize("wrapper", ["plain", "ex", "packed", "dem_ex"])
@pytest.mark.parametrize("shots", [0, 1, 63, 64, 300])
@pytest.mark.parametrize("rc,writes", [(-1, False), (-2, False), (-3, False), (-3, True), (0, True)])
def test_unwritten_results_are_zero(monkeypatch, wrapper, shots, rc, writes):
    monkeypatch.setattr(capi, "_uninit", lambda n: np.full(n, 0x5A, np.uint8))  # not zero by chance
    lib = _Lib(rc, writes)
    code, dem = synth.BB_CODES[72](), synth.random_dem(0, detectors=20, mechanisms=40, logicals=3)
    cfg = capi.GrandDecoderConfig(3, 256, 0, 64, 10, -1)
    syn = np.ones((shots, code.n), np.int32)
    extra = []
    if wrapper == "plain":
        got, res = capi.run_grand_shots_cc(lib, code.hx, code.hz, None, syn, cfg, b"x")
        res = capi.results_array(res) if shots else np.zeros(0, capi.RESULT_DTYPE)
    elif wrapper == "ex":
        got, res, dec = capi.decode_css_ex(lib, "uniform", code.hx, code.hz, None, syn, cfg, "x")
        extra = [dec]
    elif wrapper == "packed":
        got, res = capi.decode_css_packed(lib, code.hx, code.hz, capi.pack_bits(syn),
                                          capi.PACKED_SYNDROMES, cfg, "x")
    else:
        det, log = np.ones((shots, 20), np.int32), np.zeros((shots, 3), np.int32)
        got, res, dec, dlog, cost = capi.decode_dem_ex(lib, "uniform", dem.h, dem.l, det, log, cfg)
        extra = [dec, dlog, cost]
    assert got == rc and len(res) == shots
    if writes:
        assert (res["found"] == 7).all()
    else:
        assert not np.asarray(res).view(np.uint8).any()
        assert not any(a.any() for a in extra)
