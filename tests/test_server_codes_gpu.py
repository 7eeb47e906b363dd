"""Codes registered with the engine after its server was created: the server's launches read
every registered code's descriptor, so these have to be on the device before the next
batch, whether the batch uses the new code or not."""
import numpy as np
import pytest

import oracle as O
from library_s_grand_gb300 import capi, synth
from library_s_grand_gb300.engine import Engine
from library_s_grand_gb300.server import Server

pytestmark = pytest.mark.gpu

CFG = (3, 256, 0, 64, 10, -1)


@pytest.mark.parametrize("late", [(108,), (108, 144, 288, 72, 108, 144, 288, 72, 108)])
def test_codes_registered_after_the_server(gpulib, port, late):
    codes = [synth.BB_CODES[72]()]
    eng = Engine(gpulib)
    eng.add_css(codes[0].hx, codes[0].hz, "x", False, capi.GrandDecoderConfig(*CFG))
    srv = Server(eng, slots=2, max_shots_per_batch=512)

    def check(c, shots, seed):
        _, syn = synth.css_shots(codes[c].hz, shots, 0.01, seed=seed)
        rc, res, _ = srv.wait(srv.submit(syn, np.full(shots, c, np.int32)))
        prc, want, _ = port.css(O.UNIFORM, codes[c].hx, codes[c].hz, None, syn, O.Config(*CFG), "x")
        assert rc == 0 and prc == 0
        assert len(O.fields_equal(res, want)) == 0

    check(0, 100, 1)
    for n in late:
        codes.append(synth.BB_CODES[n]())
        eng.add_css(codes[-1].hx, codes[-1].hz, "x", False, capi.GrandDecoderConfig(*CFG))
    check(0, 200, 2)                      # the first code, the others registered only
    check(len(codes) - 1, 150, 3)         # the last one
    check(0, 50, 4)
    srv.close()
    eng.close()
