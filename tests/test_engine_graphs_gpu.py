"""Captured launches and the workspaces they write to: a larger batch on the stream moves the
workspace, and the same buffers on another stream have that stream's workspace, so neither may
replay a launch captured before.  Codes without a guided search, and one whose searches can
outgrow it, so that the launches use their queue, Jobs and re-run flags."""
import numpy as np
import pytest

import oracle as O
from library_s_grand_gb300 import capi, synth
from library_s_grand_gb300.engine import Engine

pytestmark = pytest.mark.gpu


def _general_code():
    rng = np.random.default_rng(1)
    h = np.zeros((60, 200), np.int32)
    for c in range(200):
        h[rng.choice(60, 9, replace=False), c] = 1  # nine ones a column: no guided tables
    return synth.CssCode("general", h, h), (3, 256, 0, 64, 10, -1)


CODES = {"general": _general_code, "guided first": lambda: (synth.BB_CODES[72](), (6, 256, 0, 64, 10, -1))}


class _Run:
    def __init__(self, gpulib, port, kind, sizes):
        import torch
        self.torch = torch
        code, cfg = CODES[kind]()
        self.eng = Engine(gpulib)
        self.eng.add_css(code.hx, code.hz, "x", False, capi.GrandDecoderConfig(*cfg))
        self.syn, self.want, self.d_rec, self.d_res = {}, {}, {}, {}
        for n in sizes:
            syn = synth.css_shots(code.hz, n, 0.01, seed=n)[1]
            prc, self.want[n], _ = port.css(O.UNIFORM, code.hx, code.hz, None, syn, O.Config(*cfg), "x")
            assert prc == 0
            self.d_rec[n] = torch.from_numpy(syn).cuda()
            self.d_res[n] = torch.zeros(n * 72, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

    def decode(self, n, stream):
        self.d_res[n].zero_()
        self.torch.cuda.synchronize()
        assert self.eng.decode_device(n, self.d_rec[n].data_ptr(), self.d_res[n].data_ptr(), stream) == 0
        assert self.eng.sync_status(stream) == 0
        got = np.frombuffer(self.d_res[n].cpu().numpy().tobytes(), dtype=capi.RESULT_DTYPE)
        bad = O.fields_equal(got, self.want[n])
        assert len(bad) == 0, (n, bad[:5])
        return self.eng.launch_stats(stream)


@pytest.mark.parametrize("kind", sorted(CODES))
def test_larger_batch_between_replays(gpulib, port, kind):
    run = _Run(gpulib, port, kind, (200, 1500, 4000))
    s = run.torch.cuda.Stream().cuda_stream
    first = run.decode(200, s)
    assert run.decode(200, s)[:4] == first[:4]
    run.decode(1500, s)
    assert run.decode(200, s)[:4] == first[:4]
    run.decode(4000, s)
    for n in (200, 1500, 200):
        run.decode(n, s)


@pytest.mark.parametrize("kind", sorted(CODES))
def test_same_buffers_on_two_streams(gpulib, port, kind):
    run = _Run(gpulib, port, kind, (300,))
    a, b = run.torch.cuda.Stream(), run.torch.cuda.Stream()
    first = run.decode(300, a.cuda_stream)
    assert sum(first[:2]) > 0
    assert run.decode(300, b.cuda_stream)[:4] == first[:4]  # b's own statistics
    assert run.decode(300, a.cuda_stream)[:4] == first[:4]
