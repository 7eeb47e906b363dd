"""The general route on the GPU: the decode kernel's classification, per-shot path, Jobs and
search tiles, first-hit and ML, for codes without guided tables, for all codes with GRAND_FAST=0,
and for what the guided search leaves.  Launches with a small light budget must have had search
tiles, so that none of these passes with the shots decoded elsewhere."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle as O
from conftest import ROOT
from library_s_grand_gb300 import capi, synth
from library_s_grand_gb300.engine import ML, PROB, UNIFORM, Engine, offsets_for
from library_s_grand_gb300.server import Server

pytestmark = pytest.mark.gpu

MASKS = [(9, 1, 0, 2, 0.5, 0.3, 0.2), (300, 0, 1, 2, 0.6, 0.3, 0.1)]


def sparse(rows, cols, weight, seed):
    rng = np.random.default_rng(seed)
    h = np.zeros((rows, cols), np.int32)
    for c in range(cols):
        h[rng.choice(rows, weight, replace=False), c] = 1
    return h


# kind: (matrix, records are errors, weight, cap); none of them has guided tables
CODES = {
    "nine ones a column": lambda: (sparse(60, 300, 9, 2), True, 3, 300),
    "rows of more than 64": lambda: (sparse(40, 500, 6, 3), False, 3, 500),
    "260 rows": lambda: (sparse(260, 700, 3, 4), False, 3, 64),
    "1100 columns": lambda: (sparse(120, 1100, 5, 5), True, 2, 1100),
}


def decode(gpulib, add, records, shots, tuning=None):
    """add(engine) registers the code; a device decode of the records: results and statistics."""
    import torch
    eng = Engine(gpulib)
    add(eng)
    if tuning:
        eng.set_tuning(*tuning)
    d_rec = torch.from_numpy(np.ascontiguousarray(records, np.int32)).cuda()
    d_res = torch.zeros(shots * 72, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert eng.decode_device(shots, d_rec.data_ptr(), d_res.data_ptr(), s, use_graph=False) == 0
    assert eng.sync_status(s) == 0
    return np.frombuffer(d_res.cpu().numpy().tobytes(), dtype=capi.RESULT_DTYPE), eng.launch_stats(s)


def css_case(kind, shots):
    h, errors, W, cap = CODES[kind]()
    rng = np.random.default_rng(11)
    e = np.zeros((shots, h.shape[1]), np.int32)
    for i in range(shots):
        e[i, rng.choice(h.shape[1], i % 5, replace=False)] = 1
    syn = (e @ h.T & 1).astype(np.int32)
    return h, e, syn, errors, W, cap


@pytest.mark.parametrize("prob", [False, True])
@pytest.mark.parametrize("kind", sorted(CODES))
def test_codes_without_tables(gpulib, port, tmp_path, kind, prob):
    h, e, syn, errors, W, cap = css_case(kind, 120)
    W = 5 if prob else W
    cap = 24 if prob else cap
    mode = 1 if prob else -1  # (weights 1 .. 5 of sets up to the cap)
    cfg = (W, 256, 0, cap, 10, mode)
    path = synth.write_phase_file(str(tmp_path / "p.txt"), MASKS) if prob else None
    prc, want, _ = port.css(O.PROB if prob else O.UNIFORM, h, h, e if errors else None,
                            None if errors else syn, O.Config(*cfg), "x", path)
    assert prc == 0

    def add(eng):
        eng.add_css(h, h, "x", errors, capi.GrandDecoderConfig(*cfg), path)
    for tuning in (None, (0, 1, 0), (2, 8, 1)):
        got, stats = decode(gpulib, add, e if errors else syn, 120, tuning)
        assert len(O.fields_equal(got, want)) == 0, tuning
        assert stats[3] > 0 or tuning is None, stats  # (the default budget may hold every search)
    rc, res, dec = capi.decode_css_ex(gpulib, "prob" if prob else "uniform", h, h, e if errors else None,
                                      None if errors else syn, capi.GrandDecoderConfig(*cfg), "x", path)
    assert rc == 0 and len(O.fields_equal(res, want)) == 0


@pytest.mark.parametrize("variant", ["uniform", "prob", "ml"])
def test_dems_without_tables(gpulib, port, tmp_path, variant):
    dem = synth.random_dem(3, detectors=90, mechanisms=420, logicals=140, col_weights=(3, 9),
                           p_range=(2e-3, 1e-2))
    det, log, _ = synth.dem_shots(dem, 300, seed=4)
    cfg = ({"uniform": 3, "prob": 6, "ml": 3}[variant], 256, 0, 24, 10, -1)
    path = {"uniform": None, "prob": synth.write_phase_file(str(tmp_path / "p.txt"), MASKS),
            "ml": synth.write_llr_file(str(tmp_path / "l.txt"), dem.llr)}[variant]
    prc, want, wdec, wlog, wcost = port.dem({"uniform": O.UNIFORM, "prob": O.PROB, "ml": O.ML}[variant],
                                            dem.h, dem.l, det, log, O.Config(*cfg), path)
    assert prc == 0

    def add(eng):
        eng.add_dem(dem.h, dem.l, capi.GrandDecoderConfig(*cfg),
                    {"uniform": UNIFORM, "prob": PROB, "ml": ML}[variant], path)
    for tuning in (None, (0, 1, 0), (2, 8, 1)):
        got, stats = decode(gpulib, add, np.concatenate([det, log], axis=1), 300, tuning)
        assert len(O.fields_equal(got, want)) == 0, tuning
        assert stats[3] > 0 or tuning is None, stats  # (the default budget may hold every search)
    rc, res, dec, dlog, cost = capi.decode_dem_ex(gpulib, variant, dem.h, dem.l, det, log,
                                                  capi.GrandDecoderConfig(*cfg), path)
    assert rc == 0 and len(O.fields_equal(res, want)) == 0
    assert np.array_equal(dec, wdec) and np.array_equal(dlog, wlog)
    if variant == "ml":
        assert np.array_equal(cost.view(np.uint32), np.asarray(wcost, np.float32).view(np.uint32))


def test_what_the_guided_search_leaves(gpulib, port):
    """A code with guided tables whose weight-4 searches outgrow them: the chunk kernel finishes the
    light shots, the decode kernel the others."""
    h = sparse(24, 230, 5, 7)
    rng = np.random.default_rng(3)
    e = np.zeros((200, 230), np.int32)
    for i in range(200):
        e[i, rng.choice(230, 1 + i % 4, replace=False)] = 1
    cfg = (4, 256, 0, 230, 10, -1)
    prc, want, wdec = port.css(O.UNIFORM, h, h, e, None, O.Config(*cfg), "x")
    assert prc == 0
    got, stats = decode(gpulib, lambda eng: eng.add_css(h, h, "x", True, capi.GrandDecoderConfig(*cfg)), e, 200)
    assert len(O.fields_equal(got, want)) == 0
    assert stats[3] > 0 and stats[0] > 0 and stats[1] > 60, stats
    rc, res, dec = capi.decode_css_ex(gpulib, "uniform", h, h, e, None, capi.GrandDecoderConfig(*cfg), "x")
    assert rc == 0 and len(O.fields_equal(res, want)) == 0 and np.array_equal(dec, wdec)


def test_server_with_codes_of_every_route(gpulib, port):
    """A closed code, one whose searches can outgrow the guided search and one without tables in
    the same requests: the slots' copies, resets and shares of the decode kernel."""
    hs = [synth.BB_CODES[72]().hz, sparse(24, 230, 5, 7), sparse(60, 300, 9, 2)]
    cfgs = [(3, 256, 0, 64, 10, -1), (4, 256, 0, 230, 10, -1), (3, 256, 0, 300, 10, -1)]
    eng = Engine(gpulib)
    for h, cfg in zip(hs, cfgs):
        eng.add_css(h, h, "x", True, capi.GrandDecoderConfig(*cfg))
    srv = Server(eng, slots=3, max_shots_per_batch=256)
    rng = np.random.default_rng(6)
    pending = []
    for _ in range(24):
        n = int(rng.integers(1, 120))
        codes = rng.integers(0, 3, n).astype(np.int32)
        errs = []
        for c in codes:
            e = np.zeros(hs[c].shape[1], np.int32)
            e[rng.choice(len(e), int(rng.integers(0, 4)), replace=False)] = 1
            errs.append(e)
        pending.append((srv.submit(np.concatenate(errs), codes), codes, errs))
    for rid, codes, errs in pending:
        rc, res, _ = srv.wait(rid)
        assert rc == 0
        for c in range(3):
            idx = np.nonzero(codes == c)[0]
            if len(idx):
                prc, want, _ = port.css(O.UNIFORM, hs[c], hs[c], np.stack([errs[i] for i in idx]), None,
                                        O.Config(*cfgs[c]), "x")
                assert prc == 0 and len(O.fields_equal(res[idx], want)) == 0
    srv.close()


def test_more_codes_than_a_block_copies(gpulib, port):
    """Twelve codes in one batch: the blocks read the descriptors past the eighth from memory."""
    import torch
    codes = [synth.BB_CODES[(72, 108, 144, 288)[i % 4]]() for i in range(12)]
    cfgs = [(2 + i // 8, 256, 0, 64, 10, (-1, 0, 1)[i % 3]) for i in range(12)]
    eng = Engine(gpulib)
    for c, cfg in zip(codes, cfgs):
        eng.add_css(c.hx, c.hz, "x", False, capi.GrandDecoderConfig(*cfg))
    syn = [synth.css_shots(c.hz, 90, 0.01, seed=i)[1] for i, c in enumerate(codes)]
    order = np.random.default_rng(1).permutation(12 * 90)
    which = (order // 90).astype(np.int32)
    flat = np.concatenate([syn[i // 90][i % 90] for i in order]).astype(np.int32)
    d_rec, d_code = torch.from_numpy(flat).cuda(), torch.from_numpy(which).cuda()
    d_off = torch.from_numpy(offsets_for(eng.rec_lens, which)).cuda()
    d_res = torch.zeros(len(order) * 72, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert eng.decode_device(len(order), d_rec.data_ptr(), d_res.data_ptr(), s, d_code.data_ptr(),
                             d_off.data_ptr()) == 0
    assert eng.sync_status(s) == 0
    got = np.frombuffer(d_res.cpu().numpy().tobytes(), dtype=capi.RESULT_DTYPE)
    for i, (c, cfg) in enumerate(zip(codes, cfgs)):
        prc, want, _ = port.css(O.UNIFORM, c.hx, c.hz, None, syn[i], O.Config(*cfg), "x")
        back = np.empty(90, capi.RESULT_DTYPE)
        back[order[which == i] % 90] = got[which == i]
        assert prc == 0 and len(O.fields_equal(back, want)) == 0, i


_CHILD = """
import json, sys
sys.path[:0] = [{root!r}, {root!r} + '/tests', {root!r} + '/oracle']
import numpy as np, torch
from library_s_grand_gb300 import capi, engine, synth
import test_general_route_gpu as T
lib = capi.load_library()
stats = {{}}
out = {{}}
c = synth.BB_CODES[72]()
e = synth.css_shots(c.hz, 150, 0.04, seed=2)[0]
dem = synth.random_dem(8, detectors=48, mechanisms=200, logicals=40, p_range=(4e-3, 3e-2))
det, log, _ = synth.dem_shots(dem, 150, seed=3)
rec = np.concatenate([det, log], axis=1)
pf = synth.write_phase_file(sys.argv[1] + '/p.txt', T.MASKS)
lf = synth.write_llr_file(sys.argv[1] + '/l.txt', dem.llr)
cfg = capi.GrandDecoderConfig
for name, add, r in (
        ('css', lambda g: g.add_css(c.hx, c.hz, 'x', True, cfg(4, 256, 0, 64, 10, -1)), e),
        ('css_prob', lambda g: g.add_css(c.hx, c.hz, 'x', True, cfg(6, 256, 0, 16, 6, 1), pf), e),
        ('dem', lambda g: g.add_dem(dem.h, dem.l, cfg(3, 256, 0, 40, 10, -1), 0), rec),
        ('dem_prob', lambda g: g.add_dem(dem.h, dem.l, cfg(6, 256, 0, 16, 10, -1), 1, pf), rec),
        ('dem_ml', lambda g: g.add_dem(dem.h, dem.l, cfg(3, 256, 0, 40, 10, -1), 2, lf), rec)):
    out[name], st = T.decode(lib, add, r, 150, (3, 4, 0))
    stats[name] = [int(v) for v in st]
np.savez(sys.argv[2], **out)
print(json.dumps(stats))
"""


def test_every_shot_through_the_per_shot_path(gpulib, tmp_path):
    """GRAND_FAST=0 (read when the library is loaded, so in processes of their own): the per-shot
    path and the Jobs give the chunk kernel's results for codes that it takes."""
    script = tmp_path / "child.py"
    script.write_text(_CHILD.format(root=ROOT))
    runs = {}
    for fast in ("1", "0"):
        out = str(tmp_path / f"out{fast}.npz")
        p = subprocess.run([sys.executable, str(script), str(tmp_path), out], capture_output=True, text=True,
                           env=dict(os.environ, GRAND_FAST=fast))
        assert p.returncode == 0, p.stderr[-2000:]
        runs[fast] = (np.load(out), json.loads(p.stdout.strip().split("\n")[-1]))
    for name, stats in runs["0"][1].items():
        assert stats[0] == 0 and stats[1] == 150 and stats[3] > 0, (name, stats)
        assert len(O.fields_equal(runs["0"][0][name], runs["1"][0][name])) == 0, name
    assert all(s[0] > 0 for s in runs["1"][1].values()), runs["1"][1]
