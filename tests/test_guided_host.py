"""CPU parity of the guided search (csrc/grand_guided.cuh) with the oracle, on the
emulated decode kernel (tests/host_guided.cpp): every deterministic field,
decoded pattern, logical flip and ML cost, at the edges of what the search takes
(4- and 8-word columns, the largest weight, both phase orders, the cap's cut sets,
duplicated and empty columns, ties and negative LLRs, levels that do not fit)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle as O
from library_s_grand_gb300 import synth
from test_host_kernels import HERE, ROOT, _compare, _cuda_include, _run, _write_code


@pytest.fixture(scope="module")
def guided(tmp_path_factory):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if cxx is None or inc is None:
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("hg") / "host_guided")
    subprocess.run([cxx, "-std=c++20", "-O2", "-pthread",
                    "-I", os.path.join(ROOT, "library_s_grand_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", inc, "-I", HERE,
                    os.path.join(HERE, "host_guided.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    return exe


def _jobs(out):
    return int(out.split()[3])


def _heavy(out):
    return int(out.split()[-1])


@pytest.mark.parametrize("n,W,mode,thr,cap,errors_input,fast,packed", [
    (72, 1, -1, 10, 64, True, True, False),
    (72, 4, -1, 10, 64, True, True, True),
    (72, 3, 0, 10, 64, False, True, False),
    (108, 6, 1, 6, 20, True, False, False),
    (144, 4, -1, 10, 64, True, True, False),
    (288, 3, -1, 10, 64, False, True, True),   # 144 rows: two word groups
])
def test_css_uniform(guided, port, tmp_path, n, W, mode, thr, cap, errors_input, fast, packed):
    code = synth.BB_CODES[n]()
    e = np.concatenate([synth.css_shots(code.hz, 30, p * 72 / n, seed=700 + i)[0]
                        for i, p in enumerate((0.01, 0.03, 0.06))])
    syn = (e.astype(np.int64) @ code.hz.T.astype(np.int64) % 2).astype(np.int32)
    rec = e if errors_input else syn
    cfg = (W, 256, 0, cap, thr, mode)
    res, dec, out = _run(guided, str(tmp_path), code.hz, code.hx, rec, errors_input, 0, cfg, [], 3,
                         packed=packed, fast=fast)
    prc, pres, pdec = port.css(O.UNIFORM, code.hx, code.hz, e if errors_input else None,
                               None if errors_input else syn, O.Config(*cfg), "x")
    assert prc == 0
    _compare(res, dec, pres, pdec)
    assert not fast or W > 4 or _jobs(out) == 0, out
    assert not fast or W == 1 or _heavy(out) > 0, out


@pytest.mark.parametrize("W,order,mode", [(6, (1, 0, 2), -1), (6, (0, 1, 2), 0), (7, (1, 0, 0), 1),
                                          (7, (2, 1, 0), -1), (5, (1, 0, 2), -1)])
def test_css_phases(guided, port, tmp_path, W, order, mode):
    # weight 6 before, after or without the weights 1..5, on a code whose weight-6
    # stabilizers let a match of a lower weight grow into one of weight 6
    code = synth.BB_CODES[72]()
    e = np.concatenate([synth.css_shots(code.hz, 25, p, seed=720 + i)[0]
                        for i, p in enumerate((0.01, 0.04))])
    masks = [(9, *order, 0.5, 0.3, 0.2), (300, 0, 1, 2, 0.6, 0.3, 0.1)]
    phase = synth.write_phase_file(str(tmp_path / "phase.txt"), masks)
    cfg = (W, 256, 0, 16, 6, mode)
    d = tmp_path / "run"
    d.mkdir()
    res, dec, out = _run(guided, str(d), code.hz, code.hx, e, True, 1, cfg, masks, 10)
    prc, pres, pdec = port.css(O.PROB, code.hx, code.hz, e, None, O.Config(*cfg), "x", phase)
    assert prc == 0
    _compare(res, dec, pres, pdec)


def _dem(kind, seed):
    dem = synth.random_dem(seed, detectors=48, mechanisms=200, logicals=40, p_range=(4e-3, 3e-2))
    if kind == "odd":  # empty and duplicated columns, weight 1 beside weight 4
        dem = synth.random_dem(seed, detectors=37, mechanisms=161, logicals=4, col_weights=(1, 4),
                               p_range=(4e-3, 3e-2))
        h = dem.h.copy()
        h[:, 7] = 0
        h[:, 31] = h[:, 30]
        h[:, 32] = h[:, 30]
        h[:, 120] = h[:, 5]
        dem = synth.Dem(h, dem.l, dem.p, dem.llr)
    return dem


@pytest.mark.parametrize("variant,kind,W,cap,llr", [
    ("uniform", "plain", 3, 24, None), ("uniform", "odd", 3, 40, None), ("uniform", "plain", 2, 0, None),
    ("prob", "plain", 6, 16, None), ("ml", "plain", 3, 24, "own"), ("ml", "odd", 3, 40, "own"),
    ("ml", "odd", 4, 14, "ties"), ("ml", "odd", 3, 24, "negative"), ("ml", "plain", 5, 12, "ties"),
])
def test_dem(guided, port, tmp_path, variant, kind, W, cap, llr):
    dem = _dem(kind, 8)
    values = dem.llr.copy()
    if llr == "ties":
        values = np.round(values)
    if llr == "negative":  # a column more costs less: lower weights do not stop the search
        values = values - 5.0
    det, log, _ = synth.dem_shots(dem, 140, seed=760)
    cfg = (W, 256, 0, cap, 10, -1)
    masks, path, v, pv = [], None, 0, O.UNIFORM
    if variant == "prob":
        masks = [(7, 1, 0, 2, 0.7, 0.2, 0.1), (300, 0, 1, 2, 0.6, 0.3, 0.1)]
        path, v, pv = synth.write_phase_file(str(tmp_path / "phase.txt"), masks), 1, O.PROB
    elif variant == "ml":
        path, v, pv = synth.write_llr_file(str(tmp_path / "llr.txt"), values), 2, O.ML
    d = tmp_path / "run"
    d.mkdir()
    res, dec, out, dlog, cost = _run(guided, str(d), dem.h, None, det, False, v, cfg, masks, 3,
                                     L=dem.l, logicals=log, llr_path=path if v == 2 else None)
    prc, pres, pdec, pdlog, pcost = port.dem(pv, dem.h, dem.l, det, log, O.Config(*cfg), path)
    assert prc == 0
    _compare(res, dec, pres, pdec)
    assert np.array_equal(dlog, pdlog)
    if variant == "ml":
        assert np.array_equal(cost.view(np.uint32), np.asarray(pcost, np.float32).view(np.uint32))


def test_capped_dem_stress(guided, port, tmp_path):
    """Random detectors of the 120 x 720 DEM: first sets of up to 64 columns, later ones
    cut to that size, every candidate ruled out without a Job."""
    from library_s_grand_gb300 import workloads
    wl = workloads.stress_dem(24, seed=11)
    res, dec, out, dlog, _ = _run(guided, str(tmp_path), wl.dem.h, None, wl.detectors, False, 0,
                                  wl.config, [], 10, L=wl.dem.l, logicals=wl.logicals)
    prc, pres, pdec, pdlog, _ = port.dem(O.UNIFORM, wl.dem.h, wl.dem.l, wl.detectors, wl.logicals,
                                         O.Config(*wl.config))
    assert prc == 0 and int(pres["found"].sum()) == 0
    _compare(res, dec, pres, pdec)
    assert np.array_equal(dlog, pdlog)
    assert _jobs(out) == 0 and _heavy(out) > 0, out


def test_levels_that_do_not_fit(guided, port, tmp_path):
    """Columns of weight 5 on 24 rows: each row meets dozens of them, so the levels of a
    weight-4 search outgrow the warp's items (of several shots together, and of one alone)
    and the shots take the general path."""
    rng = np.random.default_rng(3)
    h = np.zeros((24, 230), np.int32)
    for c in range(230):
        h[rng.choice(24, 5, replace=False), c] = 1
    assert 40 < h.sum(axis=1).max() <= 64
    e = np.zeros((40, 230), np.int32)
    for i in range(40):
        e[i, rng.choice(230, 1 + i % 5, replace=False)] = 1
    cfg = (4, 256, 0, 230, 10, -1)
    res, dec, out = _run(guided, str(tmp_path), h, h, e, True, 0, cfg, [], 10)
    prc, pres, pdec = port.css(O.UNIFORM, h, h, e, None, O.Config(*cfg), "x")
    assert prc == 0
    _compare(res, dec, pres, pdec)
    assert out.split("\n")[1].startswith("guided 1 ") and _jobs(out) > 0, out


@pytest.mark.parametrize("kind", ["bb72", "bb108", "bb288", "odd", "dense", "entries", "limit"])
def test_tables_built_on_the_device(guided, tmp_path, kind):
    """The allocation-free entry point's tables (csrc/grand_prep.cuh) equal the library's: 4-
    and 8-word columns, empty, duplicated and nested columns, codes without a guided
    search (dense, entries other than 0 and 1) and the entry point's largest matrix."""
    rng = np.random.default_rng(5)
    if kind.startswith("bb"):
        h = synth.BB_CODES[int(kind[2:])]().hz
    elif kind == "odd":
        h = _dem("odd", 8).h.copy()
        h[:, 9] |= h[:, 8]  # a column that holds another
    elif kind == "dense":
        h = (rng.random((40, 70)) < 0.4).astype(np.int32)
    elif kind == "entries":
        h = synth.BB_CODES[72]().hz.copy()
        h[3, 5] += 2
    else:
        h = synth.random_dem(2, detectors=256, mechanisms=1024).h
    _write_code(str(tmp_path / "code"), h, 0, 0, (3, 256, 0, 64, 10, -1), [], Ho=h)
    p = subprocess.run([guided, str(tmp_path / "code"), "prep"], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr
