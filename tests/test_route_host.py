"""CPU parity of whole batches planned as the library plans them (tests/host_route.cpp): which
kernel takes which shots, in chunks of what size, for codes with and without guided tables."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle as O
from library_s_grand_gb300 import capi, synth
from test_host_kernels import HERE, ROOT, _cuda_include, _write_code


@pytest.fixture(scope="module")
def route(tmp_path_factory):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if cxx is None or inc is None:
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("hr") / "host_route")
    subprocess.run([cxx, "-std=c++20", "-O2", "-pthread",
                    "-I", os.path.join(ROOT, "library_s_grand_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", inc, "-I", HERE,
                    os.path.join(HERE, "host_route.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    return exe


def sparse(rows, cols, weight, seed):
    rng = np.random.default_rng(seed)
    h = np.zeros((rows, cols), np.int32)
    for c in range(cols):
        h[rng.choice(rows, weight, replace=False), c] = 1
    return h


def decode(exe, d, codes, records, shot_code, starts=None, light=10, mode=None):
    """codes: argument tuples of _write_code after the directory, with its keywords; starts: where
    each record begins in the flat records (None: back to back).  Returns the results and the
    numbers of the program's two lines by name."""
    for k, (args, kw) in enumerate(codes):
        _write_code(str(d / f"code{k}"), *args, **kw)
    n = len(records)
    lens = np.array([len(r) for r in records])
    if starts is None:
        starts = np.concatenate([[0], np.cumsum(lens)[:-1]])
    flat = np.zeros(int((starts + lens).max()), np.int32)
    for s, r in zip(starts, records):
        flat[s:s + len(r)] = r
    with open(d / "mixed.txt", "w") as f:
        f.write(f"{len(codes)} {n} {light} 4\n")
    flat.tofile(d / "rec.bin")
    np.asarray(starts, np.int64).tofile(d / "off.bin")
    np.asarray(shot_code, np.int32).tofile(d / "code.bin")
    p = subprocess.run([exe, str(d)] + ([mode] if mode else []), capture_output=True, text=True,
                       timeout=600)
    assert p.returncode == 0, (p.returncode, p.stdout, p.stderr)
    if mode == "edge":
        return np.fromfile(d / "res.bin", dtype=capi.RESULT_DTYPE)
    first, second = p.stdout.split("\n")[:2]
    w = first.replace(",", "").split()
    info = {"jobs": int(w[3]), "slow": int(w[5])}
    w = second.split()
    info.update({w[i]: int(w[i + 1]) for i in range(0, len(w), 2)})
    return np.fromfile(d / "res.bin", dtype=capi.RESULT_DTYPE), info


@pytest.mark.parametrize("cols,errors", [(200, True), (256, True), (257, True), (300, True), (512, True),
                                         (1000, True), (300, False)])
def test_chunks_of_codes_without_tables(route, port, tmp_path, cols, errors):
    """Nine ones a column: no guided tables.  Empty records and single columns are settled in
    chunks, whatever the records' length; only the others take the per-shot path."""
    h = sparse(60, cols, 9, cols)
    rng = np.random.default_rng(2)
    e = np.zeros((70, cols), np.int32)
    for i in range(70):
        e[i, rng.choice(cols, (0, 1, 0, 1, 2)[i % 5], replace=False)] = 1
    syn = (e @ h.T & 1).astype(np.int32)
    cfg = (2, 256, 0, 64, 10, -1)
    rec = e if errors else syn
    res, info = decode(route, tmp_path, [((h, 0, 1 if errors else 0, cfg, []), {"Ho": h})], list(rec),
                       [0] * 70)
    prc, want, _ = port.css(O.UNIFORM, h, h, e if errors else None, None if errors else syn,
                            O.Config(*cfg), "x")
    assert prc == 0 and len(O.fields_equal(res, want)) == 0
    assert info["guided"] == 0 and info["settled"] == 56 and info["slow"] == 14, info


def test_long_records_of_other_codes_leave_the_chunks_alone(route, port, tmp_path):
    """Records that the chunk step does not take (more than 256 rows, or errors of more than 1024
    columns) lie between others': those are settled as without them."""
    small, long, wide = sparse(60, 100, 9, 1), sparse(300, 400, 3, 2), sparse(40, 3000, 9, 3)
    cfg = (1, 256, 0, 64, 10, -1)
    rng = np.random.default_rng(4)
    recs, codes, errs = [], [], []
    for i in range(60):
        k = (0, 0, 0, 1, 0, 2)[i % 6]
        h = (small, long, wide)[k]
        e = np.zeros(h.shape[1], np.int32)
        e[rng.integers(h.shape[1])] = 1
        errs.append(e)
        recs.append((h @ e & 1).astype(np.int32) if k == 1 else e)
        codes.append(k)
    res, info = decode(route, tmp_path, [((small, 0, 1, cfg, []), {"Ho": small}),
                                         ((long, 0, 0, cfg, []), {"Ho": long}),
                                         ((wide, 0, 1, cfg, []), {"Ho": wide})], recs, codes, mode="tables=0")
    for k, h in enumerate((small, long, wide)):
        idx = [i for i in range(60) if codes[i] == k]
        rows = np.stack([recs[i] for i in idx])
        prc, want, _ = port.css(O.UNIFORM, h, h, None if k == 1 else rows, rows if k == 1 else None,
                                O.Config(*cfg), "x")
        assert prc == 0 and len(O.fields_equal(res[idx], want)) == 0
    assert info["settled"] == 40 and info["slow"] == 20, info


@pytest.mark.parametrize("shots", [1, 63, 200])
def test_plan_of_closed_codes(route, port, tmp_path, shots):
    """Error records of 300 entries, a closed code: the plan's chunks hold them, so the chunk
    kernel decodes every shot alone."""
    h = sparse(60, 300, 3, 5)
    e = (np.random.default_rng(6).random((shots, 300)) < 0.005).astype(np.int32)
    cfg = (2, 256, 0, 64, 10, -1)
    res, info = decode(route, tmp_path, [((h, 0, 1, cfg, []), {"Ho": h})], list(e), [0] * shots)
    prc, want, _ = port.css(O.UNIFORM, h, h, e, None, O.Config(*cfg), "x")
    assert prc == 0 and len(O.fields_equal(res, want)) == 0
    assert info["guided"] == 2 and info["settled"] + info["searched"] == shots, info


@pytest.mark.parametrize("gap", [0, 1, 3])
def test_records_of_several_runs_are_kept(route, port, tmp_path, gap):
    """Requests' records in separate buffers (gap entries between groups of five): the per-shot
    path finds every record of a chunk in the cache, not those of one run only."""
    h = sparse(60, 200, 9, 7)
    dem = synth.random_dem(3, detectors=48, mechanisms=200, logicals=40, col_weights=(8, 9),
                           p_range=(4e-3, 2e-2))
    rng = np.random.default_rng(8)
    e = np.zeros((60, 200), np.int32)
    for i in range(60):
        e[i, rng.choice(200, 2, replace=False)] = 1
    det, log, _ = synth.dem_shots(dem, 60, seed=9)
    cfg = (2, 256, 0, 64, 10, -1)
    recs = [r for i in range(60) for r in (e[i], np.concatenate([det[i], log[i]]))]
    starts, at = [], 0
    for i, r in enumerate(recs):
        at += gap if i % 5 == 0 else 0
        starts.append(at)
        at += len(r)
    res, info = decode(route, tmp_path, [((h, 0, 1, cfg, []), {"Ho": h}),
                                         ((dem.h, 0, 2, cfg, []), {"L": dem.l})],
                       recs, [0, 1] * 60, np.array(starts))
    prc, want, _ = port.css(O.UNIFORM, h, h, e, None, O.Config(*cfg), "x")
    assert prc == 0 and len(O.fields_equal(res[::2], want)) == 0
    prc, want, *_ = port.dem(O.UNIFORM, dem.h, dem.l, det, log, O.Config(*cfg))
    assert prc == 0 and len(O.fields_equal(res[1::2], want)) == 0
    assert info["guided"] == 0 and info["slow"] > 60 and info["cached"] == info["slow"], info


def test_no_data_race_between_warps(route, port, tmp_path):
    """The chunk kernel under the thread sanitizer: blocks whose open shots leave groups of lanes
    without one (these must not read another warp's shot), chunks that end in every phase."""
    exe = tmp_path / "host_route_tsan"
    built = subprocess.run([shutil.which("g++"), "-std=c++20", "-O1", "-g", "-pthread", "-fsanitize=thread",
                            "-I", os.path.join(ROOT, "library_s_grand_gb300", "csrc"),
                            "-I", os.path.join(ROOT, "include"), "-I", _cuda_include(), "-I", HERE,
                            os.path.join(HERE, "host_route.cpp"), "-o", str(exe)],
                           capture_output=True, text=True)
    if built.returncode != 0 and "tsan" in built.stderr:
        pytest.skip("no thread sanitizer library")
    assert built.returncode == 0, built.stderr
    code = synth.BB_CODES[72]()
    cfg = (3, 256, 0, 64, 10, -1)
    e = synth.css_shots(code.hz, 23, 0.03, seed=3)[0]
    res, info = decode(str(exe), tmp_path, [((code.hz, 0, 1, cfg, []), {"Ho": code.hx})], list(e), [0] * 23)
    prc, want, _ = port.css(O.UNIFORM, code.hx, code.hz, e, None, O.Config(*cfg), "x")
    assert prc == 0 and len(O.fields_equal(res, want)) == 0
    assert info["guided"] == 2 and info["searched"] > 8, info


def test_last_chunk_of_the_largest_batch(route, port, tmp_path):
    """The last of INT_MAX shots, in a chunk that ends past them: its lanes' slots are not counted
    beyond the largest int, where they would be taken for shots."""
    h = sparse(3, 6, 2, 1)
    # 2^31 - 1 = 27 * 79536431 + 10 shots: the last chunk has 10, its block 10 more chunks' at most
    syn = (np.random.default_rng(2).random((10, 3)) < 0.5).astype(np.int32)
    cfg = (2, 256, 0, 64, 10, -1)
    res = decode(route, tmp_path, [((h, 0, 0, cfg, []), {"Ho": h})], list(syn), [0] * 10, mode="edge")
    prc, want, _ = port.css(O.UNIFORM, h, h, None, syn, O.Config(*cfg), "x")
    assert prc == 0 and len(O.fields_equal(res, want)) == 0


@pytest.mark.parametrize("shots", [1, 70])
def test_long_levels_go_to_the_decode_kernel(route, port, tmp_path, shots):
    """Columns of weight 5 on 24 rows: sets of three columns make levels of some 18000 pairs.
    Such a shot is left to the decode kernel's warps; those beside it in the warp are not."""
    h = sparse(24, 230, 5, 7)
    rng = np.random.default_rng(3)
    e = np.zeros((shots, 230), np.int32)
    for i in range(shots):
        e[i, rng.choice(230, 4 if i % 23 == 0 else 1 + i % 2, replace=False)] = 1
    cfg = (4, 256, 0, 230, 10, -1)
    res, info = decode(route, tmp_path, [((h, 0, 1, cfg, []), {"Ho": h})], list(e), [0] * shots)
    prc, want, _ = port.css(O.UNIFORM, h, h, e, None, O.Config(*cfg), "x")
    assert prc == 0 and len(O.fields_equal(res, want)) == 0
    long = -(-shots // 23)
    assert info["guided"] == 1 and info["slow"] == long == info["jobs"], info
    assert info["settled"] + info["searched"] == shots - long, info


def test_more_codes_than_a_block_copies(route, port, tmp_path):
    """Ten codes: the descriptors past the eighth are read from memory, guided and general alike."""
    bb = synth.BB_CODES[72]()
    hs = [bb.hz if i % 3 else sparse(60, 100, 9, i) for i in range(10)]
    cfgs = [(1 + i % 4, 256, 0, 64, 10, (-1, 0, 1)[i % 3]) for i in range(10)]
    rng = np.random.default_rng(12)
    which = rng.permutation(np.repeat(np.arange(10), 12))
    recs = []
    for k in which:
        e = np.zeros(hs[k].shape[1], np.int32)
        e[rng.choice(len(e), int(rng.integers(0, 4)), replace=False)] = 1
        recs.append(e)
    res, info = decode(route, tmp_path, [((h, 0, 1, c, []), {"Ho": h}) for h, c in zip(hs, cfgs)], recs, which)
    for k in range(10):
        idx = np.nonzero(which == k)[0]
        prc, want, _ = port.css(O.UNIFORM, hs[k], hs[k], np.stack([recs[i] for i in idx]), None,
                                O.Config(*cfgs[k]), "x")
        assert prc == 0 and len(O.fields_equal(res[idx], want)) == 0, k
    assert info["guided"] == 1 and info["searched"] > 0 and info["slow"] > 0, info


@pytest.mark.parametrize("shots", [1, 16, 17])
def test_a_warp_for_every_shot(route, port, tmp_path, shots):
    """Codes without tables, up to a shot per resident warp (16 on the plan's one SM): no chunk step;
    one shot more and empty records are settled there."""
    h = sparse(60, 120, 9, 13)
    e = np.zeros((shots, 120), np.int32)
    for i in range(shots):
        e[i, :i % 3] = 1
    cfg = (2, 256, 0, 64, 10, -1)
    res, info = decode(route, tmp_path, [((h, 0, 1, cfg, []), {"Ho": h})], list(e), [0] * shots)
    prc, want, _ = port.css(O.UNIFORM, h, h, e, None, O.Config(*cfg), "x")
    assert prc == 0 and len(O.fields_equal(res, want)) == 0
    assert info["guided"] == 0 and info["slow"] == (shots if shots <= 16 else 5), info
