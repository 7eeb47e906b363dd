"""Performance cases: the work users give this decoder, through its public entry points.

Every case decodes shots of one of the repository's own codes (BB[[72]], [[108]], [[144]],
[[288]] and the random 120 x 720 detector error model), drawn with the noise its benchmark
workloads use or a stated range around it.  A case is a dict of plain values:

  path     "host"   the C ABI on host buffers (grand_decode_*), as a ctypes caller uses it
           "device" the engine on device-resident records, replayed from its CUDA graph
           "sample" shots drawn on the device, then decoded there (error-rate runs)
           "noalloc" grand_decode_cc_noalloc on device buffers
           "server" a burst of requests through the continuous-batching server
  code     72, 108, 144, 288, "dem", or "mix" (the four BB codes, shuffled)
  variant  "uniform", "prob" or "ml"
  records  "errors" or "syndromes" (CSS), "detectors" (DEM)
  noise    "iid" (probability p per position), "loguniform" (each position's own
           probability, log-uniform in [p_lo, p]) or "random" (every check drawn by a coin
           of density p: shots nothing explains)

A result has ten deterministic fields and four measured times; the times are measurements,
not answers, so run() returns the former.  Every output is a whole number except the ML
costs, which are sums of the FP32 log-likelihoods of the decoded positions.
"""
import ctypes
import math
import tempfile

import numpy as np
import torch

from library_s_grand_gb300 import capi, engine, server, synth, workloads

FIELDS = ("found", "found_weight", "original_weight", "degenerate", "is_equal", "tam",
          "total_tested_combinations", "hibrido", "iteration")
RESULT_BYTES = 72

#: phase masks: weights 1..5 in one phase, and weight 6 after (or, for small sets, before) it
PHASES = {"one": [(300, 0, 1, 2, 1.0, 0.0, 0.0)],
          "two": [(8, 1, 0, 2, 0.3, 0.7, 0.0), (300, 0, 1, 2, 0.9, 0.1, 0.0)]}


def _case(name, path, code, variant, records, shots, W, noise, p, p_lo=0.0, cap=64, mode=-1,
          error_type="x", phases="one", packed=False, full=False):
    c = dict(path=path, code=code, variant=variant, records=records, shots=shots, W=W,
             noise=noise, p=p, p_lo=p_lo, cap=cap, mode=mode, error_type=error_type,
             phases=phases, packed=packed, full=full)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one syndrome at a time: an experiment that decodes as it measures
        _case("host_cc_bb144_1", "host", 144, "uniform", "syndromes", 1, 3, "iid", 0.01),
        # the smallest batch of the example scripts: 1024 errors of BB[[72,12,6]]
        _case("host_cc_bb72_1024", "host", 72, "uniform", "errors", 1024, 3, "iid", 0.005),
        # the headline batch from host buffers, and device-resident
        _case("host_prob_bb144_16384", "host", 144, "prob", "errors", 16384, 4, "loguniform",
              1e-2, 1e-3),
        _case("device_prob_bb144_16384", "device", 144, "prob", "errors", 16384, 4, "loguniform",
              1e-2, 1e-3),
        # bit-packed records, the largest code, Z errors, an odd number of shots
        _case("host_cc_bb288_packed_5003", "host", 288, "uniform", "errors", 5003, 4, "iid",
              0.003, error_type="z", packed=True),
        # logical error rate of a detector error model: shots drawn and decoded on the device
        _case("sample_ml_dem_65536", "sample", "dem", "ml", "detectors", 65536, 3, "loguniform",
              5e-3, 1e-4),
        # detector shots with a phase file up to weight 6, patterns and logicals returned
        _case("host_prob_dem_3001", "host", "dem", "prob", "detectors", 3001, 6, "loguniform",
              5e-3, 1e-4, cap=20, phases="two", full=True),
        # a loop that may not allocate
        _case("noalloc_bb108_2000", "noalloc", 108, "uniform", "syndromes", 2000, 3, "iid", 0.005),
        # the mixed-code batch, 25000 shots of each BB code
        _case("device_mix_100000", "device", "mix", "uniform", "syndromes", 100000, 4, "iid",
              workloads.MIX_P),
        # the upper end of a threshold sweep: many shots exhaust every pattern up to weight 4
        _case("device_cc_bb288_noisy_20000", "device", 288, "uniform", "syndromes", 20000, 4, "iid",
              0.01),
        # detectors nothing explains: every candidate of the capped active sets is ruled out
        _case("device_cln_dem_random_8192", "device", "dem", "uniform", "detectors", 8192, 3,
              "random", workloads.STRESS_DEM_DENSITY),
        # serving: a burst of 64 requests of 1-256 shots, the four BB codes and the ML DEM
        _case("server_mix_64", "server", "mix", "ml", "syndromes", 64, 3, "iid", workloads.MIX_P),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["host", "host", "host", "device", "device", "device", "sample", "noalloc",
                       "server"])
    if path == "server":
        return _case(None, path, "mix", "ml", "syndromes", rng.randint(5, 96), 3, "iid",
                     rng.choice([0.001, 0.003, 0.005]))
    if path == "noalloc":
        return _case(None, path, rng.choice([72, 108, 144]), "uniform", "syndromes",
                     _log_int(rng, 1, 6000), rng.choice([2, 3, 4]), "iid",
                     round(rng.uniform(0.001, 0.008), 4), error_type=rng.choice("xz"))
    kind = rng.choice(["css", "css", "dem", "random"] + (["mix"] if path == "device" else []))
    if path == "sample" and kind == "random":
        kind = "css"
    if kind == "mix":
        return _case(None, path, "mix", "uniform", "syndromes", 4 * _log_int(rng, 100, 25000), 4,
                     "iid", round(rng.uniform(0.001, 0.005), 4))
    if kind == "random":  # records nothing explains
        if rng.random() < 0.5:
            return _case(None, path, 144, "uniform", "syndromes", _log_int(rng, 10, 192), 4,
                         "random", 0.5)
        return _case(None, path, "dem", "uniform", "detectors", _log_int(rng, 100, 8192), 3,
                     "random", workloads.STRESS_DEM_DENSITY)
    if kind == "dem":
        variant = rng.choice(["uniform", "prob", "ml"])
        W = {"uniform": rng.choice([2, 3]), "prob": rng.choice([5, 6]), "ml": 3}[variant]
        cap = 20 if variant == "prob" else rng.choice([24, 40, 64])
        return _case(None, path, "dem", variant, "detectors",
                     _log_int(rng, 1, 4000 if variant == "prob" else 60000), W, "loguniform", 5e-3,
                     1e-4, cap=cap, mode=rng.choice([-1, -1, 1]), phases=rng.choice(["one", "two"]),
                     packed=path == "host" and rng.random() < 0.3,
                     full=path == "host" and rng.random() < 0.5)
    code = rng.choice([72, 108, 144, 288])
    variant = rng.choice(["uniform", "uniform", "prob"])
    packed = path == "host" and rng.random() < 0.3
    records = rng.choice(["errors", "syndromes"])
    p = round(rng.uniform(0.001, 0.005 if code == 288 or variant == "prob" else 0.008), 4)
    return _case(None, path, code, variant, records, _log_int(rng, 1, 20000),
                 rng.choice([3, 4]), rng.choice(["iid", "loguniform"]), p, p / 10,
                 mode=rng.choice([-1, -1, 1]), error_type=rng.choice("xz"), packed=packed,
                 full=path == "host" and not packed and rng.random() < 0.3)


# ---- inputs ------------------------------------------------------------------------------

def _config(case):
    return capi.GrandDecoderConfig(case["W"], 256, 0, case["cap"], 10, case["mode"])


def _rates(case, m):
    """Flip probability of each of the m positions (the same for every seed)."""
    if case["noise"] == "loguniform":
        r = np.random.default_rng(m)
        return np.exp(r.uniform(np.log(case["p_lo"]), np.log(case["p"]), m))
    return np.full(m, case["p"])


def _flips(rng, shots, rates):
    return (rng.random((shots, len(rates)), dtype=np.float32) < rates.astype(np.float32))


def _checks(h, flips):
    """H . e mod 2 (exact: FP32 sums of at most a few thousand ones)."""
    return (flips.astype(np.float32) @ h.T.astype(np.float32)).astype(np.int32) & 1


def _css_records(case, code, shots, rng):
    h = code.hz if case["error_type"] == "x" else code.hx
    if case["noise"] == "random":
        return (rng.random((shots, code.n)) < case["p"]).astype(np.int32)
    e = _flips(rng, shots, _rates(case, code.m))
    return e.astype(np.int32) if case["records"] == "errors" else _checks(h, e)


def _dem_records(case, dem, shots, rng):
    if case["noise"] == "random":
        det = (rng.random((shots, dem.n)) < case["p"]).astype(np.int32)
        return det, np.zeros((shots, dem.n_logicos), np.int32)
    f = _flips(rng, shots, _rates(case, dem.m))
    return _checks(dem.h, f), _checks(dem.l.T, f)


class _State:
    """What a program holds between calls."""


def _aux_file(case, directory, dem=None):
    """The phase or LLR file of the case's variant (None: it reads none)."""
    path = directory + "/aux.txt"
    if case["variant"] == "prob":
        return synth.write_phase_file(path, PHASES[case["phases"]])
    if case["variant"] == "ml":
        return synth.write_llr_file(path, dem.llr)
    return None


def _register(eng, case, code, errors):
    """Registers `code` (a CssCode or a Dem) with the engine as the case asks."""
    with tempfile.TemporaryDirectory() as d:  # the file is read at registration
        if isinstance(code, synth.Dem):
            variant = {"uniform": engine.UNIFORM, "prob": engine.PROB, "ml": engine.ML}
            return eng.add_dem(code.h, code.l, _config(case), variant[case["variant"]],
                               _aux_file(case, d, code))
        return eng.add_css(code.hx, code.hz, case["error_type"], errors, _config(case),
                           _aux_file(case, d))


def _mix_codes(case):
    """(case of the code, code) for the four BB codes with their own largest weights."""
    return [(dict(case, W=min(case["W"], W), variant="uniform"), synth.BB_CODES[n]())
            for n, W in workloads.MIX_SPEC]


def _code(case):
    return synth.random_dem(0) if case["code"] == "dem" else synth.BB_CODES[case["code"]]()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    s = _State()
    s.case, s.seed, s.passes = case, seed, 0
    if case["path"] == "host":
        _prepare_host(s, case, rng)
    elif case["path"] == "noalloc":
        s.lib = capi.load_library()
        code = _code(case)
        h = code.hz if case["error_type"] == "x" else code.hx
        s.n, s.m, s.cfg = code.n, code.m, _config(case)
        s.d_h = torch.from_numpy(h).cuda()
        s.d_rec = torch.from_numpy(_css_records(case, code, case["shots"], rng)).cuda()
        s.d_res = torch.zeros((case["shots"], RESULT_BYTES // 4), dtype=torch.int32, device="cuda")
    elif case["path"] == "server":
        _prepare_server(s, case, rng)
    else:
        _prepare_device(s, case, rng)
    return s


def _prepare_host(s, case, rng):
    s.lib = capi.load_library()
    s.cfg = _config(case)
    code = s.code = _code(case)
    s.dir = tempfile.TemporaryDirectory()
    s.file = _aux_file(case, s.dir.name, code)  # read by every call
    if case["code"] == "dem":
        s.det, s.log = _dem_records(case, code, case["shots"], rng)
        if case["packed"]:
            s.det, s.log = capi.pack_bits(s.det), capi.pack_bits(s.log)
    else:
        rec = _css_records(case, code, case["shots"], rng)
        s.rec = capi.pack_bits(rec) if case["packed"] else rec


def _prepare_device(s, case, rng):
    s.eng = engine.Engine()
    s.d_code = s.d_off = None
    if case["code"] == "mix":
        per = case["shots"] // 4
        rows, codes = [], []
        for c, code in _mix_codes(case):
            codes.append(np.full(per, _register(s.eng, c, code, False), np.int32))
            rows.extend(_css_records(c, code, per, rng))
        order = rng.permutation(len(rows))
        rec = np.concatenate([rows[i] for i in order])
        shot_code = np.concatenate(codes)[order]
        s.d_code = torch.from_numpy(shot_code).cuda()
        s.d_off = torch.from_numpy(engine.offsets_for(s.eng.rec_lens, shot_code)).cuda()
        s.shots = len(rows)
    else:
        s.shots = case["shots"]
        code = _code(case)
        errors = case["records"] == "errors"
        _register(s.eng, case, code, errors)
        if case["path"] == "sample":
            s.d_p = torch.from_numpy(_rates(case, code.m).astype(np.float32)).cuda()
            rec = np.zeros((s.shots, s.eng.rec_lens[0]), np.int32)
        elif case["code"] == "dem":
            rec = np.concatenate(_dem_records(case, code, s.shots, rng), axis=1)
        else:
            rec = _css_records(case, code, s.shots, rng)
    s.d_rec = torch.from_numpy(np.ascontiguousarray(rec)).cuda()
    s.d_res = torch.zeros((s.shots, RESULT_BYTES // 4), dtype=torch.int32, device="cuda")
    s.stream = torch.cuda.current_stream().cuda_stream


def _prepare_server(s, case, rng):
    s.eng = engine.Engine()
    codes = _mix_codes(case)
    for c, code in codes:
        _register(s.eng, c, code, False)
    dem = synth.random_dem(0)
    dem_case = dict(case, noise="loguniform", p=5e-3, p_lo=1e-4)
    _register(s.eng, dem_case, dem, False)
    s.srv = server.Server(s.eng, slots=4, max_shots_per_batch=4096)
    # the requests' sizes and codes are the case's, their shots the seed's
    shape = np.random.default_rng(case["shots"])
    s.sizes = shape.integers(1, 257, case["shots"]).astype(np.int32)
    which = shape.integers(0, 5, case["shots"])
    recs = []
    for n, c in zip(s.sizes, which):
        if c == 4:
            recs.append(np.concatenate(_dem_records(dem_case, dem, n, rng), axis=1).ravel())
        else:
            recs.append(_css_records(*codes[c], n, rng).ravel())
    s.rec = np.concatenate(recs)
    s.shot_code = np.repeat(which, s.sizes).astype(np.int32)
    s.arrival = np.zeros(case["shots"])


# ---- one pass -----------------------------------------------------------------------------

def _fields(res):
    return {f: res[f] for f in FIELDS}


def _checked(rc):
    if rc != 0:
        raise RuntimeError(f"decode failed ({rc})")


def run(state):
    case = state.case
    if case["path"] == "host":
        return _run_host(state, case)
    if case["path"] == "server":
        rc, res, _, _ = state.srv.replay(state.arrival, state.sizes, state.rec, state.shot_code)
        _checked(rc)
        return _fields(res)
    if case["path"] == "noalloc":
        _checked(state.lib.grand_decode_cc_noalloc(
            state.d_h.data_ptr(), state.n, state.m, state.d_rec.data_ptr(), case["shots"],
            ctypes.byref(state.cfg), state.d_res.data_ptr(),
            torch.cuda.current_stream().cuda_stream))
        return state.d_res[:, :10]
    if case["path"] == "sample":
        _checked(state.eng.sample(0, state.d_p.data_ptr(), state.seed, 0, state.shots,
                                  state.d_rec.data_ptr(), state.stream))
    _checked(state.eng.decode_device(
        state.shots, state.d_rec.data_ptr(), state.d_res.data_ptr(), state.stream,
        state.d_code.data_ptr() if state.d_code is not None else 0,
        state.d_off.data_ptr() if state.d_off is not None else 0))
    if case["path"] == "sample":
        return state.d_rec, state.d_res[:, :10]
    return state.d_res[:, :10]


def _run_host(s, case):
    lib, code, cfg = s.lib, s.code, s.cfg
    if case["code"] == "dem":
        if case["packed"]:
            rc, res = capi.decode_dem_packed(lib, case["variant"], code.h, code.l, s.det, s.log,
                                             cfg, s.file)
            _checked(rc)
            return _fields(res)
        if case["full"]:
            rc, res, dec, dlog, cost = capi.decode_dem_ex(lib, case["variant"], code.h, code.l,
                                                          s.det, s.log, cfg, s.file)
            _checked(rc)
            return (_fields(res), dec, dlog) + ((cost,) if case["variant"] == "ml" else ())
        call = {"uniform": capi.run_grand_shots_cln, "prob": capi.run_grand_prob_shots_cln,
                "ml": capi.run_grand_ML_shots_cln}[case["variant"]]
        more = () if s.file is None else (s.file,)
        rc, res = call(lib, code.h, code.l, s.det, s.log, code.n_logicos, cfg, *more)
    elif case["packed"]:
        kind = capi.PACKED_ERRORS if case["records"] == "errors" else capi.PACKED_SYNDROMES
        rc, res = capi.run_grand_shots_cc_packed(lib, code.hx, code.hz, s.rec, kind, cfg,
                                                 case["error_type"], s.file)
    else:
        errors, syn = (s.rec, None) if case["records"] == "errors" else (None, s.rec)
        if case["full"]:
            rc, res, dec = capi.decode_css_ex(lib, case["variant"], code.hx, code.hz, errors, syn,
                                              cfg, case["error_type"], s.file)
            _checked(rc)
            return _fields(res), dec
        et = case["error_type"].encode()
        if case["variant"] == "prob":
            rc, res = capi.run_grand_prob_shots_cc(lib, code.hx, code.hz, errors, syn, cfg, s.file,
                                                   et)
        else:
            rc, res = capi.run_grand_shots_cc(lib, code.hx, code.hz, errors, syn, cfg, et)
    _checked(rc)
    return _fields(np.frombuffer(res, dtype=capi.RESULT_DTYPE))


# ---- floors --------------------------------------------------------------------------------

def _record_bytes(case, rows, cols, logicals):
    """Bytes of one shot's record as the call takes it."""
    entries = cols if case["records"] == "errors" else rows
    if case["packed"]:
        return 4 * ((entries + 31) // 32 + (logicals + 31) // 32)
    return 4 * (entries + logicals)


def work(case):
    """Records and matrices read once, results written once.  How many patterns a shot has to
    try depends on its syndrome, so no operations are counted."""
    if case["code"] == "mix":
        shape = {n: (n // 2, n) for n, _ in workloads.MIX_SPEC}
        per = sum(4 * r for r, _ in shape.values()) / len(shape)
        if case["path"] == "server":
            sizes = np.random.default_rng(case["shots"]).integers(1, 257, case["shots"])
            return {"bytes": float(sizes.sum()) * (per + RESULT_BYTES), "flops": 0}
        return {"bytes": case["shots"] * (per + 12 + RESULT_BYTES), "flops": 0}
    rows, cols, nl = (120, 720, 12) if case["code"] == "dem" else (case["code"] // 2, case["code"], 0)
    shot = _record_bytes(case, rows, cols, nl) + RESULT_BYTES
    if case["path"] == "sample":
        shot += _record_bytes(case, rows, cols, nl)  # written by the sampler, read by the decoder
    total = case["shots"] * shot
    if case["full"]:
        total += case["shots"] * (cols + nl)
    if case["path"] == "host":
        total += 4 * (rows * cols + (cols * nl if nl else rows * cols))
    if case["path"] == "noalloc":
        total += 4 * rows * cols
    return {"bytes": total, "flops": 0}


def exact(case, seed):
    """Whole numbers throughout (and costs of the positions they name): nothing to compare in
    64 bits beyond the answers themselves."""
    return None
