"""The work that is timed: peak-group selection, scoring, quantification and run loading
through the package's public entry points, on seeded synthetic runs.

A case is a run (cycles x isolation windows x peaks per spectrum), a spectral library
(precursors x fragments), the settings of the step, and `kind`, the calls of one pass:

  search    PeakGroupSelection.search of a resident run and library, the candidates read
            into page-locked arrays (the first step of every analysis)
  resident  the same search of a program that searches again and again (calibration
            rounds): search_into with a captured graph, the candidates read back
  stream    libraries in page-locked host arrays searched one after the other against a
            resident run: every pass uploads one (SpecLibFlat.from_arrays), searches it
            and reads its candidates back
  score     PeakGroupScoring.score of candidates that the search found, features read back
  quantify  PeakGroupQuantification.quantify of one candidate per precursor, most of them
            with many of their fragments seen (what is left after the false-discovery
            filter), both tables read back
  load      DIAData.from_arrays of a run whose arrays are on the device, then the search
            of its library: what every new raw file costs before anything else
  file      a raw file in host arrays through everything: run, library, search, scoring
            of the better half of what was found

Candidates come back in arrays with room for every precursor's top n, and their number.
`exact` gives the floating outputs of the same inputs in 64 bits, from plain torch.
"""
import math

import numpy as np
import torch

import alphadia_search_rs_b200 as ads
from alphadia_search_rs_b200 import synth

WINDOW_START = 380.0


def _case(kind, cycles, windows, peaks, precursors, *, frags=(4, 24), rt=(30.0, 400.0), ppm=15.0,
          sigma=2.0, kernel=21, top_n=3, top_k=24, decoys=0.5, precision="fp32", width=2.0,
          cycle_time=1.0, name=None):
    c = dict(kind=kind, cycles=cycles, windows=windows, width=width, peaks=peaks,
             precursors=precursors, frag_min=frags[0], frag_max=frags[1], rt_lo=rt[0], rt_hi=rt[1],
             ppm=ppm, sigma=sigma, kernel=kernel, top_n=top_n, top_k=top_k, decoys=decoys,
             precision=precision, cycle_time=cycle_time)
    if name:
        c["name"] = name
    return c


# Densities, tolerances and kernels are those of the benchmark configurations (synth.CONFIGS)
# and of the default parameters; runs hold fewer isolation windows where a whole one would
# only take longer to generate (a precursor reads one or two windows whatever their number).
def listed():
    return [
        # a small targeted library on a short run: latency and launches
        _case("search", 1000, 8, 1500, 2000, frags=(12, 12), rt=(100.0, 100.0), top_k=12,
              decoys=0.0, width=25.0, name="search_small"),
        # an odd-sized library of uneven precursors with the default parameters' kernel
        # width, tolerance and top-k, RT window given per precursor
        _case("search", 2111, 37, 777, 23_457, rt=(40.0, 200.0), ppm=7.0,
              sigma=1.27, kernel=20, top_k=12, width=3.0, name="search_defaults"),
        # first pass with one RT tolerance for all and 12 fragments each, FP32
        _case("search", 3000, 100, 1000, 66_667, frags=(12, 12), rt=(150.0, 150.0), top_k=12,
              decoys=0.0, name="search_uniform"),
        # batched uneven library with decoys, plain FP32 path
        _case("search", 3000, 120, 1000, 200_000, name="search_uneven"),
        # the whole batched BF16 workload: 300 windows, half a million precursors
        _case("resident", 3000, 300, 1000, 500_000, precision="bf16", name="resident_bf16"),
        # long gradients: 6000 cycles, wide kernel, 10 ppm, top-5, BF16 storage
        _case("search", 6000, 50, 1500, 250_000, rt=(30.0, 600.0), ppm=10.0, sigma=3.0, kernel=31,
              top_n=5, width=1.5, precision="bf16", name="search_long_bf16"),
        # fast cycles searched over most of the run: RT windows of about 4000 cycles
        _case("search", 6000, 12, 600, 6_001, frags=(12, 12), rt=(1000.0, 1000.0), top_k=12,
              decoys=0.0, width=10.0, cycle_time=0.5, name="search_whole_run"),
        # library shards streamed through one selection
        _case("stream", 3000, 60, 1000, 40_000, frags=(12, 12), rt=(150.0, 150.0), top_k=12,
              decoys=0.0, name="stream_uniform"),
        # features of a first pass's candidates
        _case("score", 3000, 60, 1000, 100_000, name="score_uneven"),
        # the same for a small library
        _case("score", 1000, 8, 1500, 2000, frags=(12, 12), rt=(100.0, 100.0), top_k=12,
              decoys=0.0, width=25.0, name="score_small"),
        # quantification of one candidate per precursor
        _case("quantify", 3000, 60, 1000, 100_000, name="quantify_uneven"),
        # a new raw file: loading dominates
        _case("load", 3000, 100, 1000, 30_000, name="load_run"),
    ]


def draw(rng):
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["search", "search", "search", "resident", "stream", "score", "score",
                       "quantify", "load", "file"])
    few = 3000 if kind in ("quantify", "file") else 300
    cycles, peaks = logu(500, 6000), logu(200, 1500)
    windows = min(logu(4, 150), max(4, 300_000_000 // (cycles * peaks)))
    if kind == "file":  # host arrays: a short run
        windows = min(windows, max(4, 20_000_000 // (cycles * peaks)))
    precursors = min(logu(few, 200_000), 4000 * windows)
    frags = rng.choice([(12, 12), (4, 24), (6, 12), (3, 18), (20, 60)])
    if frags[1] > 24:
        precursors = min(precursors, 50_000)
    hi = min(0.4 * cycles, float(logu(40, 700)))
    rt = rng.choice([(hi, hi), (min(30.0, hi / 2), hi)])
    kernel = rng.choice([20, 21, 21, 31, 15])
    precision = "bf16" if kind in ("search", "resident", "stream") and rng.random() < 0.4 else "fp32"
    return _case(kind, cycles, windows, peaks, precursors, frags=frags, rt=rt,
                 ppm=rng.choice([5.0, 7.0, 10.0, 15.0, 20.0]), sigma=rng.choice([1.27, 2.0, 3.0]),
                 kernel=kernel, top_n=rng.choice([1, 3, 3, 5]),
                 top_k=rng.choice([6, 12, 12, 24, 40]), decoys=rng.choice([0.0, 0.5]),
                 precision=precision, width=rng.choice([1.5, 2.0, 4.0, 10.0, 25.0]))


# ------------------------------------------------------------------ inputs

COLUMNS = ("precursor_idx", "rank", "score", "scan_center", "scan_start", "scan_stop",
           "cycle_center", "cycle_start", "cycle_stop")


def _config(case, seed):
    lo = WINDOW_START
    return synth.SynthConfig(
        name="case", n_cycles=case["cycles"], n_windows=case["windows"], window_width=case["width"],
        window_start=lo, peaks_per_spectrum=case["peaks"], n_precursors=case["precursors"],
        frag_min=case["frag_min"], frag_max=case["frag_max"],
        precursor_mz_range=(lo, lo + case["width"] * case["windows"]), charge_range=(2, 3),
        rt_half_window=(case["rt_lo"], case["rt_hi"]), mass_tolerance=case["ppm"],
        sigma_cycles=case["sigma"], kernel_size=case["kernel"], candidate_count=case["top_n"],
        top_k_fragments=case["top_k"], decoy_fraction=case["decoys"], seed=int(seed) % (1 << 40),
        cycle_time=case["cycle_time"])


def _arrays(case, seed):
    """The run's arrays (CUDA tensors) and the library's (numpy)."""
    cfg = _config(case, seed)
    lib = synth.make_library(cfg, "torch", "cuda:0")
    run = synth.make_run(cfg, lib, "torch", "cuda:0")
    return cfg, run, synth.library_arrays(lib)


def _selection(cfg, case, **more):
    p = ads.SelectionParameters()
    p.update(cfg.params_dict())
    return ads.PeakGroupSelection(p, precision=case["precision"], verbose=False, **more)


def _pinned(n, dtype):
    return torch.zeros(n, dtype=getattr(torch, np.dtype(dtype).name), pin_memory=True).numpy()


def _out_arrays(n):
    return tuple(_pinned(max(n, 1), np.float32 if c == "score" else np.uint64) for c in COLUMNS)


def _to_score(columns, n):
    """n candidates of those found, all of them where there are as many."""
    return tuple(np.resize(c, n) for c in columns)


def _to_quantify(case, dia, lib, columns, quant):
    """One candidate for each of the case's precursors: best candidates, as many with one
    fragment seen as with two, and so on up to the longest fragment list."""
    best = tuple(np.ascontiguousarray(c[columns[1] == 0]) for c in columns)
    prec = quant.quantify(dia, lib, ads.CandidateCollection.from_arrays(*best)).to_dict_arrays()[0]
    seen = dict(zip(prec["precursor_idx"].tolist(),
                    (prec["flat_frag_stop_idx"] - prec["flat_frag_start_idx"]).tolist()))
    seen = np.array([seen.get(p, 0) for p in best[0].tolist()])
    top, n = case["frag_max"], case["precursors"]
    of = {k: np.flatnonzero(seen == k) for k in range(1, top + 1)}
    of = {k: rows for k, rows in of.items() if len(rows)}
    many = dict.fromkeys(of, 0)
    left = 0  # fragments short of the even spread, where no candidate has as many as wanted
    for k in range(1, top + 1):
        near = min(of, key=lambda v: (abs(v - k), v))
        many[near] += (n + top - k) // top
        left += (k - near) * ((n + top - k) // top)
    for k in sorted(of):  # made up for by candidates with one fragment more, or less
        more = k + (1 if left > 0 else -1)
        if left and more in of:
            move = min(abs(left), many[k])
            many[k], many[more] = many[k] - move, many[more] + move
            left -= move if left > 0 else -move
    at = np.sort(np.concatenate([np.resize(of[k], many[k]) for k in of]))
    return tuple(np.ascontiguousarray(c[at]) for c in best)


def prepare(case, seed):
    cfg, run, lib = _arrays(case, seed)
    kind = case["kind"]
    st = dict(kind=kind, case=case)
    if kind == "file":
        st["run"], st["lib_np"] = synth.run_to_numpy(run), lib
    elif kind == "load":
        st["run"], st["lib_np"] = run, lib
    else:
        st["dia"] = ads.DIAData.from_arrays(**run)
        if kind == "stream":
            st["lib_np"] = {}
            for k, v in lib.items():
                st["lib_np"][k] = _pinned(v.size, v.dtype)
                st["lib_np"][k][:] = v
        else:
            st["lib"] = ads.SpecLibFlat.from_arrays(**lib)
    del run
    torch.cuda.empty_cache()  # the engine allocates outside torch
    st["sel"] = _selection(cfg, case, use_graph=kind == "resident")
    slots = case["precursors"] * case["top_n"]
    if kind in ("search", "load"):
        st["out"] = _out_arrays(slots)
    elif kind in ("resident", "stream"):
        st["out"] = dict(zip(COLUMNS, _out_arrays(slots)))
        for c in ("scan_center", "scan_start", "scan_stop"):  # always zero, not asked for
            del st["out"][c]
        st["cand"] = st["sel"].new_candidates()
    if kind == "quantify":
        p = ads.QuantificationParameters()
        p.update(dict(tolerance_ppm=case["ppm"]))
        st["quant"] = ads.PeakGroupQuantification(p, verbose=False)
    if kind in ("score", "quantify"):
        cols = st["sel"].search(st["dia"], st["lib"]).to_arrays()
        cols = _to_score(cols, slots) if kind == "score" else \
            _to_quantify(case, st["dia"], st["lib"], cols, st["quant"])
        st["columns"] = cols
        st["cand"] = ads.CandidateCollection.from_arrays(*cols)
    if kind in ("score", "file"):
        p = ads.ScoringParameters()
        p.update(dict(mass_tolerance=case["ppm"]))
        st["scoring"] = ads.PeakGroupScoring(p, verbose=False)
    return st


def run(st):
    kind = st["kind"]
    if kind == "search":
        cand = st["sel"].search(st["dia"], st["lib"])
        cand.to_arrays(out=st["out"])
        return st["out"], len(cand)
    if kind in ("resident", "stream"):
        lib = st["lib"] if kind == "resident" else ads.SpecLibFlat.from_arrays(**st["lib_np"])
        st["sel"].search_into(st["dia"], lib, st["cand"])
        n = st["cand"].copy_out(st["out"])
        return st["out"], n
    if kind == "score":
        return st["scoring"].score(st["dia"], st["lib"], st["cand"]).to_dict_arrays()
    if kind == "quantify":
        return st["quant"].quantify(st["dia"], st["lib"], st["cand"]).to_dict_arrays()
    dia = ads.DIAData.from_arrays(**st["run"])
    lib = ads.SpecLibFlat.from_arrays(**st["lib_np"])
    cand = st["sel"].search(dia, lib)
    if kind == "load":
        cand.to_arrays(out=st["out"])
        return st["out"], len(cand)
    found = cand.to_arrays()
    order = np.argsort(-found[2], kind="stable")[:lib.num_precursors // 2]
    better = ads.CandidateCollection.from_arrays(*[c[np.sort(order)] for c in found])
    return better.to_arrays(), st["scoring"].score(dia, lib, better).to_dict_arrays()


# ------------------------------------------------------------------ work

GRID_LEN = 2_590_781  # 1-ppm bins of 150-2000 m/z


def work(case):
    """Bytes and operations of one pass, from the distributions: CSR offsets and entries of
    the (fragment, window) ranges inside the RT windows, library and results; a stencil of
    half width h and a logarithm per visited XIC cell."""
    P, W = case["precursors"], case["windows"]
    F = min((case["frag_min"] + case["frag_max"]) / 2, case["top_k"])
    raw = (case["frag_min"] + case["frag_max"]) / 2
    C = min(case["cycles"], (case["rt_lo"] + case["rt_hi"]) / case["cycle_time"] + 1)
    h = (case["kernel"] + 1) // 2
    bins = 2 * case["ppm"] + 1
    s = 4 if case["precision"] == "bf16" else 6
    noise = case["peaks"] / math.log(1800.0 / 150.0) * 2e-6 * case["ppm"]  # per cycle and fragment

    def gather(n_cand, frags, cycles):
        per = 4 * (bins + 1) + s * (noise * cycles + 0.6 * min(cycles, 33) * (1 - case["decoys"]))
        return n_cand * frags * per

    lib = P * (8 + 4 + 4 + 16 + 4) + P * raw * 10
    search = gather(P, F, C) + lib + P * case["top_n"] * 44
    flops = P * F * C * (3 * h + 2)
    peaks = case["cycles"] * W * case["peaks"]
    build = peaks * (8 + 6) + 4 * GRID_LEN * W
    n = P // 2 if case["kind"] == "file" else P * case["top_n"]
    score = gather(n, raw, 11) + n * (44 + 41 * 4 + 16) + lib
    kind = case["kind"]
    if kind == "score":
        return dict(bytes=score, flops=n * raw * 11 * 30)
    if kind == "quantify":
        return dict(bytes=gather(P, raw, 11) + P * (40 + 61) + P * raw * 63 + lib, flops=P * raw * 11 * 20)
    if kind == "load":
        return dict(bytes=build + search, flops=flops)
    if kind == "file":
        return dict(bytes=build + search + score, flops=flops + n * raw * 11 * 30)
    return dict(bytes=search + (lib if kind == "stream" else 0), flops=flops)


# ------------------------------------------------------------------ 64-bit values
#
# Decisions (bins, windows, cycle limits, kept fragments) follow the f32 definitions; every
# value computed from intensities is 64-bit.

_GRID = []


def _grid():
    if not _GRID:
        cur, step, v = np.float32(150.0), np.float32(1.0) / np.float32(1e6), []
        while True:
            v.append(cur)
            if not cur < np.float32(2000.0):
                break
            cur = np.float32(cur + np.float32(cur * step))
        _GRID.append(torch.from_numpy(np.array(v, np.float32)).cuda())
    return _GRID[0]


def _closest(mz):
    g = _grid()
    left = torch.searchsorted(g, mz)
    a, b = g[left.clamp(max=len(g) - 1)], g[(left - 1).clamp(min=0)]
    near = torch.where((a - mz).abs() < (b - mz).abs(), left, left - 1)
    near = torch.where((left < len(g)) & (a == mz), left, near)
    return torch.where(left == 0, left, torch.where(left == len(g), left - 1, near))


def _table(run):
    """Peaks sorted by (window, bin, cycle): keys, cycles, intensities; and the windows."""
    start, stop = run["spectrum_peak_start_idx"], run["spectrum_peak_stop_idx"]
    dsi, cyc = run["spectrum_delta_scan_idx"], run["spectrum_cycle_idx"]
    spec = torch.repeat_interleave(torch.arange(len(start), device="cuda"), stop - start)
    n_bin = len(_grid()) + 1
    key = (dsi[spec] * n_bin + _closest(run["peak_mz"])) * 65536 + cyc[spec]
    del spec
    key, order = torch.sort(key, stable=True)
    inten = run["peak_intensity"][order]
    del order
    n_win = int(dsi.max()) + 1
    lo, hi = torch.zeros(n_win, device="cuda"), torch.zeros(n_win, device="cuda")
    first = torch.full((n_win,), len(dsi), device="cuda", dtype=torch.int64)
    first.scatter_reduce_(0, dsi, torch.arange(len(dsi), device="cuda"), "amin")
    lo, hi = run["isolation_lower_mz"][first], run["isolation_upper_mz"][first]
    some = torch.bincount(dsi, weights=(stop - start).double(), minlength=n_win) > 0
    rt = run["spectrum_rt"][dsi == 0]
    return dict(key=key, inten=inten, n_bin=n_bin, lo=lo, hi=hi, some=some, rt=rt)


def _fragments(lib, idx, top_k):
    """Kept fragments of the precursor rows `idx`, in m/z order, padded: rows [n, F], mask."""
    fs = torch.from_numpy(lib["flat_frag_start_idx"].astype(np.int64)).cuda()[idx]
    fe = torch.from_numpy(lib["flat_frag_stop_idx"].astype(np.int64)).cuda()[idx]
    fmax = max(1, int((fe - fs).max())) if len(idx) else 1
    at = fs[:, None] + torch.arange(fmax, device="cuda")
    have = at < fe[:, None]
    at = torch.where(have, at, 0)
    inten = torch.from_numpy(lib["fragment_intensity"]).cuda()[at]
    mz = torch.from_numpy(lib["fragment_mz"]).cuda()[at]
    y1 = (torch.from_numpy(lib["fragment_type"]).cuda()[at] == 121) & \
        (torch.from_numpy(lib["fragment_number"]).cuda()[at] == 1)
    keep = have & (inten > 0) & ~y1
    by = torch.argsort(torch.where(keep, -inten, math.inf), dim=1, stable=True)
    rank = torch.argsort(by, dim=1)
    keep &= rank < top_k
    order = torch.argsort(torch.where(keep, mz, math.inf), dim=1, stable=True)
    at, keep = torch.gather(at, 1, order), torch.gather(keep, 1, order)
    F = max(1, int(keep.sum(1).max())) if len(idx) else 1
    return at[:, :F], keep[:, :F]


def _xic(T, pmz, fmz, keep, cs, ce, C, ppm, want_mz=False):
    """Dense XIC [n, F, C] (64 bits) over each row's cycles [cs, ce), and with `want_mz`
    the intensity-weighted bin m/z."""
    n, F = keep.shape
    g, nb = _grid(), T["n_bin"]
    tol = torch.tensor(ppm, dtype=torch.float32, device="cuda")
    delta = (fmz * tol) * torch.tensor(1e-6, dtype=torch.float32, device="cuda")
    b0 = torch.searchsorted(g, (fmz - delta).contiguous())
    b1 = torch.maximum(b0, torch.searchsorted(g, (fmz + delta).contiguous(), right=True))
    row, col = torch.nonzero(keep, as_tuple=True)
    xic = torch.zeros(n * F * C, dtype=torch.float64, device="cuda")
    num = torch.zeros_like(xic) if want_mz else None
    hit = (T["lo"][None] <= pmz[:, None]) & (T["hi"][None] >= pmz[:, None]) & T["some"][None]
    depth = int(hit.sum(1).max()) if n else 0
    wins = torch.argsort((~hit).to(torch.uint8), dim=1, stable=True)[:, :max(depth, 1)]
    for k in range(depth):
        ok = torch.gather(hit, 1, wins[:, k:k + 1])[:, 0][row]
        r, f = row[ok], col[ok]
        base = wins[r, k] * nb
        e0 = torch.searchsorted(T["key"], (base + b0[r, f]) * 65536)
        e1 = torch.searchsorted(T["key"], (base + b1[r, f]) * 65536)
        many = e1 - e0
        first = torch.cumsum(many, 0) - many
        total = int(many.sum())
        own = torch.repeat_interleave(torch.arange(len(r), device="cuda"), many)
        e = e0[own] + torch.arange(total, device="cuda") - first[own]
        key, rr = T["key"][e], r[own]
        c = key & 65535
        # of several entries of a bin at the window's first cycle only the last counts
        last = T["key"][(e + 1).clamp(max=len(T["key"]) - 1)] != key
        last |= e + 1 >= len(T["key"])
        use = (c >= cs[rr]) & (c < ce[rr]) & ((c > cs[rr]) | last)
        e, own, c, rr = e[use], own[use], c[use], rr[use]
        cell = (rr * F + f[own]) * C + (c - cs[rr])
        v = T["inten"][e].double()
        xic.index_add_(0, cell, v)
        if want_mz:
            num.index_add_(0, cell, v * g[(T["key"][e] >> 16) % nb].double())
    xic = xic.view(n, F, C)
    if not want_mz:
        return xic
    return xic, torch.where(xic > 0, num.view(n, F, C) / xic, 0.0)


def _taps(case):
    width = math.ceil(case["kernel"] / 2) * 2
    fwhm = float(np.float32(np.float32(case["sigma"] * 2.3548)))
    s = fwhm / 2.3548
    w = [math.exp(-0.5 * x * x / (s * s)) for x in range(-(width // 2), width // 2)]
    total = sum(w)
    return [x / total for x in w]


def _exact_search(case, T, lib):
    """Scores of the candidates in precursor_idx order, best first.  None where a precursor's
    number of candidates hangs on 32-bit rounding."""
    w = _taps(case)
    L, h = len(w), len(w) // 2
    order = torch.from_numpy(np.argsort(lib["precursor_idx"], kind="stable")).cuda()
    rt, prt = T["rt"], torch.from_numpy(lib["precursor_rt"]).cuda()
    n_rt = len(rt)
    dt = (rt[-1] - rt[0]) / (n_rt - 1)
    tol = torch.from_numpy(lib["precursor_rt_tolerance"]).cuda() if "precursor_rt_tolerance" in lib \
        else torch.full_like(prt, case["rt_hi"])
    eff = torch.maximum(tol, (10.0 + case["kernel"]) * dt)
    lower, upper = prt - eff, prt + eff
    lo = torch.where(lower <= rt[0], 0, torch.searchsorted(rt, lower))
    hi = torch.where(upper >= rt[-1], n_rt, torch.searchsorted(rt, upper))
    none = upper < rt[0]
    lo, hi = torch.where(none, 0, lo), torch.where(none, 0, hi)
    none = lower > rt[-1]
    lo, hi = torch.where(none, n_rt, lo), torch.where(none, n_rt, hi)
    pmz = torch.from_numpy(lib["precursor_mz"]).cuda()
    fint, fmz = torch.from_numpy(lib["fragment_intensity"]).cuda(), torch.from_numpy(lib["fragment_mz"]).cuda()
    # rows of similar window length together
    by_len = torch.argsort((hi - lo)[order])
    K = case["top_n"]
    best = torch.full((len(order), K), math.nan, dtype=torch.float64, device="cuda")
    a = 0
    while a < len(order):
        longest = int((hi - lo)[order[by_len[min(a, len(order) - 1)]]])
        step = max(1, int(4e7 / max(1, 24 * (longest + 64))))
        at = by_len[a:a + step]
        a += step
        idx = order[at]
        cs, ce = lo[idx], hi[idx]
        C = int((ce - cs).max()) if len(idx) else 0
        if C < max(L + 1, 5):
            continue
        rows, keep = _fragments(lib, idx, case["top_k"])
        x = _xic(T, pmz[idx], fmz[rows], keep, cs, ce, C, case["ppm"])
        j, n = torch.arange(C, device="cuda"), (ce - cs)[:, None]
        weight = torch.where(keep, fint[rows], 0.0)
        found = []
        for t in (torch.float32, torch.float64):
            y = x.to(t)
            conv = torch.zeros_like(y)
            conv[..., h:C - h] = w[h] * y[..., h:C - h]
            for d in range(1, h + 1):
                conv[..., h:C - h] += w[h - d] * (y[..., h - d:C - h - d] + y[..., h + d:C - h + d])
            conv *= (j[None] < n - h)[:, None]
            s = (torch.log(conv + 1) * weight.to(t)[..., None]).sum(1)
            del y, conv
            peak = torch.zeros_like(s, dtype=torch.bool)
            peak[:, 2:-2] = (s[:, :-4] < s[:, 1:-3]) & (s[:, 1:-3] < s[:, 2:-2]) & \
                (s[:, 2:-2] > s[:, 3:-1]) & (s[:, 3:-1] > s[:, 4:])
            peak &= (j[None] < n - 2) & (n >= max(L + 1, 5))
            found.append(peak.sum(1).clamp(max=K))
        if not torch.equal(*found):
            return None
        top = torch.sort(torch.where(peak, s, -math.inf), dim=1, descending=True, stable=True).values[:, :K]
        best[at, :top.shape[1]] = torch.where(torch.isfinite(top), top, math.nan)
    flat = best.view(-1)
    return flat[~torch.isnan(flat)].cpu().numpy()


def _median(v, mask):
    """Median over dim 1 of v [n, F, ...] where mask [n, F]."""
    m = mask.view(mask.shape + (1,) * (v.dim() - 2))
    s = torch.sort(torch.where(m, v, math.inf), dim=1).values
    R = mask.sum(1).view((-1, 1) + (1,) * (v.dim() - 2)).expand((-1, 1) + v.shape[2:])
    a = torch.gather(s, 1, ((R - 1) // 2).clamp(min=0))
    b = torch.gather(s, 1, (R // 2).clamp(max=v.shape[1] - 1))
    return torch.where(R > 0, (a + b) / 2, 0.0)[:, 0]


def _pearson(x, y, mask):
    """Correlation over the last dim where mask (broadcastable); 0 where it is undefined."""
    mask = mask.expand(torch.broadcast_shapes(x.shape, y.shape, mask.shape)).double()
    n = mask.sum(-1)
    xs, ys = (x * mask).sum(-1), (y * mask).sum(-1)
    dx, dy = (x - (xs / n)[..., None]) * mask, (y - (ys / n)[..., None]) * mask
    xv, yv = (dx * dx).sum(-1), (dy * dy).sum(-1)
    r = (dx * dy).sum(-1) / (xv.sqrt() * yv.sqrt())
    ok = (xs != 0) & (ys != 0) & (xv != 0) & (yv != 0) & torch.isfinite(r)
    return torch.where(ok, r, 0.0).clamp(-1, 1)


def _profiles(case, T, lib, idx, cs, ce, top_k):
    """What scoring and quantification share, per candidate: kept fragments, XIC, observed
    m/z, normalised profiles, the median of the non-zero ones, correlations."""
    fmz = torch.from_numpy(lib["fragment_mz"]).cuda()
    rows, keep = _fragments(lib, idx, top_k)
    C = int((ce - cs).max())
    x, mz = _xic(T, torch.from_numpy(lib["precursor_mz"]).cuda()[idx], fmz[rows], keep, cs, ce, C,
                 case["ppm"], want_mz=True)
    n = ce - cs
    j = torch.arange(C, device="cuda")
    valid = j[None] < n[:, None]
    half = n // 2
    c0, c1 = torch.where(half > 1, half - 1, 0), torch.minimum(half + 2, n)
    near = (j[None] >= c0[:, None]) & (j[None] < c1[:, None])
    mean = (x * near[:, None]).sum(-1) / (c1 - c0).clamp(min=1)[:, None]
    norm = torch.where(mean[..., None] > 0, x / mean[..., None], 0.0)
    nz = (norm != 0).any(-1) & keep
    med, med_nz = _median(norm, keep), _median(norm, nz)
    corr = _pearson(med_nz[:, None], norm, valid[:, None])
    obs = x.sum(-1)
    seen = obs > 0
    o = torch.where(seen, (mz * x).sum(-1) / obs, 0.0)
    lib_mz = fmz[rows].double()
    err = torch.where(o > 0, (o - lib_mz) / lib_mz * 1e6, 0.0)
    return dict(rows=rows, keep=keep, x=x, nz=nz, med=med, med_nz=med_nz, corr=corr, obs=obs, o=o,
                err=err, half=half, C=C, valid=valid)


def _gamma_ln(x):
    v = (x - 0.5) * torch.log(x.clamp(min=1e-300)) - x + 0.5 * 1.837877
    return torch.where((x <= 0) | ((x - 1).abs() < 1e-6) | ((x - 2).abs() < 1e-6), 0.0, v)


def _hyperscore(is_b, is_y, v, mask, w=None):
    use = mask & (v != 0)
    wi = v if w is None else v * w
    out = 0.0
    for t in (is_b, is_y):
        u = use & t
        s = torch.where(u, wi, 0.0).sum(1)
        out = out + torch.where(u.any(1), _gamma_ln(u.sum(1).double() + 1), 0.0)
        out = out + torch.where(s > 0, torch.log(s.clamp(min=1e-300)), 0.0)
    out = torch.where((use & (is_b | is_y)).any(1), out, 0.0)
    return torch.where(torch.isfinite(out), out, 0.0)


def _series(is_t, number, mask):
    """Longest run of consecutive numbers (a repeated number starts a new run)."""
    use = mask & is_t
    s = torch.sort(torch.where(use, number.long(), 100_000), dim=1).values
    longest = torch.where(use.any(1), 1, 0)
    cur = longest.clone()
    for k in range(1, s.shape[1]):
        real = s[:, k] < 100_000
        cur = torch.where(real & (s[:, k] == s[:, k - 1] + 1), cur + 1, 1)
        longest = torch.where(real, torch.maximum(longest, cur), longest)
    return longest


def _rank(v, keep):
    by = torch.argsort(torch.where(keep, -v, math.inf), dim=1, stable=True)
    return torch.argsort(by, dim=1)


def _lookup(lib, cols):
    order = np.argsort(lib["precursor_idx"], kind="stable")
    at = np.searchsorted(lib["precursor_idx"][order], cols["precursor_idx"])
    idx = torch.from_numpy(order[at]).cuda()
    i64 = {k: torch.from_numpy(cols[k].astype(np.int64)).cuda()
           for k in ("cycle_center", "cycle_start", "cycle_stop")}
    return idx, i64["cycle_center"], i64["cycle_start"], i64["cycle_stop"]


def _features(case, T, lib, cols, a, b, counts):
    c = {k: v[a:b] for k, v in cols.items()}
    idx, center, cs, ce = _lookup(lib, c)
    p = _profiles(case, T, lib, idx, cs, ce, 100)
    keep, corr, obs, rows = p["keep"], p["corr"], p["obs"], p["rows"]
    F = keep.sum(1)
    fint = torch.from_numpy(lib["fragment_intensity"]).cuda()[rows]
    ftype = torch.from_numpy(lib["fragment_type"]).cuda()[rows]
    fnum = torch.from_numpy(lib["fragment_number"]).cuda()[rows]
    is_b, is_y = (ftype == 98) & keep, (ftype == 121) & keep
    corr = torch.where(keep, corr, 0.0)
    match = (obs > 0) & keep
    cnt = counts[_closest(torch.from_numpy(lib["fragment_mz_library"]).cuda()[rows])]
    # the fragment total over the count is a 32-bit quotient by definition
    idf = torch.where(keep, torch.log((float(len(lib["fragment_mz"])) / cnt.clamp(min=1).double())), 0.0)
    mean = corr.sum(1) / F.clamp(min=1)
    dev = torch.where(keep, corr - mean[:, None], 0.0)
    std = torch.where(F > 1, ((dev * dev).sum(1) / (F - 1).clamp(min=1)).sqrt(), 0.0)
    band = torch.where(keep, _rank(fint, keep) // 6, 99)
    top6 = keep & (_rank(idf, keep) < 6)
    rt = T["rt"].double()
    half, M = p["half"], p["med_nz"]
    cen = torch.gather(M, 1, half.clamp(max=p["C"] - 1)[:, None])[:, 0]
    fwhm = torch.zeros(len(F), dtype=torch.float64, device="cuda")
    done = torch.zeros(len(F), dtype=torch.bool, device="cuda")
    for k in range(p["C"] // 2 + 1):
        lo, hi = (half - k).clamp(min=0), (half + k).clamp(max=p["C"] - 1)
        m = (torch.gather(M, 1, lo[:, None]) + torch.gather(M, 1, hi[:, None]))[:, 0] / 2
        now = (k < half) & ~done & (m <= cen / 2)
        width = rt[(cs + half + k).clamp(max=len(rt) - 1)] - rt[(cs + half - k).clamp(min=0)]
        fwhm = torch.where(now, width, fwhm)
        done |= now
    rt_obs = rt[center]
    w = torch.where(keep & (p["err"] != 0), fint.double(), 0.0)
    ws = w.sum(1)
    wmae = torch.where(ws > 0, (p["err"].abs() * w).sum(1) / ws.clamp(min=1e-300), 0.0)

    def log10(v):
        return torch.log10(v + 1e-8)

    f = {
        "score": torch.from_numpy(c["score"]).cuda(), "mean_correlation": mean,
        "median_correlation": _median(corr[..., None], keep)[:, 0], "correlation_std": std,
        "intensity_correlation": _pearson(obs, fint.double(), keep), "num_fragments": F, "num_scans": ce - cs,
        "num_profiles": F, "num_profiles_filtered": p["nz"].sum(1), "rt_observed": rt_obs,
        "delta_rt": rt_obs - torch.from_numpy(lib["precursor_rt"]).cuda()[idx].double(),
        "longest_b_series": _series(is_b, fnum, match), "longest_y_series": _series(is_y, fnum, match),
        "naa": torch.from_numpy(lib["precursor_naa"]).cuda()[idx], "weighted_mass_error": wmae,
        "hyperscore_intensity_observation": _hyperscore(is_b, is_y, obs, match),
        "hyperscore_intensity_library": _hyperscore(is_b, is_y, fint.double(), match),
        "hyperscore_inverse_mass_error": _hyperscore(is_b, is_y, obs, match, 1 / (p["err"].abs() + 0.1)),
        "log10_b_ion_intensity": log10(torch.where(is_b & match, obs, 0.0).sum(1)),
        "log10_y_ion_intensity": log10(torch.where(is_y & match, obs, 0.0).sum(1)),
        "fwhm_rt": fwhm, "idf_hyperscore": _hyperscore(is_b, is_y, idf, match),
        "idf_xic_dot_product": (idf * corr).sum(1), "idf_intensity_dot_product": log10((idf * obs).sum(1)),
        "median_profile_sum": p["med"].sum(1), "median_profile_sum_filtered": p["med_nz"].sum(1),
        "num_over_0_top6_idf": (top6 & (corr > 0)).sum(1), "num_over_50_top6_idf": (top6 & (corr > 0.5)).sum(1),
    }
    for t in (95, 90, 80, 50, 0):
        f["num_over_%d" % t] = (keep & (corr > t / 100)).sum(1)
    for t in (0, 50):
        for r in range(4):
            f["num_over_%d_rank_%d_%d" % (t, 6 * r, 6 * r + 5)] = ((band == r) & (corr > t / 100)).sum(1)
    return {k: v.double().cpu().numpy() for k, v in f.items()}


def _chunks(n, case):
    step = max(1, int(1.5e7 / (11 * max(24, case["frag_max"]))))
    return [(a, min(n, a + step)) for a in range(0, n, step)]


def _exact_score(case, T, lib, cols):
    counts = torch.bincount(_closest(torch.from_numpy(lib["fragment_mz_library"]).cuda()), minlength=len(_grid()))
    parts = [_features(case, T, lib, cols, a, b, counts) for a, b in _chunks(len(cols["rank"]), case)]
    out = {k: np.concatenate([p[k] for p in parts]) for k in parts[0]} if parts else {}
    return {"precursor_idx": None, "rank": None, **out}


def _exact_quantify(case, T, lib, cols):
    prec, frag = [], []
    rt, fmz = T["rt"].double(), torch.from_numpy(lib["fragment_mz"]).cuda().double()
    for a, b in _chunks(len(cols["rank"]), case):
        c = {k: v[a:b] for k, v in cols.items()}
        idx, center, cs, ce = _lookup(lib, c)
        p = _profiles(case, T, lib, idx, cs, ce, 10000)
        use = p["keep"] & (p["obs"] > 0)
        some = use.any(1)
        host = idx[some].cpu().numpy()
        prec.append(np.stack([c["precursor_idx"][some.cpu().numpy()].astype(np.float64),
                              lib["precursor_mz_library"][host], lib["precursor_mz"][host],
                              lib["precursor_rt_library"][host], lib["precursor_rt"][host],
                              rt[center[some]].cpu().numpy()]))
        r = p["rows"][use]
        frag.append(torch.stack([fmz[r], p["obs"][use], p["o"][use], p["corr"][use], p["err"][use]]).cpu().numpy())
    prec, frag = np.concatenate(prec, 1), np.concatenate(frag, 1)
    prec = prec[:, np.argsort(prec[0], kind="stable")]
    none = dict.fromkeys(("precursor_idx", "naa", "rank", "flat_frag_start_idx", "flat_frag_stop_idx"))
    return ({**none, "mz_library": prec[1], "mz": prec[2], "rt_library": prec[3], "rt": prec[4],
             "rt_observed": prec[5]},
            {**dict.fromkeys(("cardinality", "charge", "loss_type", "number", "position", "type",
                              "precursor_idx", "rank")),
             "mz_library": frag[0], "mz": frag[0], "intensity": frag[1], "mz_observed": frag[2],
             "correlation_observed": frag[3], "mass_error_observed": frag[4]})


def exact(case, seed):
    kind = case["kind"]
    cells = case["precursors"] * min(case["cycles"], (case["rt_lo"] + case["rt_hi"]) / case["cycle_time"]) * \
        min((case["frag_min"] + case["frag_max"]) / 2, case["top_k"])
    if kind not in ("score", "quantify") and cells > (1e8 if case["precision"] == "bf16" else 6e8):
        # among so many, some precursor's number of candidates hangs on rounding (of the
        # BF16 path's logarithm sooner), and every later row would be another one's
        return None
    cols = None
    if kind in ("score", "quantify"):  # the candidates that prepare() hands to the step
        cols = dict(zip(COLUMNS, prepare(case, seed)["columns"]))
    _, run_arrays, lib = _arrays(case, seed)
    torch.cuda.empty_cache()
    T = _table(run_arrays)
    if case["precision"] == "bf16":  # intensities as this storage holds them
        T["inten"] = T["inten"].bfloat16().float()
    del run_arrays
    torch.cuda.empty_cache()
    if kind == "score":
        return _exact_score(case, T, lib, cols)
    if kind == "quantify":
        return _exact_quantify(case, T, lib, cols)
    score = _exact_search(case, T, lib)
    if score is None:
        return None
    if kind == "file":
        half = len(lib["precursor_idx"]) // 2
        score = score[np.sort(np.argsort(-score, kind="stable")[:half])]
        return (None, None, score) + (None,) * 6, None
    score = np.pad(score, (0, max(0, case["precursors"] * case["top_n"] - len(score))))
    if kind in ("resident", "stream"):
        return {"score": score}, None
    return (None, None, score) + (None,) * 6, None
