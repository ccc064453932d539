"""GPU parity where a call meets a limit of its kernels or of the device: ranges past the
last cycle index, work done in parts, calls that fail half way, buffers and handles that
take one another's place."""
import numpy as np
import pytest

import oracle
from alphadia_search_rs_b200 import (CandidateCollection, DIAData, PeakGroupQuantification,
                                     PeakGroupScoring, PeakGroupSelection, QuantificationParameters,
                                     ScoringParameters, SpecLibFlat, mz_grid, synth)

from _util import COLS, RUN_KEYS, assert_candidates_equal, params_from
from test_gpu_quant import assert_quant_equal, quant_library
from test_gpu_scoring import assert_features_equal, build
from test_gpu_sizes import PARAMS, closest_bins, library_of, run_of, search_both

pytestmark = pytest.mark.gpu


def candidates_at(pidx, start, stop):
    start, stop = np.asarray(start, np.uint64), np.asarray(stop, np.uint64)
    c = dict(precursor_idx=np.asarray(pidx, np.uint64), rank=np.arange(len(start), dtype=np.uint64),
             score=np.linspace(1, 2, len(start), dtype=np.float32), cycle_start=start, cycle_stop=stop,
             cycle_center=(start + stop - np.uint64(1)) // np.uint64(2))
    for k in ("scan_center", "scan_start", "scan_stop"):
        c[k] = np.zeros(len(start), np.uint64)
    return c


def assert_scored_and_quantified(run, la, cands, where):
    dia, slib, od, ol = build(run, la)
    cc = CandidateCollection.from_arrays(*(cands[k] for k in COLS))
    got = PeakGroupScoring(ScoringParameters(), verbose=False).score(dia, slib, cc).to_dict_arrays()
    assert_features_equal(got, oracle.score(od, ol, cands, log_mode=oracle.LOG_RN), exact=True, where=where)
    q = PeakGroupQuantification(QuantificationParameters(), verbose=False).quantify(dia, slib, cc)
    assert_quant_equal(q, oracle.quantify(od, ol, cands, la), where=where)


@pytest.mark.parametrize("start,stop", [(65525, 65536), (65526, 65537), (65530, 65541), (65535, 65546),
                                        (65500, 65600)])
def test_cycle_ranges_past_the_last_cycle_index(start, stop):
    """A run of more than 65,536 MS1 spectra: candidates whose cycles end past 65,535, the
    last that an entry can have.  (The reference has no value for ranges that start past it:
    it searches the entries for the start's low 16 bits.)"""
    rng = np.random.default_rng(stop)
    P, F, n_rt = 5, 6, 65_600
    fmz = rng.uniform(200, 1700, (P, F))
    none = np.zeros(0)
    spectra = [(0, min(c, 65_535), none, none) for c in range(n_rt)]
    for c in range(65_490, 65_536):
        mz = np.sort(np.concatenate([rng.choice(fmz.reshape(-1), 20), rng.uniform(200, 1700, 30)]))
        spectra.append((1, c, mz, rng.lognormal(6, 1, len(mz))))
    run = run_of(spectra, 1)
    run["spectrum_rt"] = np.concatenate([np.arange(n_rt), np.arange(65_490, 65_536)]).astype(np.float32)
    la = library_of(405.0, np.full(P, float(start)), fmz, rng.uniform(0.1, 1.0, (P, F)))
    c = candidates_at(np.arange(P), np.full(P, start), np.full(P, stop))
    assert_scored_and_quantified(run, la, c, f"{start}-{stop}")


def empty_library(n, frags_of_first):
    """n precursors without fragments, but for the first."""
    la = library_of(405.0, [100.0], np.linspace(200, 1700, frags_of_first)[None], np.ones((1, frags_of_first)))
    for k in list(la):
        if k.startswith("precursor"):
            la[k] = np.arange(n, dtype=np.uint64) if k == "precursor_idx" else np.repeat(la[k], n)
    la["flat_frag_start_idx"] = np.where(np.arange(n) == 0, 0, frags_of_first).astype(np.uint64)
    la["flat_frag_stop_idx"] = np.full(n, frags_of_first, np.uint64)
    return la


def small_workload():
    cfg, lib, run = synth.make_workload("tiny", "numpy")
    return cfg, DIAData.from_arrays(*(run[k] for k in RUN_KEYS), run["cycle"]), synth.library_arrays(lib)


@pytest.mark.parametrize("into", [False, True])
def test_failed_search_leaves_nothing_behind(into):
    """A search whose workspace does not fit the device (320 GB of fragment weights) fails
    after it has queued work on its candidate buffers, here behind other work of its stream.
    Buffers that are freed with the failure have been waited for; those that stay serve the
    next search."""
    import torch

    cfg, dia, la = small_workload()
    big = SpecLibFlat.from_arrays(**empty_library(200_000, 400_000))
    lib = SpecLibFlat.from_arrays(**la)
    params = params_from(dict(cfg.params_dict(), top_k_fragments=10**6))
    stream = torch.cuda.Stream()
    sel = PeakGroupSelection(params, verbose=False, stream=stream.cuda_stream)
    want = sel.search(dia, lib).to_arrays()
    cand = sel.new_candidates()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(10**9)  # about half a second
    with pytest.raises(MemoryError):
        sel.search_into(dia, big, cand) if into else sel.search(dia, big)
    if into:
        assert cand.size() == 0
    assert stream.query()
    sel.search_into(dia, lib, cand)
    n = len(want[0])
    out = {c: np.zeros(n, w.dtype) for c, w in zip(COLS, want)}
    assert cand.copy_out(out) == n
    for c, w in zip(COLS, want):
        assert np.array_equal(out[c].view(np.uint8), w.view(np.uint8)), c


def test_candidate_buffers_that_cannot_grow():
    """Candidate buffers that would have to grow past the device's memory (214 GB) are gone
    with the failure, and come back with the next search."""
    cfg, dia, la = small_workload()
    lib = SpecLibFlat.from_arrays(**la)
    sel = PeakGroupSelection(params_from(cfg.params_dict()), verbose=False)
    want = sel.search(dia, lib).to_arrays()
    n = len(want[0])
    out = {c: np.zeros(n, w.dtype) for c, w in zip(COLS, want)}
    cand = sel.new_candidates()
    sel.search_into(dia, lib, cand)
    none = np.zeros(0)
    run = run_of([(0, c, none, none) for c in range(65_000)] + [(1, 5, [500.0], [1.0])], 1)
    long_run = DIAData.from_arrays(*(run[k] for k in RUN_KEYS), run["cycle"])
    big = SpecLibFlat.from_arrays(**empty_library(300_000, 2))
    many = PeakGroupSelection(params_from(dict(cfg.params_dict(), candidate_count=20_000,
                                               rt_tolerance=65_000.0)), verbose=False)
    with pytest.raises(MemoryError):
        many.search_into(long_run, big, cand)
    assert cand.size() == 0
    sel.search_into(dia, lib, cand)
    assert cand.copy_out(out) == n
    for c, w in zip(COLS, want):
        assert np.array_equal(out[c].view(np.uint8), w.view(np.uint8)), c


def test_replayed_graph_belongs_to_its_run():
    """Runs of equal shape and different cycle time, each in the place of the one before (its
    memory is freed first): a captured search of one is not replayed for the next."""
    cfg, lib, run = synth.make_workload("tiny_uneven", "numpy")
    la = synth.library_arrays(lib)
    slib = SpecLibFlat.from_arrays(**la)
    params = params_from(cfg.params_dict())
    sel = PeakGroupSelection(params, verbose=False, use_graph=True)
    cand = sel.new_candidates()
    for cycle_time in (1.0, 0.5, 2.0, 0.25):
        r = dict(run, spectrum_rt=(run["spectrum_rt"] * np.float32(cycle_time)).astype(np.float32))
        dia = DIAData.from_arrays(*(r[k] for k in RUN_KEYS), r["cycle"])
        want = PeakGroupSelection(params, verbose=False).search(dia, slib).to_arrays()
        for again in range(2):  # captured, replayed
            sel.search_into(dia, slib, cand)
            n = len(want[0])
            assert cand.size() == n, cycle_time
            out = {c: np.zeros(n, w.dtype) for c, w in zip(COLS, want)}
            cand.copy_out(out)
            for c, w in zip(COLS, want):
                assert np.array_equal(out[c].view(np.uint8), w.view(np.uint8)), (cycle_time, again, c)
        del dia


@pytest.mark.parametrize("span", [11, 400])
def test_fragments_without_an_mz(span):
    """NaN fragment m/z in scoring and quantification (in blocks, and the per-candidate
    kernels of whole-run ranges): last in m/z order, ties in library order, as in the search
    and the oracle."""
    rng = np.random.default_rng(span)
    P, F, n_cyc = 9, 7, 400
    fmz = rng.uniform(200, 1700, (P, F))
    none = np.zeros(0)
    spectra = []
    for c in range(n_cyc):
        mz = np.sort(np.concatenate([rng.choice(fmz.reshape(-1), 30), rng.uniform(200, 1700, 20)]))
        spectra += [(0, c, none, none), (1, c, mz, rng.lognormal(6, 1, len(mz)))]
    run = run_of(spectra, 1)
    for p in range(P):  # none to all of a precursor's fragments
        fmz[p, rng.permutation(F)[:p % 8]] = np.nan
    la = library_of(405.0, np.full(P, 200.0), fmz, rng.uniform(0.1, 1.0, (P, F)))
    la["fragment_position"] = rng.integers(0, 200, P * F).astype(np.uint8)
    start = rng.integers(0, n_cyc - span + 1, P)
    assert_scored_and_quantified(run, la, candidates_at(np.arange(P), start, start + span), f"span {span}")


@pytest.mark.parametrize("what", ["score", "search"])
def test_threads_with_different_plans(what):
    """Threads whose calls of the same kernels take different amounts of shared memory (a
    thread's candidates have 3 cycles or 60, its RT windows 80 or 1200): every call
    succeeds, with its own thread's result."""
    import threading

    cfg = synth.get_config("tiny_uneven", n_cycles=1200, n_precursors=60, rt_half_window=(40.0, 40.0),
                           frag_min=20, frag_max=24)
    lib = synth.make_library(cfg, "numpy")
    run = synth.make_run(cfg, lib, "numpy")
    la = synth.library_arrays(lib)
    dia = DIAData.from_arrays(*(run[k] for k in RUN_KEYS), run["cycle"])
    slib = SpecLibFlat.from_arrays(**la)
    scoring = PeakGroupScoring(ScoringParameters(), verbose=False)

    def call_of(i):
        if what == "search":
            sel = PeakGroupSelection(params_from(dict(cfg.params_dict(), rt_tolerance=(40.0, 900.0)[i % 2])),
                                     verbose=False)
            return lambda: sel.search(dia, slib).to_arrays()
        span = (3, 60)[i % 2]
        c = candidates_at(la["precursor_idx"][:2], [100 * i, 50 + 100 * i], [100 * i + span, 50 + 100 * i + span])
        cc = CandidateCollection.from_arrays(*(c[k] for k in COLS))
        return lambda: list(scoring.score(dia, slib, cc).to_dict_arrays().values())

    calls = [call_of(i) for i in range(8)]
    want = [f() for f in calls]
    faults = []

    def work(i):
        try:
            for _ in range(1000):
                got = calls[i]()
            for a, b in zip(got, want[i]):
                assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
        except Exception as e:  # noqa: BLE001 (told by the main thread)
            faults.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not faults, faults


def test_scoring_in_parts():
    """More candidates than one pair of launches takes (730,000 here): every copy of a
    candidate has the oracle's features, in its own row, also where the work order mixes
    precursors of few and many fragments; and the device holds little besides the results
    (all candidates' vectors at once would be 2.9 GB)."""
    import torch

    cfg, lib, run = synth.make_workload("tiny_uneven", "numpy")
    la = quant_library(synth.library_arrays(lib), seed=4)
    dia, slib, od, ol = build(run, la)
    rng = np.random.default_rng(4)
    m, n = 500, 4_000_000
    start = rng.integers(0, cfg.n_cycles - 11, m)
    few = candidates_at(la["precursor_idx"][rng.integers(0, cfg.n_precursors, m)], start, start + 11)
    ref = oracle.score(od, ol, few, log_mode=oracle.LOG_RN)
    at = rng.integers(0, m, n)
    cc = CandidateCollection.from_arrays(*(few[k][at] for k in COLS))
    free = torch.cuda.mem_get_info()[0]
    feats = PeakGroupScoring(ScoringParameters(), verbose=False).score(dia, slib, cc)
    assert free - torch.cuda.mem_get_info()[0] < n * (41 * 4 + 17) + 1.75 * 2**30
    assert_features_equal(feats.to_dict_arrays(), {k: v[at] for k, v in ref.items()}, exact=True, where="in parts")


def assert_entries_in_order(dia, spectra, n_windows, where):
    """Entries by (bin, cycle), ties in visit order."""
    grid = mz_grid()
    for w in range(1, n_windows + 1):
        rows = [s for s in spectra if s[0] == w]
        mz = np.concatenate([s[2] for s in rows]).astype(np.float32)
        cyc = np.concatenate([np.full(len(s[2]), s[1]) for s in rows])
        inten = np.concatenate([s[3] for s in rows]).astype(np.float32)
        bins = closest_bins(grid, mz)
        order = np.lexsort((np.arange(len(mz)), cyc, bins))
        got = dia.observation(w)
        starts = np.concatenate([[0], np.cumsum(np.bincount(bins, minlength=len(grid)))])
        assert np.array_equal(got["slice_starts"], starts.astype(np.uint32)), (where, w)
        assert np.array_equal(got["cycle_indices"], cyc[order].astype(np.uint16)), (where, w)
        assert np.array_equal(got["intensities"].view(np.uint32), inten[order].view(np.uint32)), (where, w)


@pytest.mark.parametrize("peaks", [2047, 2048, 2049, 4096, 10_001])
def test_build_of_long_spectra(peaks):
    """Spectra around the multiples of the 2048 peaks that a warp takes."""
    rng = np.random.default_rng(peaks)
    none = np.zeros(0)
    spectra = []
    for c in range(7):
        spectra.append((0, c, none, none))
        for w in (1, 2):
            n = peaks + (w - 1) * int(rng.integers(0, 3000))
            spectra.append((w, c, rng.uniform(150, 2000, n), rng.lognormal(5, 2, n)))
    run = run_of(spectra, 2)
    dia = DIAData.from_arrays(*(run[k] for k in RUN_KEYS), run["cycle"])
    assert_entries_in_order(dia, spectra, 2, peaks)


def device_run(cycles, windows, peaks, mz):
    """A run of device arrays: `mz(n)` gives the peaks' m/z."""
    import torch

    dsi = torch.arange(windows + 1, device="cuda").repeat(cycles)
    cyc = torch.arange(cycles, device="cuda").repeat_interleave(windows + 1)
    stop = torch.cumsum(torch.where(dsi == 0, 0, peaks), 0)
    lo = torch.where(dsi == 0, -1.0, 390.0 + 10.0 * dsi).float()
    n = cycles * windows * peaks
    return dict(spectrum_delta_scan_idx=dsi, isolation_lower_mz=lo, isolation_upper_mz=(lo + 10.0).float(),
                spectrum_peak_start_idx=stop - torch.where(dsi == 0, 0, peaks), spectrum_peak_stop_idx=stop,
                spectrum_cycle_idx=cyc, spectrum_rt=cyc.float(), peak_mz=mz(n).float(),
                peak_intensity=torch.rand(n, device="cuda") + 1.0,
                cycle=np.zeros((windows + 1, 1, 1, 1), np.float32))


def build_ms(run):
    import time

    import torch

    best = 1e9
    for _ in range(6):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        dia = DIAData.from_arrays(**run)
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t0)
        del dia
    return best * 1e3


def test_build_time_of_long_spectra():
    """24 M peaks in 160 spectra take no more than 4 times as long as in 24,000 (a warp for
    each of the 160: 20 times)."""
    import torch

    mz = lambda n: torch.rand(n, device="cuda") * 1650 + 150
    few, many = build_ms(device_run(20, 8, 150_000, mz)), build_ms(device_run(3000, 8, 1000, mz))
    assert few < 4 * many, (few, many)


@pytest.mark.parametrize("in_cycle_order", [True, False])
@pytest.mark.parametrize("widths,background", [
    ((25, 26, 64, 500), 9000),   # up to an eighth of the peaks in bins of more than 24: counted
    ((1023, 1024), 16_500),      # ... in the widest bins that a block sorts
    ((1025,), 16_500),           # wider, or more of them: sorted whole
    ((40,) * 60, 3000),
    ((3000, 7), 100),
    ((30_000, 1), 2000),
])
def test_build_of_crowded_bins(widths, background, in_cycle_order):
    """Bins of many peaks, with peaks outside the grid at both ends, three windows to a group:
    the order is the same whichever way a group is put in order."""
    rng = np.random.default_rng(len(widths) + background)
    grid = mz_grid()
    centres = grid[rng.choice(len(grid) - 2, len(widths), replace=False) + 1]
    cycles = np.arange(40) if in_cycle_order else rng.permutation(40)
    none = np.zeros(0)
    spectra = []
    for c in cycles:
        spectra.append((0, c, none, none))
        for w in (1, 2, 3):
            k = [v // 40 + (1 if c < v % 40 else 0) for v in widths]
            mz = np.concatenate([np.repeat(centres, k), rng.uniform(150, 2000, background // 40),
                                 [90.0, 149.99, 2000.5][:int(rng.integers(0, 3))]])
            mz = mz[rng.permutation(len(mz))]
            spectra.append((w, c, mz, rng.lognormal(5, 2, len(mz))))
    run = run_of(spectra, 3)
    dia = DIAData.from_arrays(*(run[k] for k in RUN_KEYS), run["cycle"])
    assert_entries_in_order(dia, spectra, 3, widths)


@pytest.mark.parametrize("share", [0.01, 0.3])
def test_build_time_of_peaks_outside_the_grid(share):
    """A run with peaks below m/z 150, which all share a bin, is loaded in no more than 5
    times the time of one without (a block to the bin: 18 times at 1 %)."""
    import torch

    def mz(n):
        inside = torch.rand(n, device="cuda") * 1650 + 150
        return torch.where(torch.rand(n, device="cuda") < share, inside * 0.05 + 50, inside)
    some = build_ms(device_run(3000, 8, 1000, mz))
    none = build_ms(device_run(3000, 8, 1000, lambda n: torch.rand(n, device="cuda") * 1650 + 150))
    assert some < 5 * none, (some, none)


@pytest.mark.parametrize("kernel_size,half", [(14, 7), (20, 10), (21, 11), (31, 16), (40, 20)])
def test_search_shortest_windows(kernel_size, half):
    """RT windows that the run's ends cut to so many cycles: from the longest that hold no
    candidate (the kernel's length) over the shortest that may hold one to 4 half widths and
    more, at both ends."""
    rng = np.random.default_rng(kernel_size)
    n_cyc, F = 300, 5
    lengths = np.arange(2 * half - 1, 4 * half + 6)
    pad = 10.0 + kernel_size  # the least tolerance, at a cycle a second
    prt = np.concatenate([lengths - 0.5 - pad, n_cyc - lengths - 0.5 + pad])
    spans = [oracle.rt_limits(np.arange(n_cyc, dtype=np.float32), 1.0, t, 1.0, kernel_size)
             for t in prt.astype(np.float32)]
    assert [b - a for a, b in spans] == [*lengths, *lengths]
    P = len(prt)
    fmz = rng.uniform(200, 1700, (P, F))
    mz = [[] for _ in range(n_cyc)]
    for (a, b), row in zip(spans, fmz):
        for f in row:
            for c in rng.integers(a, b, 12):
                mz[c].append(f * (1 + rng.uniform(-9e-6, 9e-6)))
    none = np.zeros(0)
    spectra = []
    for c in range(n_cyc):
        spectra += [(0, c, none, none), (1, c, np.sort(mz[c]), rng.lognormal(6, 2, len(mz[c])))]
    run = run_of(spectra, 1)
    la = library_of(405.0, prt, fmz, rng.uniform(0.1, 1.0, (P, F)))
    params = dict(PARAMS, kernel_size=kernel_size, rt_tolerance=1.0, fwhm_rt=1.5 if half == 7 else 3.0)
    for mode in (1, 2):
        got, ref = search_both(run, la, params, gather_mode=mode)
        assert len(set(ref["precursor_idx"])) > P // 3
        assert_candidates_equal(got, ref, exact_scores=True, where=f"kernel {kernel_size} mode {mode}")


def test_device_bytes_count_the_window_index():
    """Windows all over one another have a longer index than windows side by side."""
    none = np.zeros(0)
    spectra = [(0, 0, none, none)] + [(w, 0, [300.0 + w], [1.0]) for w in range(1, 101)]
    run = run_of(spectra, 100)
    nested = dict(run)
    w = run["spectrum_delta_scan_idx"]
    nested["isolation_lower_mz"] = np.where(w == 0, -1, 600 - w).astype(np.float32)
    nested["isolation_upper_mz"] = np.where(w == 0, -1, 600 + w).astype(np.float32)
    held = [DIAData.from_arrays(*(r[k] for k in RUN_KEYS), r["cycle"]).device_bytes() for r in (run, nested)]
    assert held[1] - held[0] > 4 * 90 * 100


def test_page_locked_tables_are_counted_while_any_view_lives():
    import gc

    from alphadia_search_rs_b200 import api

    blocks = api._HostBlocks()
    a = blocks.empty(10**6, np.float32)
    assert blocks.locked == 1 << 22
    part = a[7:9].view(np.uint8)
    del a
    gc.collect()
    b = blocks.empty(10**6, np.uint8)  # counts those that are gone: none
    assert blocks.locked == (1 << 22) + (1 << 20)
    del part, b
    gc.collect()
    blocks.empty(70_000, np.uint8)
    assert blocks.locked == 1 << 17
