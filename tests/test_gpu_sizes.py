"""GPU parity at the sizes where a kernel changes its path: entries per m/z bin in the
run's build, entries per fragment range and cycles per RT window in the search, candidates,
fragments and cycles per block in scoring and quantification.  Everything against the
oracle (or a numpy restatement of the builder's order), bit for bit."""
import numpy as np
import pytest

import oracle
from alphadia_search_rs_b200 import (CandidateCollection, DIAData, PeakGroupQuantification,
                                     PeakGroupScoring, QuantificationParameters, ScoringParameters,
                                     SelectionParameters, mz_grid, synth)

from _util import COLS, RUN_KEYS, assert_candidates_equal, oracle_inputs, oracle_search, product_search
from test_gpu_quant import assert_quant_equal, quant_library
from test_gpu_scoring import assert_features_equal, build

pytestmark = pytest.mark.gpu


def run_of(spectra, n_windows):
    """A run from (window, cycle, m/z array, intensity array) spectra; windows are 10 Th wide
    from 400 m/z, window 0 is MS1."""
    lo = np.array([-1.0 if w == 0 else 400.0 + 10.0 * (w - 1) for w, *_ in spectra], np.float32)
    n = np.array([len(s[2]) for s in spectra], np.int64)
    stop = np.cumsum(n)
    f32 = lambda k: np.concatenate([s[k] for s in spectra]).astype(np.float32)
    return dict(spectrum_delta_scan_idx=np.array([s[0] for s in spectra], np.int64),
                isolation_lower_mz=lo, isolation_upper_mz=np.where(lo < 0, lo, lo + 10.0).astype(np.float32),
                spectrum_peak_start_idx=stop - n, spectrum_peak_stop_idx=stop,
                spectrum_cycle_idx=np.array([s[1] for s in spectra], np.int64),
                spectrum_rt=np.array([s[1] for s in spectra], np.float32),
                peak_mz=f32(2), peak_intensity=f32(3),
                cycle=np.zeros((n_windows + 1, 1, 1, 1), np.float32))


def closest_bins(grid, mz):
    left = np.searchsorted(grid, mz)
    a, b = grid[np.minimum(left, len(grid) - 1)], grid[np.maximum(left - 1, 0)]
    near = np.where(np.abs(a - mz) < np.abs(b - mz), left, left - 1)
    near = np.where((left < len(grid)) & (a == mz), left, near)
    return np.where(left == 0, 0, np.where(left == len(grid), left - 1, near))


@pytest.mark.parametrize("in_cycle_order", [True, False])
@pytest.mark.parametrize("per_bin", [1, 2, 3, 4, 5, 8, 24, 25, 26, 1023, 1024, 1025, 2500])
def test_build_orders_bins_of_every_size(per_bin, in_cycle_order):
    """Entries by (bin, cycle), ties in visit order, whatever a bin holds; windows without
    peaks in between; m/z at and past both ends of the grid."""
    rng = np.random.default_rng(per_bin)
    grid = mz_grid()
    centres = grid[rng.integers(0, len(grid), 5)]
    cycles = np.arange(50) if in_cycle_order else rng.permutation(50)
    spectra = []
    for c in cycles:
        spectra.append((0, c, np.zeros(0), np.zeros(0)))
        for w in (1, 3, 4):  # window 2 holds nothing
            k = per_bin // 50 + (1 if c < per_bin % 50 else 0)  # per bin over the cycles
            mz = np.concatenate([np.repeat(centres, k), [149.0, 150.0, 2000.0, 2500.0],
                                 rng.uniform(150, 2000, 3)])
            order = rng.permutation(len(mz))
            spectra.append((w, c, mz[order], rng.lognormal(5, 2, len(mz))))
    run = run_of(spectra, 4)
    dia = DIAData.from_arrays(*(run[k] for k in RUN_KEYS), run["cycle"])
    for w in range(5):
        rows = [s for s in spectra if s[0] == w]
        mz = np.concatenate([s[2] for s in rows] or [np.zeros(0)]).astype(np.float32)
        cyc = np.concatenate([np.full(len(s[2]), s[1]) for s in rows] or [np.zeros(0)])
        inten = np.concatenate([s[3] for s in rows] or [np.zeros(0)]).astype(np.float32)
        bins = closest_bins(grid, mz) if len(mz) else np.zeros(0, np.int64)
        order = np.lexsort((np.arange(len(mz)), cyc, bins))
        got = dia.observation(w)
        starts = np.concatenate([[0], np.cumsum(np.bincount(bins, minlength=len(grid)))])
        assert np.array_equal(got["slice_starts"], starts.astype(np.uint32)), w
        assert np.array_equal(got["cycle_indices"], cyc[order].astype(np.uint16)), w
        assert np.array_equal(got["intensities"].view(np.uint32), inten[order].view(np.uint32)), w


def library_of(pmz, prt, fmz, fint, tol=None):
    """One precursor per row of fmz."""
    P, F = fmz.shape
    n = P * F
    la = dict(precursor_idx=np.arange(P, dtype=np.uint64), precursor_mz_library=np.full(P, pmz, np.float32),
              precursor_mz=np.full(P, pmz, np.float32), precursor_rt_library=np.asarray(prt, np.float32),
              precursor_rt=np.asarray(prt, np.float32), precursor_naa=np.full(P, 9, np.uint8),
              flat_frag_start_idx=np.arange(0, n, F, dtype=np.uint64),
              flat_frag_stop_idx=np.arange(F, n + 1, F, dtype=np.uint64),
              fragment_mz_library=fmz.reshape(-1).astype(np.float32),
              fragment_mz=fmz.reshape(-1).astype(np.float32),
              fragment_intensity=fint.reshape(-1).astype(np.float32))
    for k, v in dict(cardinality=1, charge=1, loss_type=0, number=3, position=1, type=98).items():
        la["fragment_" + k] = np.full(n, v, np.uint8)
    if tol is not None:
        la["precursor_rt_tolerance"] = np.asarray(tol, np.float32)
    return la


def search_both(run, la, params, **more):
    od, ol, tol = oracle_inputs(run, la)
    got, *_ = product_search(run, la, params, **more)
    return got, oracle_search(run, la, params, oracle.LOG_RN, od, ol, tol)


PARAMS = dict(fwhm_rt=4.7096, kernel_size=21, peak_length=5, mass_tolerance=15.0, rt_tolerance=250.0,
              candidate_count=3, top_k_fragments=12)


@pytest.mark.parametrize("gather_mode", [0, 1, 2])
@pytest.mark.parametrize("entries", [1, 2, 31, 33, 63, 64, 65, 95, 127, 128, 129, 191, 255, 256, 257,
                                     383, 385, 700])
def test_search_ranges_of_every_length(entries, gather_mode):
    """A fragment range of so many entries: steps of 64, staging areas of 128, the ranges
    that are searched per bin, rows that accept more cells than are recorded for clearing,
    repeated cells, and BF16 storage the same in every gather mode."""
    rng = np.random.default_rng(entries)
    n_cyc, P, F = 520, 6, 4
    fmz = rng.uniform(200, 1700, (P, F))
    mz = [[] for _ in range(n_cyc)]
    for f in fmz.reshape(-1):
        for c in rng.integers(0, n_cyc, entries):
            mz[c].append(f * (1 + rng.uniform(-12e-6, 12e-6)))
    spectra = []
    for c in range(n_cyc):
        spectra.append((0, c, np.zeros(0), np.zeros(0)))
        spectra.append((1, c, np.sort(mz[c]), rng.lognormal(6, 2, len(mz[c]))))
    run = run_of(spectra, 1)
    la = library_of(405.0, rng.uniform(200, 320, P), fmz, rng.uniform(0.1, 1.0, (P, F)))
    got, ref = search_both(run, la, PARAMS, gather_mode=gather_mode)
    assert_candidates_equal(got, ref, exact_scores=True, where=f"{entries}/{gather_mode}")
    bf16, *_ = product_search(run, la, PARAMS, gather_mode=gather_mode, precision="bf16")
    scan, *_ = product_search(run, la, PARAMS, gather_mode=1, precision="bf16")
    assert_candidates_equal(bf16, scan, exact_scores=True, where=f"bf16 {entries}/{gather_mode}")


@pytest.mark.parametrize("kernel_size,candidate_count", [(20, 1), (21, 3), (31, 9), (14, 40)])
def test_search_window_lengths(kernel_size, candidate_count):
    """RT windows of 30 to 2060 cycles around the multiples of 4 and of 128, the length
    classes and the longest window in shared memory; up to 40 candidates a precursor."""
    rng = np.random.default_rng(kernel_size)
    n_cyc, F = 2300, 3
    lengths = [30, 31, 32, 33, 34, 127, 128, 129, 130, 255, 257, 301, 511, 512, 513, 514, 767, 768, 769,
               1023, 1024, 1025, 1407, 1408, 1409, 2047, 2048, 2049, 2060]
    P = len(lengths)
    fmz = rng.uniform(200, 1700, (P, F))
    mz = [[] for _ in range(n_cyc)]
    for f in fmz.reshape(-1):
        for c in rng.integers(0, n_cyc, 400):
            mz[c].append(f * (1 + rng.uniform(-3e-6, 3e-6)))
    spectra = []
    for c in range(n_cyc):
        spectra.append((0, c, np.zeros(0), np.zeros(0)))
        spectra.append((1, c, np.sort(mz[c]), rng.lognormal(6, 2, len(mz[c]))))
    run = run_of(spectra, 1)
    tol = np.array([(k - 1) / 2.0 + 0.25 for k in lengths])
    la = library_of(405.0, np.full(P, 1150.0), fmz, rng.uniform(0.1, 1.0, (P, F)), tol)
    params = dict(PARAMS, kernel_size=kernel_size, candidate_count=candidate_count,
                  fwhm_rt=1.0 if kernel_size == 14 else 4.7096)
    got, ref = search_both(run, la, params)
    assert len(ref["rank"]) >= P
    assert_candidates_equal(got, ref, exact_scores=True, where=f"kernel {kernel_size}")


@pytest.fixture(scope="module", params=[(1, 3), (4, 24), (30, 90)], ids=["few", "usual", "many"])
def candidates(request):
    lo, hi = request.param
    cfg = synth.get_config("tiny_uneven", frag_min=lo, frag_max=hi, n_precursors=80, n_cycles=300)
    lib = synth.make_library(cfg, "numpy")
    run = synth.make_run(cfg, lib, "numpy")
    la = quant_library(synth.library_arrays(lib), seed=5)
    dia, slib, od, ol = build(run, la)
    apex = np.clip(np.round(lib["apex"]).astype(np.int64), 0, 299)
    return la, apex, dia, slib, od, ol


@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 32, 33, 240])
@pytest.mark.parametrize("span", [1, 2, 3, 4, 11, 12, 31, 64, 129, 300])
def test_scoring_and_quantification_blocks(candidates, n, span):
    """Blocks of 4 candidates (score_block_kernel) and of 32 (feature_kernel) with remainders,
    cycle ranges from one cycle to the whole run, where the per-candidate kernels take over."""
    la, apex, dia, slib, od, ol = candidates
    rng = np.random.default_rng(100 * n + span)
    row = rng.integers(0, len(apex), n)
    start = np.clip(apex[row] - span // 2, 0, 300 - span)
    stop = np.minimum(start + rng.integers(max(1, span - 2), span + 1, n), 300)
    stop[0] = start[0] + span
    c = dict(precursor_idx=la["precursor_idx"][row], rank=np.arange(n, dtype=np.uint64),
             score=rng.random(n, dtype=np.float32), cycle_center=((start + stop - 1) // 2).astype(np.uint64),
             cycle_start=start.astype(np.uint64), cycle_stop=stop.astype(np.uint64))
    for k in ("scan_center", "scan_start", "scan_stop"):
        c[k] = np.zeros(n, np.uint64)
    cc = CandidateCollection.from_arrays(*(c[k] for k in COLS))
    got = PeakGroupScoring(ScoringParameters(), verbose=False).score(dia, slib, cc).to_dict_arrays()
    assert_features_equal(got, oracle.score(od, ol, c, log_mode=oracle.LOG_RN), exact=True, where=f"{n}x{span}")
    q = PeakGroupQuantification(QuantificationParameters(), verbose=False).quantify(dia, slib, cc)
    assert_quant_equal(q, oracle.quantify(od, ol, c, la), where=f"{n}x{span}")


@pytest.mark.parametrize("n", [1, 255, 256, 257, 1024, 4096, 4097, 5000, 65536, 65537, 70000])
def test_candidates_of_many_precursors_in_order(n):
    """Eleven precursors over and over: the candidates of each are the oracle's, in order,
    whichever way they are brought together (small blocks, one launch, three launches)."""
    rng = np.random.default_rng(5)
    n_cyc, P, F = 200, 11, 3
    fmz = rng.uniform(200, 1700, (P, F))
    spectra = []
    for c in range(n_cyc):
        mz = np.sort(rng.choice(fmz.reshape(-1), 4))
        spectra.append((0, c, np.zeros(0), np.zeros(0)))
        spectra.append((1, c, mz, rng.lognormal(6, 2, len(mz))))
    run = run_of(spectra, 1)
    prt, fint = rng.uniform(20, 180, P), rng.uniform(0.1, 1.0, (P, F))
    pmz = np.where(np.arange(P) % 4 == 3, 300.0, 405.0)  # every fourth in no window
    params = dict(PARAMS, rt_tolerance=60.0)
    la = library_of(405.0, prt, fmz, fint)
    la["precursor_mz"] = pmz.astype(np.float32)
    od, ol, tol = oracle_inputs(run, la)
    ref = oracle_search(run, la, params, oracle.LOG_RN, od, ol, tol)
    rows = [np.flatnonzero(ref["precursor_idx"] == k) for k in range(P)]
    assert len({len(r) for r in rows}) > 1 and max(len(r) for r in rows) == 3
    base = np.arange(n) % P
    la = library_of(405.0, prt[base], fmz[base], fint[base])
    la["precursor_mz"] = pmz[base].astype(np.float32)
    got, *_ = product_search(run, la, params)
    at = np.concatenate([rows[k] for k in base])
    want = {k: ref[k][at] for k in COLS}
    want["precursor_idx"] = np.repeat(np.arange(n), [len(rows[k]) for k in base]).astype(np.uint64)
    assert_candidates_equal(got, want, exact_scores=True, where=f"{n} precursors")


@pytest.mark.parametrize("n_windows", [179, 184])
def test_windows_all_over_one_another(n_windows):
    """Nested windows: as many as the window index lists, and a few more, where windows are
    scanned and the per-candidate kernels score."""
    rng = np.random.default_rng(n_windows)
    n_cyc, P, F = 60, 5, 3
    fmz = rng.uniform(200, 1700, (P, F))
    spectra, lo, hi = [], [], []
    for c in range(n_cyc):
        for w in range(n_windows + 1):
            mz = np.sort(rng.choice(fmz.reshape(-1), 2 if w else 0))
            spectra.append((w, c, mz, rng.lognormal(6, 1, len(mz))))
            lo.append(-1.0 if w == 0 else 500.0 - w)
            hi.append(-1.0 if w == 0 else 500.0 + w)
    run = run_of(spectra, n_windows)
    run["isolation_lower_mz"], run["isolation_upper_mz"] = np.float32(lo), np.float32(hi)
    la = library_of(500.0, np.full(P, 30.0), fmz, rng.uniform(0.1, 1.0, (P, F)))
    la["precursor_mz"] = np.array([500.0, 400.0, 500.0 - n_windows, 620.5, 321.0], np.float32)
    got, ref = search_both(run, la, dict(PARAMS, kernel_size=14, fwhm_rt=2.0, rt_tolerance=30.0))
    assert len(ref["rank"]) > 0
    assert_candidates_equal(got, ref, exact_scores=True, where=f"{n_windows} windows")
    dia, slib, od, ol = build(run, la)
    cc = CandidateCollection.from_arrays(*(ref[k] for k in COLS))
    feats = PeakGroupScoring(ScoringParameters(), verbose=False).score(dia, slib, cc).to_dict_arrays()
    assert_features_equal(feats, oracle.score(od, ol, ref, log_mode=oracle.LOG_RN), exact=True, where="nested")
    q = PeakGroupQuantification(QuantificationParameters(), verbose=False).quantify(dia, slib, cc)
    assert_quant_equal(q, oracle.quantify(od, ol, ref, la), where="nested")
