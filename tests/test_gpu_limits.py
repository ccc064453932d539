"""GPU parity where a call meets a limit of its kernels or of the device: ranges past the
last cycle index, work done in parts, calls that fail half way, buffers and handles that
take one another's place."""
import numpy as np
import pytest

import oracle
from alphadia_search_rs_b200 import (CandidateCollection, PeakGroupQuantification, PeakGroupScoring,
                                     QuantificationParameters, ScoringParameters)

from _util import COLS
from test_gpu_quant import assert_quant_equal
from test_gpu_scoring import assert_features_equal, build
from test_gpu_sizes import library_of, run_of

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
