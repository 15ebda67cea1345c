"""Run tables of the brute fold's run form, replayed on the host with
every read checked against the padded segment, against the oracle's fold."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from oracle import lko

# (nbins, segment_len, tsamp, t_ref, frequencies): one range and several, bins
# not a multiple of 4, runs of 1 to hundreds of samples (compile-time lengths
# and longer ones), skipped bins, a run length at a whole number, segments
# shorter than a rotation, the start inside a run and on its edge
CASES = {
    "nb64_runs_5_to_49": (64, 4096, 64e-6, 0.131072, np.linspace(5.0, 50.0, 23)),
    "nb128_two_ranges": (128, 8192, 64e-6, 0.0, np.linspace(5.0, 50.0, 19)),
    "nb100_ranges_52_48": (100, 2048, 64e-6, 0.065536, np.linspace(8.0, 40.0, 17)),
    "nb50_invalid_bins": (50, 4096, 64e-6, 0.131072, np.linspace(3.0, 90.0, 31)),
    "nb33_one_bin_over": (33, 1024, 1e-3, 0.512, np.linspace(5.0, 20.0, 13)),
    "nb16_long_runs": (16, 8192, 64e-6, 0.0, np.linspace(2.0, 10.0, 9)),
    "nb8_longer_than_segment": (8, 512, 64e-6, 0.016384, np.array([0.5, 2.0, 10.0, 61.0])),
    "nb64_skipped_bins": (64, 1024, 1e-3, 0.512, np.linspace(20.0, 30.0, 11)),
    "nb256_skipped_bins": (256, 4096, 1e-3, 0.0, np.linspace(4.0, 6.0, 7)),
    "nb1024_sixteen_ranges": (1024, 4096, 64e-6, 0.0, np.linspace(5.0, 12.0, 7)),
    "whole_run_lengths": (32, 4096, 2.0**-12, 0.5, np.array([16.0, 32.0, 64.0, 25.6])),
    "ragged_segment": (48, 1236, 64e-6, 0.03, np.linspace(15.0, 70.0, 9)),
}


def _replay(freqs, seglen, nbins, tsamp, t_ref, ts):
    from loki_b200 import _capi as C

    f = np.ascontiguousarray(freqs, np.float64)
    ts = np.ascontiguousarray(ts, np.float32)
    out = np.full(f.size * nbins, np.nan, np.float32)
    applies = ctypes.c_int(-1)
    C.check(C.lib().lk_brute_fold_replay(f.ctypes.data, f.size, seglen, nbins, tsamp, t_ref, ts.ctypes.data,
                                         out.ctypes.data, ctypes.byref(applies)))
    return applies.value, out.reshape(f.size, nbins)


@pytest.mark.parametrize("name", sorted(CASES))
def test_replay_matches_oracle(name):
    nbins, seglen, tsamp, t_ref, freqs = CASES[name]
    ts = np.random.default_rng(len(name)).standard_normal(seglen).astype(np.float32)
    applies, got = _replay(freqs, seglen, nbins, tsamp, t_ref, ts)
    assert applies == 1
    want = lko.brute_fold(ts, ts, freqs, seglen, nbins, tsamp, t_ref).reshape(freqs.size, 2, nbins)[:, 0]
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))


def test_left_to_the_other_form():
    # a rotation per sample or two; too few bins for the run length
    for nbins, seglen, tsamp, f in ((64, 1024, 1e-3, 900.0), (2, 1 << 16, 64e-6, 0.9)):
        applies, _ = _replay(np.array([f]), seglen, nbins, tsamp, 0.0, np.ones(seglen, np.float32))
        assert applies == 0


# (segment_len, nsamps, samples per bin, nbins, batch, run form): segments with
# little padding, short ones padded to more than 1.5 times, long ones to more than
# twice; few segments below and above 1 GiB
FORMS = {
    "plan": (16384, 1 << 22, 9.0, 64, 1, True),
    "short_segments": (1024, 1 << 16, 6.0, 32, 1, True),
    "samples_256": (256, 1 << 20, 2.0, 64, 1, True),
    "samples_4": (4, 1 << 16, 0.8, 16, 1, False),
    "samples_64": (64, 1 << 20, 3.0, 64, 1, False),
    "samples_256_at_1.5": (256, 1 << 20, 9.0, 16, 1, True),
    "samples_256_padded": (256, 1 << 20, 20.0, 16, 1, False),
    "samples_1024_padded": (1024, 1 << 20, 60.0, 16, 1, False),
    "samples_4096": (4096, 1 << 20, 300.0, 4, 1, True),
    "samples_4096_padded": (4096, 1 << 20, 1500.0, 2, 1, False),
    "one_segment": (1 << 20, 1 << 20, 9.0, 64, 1, True),
    "one_long_segment": (1 << 23, 1 << 23, 9.0, 64, 1, False),
    "one_long_segment_of_32": (1 << 23, 1 << 23, 9.0, 64, 32, True),
}


@pytest.mark.parametrize("name", sorted(FORMS))
def test_form_and_its_memory(name):
    from loki_b200 import _capi as C

    seglen, nsamps, samples, nbins, batch, want = FORMS[name]
    f = np.array([1.0 / (samples * 64e-6 * nbins)])
    form, size = ctypes.c_int(-1), ctypes.c_uint64()
    C.check(C.lib().lk_brute_fold_form(f.ctypes.data, 1, seglen, nbins, nsamps, 64e-6, 0.0, batch,
                                       ctypes.byref(form), ctypes.byref(size)))
    assert form.value == (1 if want else 0)
    if want:  # at most twice the series' pairs, or 1 GiB
        assert 0 < size.value <= max(2 * 8 * nsamps * batch, 1 << 30)
