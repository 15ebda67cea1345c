"""Fused final level (merge + boxcar S/N) at the edges of its kernels: bins up to
128 that are no power of two (masked widths), above 128 (a block of warps per
few cells), width lists only the generic kernel takes, odd numbers of bins,
cells that are no multiple of a block, and series whose maxima are zeros."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import series
from oracle import lko

pytestmark = pytest.mark.gpu

# nbins -> widths
CASES = {
    "nb6": (6, [1, 2, 5]),
    "nb17": (17, [1, 2, 3, 4, 6, 8]),
    "nb31_wide": (31, [1, 2, 3, 5, 9, 13, 19, 30]),
    "nb33": (33, [1, 2, 3, 4, 6, 8, 12, 16]),
    "nb50_unordered": (50, [4, 1, 16, 2]),
    "nb96_w40": (96, [1, 2, 4, 8, 16, 40]),
    "nb127_w32": (127, [1, 3, 9, 17, 32]),
    "nb129": (129, [1, 2, 3, 4, 6, 8, 12, 16]),
    "nb250_17_widths": (250, [1, 2, 3, 4, 5, 6, 8, 10, 12, 14, 17, 20, 25, 30, 36, 43, 50]),
    "nb512_unordered": (512, [64, 1, 7, 100]),
    "nb1000": (1000, [1, 2, 4, 8, 16, 32, 64, 128, 200]),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("kind", ["noise", "zeros", "freq"])
def test_scores_bit_exact(cuda, name, kind):
    from loki_b200.configs import PulsarSearchConfig
    from loki_b200.ffa import FFACUDA

    nbins, widths = CASES[name]
    nsamps, tsamp = 1 << 15, 64e-6
    lims = [[20.0, 30.0]] if kind == "freq" else [[-3000.0, 3000.0], [20.0, 30.0]]
    if nbins > 256:
        lims[-1] = [5.0, 7.0] if kind == "freq" else [10.0, 11.0]
    cfg = PulsarSearchConfig(nsamps, tsamp, nbins, 4.0, np.array(lims), use_fourier=False, score_widths=widths)
    op = lko.plan_create(lko.make_cfg(nsamps, tsamp, nbins, 4.0, lims))
    e, v = series(nsamps, 31)
    if kind == "zeros":
        e = np.where(np.arange(nsamps) % 2 == 0, np.float32(0.0), np.float32(-0.0))
    got = FFACUDA(cfg).scores(e, v)
    want = lko.snr_boxcar_3d(lko.ffa(op, e, v), np.array(widths, np.uint64), nbins).ravel()
    nan = np.isnan(want)  # bins without samples: 0 / 0 on both sides
    np.testing.assert_array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got[~nan].view(np.uint32), want[~nan].view(np.uint32))
