"""Real transforms of fold rows (Fourier-domain FFA above nbins_min_lossy_bf and
back to time) at every size of the two-step kernels and at others, against
numpy in 64 bits. Bound: a value is a sum of at most 2 log2(n) rounded adds of
terms no larger than the row's largest coefficient, 8 eps log2(n) of the row's
2-norm for the two-step transforms, n eps for the direct sums."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import series
from oracle import lko

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbins", [66, 100, 128, 129, 256, 512, 1024])
def test_fold_and_back(cuda, nbins):
    from loki_b200.configs import PulsarSearchConfig
    from loki_b200.ffa import FFACOMPLEXCUDA, FFACUDA

    n, tsamp = 1 << 15, 64e-6
    lims = [[5.0, 7.0]] if nbins > 256 else [[20.0, 21.0]]
    # two levels: one merge after the transform of the level-0 fold
    cfg = PulsarSearchConfig(n, tsamp, nbins, 4.0, np.array(lims), use_fourier=True, bseg_brute=n // 2)
    e, v = series(n, nbins)
    ffa = FFACOMPLEXCUDA(cfg)
    assert ffa.lossy
    spec = ffa.execute(e, v).reshape(-1, nbins // 2 + 1).astype(np.complex128)
    back = ffa.execute_time(e, v).reshape(-1, nbins)
    eps = 2.0**-24
    tol = 8 * np.log2(nbins) * eps if nbins in (128, 256, 512, 1024) else nbins * eps
    want = np.fft.irfft(spec, n=nbins, axis=1)
    err = np.abs(back - want).max(axis=1)
    assert np.all(err <= tol * np.linalg.norm(want, axis=1))
    # forward: the final spectrum against the 64-bit merge of the level-0 folds' transforms
    op = lko.plan_create(lko.make_cfg(n, tsamp, nbins, 4.0, lims, bseg_brute=n // 2))
    fold0 = np.fft.rfft(lko.ffa(op, e, v, level=0).reshape(2, -1, 2, nbins).astype(np.float64), axis=-1)
    c = FFACUDA(cfg).plan.resolve_coordinates_freq()[1]
    ph = np.exp(-2j * np.pi * np.arange(nbins // 2 + 1)[None, :] * c["shift"].astype(np.float64)[:, None] / nbins)
    exact = fold0[0][c["idx"]] + fold0[1][c["idx"]] * ph[:, None, :]
    got = spec.reshape(exact.shape)
    scale = np.linalg.norm(exact, axis=-1, keepdims=True)
    assert np.all(np.abs(got - exact) <= (2 * tol + 16 * eps) * scale)
