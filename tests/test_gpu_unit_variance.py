"""Brute fold of series with unit variances (E alone, two segments a lane):
all ones, ones but for one sample of one group, zero variances at the end, and
batches whose lengths leave part of a group out, against the oracle bit for bit;
the executor's own count of the groups shows which way they were folded."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import series
from oracle import lko

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbins", [50, 64, 128])
@pytest.mark.parametrize("kind", ["ones", "one_other", "zero_end"])
def test_unit_variances(cuda, nbins, kind):
    from loki_b200.configs import PulsarSearchConfig
    from loki_b200.ffa import FFACUDA

    n, tsamp, lims = 1 << 19, 64e-6, [[20.0, 60.0]]
    e, _ = series(n, 17)
    v = np.ones(n, np.float32)
    if kind == "one_other":
        v[n // 2 + 12345] = 2.0
    elif kind == "zero_end":
        v[-1000:] = 0.0
    cfg = PulsarSearchConfig(n, tsamp, nbins, 1.0, np.array(lims), use_fourier=False, bseg_ffa=n // 16)
    op = lko.plan_create(lko.make_cfg(n, tsamp, nbins, 1.0, lims, bseg_ffa=n // 16))
    ffa = FFACUDA(cfg)
    got = ffa.execute(e, v)
    np.testing.assert_array_equal(got.view(np.uint32), lko.ffa(op, e, v).view(np.uint32))
    # 256 segments: four groups checked, one of them with another variance
    assert int(op.nsegments[0]) == 256
    assert ffa.unit_groups() == (4, 0 if kind == "ones" else 1)


def test_one_wave_folds_both_rows(cuda):
    """A fold whose blocks all run at once is not checked."""
    from loki_b200.configs import PulsarSearchConfig
    from loki_b200.ffa import FFACUDA

    n, lims = 1 << 16, [[20.0, 22.0]]
    cfg = PulsarSearchConfig(n, 64e-6, 32, 1.0, np.array(lims), use_fourier=False, score_widths=[1, 2])
    op = lko.plan_create(lko.make_cfg(n, 64e-6, 32, 1.0, lims))
    e, _ = series(n, 18)
    v = np.ones(n, np.float32)
    ffa = FFACUDA(cfg)
    got = ffa.execute(e, v)
    np.testing.assert_array_equal(got.view(np.uint32), lko.ffa(op, e, v).view(np.uint32))
    assert ffa.unit_groups() == (0, 0)


def test_batch_lengths(cuda):
    from loki_b200.configs import PulsarSearchConfig
    from loki_b200.ffa import FFACUDA

    t = cuda
    n, lims = 1 << 18, [[20.0, 60.0]]
    lengths = [n, int(0.7 * n) + 11, 5000]
    cfg = PulsarSearchConfig(n, 64e-6, 64, 1.0, np.array(lims), use_fourier=False, bseg_ffa=n // 8)
    op = lko.plan_create(lko.make_cfg(n, 64e-6, 64, 1.0, lims, bseg_ffa=n // 8))
    es, vs = np.zeros((3, n), np.float32), np.zeros((3, n), np.float32)
    for k, m in enumerate(lengths):
        es[k, :m] = series(n, 40 + k)[0][:m]
        vs[k, :m] = 1.0
    ffa = FFACUDA(cfg, max_batch=3)
    ffa.set_batch_lengths(t.tensor(lengths, dtype=t.int64, device="cuda"))
    got = ffa.execute_batch(t.from_numpy(es).cuda(), t.from_numpy(vs).cuda()).cpu().numpy()
    # 128 segments a series: the fourth group holds the ends of the shorter two
    assert int(op.nsegments[0]) == 128 and ffa.unit_groups() == (6, 1)
    for k in range(3):
        np.testing.assert_array_equal(got[k].view(np.uint32), lko.ffa(op, es[k], vs[k]).view(np.uint32))
