"""Merge levels two in a launch (the level between is formed in registers): even
and odd numbers of levels, bins with a kernel of their own and others, BF16
storage (the level between rounded as if it were stored) and levels that grow,
against the oracle's level-0 fold merged level by level, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import series
from oracle import lko

pytestmark = pytest.mark.gpu

# (nsamps, tsamp, nbins, limits, bseg_ffa); nbins 32 .. 1024 have kernels of their own
CASES = {
    "freq_nb32": (2**16, 64e-6, 32, [[20.0, 40.0]], None),
    "freq_nb33": (2**16, 64e-6, 33, [[20.0, 40.0]], 2**15),
    "freq_nb50": (2**16, 64e-6, 50, [[20.0, 40.0]], None),
    "accel_nb64": (2**16, 1e-3, 64, [[-300.0, 300.0], [5.0, 8.0]], None),
    "accel_nb100": (2**16, 1e-3, 100, [[-300.0, 300.0], [5.0, 6.0]], 2**15),
    "accel_nb128": (2**16, 1e-3, 128, [[-300.0, 300.0], [5.0, 6.0]], 2**14),
    "freq_nb200": (2**16, 64e-6, 200, [[20.0, 30.0]], None),
    "freq_nb256": (2**16, 64e-6, 256, [[20.0, 30.0]], 2**15),
    "freq_nb512": (2**16, 64e-6, 512, [[10.0, 14.0]], None),
    "freq_nb1000": (2**16, 64e-6, 1000, [[8.0, 10.0]], 2**15),
    "freq_nb1024": (2**16, 64e-6, 1024, [[8.0, 10.0]], None),
    "jerk_nb32": (2**16, 1e-3, 32, [[-60.0, 60.0], [-900.0, 900.0], [5.0, 6.0]], 2**15),
    "accel_nb32_growing": (2**18, 1e-3, 32, [[-20000.0, 20000.0], [5.0, 8.0]], 2**17),
}


def _bf16(x):
    """Round to nearest even to 8 significant bits."""
    u = x.view(np.uint32).astype(np.uint64)
    u = (u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000
    return u.astype(np.uint32).view(np.float32)


def _merged(op, nbins, e, v, bf16):
    fold = lko.ffa(op, e, v, level=0).reshape(int(op.nsegments[0]), -1, 2, nbins)
    coords = lko.resolve(op)
    j = np.arange(nbins)
    for level in range(1, op.n_levels):
        c = coords[op.ncoords_offsets[level]:][: int(op.ncoords[level])]

        def rot(rows, idx, shift):
            s = (shift + np.float32(0.5)).astype(np.int64) % nbins
            return np.take_along_axis(rows[:, idx], ((j[None, :] - s[:, None]) % nbins)[None, :, None, :], axis=3)

        if op.nparams == 1:
            tail, head = fold[0::2][:, c["idx"]], rot(fold[1::2], c["idx"], c["shift"])
        else:
            tail = rot(fold[0::2], c["i_tail"], c["shift_tail"])
            head = rot(fold[1::2], c["i_head"], c["shift_head"])
        fold = tail + head
        if bf16 and level + 1 < op.n_levels:
            fold = _bf16(fold)
    return fold.ravel()


@pytest.mark.parametrize("storage", ["fp32", "bf16"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_levels_match_one_at_a_time(cuda, name, storage):
    from loki_b200.configs import PulsarSearchConfig
    from loki_b200.ffa import FFACUDA

    n, tsamp, nbins, lims, bseg = CASES[name]
    cfg = PulsarSearchConfig(n, tsamp, nbins, 1.0, np.array(lims), use_fourier=False, bseg_ffa=bseg,
                             score_widths=[1, 2, 3])
    op = lko.plan_create(lko.make_cfg(n, tsamp, nbins, 1.0, lims, bseg_ffa=bseg))
    e, v = series(n, 33)
    want = _merged(op, nbins, e, v, storage == "bf16")
    if storage == "fp32":
        np.testing.assert_array_equal(want.view(np.uint32), lko.ffa(op, e, v).view(np.uint32))
    ffa = FFACUDA(cfg, fold_storage=storage)
    ffa.set_profiling(True)
    got = ffa.execute(e, v)
    # several levels in fewer launches
    assert sum(s["stage"] == "merge" for s in ffa.profile()) < op.n_levels - 1
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
    assert ffa.status() == 0
