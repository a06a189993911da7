"""I/Q demodulation of few channels and of many short records: columns of several frames in one CTA, one
thread per column, segments and their remainders; not-a-number samples.
"""

import numpy as np
import pytest

from oracle import das_fp64 as D
from tests import _golden as G
from tests._gpu import np64, require_gpu, torch

pytestmark = pytest.mark.gpu

FS, FC = 20e6, 5e6


def _iq(rf, bw=None):
    from fastsimus_gb300.beamform import rf2iq

    return np64(rf2iq(torch.as_tensor(rf, device="cuda"), FS, FC, bw))


@pytest.mark.parametrize("ns,nc,nf", [(1000, 1, 9), (33, 3, 5), (40, 5, 13), (2273, 2, 7), (5000, 1, 3),  # a warp per column
                                      (19, 64, 9), (64, 7, 300), (200, 1, 5700), (320, 8, 1121)])  # a thread per column
def test_columns_of_several_frames(ns, nc, nf):
    """Every frame and channel ends up in its own place; FP32 cascade: relative L2 <= 2e-5, as for the
    plain sizes."""
    require_gpu()
    rng = np.random.default_rng(ns + nc)
    rf = (rng.standard_normal((nf, ns, nc)) * rng.uniform(0.5, 2.0, (nf, 1, nc))).astype(np.float32)
    got = _iq(rf)
    assert got.shape == rf.shape
    for f in {0, 1, nf // 2, nf - 2, nf - 1}:
        assert G.rel_l2(got[f], D.rf2iq(rf[f].astype(np.float64), FS, FC)) < 2e-5


@pytest.mark.parametrize("ns,nc,nf", [(1000, 3, 5), (2400, 8, 1), (64, 4, 500)])
def test_nan_and_infinite_samples_spoil_their_column_only(ns, nc, nf):
    """The filter is recursive in both directions: nothing of a column with one such sample is a number, and
    the others do not see it."""
    require_gpu()
    rng = np.random.default_rng(ns)
    rf = rng.standard_normal((nf, ns, nc)).astype(np.float32)
    clean = _iq(rf)
    rf[1 % nf, 3, 0], rf[0, ns - 2, 1], rf[nf - 1, ns // 2, nc - 1] = np.nan, np.inf, np.nan
    got = _iq(rf)
    bad = np.zeros((nf, nc), dtype=bool)
    bad[1 % nf, 0] = bad[0, 1] = bad[nf - 1, nc - 1] = True
    assert not np.isfinite(got.transpose(0, 2, 1)[bad]).any()
    assert np.array_equal(got.transpose(0, 2, 1)[~bad], clean.transpose(0, 2, 1)[~bad])
