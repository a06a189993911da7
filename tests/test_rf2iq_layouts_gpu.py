"""I/Q demodulation of few channels and of many short records: columns of several frames in one CTA, one
thread per column, segments and their remainders; not-a-number samples; the filter's error against a
serial FP32 recursion."""

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


@pytest.mark.parametrize("ns,nc,nf", [(1000, 1, 9), (33, 3, 5), (40, 5, 13), (2273, 2, 7), (5000, 1, 3),  # a warp per column,
                                      (1000, 3, 50), (400, 3, 101), (700, 1, 609), (330, 7, 180),  # 1 to 8 per CTA
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


def _fma(a, b, c):
    return (np.float64(a) * b.astype(np.float64) + c).astype(np.float32)


def _serial(x, bw, dtype):
    """filtfilt's forward-backward pass (odd extension of 18 samples) of the FP32 second-order sections over
    axis 0 of the complex x's parts, one sample after the other, in `dtype`."""
    from fastsimus_gb300.beamform import _lowpass

    sos, zi = (a.astype(np.float32).astype(dtype) for a in _lowpass(FS, FC, bw))
    fma = _fma if dtype == np.float32 else lambda a, b, c: a * b + c

    def run(v):
        z = [[zi[s][k] * v[0] for k in range(2)] for s in range(len(sos))]
        out = np.empty_like(v)
        for n in range(v.shape[0]):
            u = v[n]
            for s, (b0, b1, b2, _, a1, a2) in enumerate(sos):
                y = fma(b0, u, z[s][0])
                z[s] = [fma(b1, u, fma(-a1, y, z[s][1])), fma(b2, u, -a2 * y)]
                u = y
            out[n] = u
        return out

    x = x.astype(dtype)
    ext = np.concatenate([2 * x[:1] - x[18:0:-1], x, 2 * x[-1:] - x[-2:-20:-1]])
    return 2 * run(run(ext)[::-1])[::-1][18:-18]


@pytest.mark.parametrize("ns,bw,slack", [(64, None, 1.06), (200, None, 1.06), (1015, None, 1.02), (1015, 2e5, 1.02),
                                         (1015, 1e5, 1.02)])
def test_filter_error_is_the_serial_recursions(ns, bw, slack):
    """The scan over chunks adds one rounding of the state per chunk (a 32nd part of the record, 1 to 4% of
    the error in records of up to 200 samples) and nothing else, at narrow cut-offs too."""
    require_gpu()
    rng = np.random.default_rng(ns)
    rf = rng.standard_normal((ns, 400)).astype(np.float32)
    cyc = np.arange(ns) * (FC / FS)
    e = np.exp(-2j * np.pi * (cyc - np.rint(cyc)))[:, None].astype(np.complex64)  # FS = 4 FC: exact
    x = np.concatenate([rf * e.real, rf * e.imag], axis=1)
    ref = _serial(x, bw, np.float64)
    got = _iq(rf, bw)
    got = np.concatenate([got.real, got.imag], axis=1)
    assert G.rel_l2(got, ref) < slack * G.rel_l2(_serial(x, bw, np.float32), ref)
