"""Edges of the spectrum -> RF transform and of the I/Q demodulation: element and sample remainders of
the 64 x 64 tile, one-chunk and many-chunk bands (frequency splits over a cluster of 1 to 8 CTAs),
twiddle tables beyond shared memory; channel remainders, records of one lane's chunk up to several
segments, narrow filters.  Tolerances: FP32 sums of up to 2,000 terms, relative L2 <= 2e-6; the FP32
filter cascade <= 2e-5, both as in the tests of the plain sizes."""

import numpy as np
import pytest

from oracle import das_fp64 as D
from tests import _golden as G
from tests._gpu import np64, require_gpu, torch

pytestmark = pytest.mark.gpu


class _Plan:
    def __init__(self, n_fft):
        self.n_fft = n_fft


@pytest.mark.parametrize("n_fft,k0,kc,E,nb", [(130, 3, 1, 1, 1), (258, 10, 64, 65, 2), (1023, 100, 129, 64, 1),
                                              (2030, 200, 257, 130, 1), (2030, 200, 700, 64, 9), (14001, 900, 1100, 5, 1)])
def test_irfft_tiles_and_splits(n_fft, k0, kc, E, nb):
    require_gpu()
    from fastsimus_gb300.simus import irfft_and_threshold

    rng = np.random.default_rng(n_fft + E)
    s = np.zeros((nb, n_fft // 2 + 1, E), dtype=np.complex64)
    s[:, k0:k0 + kc] = rng.standard_normal((nb, kc, E)) + 1j * rng.standard_normal((nb, kc, E))
    got = np64(irfft_and_threshold(torch.as_tensor(s, device="cuda"), _Plan(n_fft), k_first=k0, k_count=kc, gate=False))
    ref = np.fft.irfft(np.conj(s.astype(np.complex128)), n=n_fft, axis=1)[:, : (n_fft + 1) // 2]
    assert got.shape == ref.shape
    assert G.rel_l2(got, ref) < 2e-6


@pytest.mark.parametrize("ns,nc,nf,bw", [(19, 1, 1, None), (32, 7, 1, None), (33, 8, 2, None), (1015, 9, 1, None),
                                         (2272, 3, 1, None), (2273, 8, 1, None), (5003, 2, 2, 1.5e6)])
def test_rf2iq_chunks_and_segments(ns, nc, nf, bw):
    require_gpu()
    from fastsimus_gb300.beamform import rf2iq

    rng = np.random.default_rng(ns)
    rf = rng.standard_normal((nf, ns, nc)).astype(np.float32)
    got = np64(rf2iq(torch.as_tensor(rf, device="cuda"), 20e6, 5e6, bw))
    ref = np.stack([D.rf2iq(x.astype(np.float64), 20e6, 5e6, bw) for x in rf])
    assert got.shape == ref.shape
    assert G.rel_l2(got, ref) < 2e-5


@pytest.mark.parametrize("nf,n_pix,n_s", [(1, 1, 300), (4, 127, 300), (5, 128, 300), (8, 129, 300), (9, 300, 300),
                                          (17, 33, 300), (2, 40, (1 << 22) + 1), (40, 65, 300), (75, 31, 300)])
@pytest.mark.parametrize("method", ["linear", "nearest"])
def test_das_firing_groups(nf, n_pix, n_s, method):
    """Firing groups (up to four firings, full groups of eight, tails; two and four threads per pixel), pixels
    around a CTA's 128 and a record beyond the short-record floor.  FP32 phases at ~100 wavelengths of path: relative L2 <= 1e-3;
    the signal varies slowly, so that a nearest tap that rounds the other way stays within it."""
    require_gpu()
    from fastsimus_gb300.beamform import DasParam, das

    rng = np.random.default_rng(nf * 1000 + n_pix)
    E, pitch, fs, c, fc = 12, 0.3e-3, 20e6, 1540.0, 5e6
    xe = D.element_frame(E, pitch, np.inf)[0]
    iq = np.zeros((nf, n_s, E), dtype=np.complex64)
    t = np.arange(300)[None, :, None] / 300.0
    iq[:, :300] = np.exp(0.3j * np.pi * (t + rng.uniform(0, 2, (nf, 1, E)))) * rng.uniform(0.5, 1.5, (nf, 1, E))
    delays = np.stack([xe * np.sin(a) / c for a in np.linspace(-0.1, 0.1, nf)])
    delays -= delays.min(axis=1, keepdims=True)
    delays[nf // 2, 5] = np.nan
    x, z = rng.uniform(-2e-3, 2e-3, (n_pix, 1)), rng.uniform(3e-3, 9e-3, (n_pix, 1))
    param = DasParam(fc=fc, pitch=pitch, Nelements=E, width=0.25e-3, c=c, fs=fs, fnumber=1.0)
    got = np64(das(torch.as_tensor(iq, device="cuda"), x, z, delays, param, method))
    ref = D.das(iq[:, :300].astype(np.complex128), x, z, delays, n_elements=E, pitch=pitch, radius=np.inf, c=c, fs=fs,
                fc=fc, fnumber=1.0, method=method)
    assert got.shape == x.shape
    assert G.rel_l2(got, ref) < 1e-3


@pytest.mark.parametrize("baffle", ["soft", "rigid", 1.75])
@pytest.mark.parametrize("E,width,att", [(1, 0.2e-3, 0.0), (33, 0.9e-3, 0.7), (192, 0.27e-3, 0.5)])
def test_txfield_samples(E, width, att, baffle):
    """The exact transmit field for every baffle, with and without attenuation, one and more sub-elements,
    the smallest and a large array; points on a source, on the array's plane, within the clipped distance,
    behind the array and far off axis.  FP32 amplitudes and phases of up to 10^4 sources: rel-L2 < 1e-5."""
    require_gpu()
    from fastsimus_gb300 import MediumParams, TransducerParams
    from fastsimus_gb300.surrogate import TxFieldSurrogate, cfg5_box
    import oracle.fastsimus_fp64 as O

    p = TransducerParams(freq_center=5e6, pitch=1.1 * width, n_elements=E, width=width, bandwidth=0.65, baffle=baffle)
    m = MediumParams(speed_of_sound=1540.0, attenuation=att)
    sur = TxFieldSurrogate(p, m, cfg5_box(p))
    rng = np.random.default_rng(E)
    half = 0.5 * E * p.pitch
    s = np.stack([rng.uniform(-1.2 * half, 1.2 * half, 140), rng.uniform(1e-3, 40e-3, 140),
                  5e6 * rng.uniform(0.6, 1.4, 140), rng.uniform(-0.4, 0.4, 140)], axis=-1)
    s[:4, :2] = [[0.0, 0.0], [3 * half, 0.0], [1e-5, 2e-5], [0.0, -1e-3]]
    s[4, 2:] = [5e6, 0.0]  # the pulse's centre frequency, no steering
    got, ref = np64(sur.exact(torch.as_tensor(s))), O.tx_field_samples(s, p, m)
    assert got.shape == ref.shape and got[3] == 0
    # on the array's plane a rigid source is on or off by the sign of a 1e-16 in FP64: off here
    k = slice(2 if baffle == "rigid" else 0, None)
    assert np.all(np.abs(got[:2]) < 1e-6) and G.rel_l2(got[k], ref[k]) < 1e-5


def test_surrogate_forward_of_many_tiles():
    """Several tiles per CTA: the next tile's features and first products run under the last layer's
    epilogue.  Repeated calls give the same bits; every tile matches the FP64 network within the tolerance
    of the single-tile test (BF16 weights, hi + lo activations: 1e-4)."""
    require_gpu()
    import oracle.mlp_fp64 as M
    from fastsimus_gb300 import workloads as W
    from fastsimus_gb300.surrogate import TxFieldSurrogate, cfg5_box

    p = W.cfg1_probe()
    sur = TxFieldSurrogate(p, W.cfg1_medium(), cfg5_box(p), seed=2)
    u, _ = sur.inputs(sur.sample_domain(4 * 152 * 128 + 77, seed=3), with_aux=False)
    got = sur.forward_tc(u)
    for _ in range(20):
        assert torch.equal(sur.forward_tc(u), got)
    assert sur.tc_status() == 0
    ref, _, _ = M.forward(u.double().cpu().numpy(), *sur.oracle_params())
    assert G.rel_l2(np64(got), ref) < 1e-4


@pytest.mark.parametrize("step,ffd", [(0.05, False), (0.01, False), (0.01, True)])
def test_pfield_long_plans(step, ffd):
    """2,074 and 10,368 frequencies on a grid large enough for one band: the band's tables fit shared
    memory beside the geometry, or the frequencies take more bands.  Relative L2 < 1e-5, as for the
    plans of the golden vectors."""
    require_gpu()
    import fastsimus_gb300 as F
    import oracle.fastsimus_fp64 as O

    p = F.TransducerParams(freq_center=4e6, pitch=3e-4, n_elements=8, width=2.7e-4, bandwidth=0.7)
    m, d = F.MediumParams(attenuation=0.2), np.linspace(0.0, 3e-7, 8)
    grid = np.stack(np.meshgrid(np.linspace(-5e-3, 5e-3, 400), np.linspace(3e-3, 30e-3, 420)), axis=-1)
    plan = F.pfield_precompute(grid, d, p, m, frequency_step=step)
    got = np64(F.pfield_compute(grid, d, plan, p, m, full_frequency_directivity=ffd)).reshape(-1)
    at = np.random.default_rng(1).choice(got.size, 24, replace=False)
    ref = O.pfield_compute(grid.reshape(-1, 2)[at], d, plan, p, m, full_frequency_directivity=ffd)
    assert G.rel_l2(got[at], np.asarray(ref).reshape(-1)) < 1e-5
