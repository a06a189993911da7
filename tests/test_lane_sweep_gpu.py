"""simus_lane_kernel at the edges of its mapping, against the FP64 oracle: element counts around the
64 of a warp and the 32 of a lane half, scatterer counts around the points of a group and a tile,
and workspaces below the default (smaller chunks, short bands, fewer CTAs).  Tolerance: the plain
kernels' relative L2 <= 1e-5."""

import numpy as np
import pytest

import oracle.fastsimus_fp64 as O
from tests import _golden as G
from tests._gpu import np64, require_gpu, torch

pytestmark = pytest.mark.gpu

PLAIN_TOL = 1e-5


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


def _case(E, U, n, seed=0):
    from fastsimus_gb300 import MediumParams, simus_precompute
    from fastsimus_gb300.params import TransducerParams

    p = TransducerParams(freq_center=4e6, pitch=3e-4, n_elements=E, width=2.7e-4, bandwidth=0.6)
    m = MediumParams(attenuation=0.4)
    rng = np.random.default_rng(seed + E + n)
    s = np.stack([rng.uniform(-12e-3, 12e-3, n), rng.uniform(3e-3, 25e-3, n)], axis=-1)
    r = rng.standard_normal(n)
    d = np.linspace(0.0, 1e-6, E)
    d[E // 2] = np.nan
    apod = np.hanning(E + 2)[1:-1] + 0.1
    plan = simus_precompute(s, r, d, p, m, element_splitting=U)
    return p, m, s, r, d, apod, plan


@pytest.mark.parametrize("E,U,n,ffd", [(33, 1, 1, False), (63, 2, 3, False), (65, 2, 5, True), (64, 3, 2, True),
                                       (96, 4, 7, False), (127, 1, 49, True), (129, 2, 17, False),
                                       (191, 1, 33, True), (193, 2, 9, False), (255, 1, 8, False), (170, 3, 4, True)])
def test_ragged_elements_and_scatterers(E, U, n, ffd):
    from fastsimus_gb300 import simus_compute

    p, m, s, r, d, apod, plan = _case(E, U, n)
    got = np64(simus_compute(s, r, d, plan, p, m, tx_apodization=apod, full_frequency_directivity=ffd).spectrum)
    ref = O.simus_compute(s, r, d, plan, p, m, tx_apodization=apod, full_frequency_directivity=ffd).spectrum
    assert G.rel_l2(got, ref) < PLAIN_TOL


@pytest.mark.parametrize("E,U,ffd", [(64, 2, 0), (128, 2, 1), (192, 2, 0), (256, 1, 0)])
def test_small_workspaces(E, U, ffd):
    """From the default workspace down to a tenth of it: either the call runs and matches, or it is
    refused for its workspace."""
    from fastsimus_gb300 import _device, _native

    n = 400
    p, m, s, r, d, apod, plan = _case(E, U, n)
    ref = O.simus_spectrum_selected(s, r, np.nan_to_num(d), plan, p, m, tx_apodization=np.where(np.isnan(d), 0, apod),
                                    full_frequency_directivity=bool(ffd))
    lib = _native.load()
    dev = torch.device("cuda", torch.cuda.current_device())
    tabs = _device.plan_tables(plan, dev)
    probe, med, fplan = _native.make_probe(p, plan.n_sub), _native.make_medium(m), tabs.fsg_plan(plan)
    st, rc, dd, aa = (torch.as_tensor(x, device=dev) for x in (s, r, d, apod))
    full = lib.fsg_simus_workspace_size(probe, fplan, n)
    ran = 0
    for frac in (1.0, 0.7, 0.5, 0.35, 0.2, 0.1):
        ws = torch.empty(int(full * frac) // 256 * 256, dtype=torch.uint8, device=dev)
        out = torch.full((plan.selected_freqs.shape[0], E), float("nan"), dtype=torch.complex64, device=dev)
        code = lib.fsg_simus(probe, med, fplan, st.data_ptr(), rc.data_ptr(), n, dd.data_ptr(), aa.data_ptr(), ffd,
                             _native.FSG_OUT_SELECTED_RAW, out.data_ptr(), ws.data_ptr(), ws.numel(),
                             torch.cuda.current_stream(dev).cuda_stream)
        if code == _native.FSG_EWORKSPACE:
            continue
        _native.check(code)
        ran += 1
        assert G.rel_l2(np64(out), ref) < PLAIN_TOL
    assert ran >= 3


@pytest.mark.parametrize("U", [1, 3])
@pytest.mark.parametrize("x_max", [1.0, 3.99, 4.01, 6.2])
def test_directivity_polynomials(x_max, U):
    """Full-frequency directivity on both sides of the argument where its polynomial changes and near the
    largest one accepted, in the sweep of the RF spectrum and in the field (an odd number of sources)."""
    import fastsimus_gb300 as F

    E, n = 67, 21
    rng = np.random.default_rng(int(100 * x_max) + U)
    m = F.MediumParams(attenuation=0.4)
    s = np.stack([rng.uniform(-12e-3, 12e-3, n), rng.uniform(3e-3, 25e-3, n)], axis=-1)
    r, d = rng.standard_normal(n), np.linspace(0.0, 1e-6, E)

    def probe(width):
        return F.TransducerParams(freq_center=4e6, pitch=1.05 * width, n_elements=E, width=width, bandwidth=0.6)

    width = 3e-4
    for _ in range(3):  # the plan's highest frequency hardly depends on the width
        plan = F.simus_precompute(s, r, d, probe(width), m, element_splitting=U)
        width = x_max * U * m.speed_of_sound / (np.pi * float(plan.selected_freqs[-1]))
    p = probe(width)
    plan = F.simus_precompute(s, r, d, p, m, element_splitting=U)
    got = np64(F.simus_compute(s, r, d, plan, p, m, full_frequency_directivity=True).spectrum)
    ref = O.simus_compute(s, r, d, plan, p, m, full_frequency_directivity=True).spectrum
    assert G.rel_l2(got, ref) < PLAIN_TOL
    fplan = F.pfield_precompute(s, d, p, m, element_splitting=U)
    got = np64(F.pfield_compute(s, d, fplan, p, m, full_frequency_directivity=True))
    assert G.rel_l2(got, O.pfield_compute(s, d, fplan, p, m, full_frequency_directivity=True)) < PLAIN_TOL
    got = np64(F.pfield_compute(s, d, fplan, p, m))
    assert G.rel_l2(got, O.pfield_compute(s, d, fplan, p, m)) < PLAIN_TOL
