"""Last bits of the surrogate's training inputs and gradients.  The backward pass rounds its operands to
BF16, where one FP32 ulp of a target, a carrier or a factor moves a gradient by 1e-5 of its norm and more,
so the training step is held to the values recorded from the kernels whose delays, spectra and carriers
were FP64 throughout."""

from pathlib import Path

import numpy as np
import pytest

from tests import _golden as G
from tests._gpu import np64, require_gpu, torch

pytestmark = pytest.mark.gpu

RECORDED = Path(__file__).resolve().parent / "recorded" / "training_step.npz"


@pytest.fixture(scope="module")
def sur():
    require_gpu()
    from fastsimus_gb300 import workloads as W
    from fastsimus_gb300.surrogate import TxFieldSurrogate, cfg5_box

    p = W.cfg1_probe()
    return TxFieldSurrogate(p, W.cfg1_medium(), cfg5_box(p), seed=4)


def test_training_step_keeps_its_bits(sur):
    """Targets and carriers equal the recorded ones but for one in a thousand (a phase that FP64 rounds the
    other way); the gradients, projected onto one vector per layer, within 1e-7 of their norm: the
    arithmetic is the same, and of 3,072 rows none or one may carry another target bit."""
    ref = np.load(RECORDED)
    _, u, aux, field = sur.make_dataset(20000, seed=5)
    for got, key in ((field[:512], "field"), (aux[:512, :10], "carriers")):
        got = got.cpu().numpy()
        assert np.mean(got != ref[key]) < 1e-3 and G.rel_l2(got, ref[key]) < 1e-8, key
    gW, gb, _ = sur.gradients(u, aux, n_tiles=24, n_split=5, seed=11)
    for i, (w, b) in enumerate(zip(gW, gb)):
        assert G.rel_l2(w.double().cpu().numpy() @ np.cos(np.arange(w.shape[1])), ref[f"w{i}"]) < 1e-7, f"w{i}"
        assert G.rel_l2(b.cpu().numpy(), ref[f"b{i}"]) < 1e-7, f"b{i}"


def test_carriers_of_the_prediction(sur):
    """The field from one unit amplitude is the carrier itself: within FP32's half ulp below one (2^-25 in
    each part) and 1e-8 for the phase and the series, and in the norm within the rounding's uniform error
    (2.1e-8 for uniform angles) and 0.4e-8."""
    import oracle.mlp_fp64 as M

    q = sur.sample_domain(20000, seed=6)
    ref = M.carriers(q.cpu().numpy(), sur.params.n_elements, sur.params.pitch, sur.medium.speed_of_sound)
    for j in range(5):
        for part in (0, 1):
            net = torch.zeros(q.shape[0], 10, device=q.device)
            net[:, 2 * j + part] = 1.0
            out = torch.empty(q.shape[0], dtype=torch.complex64, device=q.device)
            assert sur.lib.fsg_surrogate_combine(sur.domain, q.data_ptr(), q.shape[0], net.data_ptr(), 1.0,
                                                 out.data_ptr(), sur._stream()) == 0
            want = ref[:, j] * (1j if part else 1)
            got = np64(out)
            assert np.max(np.abs(got - want)) < np.sqrt(2) * (2.0**-25 + 1e-8)
            assert G.rel_l2(got, want) < 2.5e-8


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_forward_of_queries_at_any_float(sur, offset):
    """A contiguous view need not start on a 16-byte boundary: the same bits as from an aligned copy."""
    u, _ = sur.inputs(sur.sample_domain(300, seed=8), with_aux=False)
    store = torch.empty(4 * 300 + 4, device=u.device)
    view = store[offset:offset + 4 * 300].view(300, 4)
    view.copy_(u)
    assert view.is_contiguous() and view.data_ptr() % 16 == 4 * offset
    assert torch.equal(sur.forward_tc(view), sur.forward_tc(u)) and sur.tc_status() == 0
