"""The pixel list handed to fsg_das, on the CPU: the grids' C order from any memory order, small images by
one upload."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from fastsimus_gb300 import beamform as B  # noqa: E402


@pytest.mark.parametrize("shape", [(), (1,), (7, 5), (3, 4, 2), (150, 140)])
@pytest.mark.parametrize("order", ["C", "F", "strided"])
def test_pixels_follow_the_grids_c_order(shape, order):
    rng = np.random.default_rng(1)
    x, z = rng.standard_normal(shape), rng.standard_normal(shape)
    if order == "F":
        x, z = np.asfortranarray(x), np.asfortranarray(z)
    elif order == "strided" and shape:
        x, z = np.repeat(x, 2, axis=-1)[..., ::2], z[::-1]
    got = B._interleaved(x, z, torch.device("cpu"))
    assert got.is_contiguous() and got.dtype == torch.float64
    assert np.array_equal(got.numpy(), np.stack([x.ravel(), z.ravel()], axis=1))


def test_a_small_image_is_one_upload(monkeypatch):
    calls = []
    as_tensor = torch.as_tensor
    monkeypatch.setattr(B.torch, "as_tensor", lambda *a, **k: calls.append(1) or as_tensor(*a, **k))
    B._interleaved(np.zeros((50, 40)), np.zeros((50, 40)), torch.device("cpu"))
    assert len(calls) == 1
