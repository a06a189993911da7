"""Argument checks of the surrogate's entry points that return before any launch (no GPU): rows that the
kernels read and write as 16-byte words must start on such a boundary."""

import ctypes

import pytest

from fastsimus_gb300 import _native, build


@pytest.fixture(scope="module")
def lib():
    build.build()
    return _native.load()


def _descriptor(u, aux):
    t = _native.FsgMlpTrain()
    at = 1 << 20  # never read: the check comes first
    for name, kind in t._fields_:
        if kind is ctypes.c_void_p:
            setattr(t, name, at)
        elif kind is _native._V4:
            setattr(t, name, _native._V4(at, at, at, at))
    t.u, t.aux, t.n_data, t.n_out, t.n_tiles, t.n_split = u, aux, 128, 10, 1, 1
    t.workspace_bytes = 0  # refused for its workspace if for nothing else
    return t


@pytest.mark.parametrize("u,aux,code", [(64, 64, _native.FSG_EWORKSPACE), (68, 64, _native.FSG_EINVAL),
                                        (64, 72, _native.FSG_EINVAL)])
def test_training_rows_start_on_a_word(lib, u, aux, code):
    t = _descriptor(u, aux)
    assert lib.fsg_mlp_train_gradients(ctypes.byref(t), 64, 64, None) == code
    if code == _native.FSG_EINVAL:
        assert b"16-byte" in lib.fsg_last_error_string()


def test_normalised_inputs_start_on_a_word(lib):
    dom = _native.FsgSurrogateDomain(x_lo=-1e-2, x_hi=1e-2, z_lo=5e-3, z_hi=3e-2, f_lo=2e6, f_hi=4e6, max_angle=0.3,
                                     pitch=3e-4, speed_of_sound=1540.0, n_elements=64, n_carriers=5)
    assert lib.fsg_surrogate_inputs(ctypes.byref(dom), 64, 8, None, 1.0, 68, None, None) == _native.FSG_EINVAL
    assert b"16-byte" in lib.fsg_last_error_string()
