"""Populations loaded into a handle whose last step nothing has read yet: they are
complete, so nothing of the replaced state (the band force and the wall
reflection of its last streaming) may be added to them. Against a fresh handle
given the same populations, bit for bit; after more steps with band forcing,
whose coefficients are FP64 sums in no fixed order, within their rounding."""
import numpy as np
import pytest

from droplet_gb300 import configs, _abi
from droplet_gb300.solver import Droplet, FORM_FP32, FORM_FP64
from test_gpu_fast import make_case, start

pytestmark = pytest.mark.gpu

FIELDS = ("phi", "u1", "u2", "u3", "p")


@pytest.mark.parametrize("case", ["walls", "spectral_les", "single_phase"])
@pytest.mark.parametrize("form", [FORM_FP32, FORM_FP64])
def test_loaded_populations_are_complete(case, form):
    if case == "single_phase":
        w = configs.precursor(n=32)
        shape, P, f, mode, force = (32, 32, 32), w.params, w.fields, _abi.DL_FORCE_SPECTRAL, None
        P = P.replace(eps=1e-4)
    else:
        shape = (36, 18, 20)
        P, f, mode, force = make_case(case, shape)
        P = P.replace(wall_start=1, eps=1e-4)
    single = case == "single_phase"
    a, b = (Droplet(P, shape, form, single_phase=single) for _ in range(2))
    src = Droplet(P, shape, form, single_phase=single)
    for s in (a, b, src):
        if form == FORM_FP32:
            s.set_option("lz", 16)
        start(s, f, mode, force)
    src.step(5)
    fl, gl = src.get_populations()
    a.step(3)
    if form == FORM_FP32:
        assert a.get_option("pushed") == 1
    a.set_populations(fl, gl)
    b.set_populations(fl, gl)
    for s in (a, b):
        s.step_count = 5
    for x, y in zip(a.get_populations(), b.get_populations()):
        assert np.array_equal(x, y), np.abs(x - y).max()
    x, y = a.get_fields(), b.get_fields()
    for k in FIELDS:
        assert np.array_equal(x[k], y[k]), (k, np.abs(x[k] - y[k]).max())
    for s in (a, b):
        s.step(3)
    x, y = a.get_fields(), b.get_fields()
    for k in FIELDS:
        if mode == _abi.DL_FORCE_SPECTRAL and form == FORM_FP32:
            assert np.abs(x[k] - y[k]).max() <= 1e-7 * max(1.0, np.abs(y[k]).max()), k
        else:
            assert np.array_equal(x[k], y[k]), (k, np.abs(x[k] - y[k]).max())
