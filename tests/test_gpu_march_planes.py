"""The number of z planes a block marches when no "lz" is set: between 1 and
nz, reported by get_option, restored by lz = 0, and without effect on the
values: fields after some steps equal those of one chunk over the whole height
bit for bit (no band forcing; the band projection's FP32 sums are grouped by
chunk, so there 2e-6 of the largest value)."""
import numpy as np
import pytest

from droplet_gb300.ensemble import Ensemble
from droplet_gb300.solver import Droplet, FORM_FP16, FORM_FP32
from test_gpu_fast import make_case, start

pytestmark = pytest.mark.gpu


def fields(P, f, mode, force, shape, form, lz, steps=4):
    g = Droplet(P, shape, form)
    if lz:
        g.set_option("lz", lz)
    start(g, f, mode, force)
    g.step(steps)
    used = g.get_option("lz")
    g.set_option("lz", 0)
    assert 1 <= g.get_option("lz") <= shape[2]
    out = g.get_fields()
    g.close()
    return used, out


@pytest.mark.parametrize("case", ["plain", "walls", "eta", "spectral_les"])
@pytest.mark.parametrize("form", [FORM_FP32, FORM_FP16])
@pytest.mark.parametrize("shape", [(5, 5, 6), (33, 9, 16), (40, 20, 130), (256, 17, 7)])
def test_default_march_changes_no_value(case, form, shape):
    P, f, mode, force = make_case(case, shape)
    lz, a = fields(P, f, mode, force, shape, form, 0)
    whole, b = fields(P, f, mode, force, shape, form, shape[2])
    assert 1 <= lz <= shape[2] and whole == shape[2]
    for k in a:
        if case == "spectral_les":
            tol = (2e-6 if form == FORM_FP32 else 2e-4) * np.abs(b[k]).max()
            assert np.abs(a[k] - b[k]).max() <= tol, k
        else:
            assert np.array_equal(a[k], b[k]), k


def test_ensemble_default_is_common_to_its_members():
    shapes = [(40, 20, 22), (24, 16, 12), (36, 24, 16)]
    cases = [make_case("plain", s, seed=k) for k, s in enumerate(shapes)]
    ens = Ensemble([c[0] for c in cases], shapes)
    for m, c in zip(ens.members, cases):
        start(m, *c[1:])
    lz = ens.get_option("lz")
    assert 1 <= lz <= 22
    ens.step(3)
    for m, c, s in zip(ens.members, cases, shapes):
        _, b = fields(*c, s, FORM_FP32, s[2], steps=3)
        a = m.get_fields()
        for k in a:
            assert np.array_equal(a[k], b[k]), k
    ens.close()
