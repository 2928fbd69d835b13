"""A member with band forcing takes the same steps whatever the other members of
its ensemble do: its FP32 band sums are grouped by blocks of 32 planes, so its
fields equal those that it has in an ensemble of band-forced members (FP16
storage shows any other grouping within a few steps). The groups' sums are added
in FP64 in no fixed order, which changes an FP32 coefficient with a probability of
some 1e-8 per coefficient and step: equality is asked for."""
import numpy as np
import pytest

from droplet_gb300.ensemble import Ensemble
from droplet_gb300.solver import FORM_FP16, FORM_FP32
from test_gpu_fast import make_case, start

pytestmark = pytest.mark.gpu

SHAPES = [(40, 20, 96), (64, 32, 80)]


def member_fields(first, form):
    cases = [make_case(c, s, seed=k) for k, (c, s) in enumerate(zip((first, "spectral_les"), SHAPES))]
    if first != "spectral_les":  # one LES setting in an ensemble
        cases[0] = (cases[0][0].replace(les=True, Cs=0.1, delta=1.0),) + cases[0][1:]
    with Ensemble([c[0] for c in cases], SHAPES, form) as ens:
        for m, c in zip(ens.members, cases):
            start(m, *c[1:])
        ens.step(20)
        return ens.members[1].get_fields()


@pytest.mark.parametrize("form", [FORM_FP32, FORM_FP16])
def test_band_forced_member_beside_others(form):
    a, b = member_fields("plain", form), member_fields("spectral_les", form)
    for k in a:
        assert np.array_equal(a[k], b[k]), (k, np.abs(a[k] - b[k]).max())
