"""The z planes per block of an ensemble's steps and of its members' own: an
ensemble step leaves a member's setting as it was, chosen or set, in both modes;
lz = 0 gives the ensemble's choice back."""
import pytest

from droplet_gb300 import DropletError
from droplet_gb300.ensemble import Ensemble
from droplet_gb300.solver import FORM_FP16, FORM_FP32
from test_gpu_fast import make_case, start

pytestmark = pytest.mark.gpu

SHAPES = [(40, 20, 34), (24, 16, 40), (36, 24, 16)]


@pytest.mark.parametrize("persistent", [0, 1])
@pytest.mark.parametrize("form", [FORM_FP32, FORM_FP16])
@pytest.mark.parametrize("case", ["plain", "spectral_les"])
def test_members_keep_their_planes(case, form, persistent):
    cases = [make_case(case, s, seed=k) for k, s in enumerate(SHAPES)]
    with Ensemble([c[0] for c in cases], SHAPES, form) as ens:
        ens.set_option("persistent", persistent)
        for m, c in zip(ens.members, cases):
            start(m, *c[1:])
        ens.members[1].set_option("lz", 5)
        own = [m.get_option("lz") for m in ens.members]
        assert own[1] == 5
        default = ens.get_option("lz")
        for lz in (13, 3, 0):
            ens.set_option("lz", lz)
            ens.step(3)
            assert ens.get_option("lz") == (lz or default)
            assert [m.get_option("lz") for m in ens.members] == own
        for lz in (-1, 4097):
            with pytest.raises(DropletError):
                ens.set_option("lz", lz)
