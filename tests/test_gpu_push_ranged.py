"""A viscosity ratio with the range of the previous step's phi in the push form
(calls of several steps on 2^18 sites or more; tau_g from a pass over f before
each): against the oracle on grids that end inside a tile and on the smallest
that takes it, with each body force, walls and LES; calls on either side of the
switch in turn; the range and the settled state after a call."""
import numpy as np
import pytest

from droplet_gb300 import Params
from droplet_gb300.solver import Droplet, FORM_FP32
from oracle import pyoracle
from test_gpu_fast import errors, make_case, start

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["plain", "walls", "les_static_force", "spectral_les"])
@pytest.mark.parametrize("shape", [(64, 64, 64), (33, 90, 97), (260, 37, 29)])
@pytest.mark.parametrize("calls", [(4,), (1, 4, 3, 7), (12, 1, 1, 6)])
def test_ranged_push_tracks_oracle(case, shape, calls):
    P, f, mode, force = make_case(case, shape)
    P = P.replace(nu2=0.03)
    g, o = Droplet(P, shape, FORM_FP32), pyoracle.OracleDroplet(P, shape)
    for s in (g, o):
        start(s, f, mode, force)
    for n in calls:
        g.step(n)
        assert g.get_option("pushed") == 0
        o.step(n)
    e = errors(P, g.get_fields(), o.get_fields())
    assert e["phi"] <= 2e-5 and e["u"] <= 2e-6 and e["p"] <= 2e-6, e
    span = P.phi2 - P.phi1
    assert np.allclose(g.minmax(), o.minmax(), rtol=0.0, atol=2e-5 * span)
    g.close()
    o.close()
