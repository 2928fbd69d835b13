"""The minimum that the reference's serial scan of phi leaves when every value
exceeds phi1 and the first site holds the smallest (program/lbm_drop_xy.f90
:559-571: a value that raises the maximum is not tested for the minimum): the
push form's settle and the FP64 step give what the scan over the downloaded
field gives, where the first values rise for long (several ordered rounds) and
where they do not, on domains that end inside a round."""
import numpy as np
import pytest

from droplet_gb300 import Params, init_fields
from droplet_gb300.solver import Droplet, FORM_FP32, FORM_FP64

pytestmark = pytest.mark.gpu


def serial_scan(phi, phi1, phi2):
    mx, mn = phi1, phi2
    for v in phi.reshape(-1):
        if v > mx:
            mx = v
        elif v < mn:
            mn = v
    return mn, mx


@pytest.mark.parametrize("form", [FORM_FP32, FORM_FP64])
@pytest.mark.parametrize("shape", [(5, 4, 3), (32, 8, 4), (400, 3, 3), (1400, 3, 4), (33, 21, 17)])
@pytest.mark.parametrize("noise", [0.0, 1e-4])
def test_scan_minimum(form, shape, noise):
    nx, ny, nz = shape
    P = Params.lbm_drop_xy().replace(tauf=0.7, nu1=0.1, nu2=0.1, kappaf=0.0, kappag=0.0)
    x = np.arange(nx)[None, None, :]
    y = np.arange(ny)[None, :, None]
    z = np.arange(nz)[:, None, None]
    # lowest at site 0, rising along the whole first half row
    phi = P.phi1 + 0.3 + 0.2 * (3.0 - np.cos(2 * np.pi * x / nx) - np.cos(2 * np.pi * y / ny) - np.cos(2 * np.pi * z / nz))
    rng = np.random.default_rng(1)
    phi += noise * rng.random(phi.shape)
    phi[0, 0, 0] -= 0.05
    g = Droplet(P, shape, form)
    g.set_fields(**init_fields.fields(phi))
    g.init_equilibrium()
    g.step(1)
    mn, mx = g.minmax()
    out = g.get_fields()["phi"]
    g.close()
    if form == FORM_FP32:  # the range is taken of float phi1 + dphi
        out = (np.float32(P.phi1) + (out - P.phi1).astype(np.float32)).astype(np.float64)
    assert out.min() > P.phi1 and out.reshape(-1)[0] == out.min() and np.sum(out == out.min()) == 1
    assert (mn, mx) == serial_scan(out, P.phi1, P.phi2)
