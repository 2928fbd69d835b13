"""The FP64 band force is bitwise the oracle's for every band (kc 2 to 5) at
sizes that end inside a block of 32 rows, 32 columns or 16 terms, and at the
smallest box that holds the band."""
import numpy as np
import pytest

from droplet_gb300 import Params, _abi, init_fields
from droplet_gb300.solver import Droplet, FORM_FP64
from oracle import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kc,shape", [(2, (3, 3, 4)), (2, (33, 7, 32)), (3, (5, 5, 6)), (3, (37, 11, 35)),
                                      (3, (64, 16, 16)), (4, (7, 19, 8)), (5, (9, 9, 10)), (5, (70, 17, 66))])
def test_fp64_band_force_bitwise(kc, shape):
    P = Params.lbm_drop_xy().replace(tauf=0.7, nu1=0.1, nu2=0.1, kappag=2e-3, eps=1e-5, kc=kc)
    rng = np.random.default_rng(kc)
    phi = init_fields.tanh_droplets(shape, P, [tuple(n / 2 for n in shape)], [min(shape) / 3], width=1.0)
    f = init_fields.fields(phi, *[0.02 * rng.standard_normal(phi.shape) for _ in range(3)])
    out = []
    for s in (Droplet(P, shape, FORM_FP64), pyoracle.OracleDroplet(P, shape)):
        s.set_fields(**f)
        s.init_equilibrium()
        s.set_force(_abi.DL_FORCE_SPECTRAL)
        s.step(3)
        out.append(s.get_fields())
        s.close()
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
