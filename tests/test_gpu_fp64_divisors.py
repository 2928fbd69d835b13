"""The FP64 form is bitwise the oracle whichever way its known divisors take
(tau_f and a uniform tau_g 1, a power of two, short, general; ds other than
1; tau_g per site from LES, a viscosity ratio in both modes, and A_nu), on a
grid whose sites do not fill the last block."""
import numpy as np
import pytest

from droplet_gb300 import Params, init_fields
from droplet_gb300.solver import Droplet, FORM_FP64
from oracle import pyoracle

pytestmark = pytest.mark.gpu

CASES = {
    "tauf_one": dict(tauf=1.0),
    "tauf_two": dict(tauf=2.0),
    "tauf_short": dict(tauf=0.75),
    "tauf_general": dict(tauf=0.8130000000000001),
    "taug_one": dict(nu1=0.5 / 3.0, nu2=0.5 / 3.0),
    "taug_short": dict(nu1=0.25, nu2=0.25),
    "ds": dict(ds=0.37),
    "les": dict(les=True, Cs=0.2, delta=1.0),
    "ratio": dict(nu2=0.03),
    "ratio_fixed": dict(nu2=0.03, visc_mode=1),
    "anu": dict(Anu=0.05, nu2=0.05),
    "les_walls": dict(les=True, Cs=0.2, delta=1.0, walls=True, wall_u=(0.02, -0.01, 0.0)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_fp64_bitwise_for_every_divisor(name):
    shape = (19, 7, 5)
    P = Params.lbm_drop_xy().replace(**{**dict(tauf=0.7, nu1=0.1, nu2=0.1, kappag=2e-3), **CASES[name]})
    rng = np.random.default_rng(5)
    phi = init_fields.tanh_droplets(shape, P, [(9.0, 3.2, 2.1)], [2.3], width=1.0)
    f = init_fields.fields(phi, *[0.02 * rng.standard_normal(phi.shape) for _ in range(3)])
    out = []
    for s in (Droplet(P, shape, FORM_FP64), pyoracle.OracleDroplet(P, shape)):
        s.set_fields(**f)
        s.init_equilibrium()
        s.step(5)
        d = s.get_fields()
        d["f"], d["g"] = s.get_populations()
        out.append(d)
        s.close()
    for k, v in out[0].items():
        assert np.array_equal(v, out[1][k]), k
