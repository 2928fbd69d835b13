"""A viscosity ratio with the range of the previous step's phi: which form steps a
handle depends on its size and options alone. One call of n steps, n calls of one,
calls of several, a run with a phi-range mirror and the same domain in an ensemble
have the same bits (with band forcing, whose coefficients are FP64 sums in no fixed
order, agree within FP32 rounding), and the launches of a call are those of the form
that the size asks for."""
import numpy as np
import pytest

from droplet_gb300 import _abi
from droplet_gb300.ensemble import Ensemble
from droplet_gb300.solver import Droplet, FORM_FP32
from test_gpu_fast import make_case, start

pytestmark = pytest.mark.gpu

N = 9


def run(P, f, mode, force, shape, calls, mirror=None, push=1):
    g = Droplet(P, shape, FORM_FP32)
    g.set_option("push", push)
    start(g, f, mode, force)
    if mirror is not None:
        g.set_minmax_mirror(mirror.data_ptr(), mirror.shape[0])
    for n in calls:
        g.step(n)
    out = g.get_fields(), g.minmax()
    g.close()
    return out


@pytest.mark.parametrize("case", ["plain", "walls", "les_static_force", "spectral_les"])
@pytest.mark.parametrize("shape", [(64, 64, 64), (33, 90, 97), (64, 64, 63)])
def test_grouping_of_steps_changes_nothing(case, shape):
    import torch

    P, f, mode, force = make_case(case, shape)
    P = P.replace(nu2=0.03)
    a, ra = run(P, f, mode, force, shape, (N,))

    def same(b, what):
        for k in a:
            if case == "spectral_les":
                assert np.abs(a[k] - b[k]).max() <= 1e-6 * max(1.0, np.abs(a[k]).max()), (what, k)
            else:
                assert np.array_equal(a[k], b[k]), (what, k, np.abs(a[k] - b[k]).max())

    for calls in ((1,) * N, (4, 3, 2), (1, 5, 3)):
        b, rb = run(P, f, mode, force, shape, calls)
        same(b, calls)
        assert case == "spectral_les" or ra == rb
    slots = torch.zeros((16, 2), dtype=torch.float64).pin_memory()
    b, rb = run(P, f, mode, force, shape, (4, 5), slots)
    same(b, "mirror")
    torch.cuda.synchronize()
    assert tuple(slots[N].tolist()) == rb
    with Ensemble([P, P], [shape, (24, 16, 12)], FORM_FP32) as ens:
        small = make_case(case, (24, 16, 12))
        start(ens.members[0], f, mode, force)
        start(ens.members[1], *small[1:])
        ens.step(4)
        ens.step(5)
        same(ens.members[0].get_fields(), "ensemble")


@pytest.mark.parametrize("shape,ranged", [((64, 64, 64), True), ((64, 64, 63), False)])
def test_launches_are_those_of_the_form(shape, ranged):
    P, f, mode, force = make_case("plain", shape)
    for push, nu2, want in ((1, 0.03, {1: 2, 4: 8} if ranged else {1: 1, 4: 4}),  # step, range between two, settle
                            (0, 0.03, {1: 1, 4: 4}), (1, 0.1, {1: 1, 4: 4})):
        g = Droplet(P.replace(nu2=nu2), shape, FORM_FP32)
        g.set_option("push", push)
        start(g, f, mode, force)
        for n in (1, 4):
            g.profile(True)
            g.step(n)
            assert g.profile_read()["launches"] == want[n], (push, nu2, n)
        g.close()
