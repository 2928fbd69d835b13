"""Every quantity of dl_reduce, dl_reduce_static and the free-energy sums of
dl_energy against NumPy sums over the fields that the handle holds, where the tile
march (32 x 8 columns, some planes at a time, chunks shared out over the blocks) has
an edge: domains narrower than a tile, sides that end inside one, nz that ends inside
a chunk, more tiles than blocks, one block for all of them, a NaN in phi (left out of
the counts and the range, in the sums of phi).

Tolerances: the sums are FP64 over at most some 500 terms per thread and then
pairwise: 1e-12 of the sum of the terms' magnitudes covers their rounding and
NumPy's. S:S of FP32 fields is formed in FP32 (20 operations of relative error 6e-8 on
sums of ten terms): 2e-6."""
import numpy as np
import pytest

from droplet_gb300 import Params, init_fields
from droplet_gb300.solver import Droplet, FORM_FP16, FORM_FP32, FORM_FP64
from oracle import np_energy

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (5, 9, 40), (48, 10, 19), (33, 7, 21), (32, 8, 64), (40, 17, 130), (7, 100, 3), (129, 3, 5), (65, 33, 37),
          (330, 250, 5)]


def made(form, shape, nan=False):
    nx, ny, nz = shape
    P = Params.lbm_drop_xy().replace(tauf=0.8, nu1=0.1, nu2=0.05, kappag=2e-3)
    rng = np.random.default_rng(nx + 1000 * ny + nz)
    phi = P.phi1 + (P.phi2 - P.phi1) * rng.uniform(0.0, 1.0, (nz, ny, nx))
    if nan:
        phi[nz // 2, ny - 1, nx // 2] = np.nan
    u = [0.02 * rng.standard_normal((nz, ny, nx)) for _ in range(3)]
    f = init_fields.fields(phi, *u)
    f["p"] = f["p"] + 1e-3 * rng.standard_normal((nz, ny, nx))
    g = Droplet(P, shape, form)
    g.set_fields(**f)
    return P, g, g.get_fields()


def expected(P, f):
    """name -> (value, sum of the magnitudes of its terms)"""
    phi, p, u = f["phi"], f["p"], [f["u1"], f["u2"], f["u3"]]
    nz, ny, nx = phi.shape
    z, y, x = (a.astype(np.float64) for a in np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij"))
    w = (phi - P.phi1) / (P.phi2 - P.phi1)
    with np.errstate(invalid="ignore"):
        inside, outside, drop = w > 0.95, w < 0.05, phi > 0.5 * (P.phi1 + P.phi2)
    terms = {"phi_sum": phi, "p_sum": p, "ke": 0.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2), "vol_smooth": w, "w_sum": w,
             "vol_count": drop * 1.0, "p_in": p[inside], "n_in": inside * 1.0, "p_out": p[outside], "n_out": outside * 1.0}
    terms.update({("mom", k): v for k, v in enumerate(u)})
    terms.update({("w_x", k): w * v for k, v in enumerate((x, y, z))})
    terms.update({("w_xx", k): w * v for k, v in enumerate((x * x, y * y, z * z, x * y, x * z, y * z))})
    out = {k: (float(v.sum()), float(np.nansum(np.abs(v)))) for k, v in terms.items()}
    out["diss"] = (np_energy.dissipation_sum(P, *u, phi),) * 2
    return out


def check(P, d, want, f, rel_diss):
    for k, (v, mag) in want.items():
        got = d[k] if isinstance(k, str) else d[k[0]][k[1]]
        if np.isnan(v):
            assert np.isnan(got), (k, got)
        elif k in ("vol_count", "n_in", "n_out"):
            assert got == v, k
        else:
            assert abs(got - v) <= (rel_diss if k == "diss" else 1e-12) * mag, (k, got, v, mag)
    assert d["phi_min"] == np.nanmin(f["phi"]) and d["phi_max"] == np.nanmax(f["phi"])


@pytest.mark.parametrize("form", [FORM_FP64, FORM_FP32, FORM_FP16])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("nan", [False, True])
def test_reductions_match_numpy(form, shape, nan):
    P, g, f = made(form, shape, nan)
    want = expected(P, f)
    rel = 1e-12 if form == FORM_FP64 else 2e-6
    check(P, g.reduce(), want, f, rel)
    for nblocks in (0, 1, 3):
        check(P, g.reduce_static(nblocks), want, f, rel)
    g.close()


@pytest.mark.parametrize("form", [FORM_FP64, FORM_FP32])
@pytest.mark.parametrize("shape", SHAPES)
def test_free_energy_matches_numpy(form, shape):
    P, g, f = made(form, shape)
    d = g.energy(0)
    phi = f["phi"]
    lg = np.log(phi / (1.0 - P.b * phi))
    mag = np.abs(phi * P.T * lg).sum() + np.abs(P.a * phi * phi).sum()
    psi, mu, gsq = np_energy.free_energy_sums(P, phi)
    assert abs(d["psi_sum"] - psi) <= 1e-12 * mag
    mag = (np.abs(P.T * lg) + P.T / (1.0 - P.b * phi) + 2.0 * P.a * phi + P.kappag * 28.0 * phi / (5.0 * P.ds ** 2)).sum()
    assert abs(d["mu_sum"] - mu) <= 1e-12 * mag
    # the gradient cancels: ten terms of up to phi2 for a sum of their differences
    assert abs(d["grad_sq_sum"] - gsq) <= 1e-11 * gsq
    g.close()
