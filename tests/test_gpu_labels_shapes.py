"""Labelling where runs, warps and rows meet: rows shorter and longer than a
warp's 32 sites and ending inside one, runs over several warps and over the
periodic ends, a percolating random medium, a full and an empty domain; the
partition and volumes of the NumPy labelling."""
import numpy as np
import pytest

from droplet_gb300 import Params, init_fields
from droplet_gb300.solver import Droplet, FORM_FP32
from oracle import np_labels
from test_gpu_labels import same_partition

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 3, 3), (5, 7, 9), (33, 6, 5), (64, 32, 4), (100, 3, 3), (31, 8, 8), (129, 5, 4)])
@pytest.mark.parametrize("fill", [0.0, 0.15, 0.4, 0.9, 1.0])
@pytest.mark.parametrize("conn", [6, 14, 26])
def test_labels_of_random_media(shape, fill, conn):
    P = Params.lbm_drop_xy()
    rng = np.random.default_rng([shape[0], conn, int(100 * fill)])
    mask = rng.random(shape[::-1]) < fill
    if 0.0 < fill < 0.5:  # whole rows and a column as well: long runs
        mask[0, 0, :] = True
        mask[:, -1, -1] = True
    g = Droplet(P, shape, FORM_FP32)
    g.set_fields(**init_fields.fields(np.where(mask, P.phi2, P.phi1)))
    vols, lab = g.label_droplets(conn, labels=True)
    g.close()
    rv, rl = np_labels.label(mask, conn)
    assert np.array_equal(vols, rv)
    assert np.array_equal(lab > 0, mask) and same_partition(lab, rl)
    # labels are ranks: the volume of label k is vols[k - 1]
    assert np.array_equal(np.bincount(lab.reshape(-1), minlength=len(vols) + 1)[1:], vols.astype(np.int64))
