"""Component tiles cut to the table: models smaller than a tile, and counts about
the tiles' edges, on the recurrence kernels (short channel runs) against the
FP64 oracle within the parity bound, and against an asked-for tile of 128, whose
sums differ by FP32 rounding of the folds alone.  (A lone Gaussian tapered by
e^-40 is off by the rounding of its exponent, whatever the tile: Gaussians are
compared with the other tile only.)"""
import numpy as np
import pytest

from helpers import TOL_REL, gpu_model, model_error, small
from obit_b200 import uvdata as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mt", [U.MOD_POINT, U.MOD_POINT_SPEC, U.MOD_GAUSS_SPEC, U.MOD_POINT_TSPEC])
@pytest.mark.parametrize("nchan, nif", [(1, 2), (40, 1)])
@pytest.mark.parametrize("ncomp", [1, 2, 9, 13, 129, 161, 321])
def test_small_and_uneven_tables(mt, nchan, nif, ncomp):
    uv, sky = small(mt, nrow=33, nchan=nchan, nif=nif, ncomp=ncomp, seed=ncomp)
    if mt != U.MOD_GAUSS_SPEC:
        assert model_error(uv, sky)[0] < TOL_REL
    a, b = gpu_model(uv, sky), gpu_model(uv, sky, ct=128)
    assert np.abs(a - b).max() <= 1e-6 * np.abs(sky.comps[:, 0]).sum()
