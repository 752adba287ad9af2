"""The outer-product tensor-core form of the beam-corrected DFT at the edges of
its grids (runs that end inside and past a warp's 128 or 256 channels, Jones
planes cutting them, component counts at chunk edges and past the merge of the
totals, one, two and four correlations) against the FP64 beam oracle, with the
bound of the other beam tests."""
import numpy as np
import pytest

import oracle
from obit_b200 import uvdata as U
from obit_b200.skymodel import OP_SUB, SkyModelParams
from test_beam_gpu import _check, _run_beam
from test_beam_oracle_cpu import beam_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mt", [U.MOD_POINT, U.MOD_POINT_SPEC, U.MOD_GAUSS, U.MOD_GAUSS_SPEC])
@pytest.mark.parametrize("nstok, nchan, nif, njc, ncomp", [
    (4, 128, 1, 1, 48), (4, 129, 1, 1, 65), (4, 257, 1, 2, 97), (2, 300, 2, 3, 70), (4, 64, 8, 1, 530),
    (1, 200, 1, 2, 64), (2, 512, 1, 1, 550)])
def test_beam_grid_edges(mt, nstok, nchan, nif, njc, ncomp):
    torch = pytest.importorskip("torch")
    uv, sky, beam = beam_case(mt=mt, nstok=nstok, nrow=7, nchan=nchan, nif=nif, ncomp=ncomp, njc=njc, ntype=3,
                              seed=nchan + ncomp, flag_frac=0.05)
    info = {}
    got = _run_beam(uv, sky, SkyModelParams(op=OP_SUB), beam, torch, info=info)
    assert info["form"] == 1
    want, l1 = oracle.apply_beam_fp64(uv, sky, SkyModelParams(op=OP_SUB), beam)
    _check(uv, got, want, l1, OP_SUB)


def test_beam_mixed_model_in_table_order():
    """Points and Gaussians interleaved, indices unordered: the Jones table stays
    in the caller's order while the kernel reads an ordered copy of the model."""
    torch = pytest.importorskip("torch")
    uv, sky, beam = beam_case(mt=U.MOD_GAUSS_SPEC, nrow=9, nchan=256, nif=1, ncomp=400, njc=2, seed=77)
    sky.comps[::2, 4:7] = 0.0
    r = np.random.default_rng(1)
    order = r.permutation(sky.ncomp)
    sky.comps = np.ascontiguousarray(sky.comps[order])
    got = _run_beam(uv, sky, SkyModelParams(op=OP_SUB), beam, torch)
    want, l1 = oracle.apply_beam_fp64(uv, sky, SkyModelParams(op=OP_SUB), beam)
    _check(uv, got, want, l1, OP_SUB)
