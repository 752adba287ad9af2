"""The tensor-core form of the DFT against the FP64 oracle at the edges of its
tiles (rows, columns, chunks of components, merged totals, several runs, the
smallest model it takes), and which calls it takes.

The bound is the parity bound of every kernel, 1e-5 of the L1 norm: the form
drops less than 2^-22 of each term's scale, and the planner bounds what a
spectrum or taper leaves out by 2.5e-6 of a term."""
import numpy as np
import pytest

import oracle
from helpers import OBIT_DFT_RECUR, TOL_REL, gpu_model, run_gpu, small
from obit_b200 import uvdata as U
from obit_b200.skymodel import OP_DIV, OP_REPL, OP_SUB, GPUSkyModel, SkyModelParams

pytestmark = pytest.mark.gpu

FAMILIES = [U.MOD_POINT, U.MOD_POINT_SPEC, U.MOD_GAUSS, U.MOD_GAUSS_SPEC]


def _plan(uv, sky, params=None, xyz=None, **kernel):
    gm = GPUSkyModel("plan")
    try:
        gm.DFTInit(sky, uv, params or SkyModelParams(nVisPIO=1))
        if kernel:
            gm.set_kernel(**kernel)
        gm.DFTSetMod(sky)
        if xyz is not None:
            gm.set_positions_fp64(xyz)
        return gm.plan_info()
    finally:
        gm.close()


def _error(uv, sky):
    g = gpu_model(uv, sky)
    m, l1 = oracle.model_fp64(uv, sky)
    ok = ~np.isnan(l1)
    return float((np.abs(g - m)[ok] / l1[ok]).max())


@pytest.mark.parametrize("mt", FAMILIES)
@pytest.mark.parametrize("nchan, nif, ncomp", [
    (128, 1, 48), (129, 1, 65), (255, 1, 100), (256, 1, 511), (257, 2, 97), (512, 1, 64), (300, 2, 130),
    (513, 1, 33 + 16), (64, 8, 530), (256, 4, 1100), (1030, 1, 70)])
def test_tile_edges(mt, nchan, nif, ncomp):
    """Runs that end inside, at and past a warp's grid and a team; component
    counts at chunk edges and past the first merge of the totals.  (With a few
    components of widely spread indices a spectrum may exceed the bounds, and the
    recurrence runs.)"""
    uv, sky = small(mt, nrow=5, nchan=nchan, nif=nif, ncomp=ncomp, dnu=2.0e8 / (nchan * nif), seed=nchan + ncomp)
    if mt == U.MOD_POINT:
        assert _plan(uv, sky)["tensorChannels"] > 0
    assert _error(uv, sky) < TOL_REL


@pytest.mark.parametrize("mt", FAMILIES)
def test_separate_runs(mt):
    """IFs apart, and a descending frequency axis: a run per IF, negative increments."""
    uv, sky = small(mt, nrow=6, nchan=160, nif=3, ncomp=200, dnu=5e5)
    uv.freqArr = U.freq_axis(160, 3, 1.3e9, 5e5, 1.2e8)
    assert _plan(uv, sky)["tensorChannels"] > 0
    assert _error(uv, sky) < TOL_REL
    uv.freqArr = uv.freqArr[::-1].copy()
    assert _plan(uv, sky)["tensorChannels"] > 0
    assert _error(uv, sky) < TOL_REL


def test_mixed_model_and_wide_index_spread():
    """Points and Gaussians in one table, few components over a wide index range
    (the cross product), long baselines that taper Gaussians to nothing."""
    uv, sky = small(U.MOD_GAUSS_SPEC, nrow=40, nchan=256, nif=1, ncomp=333, gauss_frac=0.3, max_bl=1e6)
    assert _plan(uv, sky)["tensorChannels"] > 0
    assert _error(uv, sky) < TOL_REL


def test_flux_range():
    """Fluxes over twelve decades, zero and negative ones among them."""
    uv, sky = small(U.MOD_POINT, nrow=6, nchan=256, nif=1, ncomp=300)
    sky.comps[:, 0] = np.logspace(6, -6, 300) * np.where(np.arange(300) % 3 == 0, -1, 1)
    sky.comps[40:44, 0] = 0.0
    assert _plan(uv, sky)["tensorChannels"] > 0
    assert _error(uv, sky) < TOL_REL


@pytest.mark.parametrize("op", [OP_SUB, OP_DIV, OP_REPL])
def test_operations_and_selection(op):
    """Every operation with flags and an uneven channel selection: the selected
    data follow the oracle, the rest stays bit for bit."""
    uv, sky = small(U.MOD_POINT_SPEC, nrow=30, nchan=200, nif=2, nstok=4, ncomp=90, flag_frac=0.1)
    p = SkyModelParams(op=op, startChannel=11, numberChannel=150, startPoln=2, numberPoln=2, stokFactor=-1.0, doFlip=True)
    assert _plan(uv, sky, SkyModelParams(**{**p.__dict__, "nVisPIO": 1}))["tensorChannels"] > 0
    got, want = run_gpu(uv, sky, p), oracle.apply_fp64(uv, sky, p)
    a, b = got.vis_view(), want[:, uv.nrparm:].reshape(uv.vis_view().shape)
    m, l1 = oracle.model_fp64(uv, sky, p)
    scale = np.nanmax(l1) if op != OP_DIV else np.abs(b[..., :2]).max() / np.nanmin(np.abs(m)) * np.nanmax(l1)
    assert np.abs(a - b).max() < 2 * TOL_REL * max(scale, 1.0)
    keep = np.ones(a.shape, bool)
    keep[:, :, 10:160, 1:3] = False
    assert np.array_equal(a[keep], uv.vis_view()[keep])


def test_fp64_positions():
    uv, sky = small(U.MOD_POINT, nrow=8, nchan=256, nif=1, ncomp=150, max_bl=8e6, freq=22e9, radius_deg=0.3)
    gm = GPUSkyModel("lo")
    out = uv.copy()
    try:
        gm.DFTInit(sky, out, SkyModelParams(op=OP_REPL, nVisPIO=uv.nvis))
        gm.DFTSetMod(sky)
        gm.set_positions_fp64(sky.xyz)
        assert gm.plan_info()["tensorChannels"] > 0
        gm.DFTCalc(out)
    finally:
        gm.close()
    v = out.vis_view()[..., 0, :]
    uvw = uv.vis[:, :3].astype(np.float64)
    ph = (uvw @ sky.xyz.T)[:, None, :] * (uv.freqArr / uv.freq)[None, :, None]
    want = (sky.comps[:, 0].astype(np.float64) * np.exp(1j * ph)).sum(2).reshape(v.shape[:3])
    assert np.abs(v[..., 0] + 1j * v[..., 1] - want).max() < TOL_REL * np.abs(sky.comps[:, 0]).sum()


def test_what_it_leaves_to_the_recurrence():
    """Short runs, small models, growing tapers, several spectral terms, tables
    that are not finite and any asked-for kernel keep the recurrence kernels."""
    uv, sky = small(U.MOD_POINT, nrow=4, nchan=256, nif=1, ncomp=100)
    assert _plan(uv, sky)["tensorChannels"] == 256
    assert _plan(uv, sky, flavor=OBIT_DFT_RECUR, chan_per_thread=32)["tensorChannels"] == 0
    short, s2 = small(U.MOD_POINT, nrow=4, nchan=48, nif=1, ncomp=100)
    assert _plan(short, s2)["tensorChannels"] == 0
    few, s3 = small(U.MOD_POINT, nrow=4, nchan=256, nif=1, ncomp=20)
    assert _plan(few, s3)["tensorChannels"] == 0
    terms, s4 = small(U.MOD_POINT_SPEC, nrow=4, nchan=256, nif=1, ncomp=100, nterm=2)
    assert _plan(terms, s4)["tensorChannels"] == 0
    sky.comps[3, 1] = np.inf
    assert _plan(uv, sky)["tensorChannels"] == 0
    g, s5 = small(U.MOD_GAUSS, nrow=4, nchan=256, nif=1, ncomp=100)
    s5.comps[7, 4] = 1e-12
    assert _plan(g, s5)["tensorChannels"] == 0


def test_batch_facets_on_the_tensor_cores():
    """Facets that the tensor-core form takes (in branches of the batch's graph)
    beside ones it does not: each against the oracle, and the streamed run over
    host records bit for bit the same."""
    torch = pytest.importorskip("torch")
    from obit_b200.batch import DFTBatch, Facet

    cases, facets, keep = [], [], []
    for i, (mt, nrow, nchan, nif, ncomp) in enumerate([
            (U.MOD_POINT, 40, 256, 1, 200), (U.MOD_POINT, 7, 130, 3, 900), (U.MOD_POINT, 33, 32, 1, 60),
            (U.MOD_POINT_SPEC, 12, 128, 2, 75), (U.MOD_GAUSS_SPEC, 9, 512, 1, 120), (U.MOD_POINT, 64, 256, 2, 20)]):
        uv, sky = small(mt, nrow=nrow, nchan=nchan, nif=nif, ncomp=ncomp, dnu=1e8 / (nchan * nif), seed=60 + i)
        d, c = torch.from_numpy(uv.vis.copy()).cuda(), torch.from_numpy(sky.comps).cuda()
        keep.append((d, c))
        cases.append((uv, sky))
        facets.append(Facet(uv, sky, SkyModelParams(op=OP_SUB), d.data_ptr(), nrow, c.data_ptr()))
    b = DFTBatch(facets)
    try:
        host = [torch.from_numpy(uv.vis.copy()).pin_memory() for uv, _ in cases]
        b.run()
        b.check()
        b.run_host([h.data_ptr() for h in host], 1 << 20)
        b.check()
        for (uv, sky), (d, _), h in zip(cases, keep, host):
            got = d.cpu().numpy()
            assert np.array_equal(got, h.numpy())
            _, l1 = oracle.model_fp64(uv, sky)
            want = oracle.apply_fp64(uv, sky, SkyModelParams(op=OP_SUB))
            err = np.abs(got - want)[:, uv.nrparm:].reshape(uv.vis_view().shape)[..., :2, :2]
            assert (err / l1[..., None, None]).max() < TOL_REL
    finally:
        b.close()


@pytest.mark.parametrize("mt", [U.MOD_POINT_TSPEC, U.MOD_GAUSS_TSPEC])
@pytest.mark.parametrize("nchan, nif, nplanes, ncomp", [(256, 1, 4, 300), (512, 2, 16, 1100), (300, 1, 3, 64), (256, 4, 1, 99),
                                                        (1000, 1, 5, 48)])
def test_tabulated_spectra(mt, nchan, nif, nplanes, ncomp):
    """Coarse planes that fall on the grid's rows and ones that cut it, a zero
    flux and a negative one in a plane."""
    uv, sky = small(mt, nrow=6, nchan=nchan, nif=nif, ncomp=ncomp, dnu=1.5e8 / (nchan * nif), nplanes=nplanes,
                    seed=nchan + ncomp, gauss_frac=0.4)
    first = 5 if mt == U.MOD_POINT_TSPEC else 8
    sky.comps[3, first] = 0.0
    sky.comps[5, first:] *= -1.0
    if mt == U.MOD_POINT_TSPEC and nplanes != 3 and nplanes != 5:
        assert _plan(uv, sky)["tensorChannels"] > 0
    assert _error(uv, sky) < TOL_REL
