"""The work that programs have this framework do, as cases to be timed: model
subtraction, division and prediction by the DFT on device-resident records
(every model family, one field at a time and as a multi-facet batch), the
beam-corrected DFT and the Jones tables it reads, the gridded model and its
per-field set-up, and the call on host records.  Records, component tables and
beams are synthetic, drawn from a seed, with the geometry of real arrays.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from obit_b200 import uvdata as U
from obit_b200.batch import DFTBatch, Facet
from obit_b200.beam import Beam, BeamImages, baseline_codes, jones_from_images
from obit_b200.comps import CCField, CCModel
from obit_b200.grid import GridField, GridImage
from obit_b200.skymodel import OP_DIV, OP_REPL, OP_SUB, GPUSkyModel, SkyModelParams

OPS = {"sub": OP_SUB, "div": OP_DIV, "repl": OP_REPL}
MODELS = {"point": U.MOD_POINT, "pointspec": U.MOD_POINT_SPEC, "pointtspec": U.MOD_POINT_TSPEC,
          "gauss": U.MOD_GAUSS, "gaussspec": U.MOD_GAUSS_SPEC, "gausstspec": U.MOD_GAUSS_TSPEC}
MAX_EVALS = 4.0e11  # component-visibility evaluations of the largest listed case

# Fields every DFT case has; a case states what differs.
DFT = {"kind": "dft", "rows": 20160, "nant": 64, "max_bl_m": 36e3, "freq": 1.4e9, "dnu": 1e6, "nchan": 256,
       "nif": 4, "if_gap": 0.0, "nstok": 4, "model": "point", "ncomp": 20000, "nplanes": 0, "gauss_frac": 1.0,
       "radius_deg": 1.0, "offset_deg": 0.0, "op": "sub", "flag_frac": 0.0, "fp64_positions": False}


def listed():
    return [
        # self-calibration of a compact calibrator: a few components divided into
        # continuum data of two wide channels; the shortest calls there are
        {**DFT, "name": "calibrator", "rows": 15949, "nant": 27, "freq": 1.465e9, "dnu": 50e6, "nchan": 1, "nif": 2,
         "ncomp": 13, "radius_deg": 0.05, "op": "div"},
        # a whole continuum track of a small array, a modest CLEAN model
        {**DFT, "name": "small_track", "rows": 42120, "nant": 27, "nchan": 64, "nif": 1, "nstok": 2, "ncomp": 1000,
         "radius_deg": 0.5},
        # a chunk of a wide-band survey field: points with a spectral index
        {**DFT, "name": "survey_chunk", "rows": 19600, "model": "pointspec", "flag_frac": 0.02},
        # the same coverage with a multi-scale model: 70 % points, 30 % Gaussians
        {**DFT, "name": "multiscale_chunk", "rows": 8064, "model": "gaussspec", "ncomp": 49000, "gauss_frac": 0.3},
        # VLBI at 22 GHz: phases of 1e7 radians, a field off the phase centre
        {**DFT, "name": "vlbi", "rows": 23808, "nant": 32, "max_bl_m": 8.0e6, "freq": 22e9, "dnu": 2e6, "nchan": 64,
         "nif": 8, "nstok": 2, "ncomp": 10000, "radius_deg": 2.0 / 60.0, "offset_deg": 0.3},
        # wide-band imaging: fluxes tabulated per coarse plane, data predicted
        {**DFT, "name": "wideband_planes", "rows": 10080, "model": "pointtspec", "ncomp": 4999, "nplanes": 16,
         "op": "repl"},
        # a mosaic's uneven facets in one launch
        {"kind": "batch", "name": "mosaic", "nfacet": 96, "row_scale": 0.0002},
        # primary-beam-corrected model, four correlations, two antenna types
        {"kind": "beam", "name": "beam_corrected", "rows": 8064, "nchan": 256, "nif": 4, "model": "pointspec",
         "ncomp": 4000, "ntype": 2, "njones": 3},
        # the Jones table of that model, interpolated from beam images each parallactic angle
        {"kind": "jones", "name": "beam_images", "ncomp": 4000, "ntype": 2, "nplane": 8, "npix": 61, "hwidth": 2},
        # a dense model through the gridded path: many records on a ready field
        {"kind": "grid", "name": "gridded_apply", "rows": 20160, "npix": 4096, "ncomp": 20000, "nchan": 256, "nif": 4,
         "setup": False},
        # one field of a major cycle: grid its components, transform, apply to a buffer
        {"kind": "grid", "name": "gridded_field", "rows": 2016, "npix": 2048, "ncomp": 50000, "nchan": 64, "nif": 4,
         "setup": True},
        # the reference's calling sequence: a new model, then a buffer of host records
        {**DFT, "kind": "host", "name": "host_buffer", "rows": 10000, "nant": 27, "nchan": 64, "nif": 2, "nstok": 2,
         "ncomp": 1000, "radius_deg": 0.5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dft"] * 6 + ["batch", "beam", "jones", "grid", "grid", "host"])
    if kind in ("dft", "host"):
        c = dict(DFT, kind=kind)
        c["nant"] = rng.randint(12, 64)
        c["max_bl_m"] = math.exp(rng.uniform(math.log(3e3), math.log(1e5)))
        c["freq"] = math.exp(rng.uniform(math.log(0.7e9), math.log(9e9)))
        vlbi = rng.random() < 0.15
        if vlbi:
            c.update(nant=rng.randint(8, 32), max_bl_m=8.0e6, freq=22e9, offset_deg=0.3, radius_deg=2.0 / 60.0)
        else:
            c["radius_deg"] = rng.uniform(0.05, 1.0)
        c["nchan"] = _log_int(rng, 1, 512)
        c["nif"] = rng.randint(1, 8)
        band = min(c["freq"] * 0.5, rng.choice([32e6, 128e6, 512e6, 1e9]))  # whole bandwidth
        c["dnu"] = band / (c["nchan"] * c["nif"])
        c["if_gap"] = rng.choice([0.0, 0.0, 0.25])  # of an IF's width, between IFs
        c["nstok"] = rng.choice([1, 2, 4])
        c["model"] = rng.choice(sorted(MODELS))
        c["gauss_frac"] = rng.choice([0.3, 1.0])
        if c["model"].endswith("tspec"):
            c["nplanes"] = rng.randint(2, 16)
        c["op"] = rng.choice(["sub", "sub", "div", "repl"])
        c["flag_frac"] = rng.choice([0.0, 0.05])
        c["fp64_positions"] = kind == "dft" and rng.random() < (0.5 if vlbi else 0.15)
        c["ncomp"] = _log_int(rng, 10, 2000 if kind == "host" else 50000)
        rows = _log_int(rng, 351, 10000 if kind == "host" else 40000)
        most = MAX_EVALS / (0.5 if c["model"].startswith("gauss") else 0.25) * 0.2
        width = c["nchan"] * c["nif"]
        c["rows"] = max(1, int(min(rows, most / (c["ncomp"] * width), 2.4e8 / (3 * c["nstok"] * width))))
        return c
    if kind == "batch":
        return {"kind": "batch", "nfacet": rng.randint(8, 96), "row_scale": rng.uniform(2e-5, 2e-4)}
    if kind == "beam":
        nchan, nif = _log_int(rng, 16, 300), rng.randint(1, 4)
        ncomp = _log_int(rng, 50, 5000)
        rows = int(min(_log_int(rng, 351, 20000), 3e10 / (ncomp * nchan * nif)))
        return {"kind": "beam", "rows": max(8, rows), "nchan": nchan, "nif": nif,
                "model": rng.choice(["point", "pointspec", "gaussspec"]), "ncomp": ncomp, "ntype": rng.randint(1, 3),
                "njones": rng.randint(1, 6)}
    if kind == "jones":
        return {"kind": "jones", "ncomp": _log_int(rng, 50, 50000), "ntype": rng.randint(1, 3),
                "nplane": rng.randint(1, 16), "npix": rng.randint(41, 201), "hwidth": rng.randint(1, 4)}
    nchan, nif = _log_int(rng, 8, 300), rng.randint(1, 4)
    return {"kind": "grid", "rows": max(64, int(min(_log_int(rng, 351, 20160), 2e7 / (nchan * nif)))),
            "npix": rng.choice([512, 768, 1024, 2000, 2048, 3000, 4096]), "ncomp": _log_int(rng, 100, 200000),
            "nchan": nchan, "nif": nif, "setup": rng.random() < 0.6}


# ---- inputs --------------------------------------------------------------------


def _uvw(rows, nant, max_bl_m, freq, seed):
    """rows of a time-major track, the integrations spread over eight hours."""
    pos = U.array_layout(nant, max_bl_m, np.random.default_rng(seed))
    nint = -(-rows // (nant * (nant - 1) // 2))
    return U.make_uvw(pos, nint, 45.0, 4.0, 34.0, freq)[:rows].astype(np.float32)


def _records(uvw, nstok, width, seed, flag_frac=0.0):
    """Noise visibilities of unit weight on the GPU, a share of them flagged."""
    rows, ncorr = len(uvw), nstok * width
    g = torch.Generator(device="cuda").manual_seed(seed)
    vis = torch.empty((rows, 5 + 3 * ncorr), dtype=torch.float32, device="cuda")
    c = vis[:, 5:].view(rows, ncorr, 3)
    c[:, :, :2] = 0.01 * torch.randn((rows, ncorr, 2), generator=g, device="cuda")
    c[:, :, 2] = 1.0
    if flag_frac > 0:
        c[:, :, 2][torch.rand((rows, ncorr), generator=g, device="cuda") < flag_frac] = -1.0
    vis[:, 0:3] = torch.from_numpy(uvw).cuda()
    vis[:, 3] = 256.0
    vis[:, 4] = 0.0
    return vis


def _freqs(c):
    width = c["nchan"] * c["dnu"]
    step = width * (1.0 + c.get("if_gap", 0.0))
    return U.freq_axis(c["nchan"], c["nif"], c["freq"] - 0.5 * (c["nif"] * step), c["dnu"], step)


def _sky(c, fa, seed):
    kw = {}
    if c["model"].endswith("tspec"):
        edges = np.linspace(fa.min(), fa.max() + 1.0, c["nplanes"] + 1)
        kw = {"spec_freq": 0.5 * (edges[:-1] + edges[1:]),
              "spec_index": np.clip(np.searchsorted(edges, fa, side="right") - 1, 0, c["nplanes"] - 1)}
    o = c["offset_deg"] * U.DG2RAD / math.sqrt(2.0)
    return U.make_comps(MODELS[c["model"]], c["ncomp"], np.random.default_rng(seed), radius_deg=c["radius_deg"],
                        center=(o, o), gauss_frac=c["gauss_frac"], ref_freq=c["freq"], **kw)


def _dft_inputs(case, seed):
    fa = _freqs(case)
    uvw = _uvw(case["rows"], case["nant"], case["max_bl_m"], case["freq"], seed)
    vis = _records(uvw, case["nstok"], case["nchan"] * case["nif"], seed, case["flag_frac"])
    return fa, vis, _sky(case, fa, seed + 1)


def _layout(case, fa, nstok, vis):
    """The record layout with no records of its own."""
    return U.UVData(np.zeros((1, vis.shape[1]), np.float32), nstok, case["nchan"], case["nif"], case["freq"], fa)


def _beam_inputs(case, seed):
    c = dict(DFT, **{k: case[k] for k in ("rows", "nchan", "nif", "model", "ncomp")})
    c["dnu"] = 1e6 * 256 / case["nchan"]
    fa = _freqs(c)
    uvw = _uvw(c["rows"], 64, 36e3, c["freq"], seed)
    vis = _records(uvw, 4, c["nchan"] * c["nif"], seed)
    vis[:, 3] = torch.from_numpy(baseline_codes(64, c["rows"])).cuda()
    sky = _sky(c, fa, seed + 1)
    r = np.random.default_rng(seed + 2)
    jones = np.zeros((case["ntype"], sky.ncomp, case["njones"], 8), np.float32)
    jones[..., 0] = jones[..., 6] = 1.0
    jones += (0.1 * r.standard_normal(jones.shape)).astype(np.float32)
    width = c["nchan"] * c["nif"]
    beam = Beam(np.arange(64) % case["ntype"], (np.arange(width) * case["njones"] // width).astype(np.int32), jones)
    return c, fa, vis, sky, beam


def _jones_inputs(case, seed):
    """Smooth beams near one, tapering outwards, small cross terms; positions
    over the central part of the image."""
    n, r = case["npix"], np.random.default_rng(seed)
    y, x = (np.mgrid[0:n, 0:n] - n // 2) / (n // 2)
    px = np.empty((case["ntype"], 8, case["nplane"], n, n), np.float32)
    for t in range(case["ntype"]):
        for k in range(case["nplane"]):
            for q in range(8):
                a, b, c = r.uniform(-1, 1, 3)
                base = 0.95 * np.exp(-0.3 * (x * x + y * y)) if q in (0, 2) else 0.05
                px[t, q, k] = base + 0.02 * (a * x + b * y + c * x * y)
    half = 1.5
    im = BeamImages(px, np.linspace(1.2e9, 1.6e9, case["nplane"]), crpix=(n // 2 + 1, n // 2 + 1),
                    cdelt=(half / (n // 2), half / (n // 2)), hwidth=case["hwidth"], refSizeFact=3.0e-10)
    pos = r.uniform(-0.9, 0.9, (case["ncomp"], 2)).astype(np.float32)
    return im, pos, 0.37


def _grid_inputs(case, seed):
    """CLEAN components on cells of the central half of the image, the pixels
    sized so that the plane reaches past the longest baseline."""
    n, r = case["npix"], np.random.default_rng(seed)
    cell = 0.25 / 3600.0
    ix, iy = r.integers(-n // 4, n // 4, (2, case["ncomp"]))
    flux = np.exp(r.uniform(math.log(1e-3), 0.0, case["ncomp"])).astype(np.float32)
    field = CCField(flux=flux, deltaX=(ix * -cell).astype(np.float32), deltaY=(iy * cell).astype(np.float32),
                    crvalRA=0.0, crvalDec=34.0, do3D=False, cdeltX=-cell, cdeltY=cell)
    c = dict(DFT, nchan=case["nchan"], nif=case["nif"], dnu=256e6 / case["nchan"])
    fa = _freqs(c)
    vis = _records(_uvw(case["rows"], 64, 36e3, 1.4e9, seed), 4, case["nchan"] * case["nif"], seed)
    return c, fa, vis, field, GridImage(n, n, n / 2 + 1, n / 2 + 1), CCModel(uvRA=0.0, uvDec=34.0)


def _batch_inputs(case, seed):
    """Facets of uneven rows, components, IFs and channels about 1 GHz."""
    rng = np.random.default_rng(seed)
    pos = U.array_layout(64, 36e3, rng)
    track = U.make_uvw(pos, 40, 45.0, 4.0, 34.0, 1.4e9).astype(np.float32)
    out = []
    # the sizes of the facets are the workload's own; what they hold is the seed's
    for k, (nr, nc, nif, nch) in enumerate(U.config5_facets(case["nfacet"], row_scale=case["row_scale"])):
        fa = U.freq_axis(nch, nif, 1.0e9, 128e6 / nch)
        uvw = track[rng.integers(0, len(track), nr)]
        vis = _records(uvw, 2, nch * nif, seed + k)
        centre = rng.uniform(-1.0, 1.0, 2) * U.DG2RAD
        sky = U.make_comps(U.MOD_POINT, nc, np.random.default_rng([seed, k]), radius_deg=0.5, center=centre)
        out.append((fa, vis, sky, nch, nif))
    return out


# ---- the cases --------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dft":
        fa, vis, sky = _dft_inputs(case, seed)
        gm = GPUSkyModel(case["kind"])
        gm.DFTInit(sky, _layout(case, fa, case["nstok"], vis), SkyModelParams(op=OPS[case["op"]], nVisPIO=1))
        gm.DFTSetMod(sky)
        if case["fp64_positions"]:
            gm.set_positions_fp64(sky.xyz)
        return {"kind": kind, "gm": gm, "vis": vis}
    if kind == "host":
        fa, vis, sky = _dft_inputs(case, seed)
        uv = U.UVData(vis.cpu().numpy(), case["nstok"], case["nchan"], case["nif"], case["freq"], fa)
        gm = GPUSkyModel(case["kind"])
        gm.DFTInit(sky, uv, SkyModelParams(op=OPS[case["op"]]))
        return {"kind": kind, "gm": gm, "uv": uv, "sky": sky}
    if kind == "batch":
        inputs = _batch_inputs(case, seed)
        facets, keep = [], []
        for fa, vis, sky, nch, nif in inputs:
            comps = torch.from_numpy(sky.comps).cuda()
            uv = U.UVData(np.zeros((1, vis.shape[1]), np.float32), 2, nch, nif, float(fa[0]), fa)
            facets.append(Facet(uv, sky, SkyModelParams(), vis.data_ptr(), vis.shape[0], comps.data_ptr()))
            keep.append((vis, comps))
        return {"kind": kind, "batch": DFTBatch(facets), "keep": keep}
    if kind == "beam":
        c, fa, vis, sky, beam = _beam_inputs(case, seed)
        d_jones = torch.from_numpy(beam.jones).cuda()
        gm = GPUSkyModel(kind)
        gm.DFTInit(sky, _layout(c, fa, 4, vis), SkyModelParams(nVisPIO=1))
        gm.set_beam(beam, d_jones.data_ptr())
        gm.DFTSetMod(sky)
        return {"kind": kind, "gm": gm, "vis": vis, "jones": d_jones, "beam": beam}
    if kind == "jones":
        im, pos, angle = _jones_inputs(case, seed)
        return {"kind": kind, "images": im, "pixels": torch.from_numpy(im.pixels).cuda(),
                "pos": torch.from_numpy(pos).cuda(), "angle": angle,
                "jones": torch.empty((case["ntype"], case["ncomp"], case["nplane"], 8), device="cuda")}
    c, fa, vis, field, image, model = _grid_inputs(case, seed)
    uv = _layout(c, fa, 4, vis)
    state = {"kind": kind, "uv": uv, "vis": vis, "setup": (field, image, model) if case["setup"] else None,
             "fscale": torch.from_numpy(np.ascontiguousarray(uv.fscale)).cuda()}
    if not case["setup"]:
        state["grid"] = GridField(field, image, model)
    return state


def _split(vis):
    return {"params": vis[:, :5], "corr": vis[:, 5:]}


def run(state):
    kind = state["kind"]
    if kind in ("dft", "beam"):
        state["gm"].calc_device(state["vis"].data_ptr(), state["vis"].shape[0])
        return _split(state["vis"])
    if kind == "host":
        state["gm"].DFTSetMod(state["sky"])
        state["gm"].DFTCalc(state["uv"])
        return _split(state["uv"].vis)
    if kind == "batch":
        state["batch"].run()
        return [v[:, 5:] for v, _ in state["keep"]][:64]
    if kind == "jones":
        jones_from_images(state["images"], state["pixels"].data_ptr(), state["pos"].data_ptr(),
                          state["pos"].shape[0], state["angle"], state["jones"].data_ptr())
        return state["jones"]
    grid = state.get("grid") or GridField(*state["setup"])
    grid.FTGrid_device(state["uv"], state["vis"].data_ptr(), state["vis"].shape[0],
                       d_fscale=state["fscale"].data_ptr())
    if state["setup"]:
        grid.close()
    return _split(state["vis"])


def work(case):
    """Complex rotate (6) and accumulate (4) per component and model
    visibility; a record's u, v, w and the selected correlations read and
    written once; component tables and images read once."""
    kind = case["kind"]
    width = case["nchan"] * case["nif"] if "nchan" in case else 0
    if kind in ("dft", "host"):
        npol = min(2, case["nstok"])
        rec = 12 + width * npol * (12 + (12 if case["op"] == "div" else 8))
        return {"bytes": case["rows"] * rec + case["ncomp"] * 4 * (8 + case["nplanes"]),
                "flops": 10.0 * case["rows"] * width * case["ncomp"]}
    if kind == "batch":
        draws = U.config5_facets(case["nfacet"], row_scale=case["row_scale"])
        return {"bytes": sum(r * (12 + 2 * 20 * i * n) + 16 * c for r, c, i, n in draws),
                "flops": 10.0 * sum(float(r) * c * i * n for r, c, i, n in draws)}
    if kind == "beam":
        return {"bytes": case["rows"] * (16 + width * 4 * 20) +
                case["ncomp"] * (32 + 32 * case["ntype"] * case["njones"]),
                "flops": (6.0 + 8.0 * 4) * case["rows"] * width * case["ncomp"]}
    if kind == "jones":
        out, taps = case["ntype"] * case["nplane"] * 8, (2 * case["hwidth"] + 1) ** 2
        return {"bytes": 4 * out * (case["npix"] ** 2 + case["ncomp"]) + 8 * case["ncomp"],
                "flops": 2.0 * out * taps * case["ncomp"]}
    n2 = 2 * case["npix"]
    flops = 2.0 * 25 * 26 * 2 * case["rows"] * width
    nbytes = case["rows"] * (12 + width * 2 * 20) + 4 * n2 * n2
    if case["setup"]:
        flops += 2.5 * n2 * n2 * 2 * math.log2(n2)
        nbytes += 12 * case["ncomp"]
    return {"bytes": nbytes, "flops": flops}


# ---- the same in 64 bits ---------------------------------------------------------


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", torch.float64)


def _phasors(uvw, xyz, f):
    return torch.polar(torch.ones((), dtype=torch.float64, device="cuda"), (uvw @ xyz.T) * f)


def _model64(uvw, sky, xyz, fa, freq, nchan, nif, coef=None):
    """Model of the rows uvw (float64): complex (rows, nif * nchan), or with
    coef(channel) -> (ncomp, k) complex factors (rows, nif * nchan, k)."""
    t = _dev(sky.comps)
    gauss, spec, tspec = sky.modType % 10 == 1, sky.modType // 10 == 1, sky.is_tspec
    f64 = fa / freq
    taper = None
    if gauss:
        q = torch.stack([uvw[:, 0] ** 2, uvw[:, 1] ** 2, uvw[:, 0] * uvw[:, 1]], 1) @ t[:, 4:7].T
        taper = None if not bool((q != 0).any()) else q
    a_at = 7 if gauss else 4
    out = []
    for i in range(nif):
        ks = range(i * nchan, (i + 1) * nchan)
        z = _phasors(uvw, xyz, f64[ks[0]])
        s = _phasors(uvw, xyz, f64[ks[0] + 1] - f64[ks[0]]) if nchan > 1 else None
        for k in ks:
            if k > ks[0]:
                z *= s
            if tspec:
                p = int(sky.specIndex[k])
                amp = t[:, a_at + 1 + p] * torch.exp(t[:, a_at] * math.log(fa[k] / sky.specFreq[p]))
            elif spec:
                amp = t[:, 0] * torch.exp(t[:, a_at] * math.log(fa[k] / sky.refFreq))
            else:
                amp = t[:, 0]
            zk = z if taper is None else z * torch.exp(taper * f64[k] ** 2)
            if coef is None:
                out.append(torch.mv(zk, amp.to(torch.complex128)))
            else:
                out.append(zk @ (coef(k) * amp[:, None]))
    return torch.stack(out, 1)


def _sky_model64(uvw, sky, fp64_positions, fa, freq, nchan, nif):
    xyz = _dev(sky.xyz if fp64_positions else sky.comps[:, 1:4])
    parts = [np.arange(sky.ncomp)]
    if sky.modType % 10 == 1:  # the untapered components need no exponential per row
        point = ~sky.comps[:, 4:7].any(axis=1)
        parts = [p for p in (np.nonzero(point)[0], np.nonzero(~point)[0]) if len(p)]
    rows = max(1, min(len(uvw), int(2.0e7 / sky.ncomp)))
    chunks = []
    for r in range(0, len(uvw), rows):
        total = 0
        for p in parts:
            sub = U.SkyComps(sky.modType, sky.comps[p], sky.nterm, sky.refFreq, sky.specFreq, sky.specIndex)
            total = total + _model64(uvw[r:r + rows], sub, xyz[p], fa, freq, nchan, nif)
        chunks.append(total)
    return torch.cat(chunks)


def _apply64(vis, model, nstok, op):
    """model (rows, channels, polarizations) applied to the first of them."""
    out = vis.to(torch.float64)
    c = out[:, 5:].view(out.shape[0], -1, nstok, 3)[:, :, :model.shape[2]]
    v = torch.complex(c[..., 0].clone(), c[..., 1].clone())
    good = c[..., 2] > 0
    if op == "repl":
        v = model
    elif op == "sub":
        v = torch.where(good, v - model, v)
    else:
        v = torch.where(good, v / model, v)
        c[..., 2] = torch.where(good, c[..., 2] * model.abs(), c[..., 2])
    c[..., 0], c[..., 1] = v.real, v.imag
    return out


def _exact_jones(case, seed):
    im, pos, angle = _jones_inputs(case, seed)
    iw, hw, n = 2 * case["hwidth"] + 1, case["hwidth"], case["npix"]
    p = _dev(pos)
    ca, sa = math.cos(angle), math.sin(angle)
    off = torch.stack([p[:, 0] * ca + p[:, 1] * sa, p[:, 1] * ca - p[:, 0] * sa], 1)
    pix = off / torch.tensor(im.cdelt, dtype=torch.float64, device="cuda") + n // 2 + 1
    first = (torch.clamp(torch.floor(pix + 0.5).long() - hw, 1, n - iw + 1) - 1)
    x = pix - first
    w = torch.ones((len(pos), 2, iw), dtype=torch.float64, device="cuda")
    for j in range(iw):
        for i in range(iw):
            if i != j:
                w[:, :, j] *= (x - (i + 1)) / (j - i)
    px = _dev(im.pixels)
    out = []
    gain_at = torch.linalg.norm(p, dim=1)[:, None] * _dev(im.planeFreq.astype(np.float32)) * im.refSizeFact
    gain = (1.0 - 4.0 * gain_at ** 2) / torch.cos(math.pi * gain_at)
    for t in range(case["ntype"]):
        v = torch.zeros((len(pos), case["nplane"], 8), dtype=torch.float64, device="cuda")
        for j in range(iw):
            for i in range(iw):
                tap = px[t][:, :, first[:, 1] + j, first[:, 0] + i]  # (8, plane, comp)
                v += tap.permute(2, 1, 0) * (w[:, 0, i] * w[:, 1, j])[:, None, None]
        v = (v * gain[..., None])[..., [0, 1, 4, 5, 6, 7, 2, 3]]
        unit = torch.tensor([1.0, 0, 0, 0, 0, 0, 1, 0], dtype=torch.float64, device="cuda")
        off_limit = (gain >= 10.0) | (v[..., 0].abs() > 1.3) | (v[..., 6].abs() > 1.3)
        out.append(torch.where(off_limit[..., None], unit, v))
    return torch.stack(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "grid":  # the reference's single-precision choice of windows and table rows has no 64-bit value
        return None
    if kind == "jones":
        return _exact_jones(case, seed)
    if kind == "batch":
        out = []
        for fa, vis, sky, nch, nif in _batch_inputs(case, seed)[:64]:
            m = _sky_model64(vis[:, :3].double(), sky, False, fa, float(fa[0]), nch, nif)
            out.append(_apply64(vis, m[:, :, None].expand(-1, -1, 2), 2, "sub")[:, 5:])
        return out
    if kind == "beam":
        c, fa, vis, sky, beam = _beam_inputs(case, seed)
        j = torch.view_as_complex(_dev(beam.jones).view(case["ntype"], sky.ncomp, case["njones"], 4, 2).contiguous())
        code = vis[:, 3].double()
        a1 = torch.floor(code / 256.0)
        t1, t2 = ((a - 1).long() % case["ntype"] for a in (a1, code - 256.0 * a1))
        model = torch.zeros((c["rows"], c["nchan"] * c["nif"], 4), dtype=torch.complex128, device="cuda")
        xyz = _dev(sky.comps[:, 1:4])
        for p in range(case["ntype"]):
            for q in range(case["ntype"]):
                def coef(k):
                    x, y = j[p, :, beam.jchan[k]], j[q, :, beam.jchan[k]].conj()
                    xx, xy = x[:, 0] * y[:, 0] + x[:, 1] * y[:, 1], x[:, 1] * y[:, 3] + x[:, 0] * y[:, 2]
                    yx, yy = x[:, 2] * y[:, 0] + x[:, 3] * y[:, 1], x[:, 2] * y[:, 2] + x[:, 3] * y[:, 3]
                    return torch.stack([xx, yy, xy, yx], 1)
                rows = torch.nonzero((t1 == p) & (t2 == q))[:, 0]
                for r in rows.split(max(1, int(2.0e7 / sky.ncomp))):
                    model[r] = _model64(vis[r, :3].double(), sky, xyz, fa, c["freq"], c["nchan"], c["nif"], coef)
        return _split(_apply64(vis, model, 4, "sub"))
    fa, vis, sky = _dft_inputs(case, seed)
    m = _sky_model64(vis[:, :3].double(), sky, case["fp64_positions"], fa, case["freq"], case["nchan"], case["nif"])
    return _split(_apply64(vis, m[:, :, None].expand(-1, -1, min(2, case["nstok"])), case["nstok"], case["op"]))
