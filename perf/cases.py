"""The workloads this library is measured on: GPP sigma reductions as a GW code
makes them, through the public entry points.

A case is one call (or the reference program's call sequence) on one problem:

* kind "sigma":  gppsigma.ops.sigma, the whole problem from device arrays;
* kind "dropin": d_till_nvband + d_noFlagOCCSolver, the call sequence of the
  reference's CUDA driver, accumulating into zeroed outputs, one row of
  frequencies for every band;
* kind "kernel": gppKernelGPU, every band unoccupied, with an index remap;
* kind "batch":  a gpp_batch plan over several uneven states, one run;
* kind "host":   HostContext.sigma from pinned host arrays, copies included.

Sizes: the reference mini-app's own argument lists (512 bands, 2 of them
occupied, ncouls 800 to 32768, ngpown = ncouls / 20, 3 frequencies), the
32-frequency sweep and the batched states at part of their size, and odd sizes
between.  Values: uniform coefficients, wtilde in a plasmon band
(re 0.5..2, im -0.05..0.05), band energies over 20 Ry, optionally a share of
wtilde placed next to a band's frequency (near the plasmon pole).
"""
from __future__ import annotations

import ctypes as C
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "doe-csfg-hackathon_gb300"))

from gppsigma import capi, ops  # noqa: E402

TO1 = 1e-6


def _case(name, kind, precision, bands, occupied, ncouls, ngpown, nw, **more):
    c = {"kind": kind, "precision": precision, "bands": bands, "occupied": occupied,
         "ncouls": ncouls, "ngpown": ngpown, "nw": nw, "dw": 1.0, "per_band_wx": True,
         "near_pole": 0.0, "per_band_out": False, "static_out": False,
         "semantics": "complex_seq", "states": 1}
    c.update(more)
    if name:
        c = {"name": name, **c}
    return c


def listed():
    return [
        # The smallest call: a test system, latency and launches count.
        _case("sigma_fp64_tiny", "sigma", "fp64", 16, 2, 256, 24, 3, static_out=True),
        # The reference README's smallest job through the drop-in calls.
        _case("dropin_fp64_small_job", "dropin", "fp64", 512, 2, 800, 40, 3, per_band_wx=False),
        # A small full calculation: every output, FP64.
        _case("sigma_fp64_all_outputs", "sigma", "fp64", 512, 2, 2048, 128, 3,
              per_band_out=True, static_out=True),
        # A medium FP64 state with its own frequencies per band.
        _case("sigma_fp64_medium", "sigma", "fp64", 512, 2, 8192, 409, 3),
        # The production job of the reference's CUDA driver, FP64 and mixed.
        _case("dropin_fp64_production", "dropin", "fp64", 512, 2, 32768, 1638, 3,
              per_band_wx=False),
        _case("dropin_mixed_production", "dropin", "mixed", 512, 2, 32768, 1638, 3,
              per_band_wx=False),
        # The same sizes in one call, one frequency row, sums only.
        _case("sigma_fp64_one_wx_row", "sigma", "fp64", 512, 2, 32768, 1638, 3,
              per_band_wx=False),
        # Odd sizes, five frequencies, more occupied bands, the other semantics.
        _case("sigma_mixed_one_wx_row_odd", "sigma", "mixed", 403, 5, 12347, 617, 5,
              per_band_wx=False, semantics="kerseq", per_band_out=True),
        # The largest: the production state, per-band frequencies, 1% of wtilde
        # near a pole, mixed precision (the library's headline).
        _case("sigma_mixed_production", "sigma", "mixed", 512, 2, 32768, 1638, 3,
              near_pole=0.01),
        # A frequency sweep: 32 frequencies, 8 occupied bands.
        _case("sigma_mixed_sweep", "sigma", "mixed", 128, 8, 16384, 819, 32, dw=0.25,
              per_band_out=True),
        # Uneven quasiparticle states in one batch.
        _case("batch_mixed", "batch", "mixed", 256, 4, 8192, 409, 3, states=6),
        # End to end from pinned host memory.
        _case("host_mixed", "host", "mixed", 256, 4, 16384, 819, 3),
    ]


def _seconds(c):
    """A rough cost, to keep drawn cases below the largest listed one."""
    cells = c["ngpown"] * c["ncouls"] * c["states"]
    occ = cells * c["occupied"] * c["nw"]
    un = cells * (c["bands"] - (0 if c["kind"] == "kernel" else c["occupied"]))
    fp64 = c["precision"] == "fp64"
    if c["per_band_wx"]:
        s = un * c["nw"] / (5.0e10 if fp64 else 3.8e11)
    else:
        s = un / 4e12 + cells * c["nw"] / 4e10
    return s + occ / (2e10 if fp64 else 1e11)


def draw(rng):
    def logint(lo, hi):
        return min(hi, int(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["sigma", "sigma", "sigma", "dropin", "dropin", "kernel", "batch", "host"])
    precision = rng.choice(["fp64", "mixed"])
    per_band = kind in ("batch", "host") or (kind == "sigma" and rng.random() < 0.5)
    nw = 3 if kind == "dropin" else rng.choice([1, 2, 3, 3, 3, 4, 5, 8, 13, 32])
    bands = logint(16, 900)
    # A kernel call has no occupied bands; the others 0 to 8.
    occupied = 0 if kind == "kernel" else rng.choice([0, 1, 2, 2, 3, 4, 8])
    if kind == "dropin":
        occupied = max(1, occupied)
    ncouls = logint(256, 32768)
    ngpown = max(1, min(ncouls, logint(max(1, ncouls // 40), max(2, ncouls // 10))))
    near_pole = rng.choice([0.0, 0.0, 0.01])
    c = _case(None, kind, precision, bands, occupied, ncouls, ngpown, nw,
              dw=rng.choice([1.0, 0.25]), per_band_wx=per_band, near_pole=near_pole,
              per_band_out=kind != "kernel" and nw >= 3 and rng.random() < 0.5,
              static_out=kind in ("sigma", "host") and rng.random() < 0.3,
              semantics=rng.choice(["complex_seq", "complex_seq", "kerseq"])
              if kind in ("sigma", "batch", "host") else "complex_seq",
              states=rng.choice([2, 3, 5, 8]) if kind == "batch" else 1)
    while _seconds(c) > 0.2 and c["ngpown"] > 1:
        c["ngpown"] = max(1, int(c["ngpown"] * 0.7))
    while _seconds(c) > 0.2 and c["bands"] > 16:
        c["bands"] = max(16, int(c["bands"] * 0.7))
    return c


# ---------------------------------------------------------------------------
# Inputs.

def _state_case(c, k):
    """State k of a batch: uneven sizes around the case's own."""
    if c["kind"] != "batch":
        return c
    f = 1.0 - 0.09 * k
    s = dict(c)
    s["bands"] = max(c["occupied"], int(c["bands"] * (1.0 - 0.06 * ((3 * k) % 8))))
    s["ncouls"] = max(16, int(c["ncouls"] * f))
    s["ngpown"] = max(1, int(c["ngpown"] * f))
    return s


def _inputs(c, seed):
    nb, nc, ng, nw = c["bands"], c["ncouls"], c["ngpown"], c["nw"]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def u(shape, lo, hi):
        return torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen) * (hi - lo) + lo

    def z(rows, cols, re, im):
        out = torch.empty((rows, cols), dtype=torch.complex128, device="cuda")
        v = torch.view_as_real(out)
        v[..., 0] = u((rows, cols), *re)
        v[..., 1] = u((rows, cols), *im)
        return out

    t = {"aqsm": z(nb, nc, (-0.5, 0.5), (-0.5, 0.5)), "aqsn": z(nb, nc, (-0.5, 0.5), (-0.5, 0.5)),
         "ieps": z(ng, nc, (-0.5, 0.5), (-0.5, 0.5)), "wt": z(ng, nc, (0.5, 2.0), (-0.05, 0.05)),
         "vcoul": u((nc,), 0.1, 1.0)}
    igp = torch.sort(torch.randperm(nc, device="cuda", generator=gen)[:ng]).values
    if ng > 2:
        igp[-1] = nc + 3  # past ncouls: clamped to the last column
    t["igp"] = igp.to(torch.int32)
    t["indinv"] = None
    if c["kind"] == "kernel":
        t["indinv"] = torch.randperm(nc, device="cuda", generator=gen).to(torch.int32)
    # Band energies over 20 Ry, every frequency row 10 + dw (iw + 1) - e_n1.
    rows = nb if c["per_band_wx"] else 1
    wx = 10.0 + c["dw"] * torch.arange(1, nw + 1, dtype=torch.float64, device="cuda")[None, :] \
        - u((rows, 1), 0.0, 20.0)
    t["wx"] = torch.where(wx.abs() < TO1, TO1, wx).contiguous()
    if c["near_pole"] > 0:
        flat = torch.view_as_real(t["wt"]).view(-1, 2)
        at = torch.nonzero(u((ng * nc,), 0.0, 1.0) < c["near_pole"]).flatten()
        n = at.numel()
        pick = t["wx"].reshape(-1)[torch.randint(rows * nw, (n,), device="cuda", generator=gen)]
        flat[at, 0] = pick + u((n,), -7e-5, 7e-5)
        flat[at, 1] = u((n,), -7e-5, 7e-5)
    return t


def _device_inputs(c, t):
    one_row = not c["per_band_wx"]
    return ops.DeviceInputs(c["bands"], c["occupied"], c["ncouls"], c["ngpown"], c["nw"],
                            t["aqsm"], t["aqsn"], t["ieps"], t["wt"], t["vcoul"], t["igp"],
                            t["indinv"], t["wx"], 0 if one_row else c["nw"])


class _Batch:
    """A gpp_batch plan with the arrays it points to."""

    def __init__(self, c, seed):
        self.lib = capi.load()
        self.handle = C.c_void_p()
        n = c["states"]
        self.inputs, self.outs = [], []
        problems, outs = (capi.GppProblem * n)(), (capi.GppOutputs * n)()
        for k in range(n):
            s = _state_case(c, k)
            d = _device_inputs(s, _inputs(s, seed + 1000 * k))
            self.inputs.append(d)
            problems[k] = ops.problem_struct(d, c["precision"], c["semantics"], 1.0)
            o = [torch.empty(m, dtype=torch.complex128, device="cuda")
                 for m in [s["nw"], s["nw"]] + ([s["bands"]] if c["per_band_out"] else [])]
            self.outs.append(o)
            outs[k].achtemp, outs[k].asxtemp = o[0].data_ptr(), o[1].data_ptr()
            outs[k].acht_n1_loc = o[2].data_ptr() if c["per_band_out"] else None
        torch.cuda.synchronize()
        capi.check(self.lib.gpp_batch_create(C.byref(self.handle), problems, outs, n),
                   "gpp_batch_create")

    def run(self):
        capi.check(self.lib.gpp_batch_run(self.handle, torch.cuda.current_stream().cuda_stream),
                   "gpp_batch_run")
        return [list(o) for o in self.outs]

    def __del__(self):
        if self.handle:
            self.lib.gpp_batch_destroy(self.handle)


class _Shape:
    def __init__(self, c):
        self.number_bands, self.nvband, self.ncouls = c["bands"], c["occupied"], c["ncouls"]
        self.ngpown, self.nw = c["ngpown"], c["nw"]


def prepare(case, seed):
    if case["kind"] == "batch":
        return {"case": case, "batch": _Batch(case, seed)}
    t = _inputs(case, seed)
    if case["kind"] == "host":
        names = {"aqsmtemp": "aqsm", "aqsntemp": "aqsn", "I_eps_array": "ieps",
                 "wtilde_array": "wt", "vcoul": "vcoul", "inv_igp_index": "igp", "wx_array": "wx"}
        keep, arrays = [], {}
        for k, v in names.items():
            h = torch.empty(t[v].shape, dtype=t[v].dtype, pin_memory=True)
            h.copy_(t[v])
            keep.append(h)
            arrays[k] = h.numpy()
        return {"case": case, "arrays": arrays, "keep": keep, "shape": _Shape(case),
                "ctx": ops.HostContext()}
    return {"case": case, "in": _device_inputs(case, t)}


def run(state):
    c = state["case"]
    if c["kind"] == "batch":
        return state["batch"].run()
    if c["kind"] == "host":
        return state["ctx"].sigma(state["arrays"], state["shape"], c["precision"], c["semantics"],
                                  acht_n1=c["per_band_out"], achstemp=c["static_out"])
    d = state["in"]
    if c["kind"] == "sigma":
        r = ops.sigma(d, c["precision"], c["semantics"], acht_n1=c["per_band_out"],
                      achstemp=c["static_out"])
        return [x for x in (r.achtemp, r.asxtemp, r.acht_n1_loc, r.achstemp) if x is not None]
    lib = capi.load()
    capi.check(lib.gpp_set_dropin_precision(capi.PRECISION[c["precision"]]), "precision")
    zeros = lambda n, t: torch.zeros(n, dtype=t, device="cuda")  # noqa: E731
    re, im = zeros(c["nw"], torch.float64), zeros(c["nw"], torch.float64)
    if c["kind"] == "kernel":
        ops.gppKernelGPU(d.wtilde_array, d.aqsntemp, d.aqsmtemp, d.I_eps_array, d.ncouls, d.ngpown,
                         d.number_bands, d.wx_array, re, im, d.vcoul, 0, d.nw, d.indinv,
                         d.inv_igp_index)
        out = [re, im]
    else:
        asx, n1 = zeros(c["nw"], torch.complex128), zeros(c["bands"], torch.complex128)
        ops.d_till_nvband(d.nvband, d.ngpown, d.ncouls, d.inv_igp_index, d.wx_array,
                          d.wtilde_array, d.aqsmtemp, d.aqsntemp, d.I_eps_array, asx, d.vcoul, n1,
                          re, im)
        ops.d_noFlagOCCSolver(d.number_bands, d.nvband, d.ngpown, d.ncouls, d.inv_igp_index,
                              d.wx_array, d.wtilde_array, d.aqsmtemp, d.aqsntemp, d.I_eps_array,
                              d.vcoul, re, im, n1)
        out = [re, im, asx, n1]
    capi.check(lib.gpp_set_dropin_precision(-1), "precision")
    return out


# ---------------------------------------------------------------------------
# Work and exact values.

def work(case):
    read = written = flops = 0.0
    for k in range(case["states"]):
        c = _state_case(case, k)
        nb, nc, ng, nw = c["bands"], c["ncouls"], c["ngpown"], c["nw"]
        nv = 0 if c["kind"] == "kernel" else c["occupied"]
        cells = float(ng) * nc
        # aqsn, wtilde and I_eps whole; of aqsm and vcoul the G' columns.
        read += 16.0 * (nb * nc + 2 * cells + nb * ng) + 8.0 * ng + 4.0 * ng \
            + 8.0 * nw * (nb if c["per_band_wx"] else 1)
        written += 16.0 * (2 * nw + (nb if c["per_band_out"] or c["kind"] == "dropin" else 0))
        # Unoccupied: 20 flops a term and 12 shared by the frequencies; with one
        # frequency row the band sum is a complex product and the frequency
        # factor is applied once per (row, column).  Occupied: about 60 a term.
        if c["per_band_wx"]:
            flops += (nb - nv) * cells * (20.0 * nw + 12.0)
        else:
            flops += 8.0 * (nb - nv) * cells + cells * (20.0 * nw + 12.0)
            if c["per_band_out"] or c["kind"] == "dropin":
                flops += 8.0 * (nb - nv) * cells
        flops += 60.0 * nv * cells * nw
    return {"bytes": read + written, "flops": flops}


def _sigma64(c, t):
    """achtemp, asxtemp, per-band iw = 2 column and static term by plain torch."""
    nb, nc, nw = c["bands"], c["ncouls"], c["nw"]
    nv = 0 if c["kind"] == "kernel" else c["occupied"]
    igp = torch.clamp(t["igp"].long(), max=nc - 1)
    if t["indinv"] is not None:
        igp = t["indinv"].long()[igp]
    wt, ie = t["wt"], t["ieps"]
    weight = t["vcoul"][igp]
    ach = torch.zeros(nw, dtype=torch.complex128, device="cuda")
    asx = torch.zeros(nw, dtype=torch.complex128, device="cuda")
    n1 = torch.zeros(nb, dtype=torch.complex128, device="cuda")
    q = wt * ie
    wt2 = wt * wt
    om2 = wt2 * ie
    ie2 = ie.real ** 2 + ie.imag ** 2
    inv = {}
    for n in range(nb):
        m = t["aqsm"][n, igp].conj()
        for w in range(nw):
            x = float(t["wx"][n if c["per_band_wx"] else 0, w])
            if n < nv:
                wd = x - wt
                wdr = wd.real ** 2 + wd.imag ** 2
                delw = wt * wd.conj() / wdr
                delwr = delw.real ** 2 + delw.imag ** 2
                a = (wdr > 0.25) & (delwr < 1.0 / (TO1 * 4.0))
                b = ~a & (delwr > TO1)
                cden = 4.0 * wt2 * (delw + 0.5)
                ssx_b = -om2 * cden.conj() / (cden.real ** 2 + cden.imag ** 2) * delw
                zero = torch.zeros((), dtype=torch.complex128, device="cuda")
                sch = torch.where(a, delw * ie, zero)
                ssx = torch.where(a, om2 / (x * x), torch.where(b, ssx_b, zero))
                if c["semantics"] == "complex_seq" and x < 0.0:
                    cut = (ssx.real ** 2 + ssx.imag ** 2) > 16.0 * ie2
                    ssx = torch.where(cut, zero, ssx)
                asx[w] += (m * weight * (ssx @ t["aqsn"][n])).sum()
                s = (0.5 * m * weight * (sch @ t["aqsn"][n])).sum()
            else:
                if c["per_band_wx"]:
                    f = q / (x - wt)
                else:
                    f = inv.get(w)
                    if f is None:
                        f = inv[w] = q / (x - wt)
                s = (0.5 * m * weight * (f @ t["aqsn"][n])).sum()
            ach[w] += s
            if w == 2:
                n1[n] = s
    m = t["aqsm"][:, igp].conj()
    an = t["aqsn"][:, igp]
    own = ie[torch.arange(c["ngpown"], device="cuda"), igp]
    own = torch.where(own.abs() > TO1, -own, torch.zeros_like(own))
    static = (m * an * (own * 0.5 * weight)[None, :]).sum().reshape(1)
    return ach, asx, n1, static


def exact(case, seed):
    if case["kind"] == "batch":
        out = []
        for k in range(case["states"]):
            s = _state_case(case, k)
            ach, asx, n1, _ = _sigma64(s, _inputs(s, seed + 1000 * k))
            out.append([ach, asx] + ([n1] if case["per_band_out"] else []))
        return out
    ach, asx, n1, static = _sigma64(case, _inputs(case, seed))
    if case["kind"] == "host":
        out = {"achtemp": ach, "asxtemp": asx}
        if case["per_band_out"]:
            out["acht_n1_loc"] = n1
        if case["static_out"]:
            out["achstemp"] = static
        return out
    if case["kind"] == "kernel":
        return [ach.real.contiguous(), ach.imag.contiguous()]
    if case["kind"] == "dropin":
        return [ach.real.contiguous(), ach.imag.contiguous(), asx, n1]
    return [ach, asx] + ([n1] if case["per_band_out"] else []) \
        + ([static] if case["static_out"] else [])
