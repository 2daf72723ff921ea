"""Workloads of the library through its Python binding, for timing.

Each case is one call (or one forward and backward) that a program built on
clblm_gb300 makes again and again: layer optical depths, nadir radiances,
Jacobians, gradients, batches of profiles and the instrument scan.  Sizes and
distributions are those of synth.py and bench.py (uniform line centres at
about 250 lines per cm-1, seven absorbers, 1013 hPa upwards), from a one-layer
window of 15 cm-1 to whole columns.

  listed()            the cases
  draw(rng)           another case of the same ranges
  prepare(case, seed) lines, atmosphere, handle and output buffers
  run(state)          one pass, its outputs
  work(case)          bytes and operations of one pass
  exact(case, seed)   the instrument scan in plain numpy

Outputs of the mixed path are returned in binary32: its line shapes, merges
and derivatives are computed in binary32, and the library widens each value to
binary64 as it stores it, so a program that keeps such spectra keeps the four
bytes.  The FP64 path and the scans return binary64.
"""
import math

import numpy as np
import torch

from clblm_gb300 import capi, synth, torch_ops
from clblm_gb300 import capi_types as T

DENSITY = 250.0  # lines per cm-1 (500,000 on 500-2500 cm-1)
WING = 25.0      # the line wing cut-off, cm-1


def listed():
    return [
        # one layer of a narrow channel, called from a host program that takes
        # the spectrum back in host memory: latency and launches
        {"name": "layer_channel", "kind": "layer", "precision": "mixed", "out": "host", "level": "surface",
         "v1": 600.0, "width": 15.0, "density": 200.0, "dv_out": 0.0},
        # a homogeneous surface layer, 20,000 lines on 100 cm-1, on the device
        {"name": "layer_100cm", "kind": "layer", "precision": "mixed", "out": "device", "level": "surface",
         "v1": 600.0, "width": 100.0, "density": 200.0, "dv_out": 0.0},
        # the same in the reference's arithmetic, onto a uniform output grid
        {"name": "layer_100cm_fp64", "kind": "layer", "precision": "fp64", "out": "device", "level": "surface",
         "v1": 600.0, "width": 100.0, "density": 200.0, "dv_out": 0.004},
        # a 0.1 hPa layer over 1000 cm-1: millions of points, narrow lines,
        # a window high enough that the radiation term is in the line strengths
        {"name": "layer_top_1000cm", "kind": "layer", "precision": "mixed", "out": "device", "level": "top",
         "v1": 1200.0, "width": 1000.0, "density": 250.0, "dv_out": 0.0},
        # the radiance of a retrieval window, a coarse atmosphere
        {"name": "column_50cm", "kind": "column", "precision": "mixed", "nlay": 20, "p_top": 0.1, "v1": 650.0,
         "width": 50.0, "density": 250.0},
        # the radiance of a whole infrared sounder band
        {"name": "column_2000cm", "kind": "column", "precision": "mixed", "nlay": 60, "p_top": 0.1, "v1": 500.0,
         "width": 2000.0, "density": 250.0},
        # a reference calculation: the same atmosphere in FP64
        {"name": "column_100cm_fp64", "kind": "column", "precision": "fp64", "nlay": 60, "p_top": 0.1, "v1": 667.3,
         "width": 100.0, "density": 250.0},
        # far infrared, 100 layers to 0.01 hPa, the broadband list's density
        {"name": "column_far_ir", "kind": "column", "precision": "mixed", "nlay": 100, "p_top": 0.01, "v1": 10.0,
         "width": 590.0, "density": 860.0},
        # radiance with level temperature and ln q(H2O) Jacobians of a column
        {"name": "jacobian_500cm", "kind": "jacobian", "precision": "mixed", "nlay": 60, "p_top": 0.1, "v1": 600.0,
         "width": 500.0, "density": 250.0},
        # a training step's layer: radiance forward and its gradient with
        # respect to the level profile backward, through torch.autograd
        {"name": "gradient_60cm", "kind": "gradient", "precision": "mixed", "nlay": 30, "p_top": 0.1, "v1": 700.0,
         "width": 60.0, "density": 250.0},
        # many uneven profiles in one call, radiance and Jacobians of each
        {"name": "batch_6_profiles", "kind": "batch", "precision": "mixed", "profiles": 6, "nlay_min": 20,
         "nlay_max": 60, "v1": 600.0, "width_min": 10.0, "width_max": 60.0, "density": 250.0},
        # a monochromatic spectrum to instrument resolution (sinc, OPD 0.8 cm)
        {"name": "scan_sinc_2M", "kind": "scan", "function": 5, "hwhm": 0.3771, "v1": 600.0, "dv": 3.0e-4,
         "points": 2000000},
    ]


def draw(rng):
    def logu(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    kind = rng.choice(["layer", "layer", "layer", "column", "column", "column", "jacobian", "gradient", "batch",
                       "scan"])
    fp64 = rng.random() < 0.3
    prec = "fp64" if fp64 else "mixed"
    v1 = round(rng.uniform(500.0, 1400.0), 3)
    density = round(logu(100.0, 500.0), 1)
    if kind == "layer":
        return {"kind": kind, "precision": prec, "out": rng.choice(["host", "device"]),
                "level": rng.choice(["surface", "middle", "top"]), "v1": v1,
                "width": round(logu(8.0, 200.0 if fp64 else 900.0), 3), "density": density,
                "dv_out": rng.choice([0.0, 0.003]) if fp64 else 0.0}
    if kind == "column":
        if fp64:
            return {"kind": kind, "precision": prec, "nlay": rng.randint(20, 60), "p_top": 0.1, "v1": v1,
                    "width": round(logu(8.0, 60.0), 3), "density": round(logu(100.0, 250.0), 1)}
        return {"kind": kind, "precision": prec, "nlay": rng.randint(20, 100),
                "p_top": rng.choice([0.1, 0.01]), "v1": round(rng.uniform(10.0, 1400.0), 3),
                "width": round(logu(10.0, 500.0), 3), "density": density}
    if kind == "jacobian":
        return {"kind": kind, "precision": "mixed", "nlay": rng.randint(20, 70), "p_top": 0.1, "v1": v1,
                "width": round(logu(10.0, 200.0), 3), "density": density}
    if kind == "gradient":
        return {"kind": kind, "precision": "mixed", "nlay": rng.randint(20, 60), "p_top": 0.1, "v1": v1,
                "width": round(logu(10.0, 150.0), 3), "density": density}
    if kind == "batch":
        return {"kind": kind, "precision": "mixed", "profiles": rng.randint(2, 10), "nlay_min": 20,
                "nlay_max": rng.randint(30, 80), "v1": v1, "width_min": 10.0,
                "width_max": round(logu(20.0, 80.0), 3), "density": 250.0}
    fn = rng.choice([3, 5])
    return {"kind": "scan", "function": fn, "hwhm": round(logu(0.2, 0.6), 4), "v1": v1,
            "dv": round(logu(2.0e-4, 2.0e-3), 6), "points": int(logu(500000, 6000000))}


# ---- inputs -------------------------------------------------------------------

def _lines(case, seed, width, mols=synth.SEVEN):
    lo, hi = max(1.0, case["v1"] - WING - 5.0), case["v1"] + width + WING + 5.0
    return synth.line_list(int(round(case["density"] * (hi - lo))), lo, hi, seed, mols=mols)


def _atmosphere(nlay, p_top, v1, v2, rng):
    """The synthetic lapse atmosphere with the absorbers other than H2O
    scaled by factors near 1, so that another seed is another atmosphere.
    Pressures, temperatures and H2O stay: they set the spectral grids, and so
    the sizes of the outputs."""
    col = synth.atmosphere(nlay, p_top, v1, v2)
    f = np.exp(rng.normal(0.0, 0.2, len(col.mol_id)))
    f[col.mol_id == 1] = 1.0
    col.w = col.w * f
    col.vmr_lev = col.vmr_lev * f
    return col


def _precision(case):
    return T.CLBLM_PREC_PLAIN if case["precision"] == "fp64" else T.CLBLM_PREC_MIXED


def _spectrum(case, seed):
    """A radiance-like spectrum: a smooth background with narrow lines."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, dv = case["points"], case["dv"]
    x = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    k = max(1, int(0.01 / dv))
    x = torch.nn.functional.avg_pool1d(x[None, None], 2 * k + 1, stride=1, padding=k)[0, 0]
    t = torch.arange(n, dtype=torch.float64, device="cuda") * dv
    return 1.0e-5 * (1.0 + 0.3 * torch.sin(2.0 * math.pi * t / 7.0) + x)


def _scan(case):
    v2 = case["v1"] + case["dv"] * (case["points"] - 1)
    margin = 0.05 * (v2 - case["v1"])
    return T.scan_struct(case["function"], case["hwhm"], case["v1"] + margin, v2 - margin)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "scan":
        h = capi.Handle(synth.line_list(1000, 600.0, 700.0, seed))
        sc = _scan(case)
        _, _, n = capi.fftscn_size(sc, case["v1"], case["dv"], case["points"])
        return {"case": case, "h": h, "scan": sc, "x": _spectrum(case, seed),
                "out": torch.empty(n, dtype=torch.float64, device="cuda")}
    if kind == "batch":
        n = case["profiles"]
        fixed = np.random.default_rng(n)  # windows and layer counts: the case's own
        widths = 10.0 ** fixed.uniform(math.log10(case["width_min"]), math.log10(case["width_max"]), n)
        h = capi.Handle(_lines(case, seed, case["width_max"] * 2.0), synth.continuum())
        cols = []
        for i in range(n):
            a = case["v1"] + float(np.round(fixed.uniform(0.0, case["width_max"]), 3))
            nlay = int(fixed.integers(case["nlay_min"], case["nlay_max"] + 1))
            cols.append(_atmosphere(nlay, 0.1, a, a + float(np.round(widths[i], 3)), rng))
        jacs = [synth.jac_profile(c) for c in cols]
        ctrl = T.rt_ctrl(precision=_precision(case), grid_type=1)
        npts, _ = h.batch_size(cols, ctrl, jacs)
        bufs = [_jac_buffers(m, c.nlay) for m, c in zip(npts, cols)]
        return {"case": case, "h": h, "cols": cols, "jacs": jacs, "ctrl": ctrl, "bufs": bufs,
                "outs": [{k: t.data_ptr() for k, t in b.items()} | {"cap": m} for b, m in zip(bufs, npts)]}
    v1, v2 = case["v1"], case["v1"] + case["width"]
    if kind == "layer":
        mols = np.array([1], np.int32) if case["level"] == "surface" else synth.SEVEN
        h = capi.Handle(_lines(case, seed, case["width"], mols), synth.continuum())
        if case["level"] == "surface":  # 1 km of air at 1013.25 hPa
            t, wtot = 296.0, 2.479e24
            col = T.Column(mols, [1013.25], [t], [t], [t], np.array([[1.0e22]]), [wtot],
                           [synth.SECANT_DIFFUSE * wtot], v1, v2, t, 1.0)
            i = 0
        else:
            col = _atmosphere(60, 0.1, v1, v2, rng)
            i = 59 if case["level"] == "top" else 30
        dn, df, _ = capi.setDV(col)
        ctrl = T.od_ctrl(precision=_precision(case))
        grid = T.grid_struct(v1, v2, dn[i], df[i], case["dv_out"] if case["dv_out"] > 0 else -999.9)
        lay = col.layer(i)
        n, _ = h.od_size(lay, grid, ctrl)
        out = torch.empty(n, dtype=torch.float64, device="cuda") if case["out"] == "device" else np.empty(n)
        return {"case": case, "h": h, "layer": lay, "grid": grid, "ctrl": ctrl, "out": out}
    h = capi.Handle(_lines(case, seed, case["width"]), synth.continuum())
    col = _atmosphere(case["nlay"], case["p_top"], v1, v2, rng)
    if kind == "column":
        ctrl = T.rt_ctrl(precision=_precision(case))
        n, _ = h.rt_size(col, ctrl)
        return {"case": case, "h": h, "col": col, "ctrl": ctrl,
                "out": torch.empty(n, dtype=torch.float64, device="cuda")}
    ctrl = T.rt_ctrl(precision=_precision(case), grid_type=1)
    if kind == "jacobian":
        jac = synth.jac_profile(col)
        n, _ = h.jac_size(col, ctrl, jac)
        return {"case": case, "h": h, "col": col, "ctrl": ctrl, "jac": jac, "n": n,
                "buf": _jac_buffers(n, col.nlay)}
    p = torch_ops.RadianceProblem.from_column(h, ctrl, col)
    t, q = p.levels(np.append(col.tbot, col.ttop[-1]))
    f = lambda x: torch.tensor(float(x), device="cuda")
    n, _ = h.jac_size(col, p.ctrl, synth.jac_profile(col, jac_mol=0, do_temp=0))
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    return {"case": case, "h": h, "problem": p, "t": t.float(), "q": q.float(), "ts": f(col.tskin), "em": f(col.emis),
            "w": w}


def _jac_buffers(n, nlay):
    e = lambda *s: torch.empty(s, dtype=torch.float64, device="cuda")
    return {"rad": e(n), "dtlev": e(nlay + 1, n), "dqlev": e(nlay + 1, n), "dtsfc": e(n), "demis": e(n)}


# ---- one pass -------------------------------------------------------------------

def _kept(case, x):
    """A spectrum as the program keeps it (see the module's docstring)."""
    if case["precision"] == "fp64":
        return x
    return x.float() if torch.is_tensor(x) else x.astype(np.float32)


def run(s):
    c, h = s["case"], s["h"]
    kind = c["kind"]
    if kind == "layer":
        if c["out"] == "host":
            od, _ = h.odlay(s["layer"], s["grid"], s["ctrl"], s["out"])
            return _kept(c, od)
        h.od_device(s["layer"], s["grid"], s["ctrl"], s["out"].data_ptr(), len(s["out"]))
        return _kept(c, s["out"])
    if kind == "column":
        h.rt_mode2_device(s["col"], s["ctrl"], s["out"].data_ptr(), len(s["out"]))
        return _kept(c, s["out"])
    if kind == "jacobian":
        b = s["buf"]
        h.jac_device(s["col"], s["ctrl"], s["jac"], b["rad"].data_ptr(), b["dtlev"].data_ptr(),
                     b["dqlev"].data_ptr(), b["dtsfc"].data_ptr(), b["demis"].data_ptr(), s["n"])
        return {k: _kept(c, v) for k, v in b.items()}
    if kind == "batch":
        h.batch_device(s["cols"], s["ctrl"], s["jacs"], s["outs"])
        return [{k: _kept(c, v) for k, v in b.items()} for b in s["bufs"]]
    if kind == "scan":
        h.fftscn_device(s["scan"], s["x"].data_ptr(), len(s["x"]), c["v1"], c["dv"], s["out"].data_ptr(),
                        len(s["out"]))
        return s["out"]
    leaves = [s[k].detach().requires_grad_() for k in ("t", "q", "ts", "em")]
    rad = torch_ops.nadir_radiance(s["problem"], *leaves)
    rad.backward(s["w"])
    return {"rad": _kept(c, rad.detach()), "grads": [x.grad for x in leaves]}


# ---- what a pass cannot do without -------------------------------------------------

def _od_work(col, n_lines, grid_type, v1, v2):
    """(points, operations) of one OD of every layer: per line about 45 steps
    of 19 operations on the three panel grids, and per point of the far-wing
    grid (64 DV) 9 operations for each far-wing record within 25 cm-1 (about
    half the lines are left after they are merged)."""
    dn, df, do = capi.setDV(col, grid_type=grid_type)
    width = v2 - v1
    density = n_lines / (width + 2 * WING)
    pts = flops = 0.0
    for i in range(col.nlay):
        dv = dn[i] if abs(dn[i] - df[i]) / dn[i] > 0.2 else df[i]
        pts += width / dv
        flops += 19.0 * 45.0 * n_lines + 9.0 * (width / (64.0 * dv)) * 2.0 * WING * 0.5 * density
    return pts, flops, do


def work(case):
    rng = np.random.default_rng(0)
    kind = case["kind"]
    if kind == "scan":
        n = case["points"]
        return {"bytes": 8.0 * 2 * n, "flops": 10.0 * n * math.log2(n)}
    total = {"bytes": 0.0, "flops": 0.0}
    if kind == "batch":
        parts = []
        for _ in range(case["profiles"]):
            nlay = int(round(0.5 * (case["nlay_min"] + case["nlay_max"])))
            parts.append((nlay, 0.1, math.sqrt(case["width_min"] * case["width_max"])))
    elif kind == "layer":
        parts = [(60, 0.1, case["width"])]
    else:
        parts = [(case["nlay"], case["p_top"], case["width"])]
    for nlay, p_top, width in parts:
        v1, v2 = case["v1"], case["v1"] + width
        col = _atmosphere(nlay, p_top, v1, v2, rng)
        if kind == "layer":
            col = col.sub([{"surface": 0, "middle": 30, "top": 59}[case["level"]]])
        lines = case["density"] * (width + 2 * (WING + 5.0))
        uniform = kind not in ("layer", "column")
        pts, flops, dv_out = _od_work(col, lines, 1 if uniform else 0, v1, v2)
        total["bytes"] += 40.0 * lines
        if not uniform:
            n_out = pts if kind == "layer" else width / min(capi.setDV(col)[1])
            total["bytes"] += 8.0 * n_out
            total["flops"] += flops + (0.0 if kind == "layer" else 60.0 * pts)
            continue
        n = width / dv_out
        # four ODs per layer (the molecule alone has a seventh of the lines),
        # with a gradient the radiance's own besides
        ods = (3.0 + 1.0 / 7.0) + (1.0 if kind == "gradient" else 0.0)
        rows = 2.0 if kind == "gradient" else 3.0 + 2.0 * (col.nlay + 1)
        total["bytes"] += 8.0 * rows * n
        total["flops"] += ods * flops + 200.0 * col.nlay * n
    return total


# ---- 64-bit values ---------------------------------------------------------------------

def exact(case, seed):
    """The FFT scan: the circular convolution of the zero-padded spectrum with
    the scanning function through its apodization.  The optical depths,
    radiances and Jacobians have no value apart from the reference's own
    algorithm (nested grids, tabulated shapes, merged far-wing lines), whose
    64-bit restatement is thousands of lines: none here."""
    if case["kind"] != "scan":
        return None
    x = _spectrum(case, seed).cpu().numpy()
    sc = _scan(case)
    v1c, dv, hw, rec = case["v1"], case["dv"], case["hwhm"], 65536
    limit = {3: 3.0, 5: 160.0}[case["function"]]
    a = {3: 0.849322, 5: 3.3148}[case["function"]] * hw
    v2c = v1c + dv * (len(x) - 1)
    v1z = max(v1c, v1c + int((sc.v1out - hw * limit - v1c) / dv) * dv)
    v2z = min(v2c, v1c + int((sc.v2out + hw * limit - v1c) / dv + 1.01) * dv)
    total = int((v2z - v1z) / dv + 1.1)
    first = int((v1z - v1c) / dv + 1.00001)
    nrec = 4 * 2 ** math.ceil(math.log2(math.ceil(total / rec)))
    n = nrec * rec
    y = np.zeros(n)
    y[:total] = x[first - 1:first - 1 + total]
    f = np.fft.rfft(y)
    dx = 1.0 / (n * dv)
    k = np.arange(n // 2 + 1)
    opd = k * dx
    if case["function"] == 3:
        ap = np.exp(-np.minimum(2.0 * (math.pi * opd * a) ** 2, 34.0))
    else:  # a rectangle to 1/A with an interpolated end point in its record
        ap = np.where(opd < 1.0 / a, 1.0, 0.0)
        for j in range(nrec):
            x0 = j * (rec // 2) * dx
            m = int((1.0 / a - x0) / dx) + 1
            r = (1.0 / a - x0) / dx + 1 - m
            if r <= 0.5:
                r, m = r + 1.0, m - 1
            if 1 <= m <= rec // 2 - 1:
                ap[j * (rec // 2) + m] = r - 0.5
    ap[n // 2] = 0.0
    y = np.fft.irfft(f * ap, n=n)
    n1 = max(1, int((sc.v1out - v1z) / dv))
    n2 = int((sc.v2out - v1z) / dv + 3.01)
    if v1z + (n2 - 1) * dv > v1z + dv * (total - 1):
        n2 = total
    return y[n1 - 1:n2]
