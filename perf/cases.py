"""Workloads of the sigma GPP / FF library, through its public entry points.

`listed()` names the calls a sigma calculation makes with this library, at
the sizes of its benchmark, tests and job scripts; `draw(rng)` gives more of
the same ranges.  `prepare` makes the inputs on the GPU (on the host for the
host-pointer drop-in) and the plan a program keeps, `run` is one pass, `work`
what a pass cannot do without, `exact` the same outputs from complex128 /
float64 torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "fortkernels-_gb300"))
import sigma_gb300 as S  # noqa: E402
import autotune  # noqa: E402
import workload as W  # noqa: E402

PREC = {"fp64": S.PREC_FP64, "mixed": S.PREC_MIXED, "tensor": S.PREC_TENSOR}
MODE = {"fp64": S.FF_MODE_FP64, "tensor": S.FF_MODE_OZAKI_BF16}
TO1, LIMITONE, LIMITTWO = 1e-6, 1.0 / 4e-6, 0.25


def listed():
    return [
        # the smallest call: the host-pointer drop-in of one small instance, as a driver that replaces the
        # reference's loop nest makes it (inputs and outputs in host memory)
        {"name": "host_fp64_tiny", "kind": "host", "form": "fp64", "nb": 24, "nvb": 2, "nc": 1024, "ng": 40, "stress": False},
        # the reference's small problem (128 2 8192 20) with inputs on the device
        {"name": "gpp_fp64_small", "kind": "gpp", "form": "fp64", "nb": 128, "nvb": 2, "nc": 8192, "ng": 409, "stress": False, "per_band": False},
        # the job scripts' production problem (512 2 32768 20): the headline
        {"name": "gpp_fp64_production", "kind": "gpp", "form": "fp64", "nb": 512, "nvb": 2, "nc": 32768, "ng": 1638, "stress": False, "per_band": False},
        # frequencies that depend on the band, as in the Fortran original; sizes that divide nothing
        {"name": "gpp_fp64_perband_odd", "kind": "gpp", "form": "fp64", "nb": 133, "nvb": 5, "nc": 5003, "ng": 167, "stress": False, "per_band": True},
        # the FP32 form at the production problem
        {"name": "gpp_mixed_production", "kind": "gpp", "form": "mixed", "nb": 512, "nvb": 2, "nc": 32768, "ng": 1638, "stress": False, "per_band": False},
        # the tensor-core form at the production problem with poles close to the frequencies
        {"name": "gpp_tensor_stress", "kind": "gpp", "form": "tensor", "nb": 512, "nvb": 2, "nc": 32768, "ng": 1638, "stress": True, "per_band": False},
        # q-points and band windows of uneven shape in one queue, replayed as a graph
        {"name": "batch_fp64", "kind": "batch", "form": "fp64", "n": 12, "shapes": 3},
        {"name": "batch_tensor", "kind": "batch", "form": "tensor", "n": 12, "shapes": 3},
        # full-frequency contraction schDt at the benchmark's size
        {"name": "ff_schdt_fp64", "kind": "ff", "mode": "fp64", "nb": 512, "nc": 16384, "ng": 820, "nf": 15},
        # full-frequency band loop around two contractions, tensor-core form
        {"name": "ff_sigma_tensor", "kind": "ff_sigma", "mode": "tensor", "nb": 512, "nvb": 2, "nc": 16384, "ng": 820, "nf": 15, "ne": 15},
        # gppsum = 1 half sum with its static remainder
        {"name": "halfsum_fp64_production", "kind": "halfsum", "tensor": False, "nb": 512, "nvb": 2, "nc": 32768, "ng": 1638},
        # real-valued GPP (systems with inversion symmetry)
        {"name": "real_fp64_production", "kind": "real", "nb": 512, "nvb": 2, "nc": 32768, "ng": 1638},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "gpp", "gpp", "gpp", "batch", "ff", "ff_sigma", "halfsum", "real"])
    if kind == "batch":
        while True:
            c = {"kind": "batch", "form": rng.choice(["fp64", "mixed", "tensor"]), "n": rng.randint(3, 12),
                 "shapes": rng.randint(4, 10 ** 6)}
            if work(c)["flops"] <= 1.9e12 and work(c)["bytes"] <= 1e10:
                return c
    while True:
        nb = _log(rng, 16, 128 if kind == "host" else 512)
        nc = _log(rng, 512, 8192 if kind == "host" else 32768)
        ng = max(20, nc // rng.randint(10, 40))
        nvb = min(nb, rng.randint(0, 8))
        if kind == "host":
            return {"kind": kind, "form": rng.choice(["fp64", "fp64", "mixed", "tensor"]), "nb": nb, "nvb": nvb,
                    "nc": nc, "ng": ng, "stress": rng.random() < 0.3}
        if kind == "gpp":
            form = rng.choice(["fp64", "fp64", "mixed", "tensor"])
            per_band = form == "fp64" and rng.random() < 0.25
            if 3.0 * nb * ng * nc > (5e9 if per_band else 9e10):
                continue
            return {"kind": kind, "form": form, "nb": nb, "nvb": nvb, "nc": nc, "ng": ng,
                    "stress": rng.random() < 0.3, "per_band": per_band}
        if kind in ("halfsum", "real"):
            if 3.0 * nb * ng * nc > 9e10:
                continue
            c = {"kind": kind, "nb": nb, "nvb": nvb, "nc": nc, "ng": ng}
            return dict(c, tensor=rng.random() < 0.5) if kind == "halfsum" else c
        nf = rng.randint(5, 15)
        if float(nf) * nb * ng * nc > 1e11 or 16.0 * nf * ng * nc > 4e9:
            continue
        c = {"kind": kind, "nb": nb, "nc": nc, "ng": ng, "nf": nf}
        if kind == "ff":
            return dict(c, mode=rng.choice(["fp64", "fp64", "tensor"]))
        return dict(c, nvb=nvb, ne=rng.randint(5, 15), mode=rng.choice(["fp64", "tensor"]))


# ---------------------------------------------------------------- inputs
# The value ranges of the repository's seeded workloads: aqsm, aqsn, I_eps
# U(-1, 1) per part, wtilde U(0.5, 5) + i U(-0.1, 0.1), vcoul U(0.1, 10).
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _real(g, shape, lo, hi):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64).mul_(hi - lo).add_(lo)


def _complex(g, shape, re=(-1.0, 1.0), im=(-1.0, 1.0)):
    """[..., 2] float64: interleaved complex128."""
    t = torch.rand((*shape, 2), generator=g, device="cuda", dtype=torch.float64)
    t[..., 0].mul_(re[1] - re[0]).add_(re[0])
    t[..., 1].mul_(im[1] - im[0]).add_(im[0])
    return t


def _gpp_inputs(seed, nb, nc, ng, stress=False):
    g = _gen(seed)
    d = {"aqsm": _complex(g, (nb, nc)), "aqsn": _complex(g, (nb, nc)), "ieps": _complex(g, (ng, nc)),
         "wt": _complex(g, (ng, nc), (0.5, 5.0), (-0.1, 0.1)), "vcoul": _real(g, (nc,), 0.1, 10.0),
         "wx": torch.tensor(W.wx_frequencies(), dtype=torch.float64, device="cuda")}
    if stress:  # 5 % of the poles within 1e-3 of a frequency
        near = torch.rand((ng, nc), generator=g, device="cuda") < 0.05
        k = torch.randint(0, 3, (ng, nc), generator=g, device="cuda")
        off = _real(g, (ng, nc), -1e-3, 1e-3)
        d["wt"][..., 0] = torch.where(near, d["wx"][k] + off, d["wt"][..., 0])
    return d


def _band_frequencies(g, nb, wx):
    """One frequency set per band: the mini-app's, each band shifted by up to one spacing."""
    return (wx[None, :] + _real(g, (nb, 1), -0.5, 0.5)).contiguous()


def _zeros(*shape):
    return torch.zeros(shape, dtype=torch.float64, device="cuda")


def _shapes(c):
    return W.batched_shapes(c["n"], seed=c["shapes"])


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    s = {"case": c, "kind": kind}
    if kind == "host":
        d = _gpp_inputs(seed, c["nb"], c["nc"], c["ng"], c["stress"])
        h = {k: v.cpu().numpy() for k, v in d.items()}
        z = lambda a: a.view(np.complex128)[..., 0]  # noqa: E731
        inv, indinv = W.gpp_index_maps(c["nc"], c["ng"])
        s["prob"] = W.GppProblem(c["nb"], c["nvb"], c["nc"], c["ng"], inv, indinv, h["wx"], z(h["aqsm"]), z(h["aqsn"]),
                                 z(h["ieps"]), z(h["wt"]), h["vcoul"])
    elif kind in ("gpp", "halfsum"):
        d = _gpp_inputs(seed, c["nb"], c["nc"], c["ng"], c.get("stress", False))
        if c.get("per_band"):
            d["wx"] = _band_frequencies(_gen(seed + 1), c["nb"], d["wx"])
        inv, indinv = W.gpp_index_maps(c["nc"], c["ng"])
        if kind == "gpp":
            s["plan"] = S.GppPlan(c["nb"], c["nvb"], c["nc"], c["ng"], inv, indinv, precision=PREC[c["form"]])
        else:
            s["plan"] = S.GppHalfSumPlan(c["nb"], c["nvb"], c["nc"], c["ng"], inv, indinv,
                                         flags=S.HALFSUM_STATIC | (S.HALFSUM_TENSOR if c["tensor"] else 0))
        s["d"] = d
        s["out"] = {"achtemp": _zeros(3, 2), "asxtemp": _zeros(3, 2), "acht_n1_loc": _zeros(c["nb"], 2)}
        if kind == "halfsum":
            s["out"]["achstemp"] = _zeros(1, 2)
    elif kind == "real":
        g = _gen(seed)
        nb, nc, ng = c["nb"], c["nc"], c["ng"]
        s["d"] = {"aqsm": _real(g, (nb, nc), -1, 1), "aqsn": _real(g, (nb, nc), -1, 1), "ieps": _real(g, (ng, nc), -1, 1),
                  "wt": _real(g, (ng, nc), 0.5, 5.0), "vcoul": _real(g, (nc,), 0.1, 10.0),
                  "wx": torch.tensor(W.wx_frequencies(), dtype=torch.float64, device="cuda")}
        s["plan"] = S.GppRealPlan(nb, c["nvb"], nc, ng, *W.gpp_index_maps(nc, ng))
        s["out"] = {"achtemp": _zeros(3), "asxtemp": _zeros(3), "acht_n1_loc": _zeros(nb)}
    elif kind == "batch":
        s["in"], s["outs"], inst = [], [], []
        shapes = _shapes(c)
        for i, q in enumerate(shapes):
            nb, nc, ng = q["number_bands"], q["ncouls"], q["ngpown"]
            d = _gpp_inputs(seed * 64 + i, nb, nc, ng)
            o = {"achtemp": _zeros(3, 2), "asxtemp": _zeros(3, 2), "acht_n1_loc": _zeros(nb, 2)}
            inv, indinv = W.gpp_index_maps(nc, ng)
            inst.append(dict(number_bands=nb, nvband=q["nvband"], ncouls=nc, ngpown=ng, inv_igp_index=inv, indinv=indinv,
                             wx_array=d["wx"], aqsmtemp=d["aqsm"], aqsntemp=d["aqsn"], I_eps_array=d["ieps"],
                             wtilde_array=d["wt"], vcoul=d["vcoul"], **o))
            s["in"].append(d)
            s["outs"].append(o)
        tiles = [autotune.tile_for(q["number_bands"], q["ngpown"], shared=True) for q in shapes]
        form = c["form"]
        s["batch"] = S.GppBatch(inst, PREC[form], tiles=tiles if form == "fp64" else None,
                                items_per_cta=autotune.sizing_for(form) if form != "tensor" else 0,
                                tensor_split_tiles=autotune.sizing_for("tensor") if form == "tensor" else 0)
        s["stream"] = torch.cuda.Stream()
    else:  # ff, ff_sigma
        g = _gen(seed)
        nb, nc, ng, nf = c["nb"], c["nc"], c["ng"], c["nf"]
        s["d"] = d = {"aqsm": _complex(g, (nb, nc)), "aqsn": _complex(g, (nb, nc)), "epsr": _complex(g, (nf, ng, nc))}
        inv, indinv = W.ff_index_maps(nc, ng)
        if kind == "ff":
            s["plan"] = S.FfPlan(nb, nc, ng, nf, inv, indinv, MODE[c["mode"]])
            s["out"] = _zeros(nb, nf, 2)
        else:
            d["epsa"] = _complex(g, (nf, ng, nc))
            d["vcoul"] = _real(g, (nc,), 0.1, 10.0)
            ekq, grid, brd, pref = W.ff_sigma_grid(nb, nf)
            dev = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
            d.update(ekq=dev(ekq), grid=dev(grid), brd=torch.view_as_real(dev(brd)).contiguous(), pref=dev(pref))
            s["plan"] = S.FfSigmaPlan(nb, c["nvb"], nc, ng, nf, c["ne"], inv, indinv, MODE[c["mode"]])
            s["out"] = _zeros(1 + 5 * c["ne"], 2)
    torch.cuda.synchronize()
    return s


PREF_ZB, FMIN, FSTEP = 0.5 / 3.14, 0.0, 0.5


def run(s):
    kind = s["kind"]
    if kind == "host":
        ach, asx, n1 = S.gpp_host(s["prob"], PREC[s["case"]["form"]])
        return {"achtemp": ach, "asxtemp": asx, "acht_n1_loc": n1}
    if kind == "batch":
        s["batch"].launch_graph(s["stream"].cuda_stream)
        return s["outs"]
    d, o = s["d"], s["out"]
    if kind == "gpp":
        s["plan"].execute(d["wx"], d["aqsm"], d["aqsn"], d["ieps"], d["wt"], d["vcoul"], o["achtemp"], o["asxtemp"],
                          o["acht_n1_loc"], wx_band_stride=3 if s["case"]["per_band"] else 0)
    elif kind == "halfsum":
        s["plan"].execute(d["wx"], d["aqsm"], d["aqsn"], d["ieps"], d["wt"], d["vcoul"], o["achtemp"], o["asxtemp"],
                          o["acht_n1_loc"], o["achstemp"])
    elif kind == "real":
        s["plan"].execute(d["wx"], d["aqsm"], d["aqsn"], d["ieps"], d["wt"], d["vcoul"], o["achtemp"], o["asxtemp"],
                          o["acht_n1_loc"])
    elif kind == "ff":
        s["plan"].execute(d["epsr"], d["aqsn"], d["aqsm"], o)
    else:
        s["plan"].execute(d["aqsm"], d["aqsn"], d["epsr"], d["epsa"], d["vcoul"], d["ekq"], d["grid"], d["brd"], d["pref"],
                          PREF_ZB, FMIN, FSTEP, 1.0, None, o)
    return o


def _gpp_work(nb, nc, ng, cplx=True):
    n = 2 if cplx else 1
    return 8.0 * n * (2.0 * nb * nc + 2.0 * ng * nc) + 8.0 * nc + 8.0 * n * (nb + 6), (8.0 if cplx else 2.0) * 3 * nb * ng * nc


def work(case):
    """Each input read once, each output written once; one multiply-add (8
    flops when complex) per term of the band sums."""
    c = case
    kind = c["kind"]
    if kind == "batch":
        p = [_gpp_work(q["number_bands"], q["ncouls"], q["ngpown"]) for q in _shapes(c)]
        return {"bytes": sum(x[0] for x in p), "flops": sum(x[1] for x in p)}
    nb, nc, ng = c["nb"], c["nc"], c["ng"]
    if kind in ("host", "gpp", "real"):
        b, f = _gpp_work(nb, nc, ng, kind != "real")
        return {"bytes": b, "flops": f}
    if kind == "halfsum":
        # two sums (term and partner) of three frequencies and the static one, over g-vectors below igp
        igp = float(W.gpp_index_maps(nc, ng)[0].astype(np.float64).sum())
        return {"bytes": _gpp_work(nb, nc, ng)[0], "flops": 8.0 * nb * igp * 2 * 4}
    eps = 16.0 * c["nf"] * ng * nc
    b, f = 32.0 * nb * nc + eps + 16.0 * nb * c["nf"], 8.0 * c["nf"] * ng * nb * nc
    return {"bytes": b, "flops": f} if kind == "ff" else {"bytes": b + eps + 8.0 * nc, "flops": 2 * f}


# ---------------------------------------------------------------- 64-bit values
def _z(t):
    return torch.view_as_complex(t.contiguous())


def _blocks(ng, nc, planes=10):
    step = max(1, min(ng, int(3e9 / (16.0 * nc * planes))))
    return [(a, min(ng, a + step)) for a in range(0, ng, step)]


def _pole_factors(wx, wt, ieps):
    """(sch, ssx) of the plasmon-pole term for one frequency."""
    wdiff = wx - wt
    w2 = wdiff.real ** 2 + wdiff.imag ** 2 if wdiff.is_complex() else wdiff ** 2
    delw = wt / wdiff
    d2 = delw.real ** 2 + delw.imag ** 2 if delw.is_complex() else delw ** 2
    keep = (w2 > LIMITTWO) & (d2 < LIMITONE)
    zero = torch.zeros((), dtype=wt.dtype, device=wt.device)
    omega2 = wt * wt * ieps
    other = torch.where(d2 > TO1, -omega2 * delw / (4.0 * wt * wt * (delw + 0.5)), zero)
    return torch.where(keep, delw * ieps, zero), torch.where(keep, omega2 / (wx * wx), other)


def _gpp_exact(d, nb, nvb, nc, ng, per_band=False, real=False):
    cv = (lambda t: t) if real else _z
    aqsm, aqsn, vcoul = cv(d["aqsm"]), cv(d["aqsn"]), d["vcoul"]
    igp = torch.tensor(W.gpp_index_maps(nc, ng)[0].astype(np.int64), device="cuda")
    igp = torch.clamp(igp, max=nc - 1)
    m = aqsm[:, igp] if real else aqsm[:, igp].conj()
    v = vcoul[igp]
    dt = aqsm.dtype
    band = torch.zeros((3, nb), dtype=dt, device="cuda")
    occ = torch.zeros((3, max(nvb, 1)), dtype=dt, device="cuda")
    for a, b in _blocks(ng, nc):
        wt, ie = cv(d["wt"][a:b]), cv(d["ieps"][a:b])
        for iw in range(3):
            if not per_band:
                sch, ssx = _pole_factors(float(d["wx"][iw]), wt, ie)
                band[iw] += ((aqsn @ sch.T) * m[:, a:b]) @ (0.5 * v[a:b]).to(dt)
                if nvb:
                    occ[iw, :nvb] += ((aqsn[:nvb] @ ssx.T) * m[:nvb, a:b]) @ v[a:b].to(dt)
            else:
                for n in range(nb):
                    sch, ssx = _pole_factors(d["wx"][n, iw], wt, ie)
                    band[iw, n] += ((sch @ aqsn[n]) * m[n, a:b] * (0.5 * v[a:b])).sum()
                    if n < nvb:
                        occ[iw, n] += ((ssx @ aqsn[n]) * m[n, a:b] * v[a:b]).sum()
    out = {"achtemp": band.sum(1), "asxtemp": occ.sum(1), "acht_n1_loc": band[2]}
    return out if real else {k: torch.view_as_real(x) for k, x in out.items()}


def _halfsum_exact(d, nb, nvb, nc, ng):
    aqsm, aqsn, vcoul = _z(d["aqsm"]), _z(d["aqsn"]), d["vcoul"]
    igp = torch.tensor(W.gpp_index_maps(nc, ng)[0].astype(np.int64), device="cuda")
    igp = torch.clamp(igp, max=nc - 1)
    band = torch.zeros((3, nb), dtype=torch.complex128, device="cuda")
    occ = torch.zeros(3, dtype=torch.complex128, device="cuda")
    stat = torch.zeros((), dtype=torch.complex128, device="cuda")
    ig = torch.arange(nc, device="cuda")
    zero = torch.zeros((), dtype=torch.complex128, device="cuda")
    for a, b in _blocks(ng, nc, 14):
        wt, ie, p, v = _z(d["wt"][a:b]), _z(d["ieps"][a:b]), igp[a:b], vcoul[igp[a:b]].to(torch.complex128)
        m, n, below = aqsm[:, p], aqsn[:, p], ig[None, :] < p[:, None]
        at = torch.arange(b - a, device="cuda")

        def both(rows, z, partner, paired=None):
            """sum over ig of conj(m_p) aqsn z + partner conj(aqsm z), per band of `rows`; `paired`: z of the second part"""
            zz = z if paired is None else paired
            return (aqsn[rows] @ z.T) * m[rows].conj() + partner[rows] * (aqsm[rows] @ zz.T).conj()

        every = slice(0, nb)
        schs = torch.where(below, -ie, zero)
        one = -ie[at, p]
        one = torch.where(one.abs() > TO1, one, zero)
        stat += (((both(every, schs, n) + n * m.conj() * one) @ v) * 0.5).sum()
        unocc, o = slice(nvb, nb), slice(0, nvb)
        cut = torch.cumsum(((wt * wt * ie).abs() < TO1).to(torch.int32), 1) == 0
        for iw in range(3):
            wx = float(d["wx"][iw])
            wdiff = wx - wt
            delw = wt / wdiff
            w2, d2 = wdiff.real ** 2 + wdiff.imag ** 2, delw.real ** 2 + delw.imag ** 2
            z = torch.where((w2 < LIMITTWO) | (d2 > LIMITONE), delw * ie, zero)
            alone = torch.where((p % 512 == 0) & (p > 0), z[at, p], zero)
            z = torch.where((ig[None, :] < p[:, None] - 1) & (ig[None, :] % 512 != 511), z, zero)
            band[iw, nvb:] += 0.5 * ((both(unocc, z, m) + n[unocc] * m[unocc].conj() * alone) @ v)
            if nvb:
                dw = wdiff * 0.5 / wt
                low = (w2 < LIMITTWO) | (dw.real ** 2 + dw.imag ** 2 < TO1)
                ok = below & cut
                sch = torch.where(ok & ~low, wt * ie / wdiff, zero)
                small = torch.where(wt.abs() > TO1, -ie / (4.0 * (1.0 + dw)), zero)
                ssx = torch.where(ok, torch.where(low, small, wt * wt * ie / (wx * wx - wt * wt)), zero)
                pair = ig[None, :] != p[:, None] - 1
                band[iw, :nvb] += 0.5 * (both(o, sch, m, torch.where(pair, sch, zero)) @ v)
                occ[iw] += (both(o, ssx, m, torch.where(pair, ssx, zero)) @ v).sum()
    r = torch.view_as_real
    return {"achtemp": r(band.sum(1)), "asxtemp": r(occ), "acht_n1_loc": r(band[2]), "achstemp": r(stat.reshape(1))}


def _contract(d, name, nf, ng, nc, weight):
    aqsm, aqsn = _z(d["aqsm"]), _z(d["aqsn"])
    m = aqsm[:, :ng].conj() * weight[None, :ng].to(torch.complex128)
    return torch.stack([((aqsn @ _z(d[name][f]).T) * m).sum(1) for f in range(nf)], 1)


def _ff_sigma_exact(s):
    c, d = s["case"], s["d"]
    nb, nf, ne, nvb = c["nb"], c["nf"], c["ne"], c["nvb"]
    one = torch.ones(c["nc"], dtype=torch.float64, device="cuda")
    h = lambda t: t.cpu().numpy()  # noqa: E731
    cr, ca, sd = (h(_contract(d, n, nf, c["ng"], c["nc"], w)) for n, w in
                  (("epsr", d["vcoul"]), ("epsa", d["vcoul"]), ("epsr", one)))
    ekq, grid, pref, brd = h(d["ekq"]), h(d["grid"]), h(d["pref"]), h(_z(d["brd"]))
    occ = (np.arange(nb) < nvb)[:, None]
    e = FMIN - ekq[:, None] + FSTEP * np.arange(ne)[None, :]
    n1 = np.arange(nb)[:, None]
    f = np.searchsorted(grid, np.abs(e), side="right") - 1
    f = np.where((f < 0) | (f > nf - 2), nf - 2, f)
    g0, g1 = grid[f], grid[f + 1]
    w, pos = np.abs(e), e >= 0
    a1, a2 = (g1 - w) / (g1 - g0), np.where(pos, w - g0, -g0 - e) / (g1 - g0)
    asx = np.where(occ, np.where(pos, cr[n1, f] * a1 + cr[n1, f + 1] * a2, ca[n1, f] * a1 + ca[n1, f + 1] * a2), 0)
    delta = -0.5 * ((cr - ca)[n1, f] * a1 + (cr - ca)[n1, f + 1] * (w - g0) / (g1 - g0))
    ach, cor, corb, ach2 = (np.zeros((nb, ne), complex) for _ in range(4))
    for k in range(nf):
        z = sd[:, k][:, None]
        if k < nf - 1:
            ach -= 1j * pref[k] * z / (e - (grid[k] - brd[k]))
            corb -= 1j * pref[k] * z / (e - (np.where(occ, -grid[k], grid[k]) - brd[k]))
        if k > 0:
            zr, zl, left = grid[k], grid[k - 1], sd[:, k - 1][:, None]
            with np.errstate(divide="ignore"):
                t = -np.log(np.clip(np.abs((e - zr) / (e - zl)), 1e-4, 1e4))
                t4 = np.log(np.clip(np.abs((e + zr) / (e + zl)), 1e-4, 1e4))
            ach2 -= 1j * PREF_ZB * 0.5 * (z + left) * t
            slope = (z - left) / (zr - zl)
            lin = np.where(occ, (left + slope * (-FMIN - ekq[:, None] + FSTEP * np.arange(ne) - zl)) * t4,
                           (left + slope * (e - zl)) * t)
            cor -= 1j * PREF_ZB * (lin + z - left)
    ach2 += np.where(pos, delta, 0)
    cor += np.where(pos & ~occ, delta, 0) + np.where(~pos & occ, delta, 0)
    out = np.concatenate([[-0.5 * cr[:, 0].sum()]] + [x.sum(0) for x in (asx, ach, cor, corb, ach2)])
    return torch.view_as_real(torch.tensor(out))


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "host":
        d = _gpp_inputs(seed, c["nb"], c["nc"], c["ng"], c["stress"])
        o = _gpp_exact(d, c["nb"], c["nvb"], c["nc"], c["ng"])
        return {k: v.cpu().numpy().view(np.complex128)[..., 0] for k, v in o.items()}
    if kind == "batch":
        return [_gpp_exact(_gpp_inputs(seed * 64 + i, q["number_bands"], q["ncouls"], q["ngpown"]),
                           q["number_bands"], q["nvband"], q["ncouls"], q["ngpown"]) for i, q in enumerate(_shapes(c))]
    s = prepare(case, seed)
    d = s["d"]
    if kind == "gpp":
        return _gpp_exact(d, c["nb"], c["nvb"], c["nc"], c["ng"], per_band=c["per_band"])
    if kind == "real":
        return _gpp_exact(d, c["nb"], c["nvb"], c["nc"], c["ng"], real=True)
    if kind == "halfsum":
        return _halfsum_exact(d, c["nb"], c["nvb"], c["nc"], c["ng"])
    if kind == "ff":
        one = torch.ones(c["nc"], dtype=torch.float64, device="cuda")
        return torch.view_as_real(_contract(d, "epsr", c["nf"], c["ng"], c["nc"], one))
    return _ff_sigma_exact(s)
