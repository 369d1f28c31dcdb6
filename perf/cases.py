"""The work that is timed when this library is tuned: cases over the range it is used in.

Each case is one call (or the short sequence of calls) that a program makes on data it holds on
the GPU, through the package's public functions:

    chain    ``DsChain.run`` with a plan kept between calls: the whole distributed-scatterer
             chain of one tile or scene (FP64 Gram, refined or FP64 EMI)
    ks       ``ks_test`` then ``select_shp``: the SHP step on its own
    coh      ``emperical_co_pc``: coherence of the DS points, FP32 (the default) or FP64
    raster   ``emperical_co``: covariance and coherence of every pixel
    emi      ``emi``: phase linking of compressed coherence, FP64 (the default) or refined
    tcoh     ``ds_temp_coh`` of a phase history
    ampdisp  ``amp_disp``: the PS-side statistic of a stack

Stacks come from the package's seeded scene generator with the benchmark's scene models (c0 to
c3). The all-FP32 EMI is left out: on these scenes a third of its phases are decided by rounding
(cond(|Gamma|) / gap above 1e6), so two correct builds do not agree on them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import moraine_b200 as mb
from moraine_b200.chain import DsChain
from moraine_b200.synth import CONFIGS, make_stack

P_MAX = 0.05


def listed():
    return [
        # a small tile of the 17-image scene: launches and host work count
        _chain("chain_small_n17", "c0", 64, 64, 17, 5, 5, 20, "refine"),
        # an ordinary request of a tile server, odd sides
        _chain("chain_tile_n50", "c0", 257, 251, 50, 5, 10, 50, "refine"),
        # the benchmark's scene model at a quarter of its area: the largest pass
        _chain("chain_scene_n100", "c2", 1000, 1000, 100, 5, 10, 50, "refine"),
        # a long stack of the tile server (above 128 images), FP64 throughout
        _chain("chain_tile_n150", "c0", 72, 81, 150, 7, 15, 50, "fp64"),
        # SHP selection as the API notebooks run it, p kept, three no-data lines
        {"name": "ks_n41", "kind": "ks", "scene": "c0", "lines": 251, "pixels": 333, "images": 41, "az": 5, "r": 10,
         "nodata": 3},
        # coherence of the DS points: the 15 x 31 window in FP32, the 11 x 21 window in FP64
        {"name": "coh_fp32_n50", "kind": "coh", "scene": "c1", "lines": 200, "pixels": 211, "images": 50, "az": 7,
         "r": 15, "points": 30011, "precision": "fp32"},
        {"name": "coh_fp64_n100", "kind": "coh", "scene": "c2", "lines": 300, "pixels": 300, "images": 100, "az": 5,
         "r": 10, "points": 20000, "precision": "fp64"},
        # full covariance of a raster crop
        {"name": "raster_n20", "kind": "raster", "scene": "c0", "lines": 123, "pixels": 131, "images": 20, "az": 5,
         "r": 5},
        # phase linking of stored coherence: a small batch of a short stack, a large one of a long stack
        {"name": "emi_fp64_n17", "kind": "emi", "points": 1003, "images": 17, "precision": "fp64"},
        {"name": "emi_fp64_n100", "kind": "emi", "points": 4001, "images": 100, "precision": "fp64"},
        # temporal coherence of a long stack, and the amplitude dispersion of a short one
        {"name": "tcoh_n100", "kind": "tcoh", "points": 20011, "images": 100},
        {"name": "ampdisp_n30", "kind": "ampdisp", "scene": "c0", "lines": 700, "pixels": 701, "images": 30},
    ]


def _chain(name, scene, lines, pixels, images, az, r, min_shp, emi):
    return {"name": name, "kind": "chain", "scene": scene, "lines": lines, "pixels": pixels, "images": images,
            "az": az, "r": r, "min_shp": min_shp, "emi": emi}


WINDOWS = ((5, 5), (5, 10), (7, 15))  # the half windows of the scene configurations


def draw(rng):
    kind = rng.choice(("chain",) * 4 + ("ks",) * 2 + ("coh",) * 3 + ("raster", "tcoh", "ampdisp") + ("emi",) * 3)
    n = _log(rng, 12, 128)
    az, r = rng.choice(WINDOWS)
    case = {"kind": kind, "images": n}
    if kind == "chain":
        if rng.random() < 0.25:
            n = case["images"] = _log(rng, 129, 200)
        emi = "refine" if n <= 128 and rng.random() < 0.7 else "fp64"
        most = 6e3 * (150 / n) ** 3 if n > 128 else (2.5e5 if emi == "refine" else 1e5) * min(4.0, (100 / n) ** 2)
        case.update(scene=rng.choice(("c0", "c1", "c2")), az=az, r=r, min_shp=rng.choice((20, 50)), emi=emi,
                    **_sides(rng, 48 * 48, most))
    elif kind == "ks":
        case.update(scene="c0", az=az, r=r, nodata=rng.choice((0, 3)), **_sides(rng, 48 * 48, 1.5e5))
    elif kind == "coh":
        case.update(scene=rng.choice(("c0", "c1", "c2")), az=az, r=r, precision=rng.choice(("fp32", "fp64")),
                    **_sides(rng, 64 * 64, 9e4))
        case.update(points=_log(rng, 200, case["lines"] * case["pixels"] // 3))
    elif kind == "raster":
        n = case["images"] = _log(rng, 8, 40)
        case.update(scene="c0", az=az, r=r, **_sides(rng, 32 * 32, 6.4e6 / n ** 2))
    elif kind == "emi":
        if rng.random() < 0.15:
            n = case["images"] = _log(rng, 129, 200)
        most = 2e3 if n > 128 else min(5e4, 4e3 * (100 / n) ** 2)
        case.update(points=_log(rng, 200, int(most)), precision=rng.choice(("fp64", "refine")))
    elif kind == "tcoh":
        case.update(points=_log(rng, 300, int(min(2e5, 2e4 * (100 / n) ** 2))))
    else:
        case.update(scene="c0", **_sides(rng, 64 * 64, 1.5e7 / n))
    return case


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    area = math.exp(rng.uniform(math.log(lo), math.log(max(hi, lo + 1))))
    lines = max(16, int(math.sqrt(area * math.exp(rng.uniform(-0.7, 0.7)))))
    return {"lines": lines, "pixels": max(16, int(area / lines))}


# ------------------------------------------------------------------ what a program has in hand
def _stack(case, seed):
    """The scene model's stack at this case's size, with its patch density."""
    base = CONFIGS[case["scene"]]
    lines, pixels = case["lines"], case["pixels"]
    patches = max(4, round(base.n_patches * lines * pixels / (base.nlines * base.width)))
    return make_stack(base.scaled(nlines=lines, width=pixels, nimages=case["images"], n_patches=patches, seed=seed),
                      "cuda")


def _intensity(rslc):
    re, im = rslc.real.contiguous(), rslc.imag.contiguous()
    return re * re + im * im


def _shps(case, rslc):
    return mb.select_shp(mb.ks_test(_intensity(rslc), case["az"], case["r"]), P_MAX)


def _coherence_points(case, seed):
    """Compressed coherence (points, pairs) of points with 50 to 231 looks each, from circular
    Gaussian looks of the c2 model's temporal covariance and a deformation ramp."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n, points = case["images"], case["points"]
    t = np.arange(n) * 12.0
    lag = np.abs(t[:, None] - t[None, :])
    gamma = np.where(lag == 0, 1.0, 0.5 * np.exp(-lag / 36.0) + 0.05)
    chol = torch.from_numpy(np.linalg.cholesky(gamma)).to("cuda", torch.complex128)
    m, j = np.triu_indices(n, 1)
    m, j = torch.from_numpy(m).cuda(), torch.from_numpy(j).cuda()
    out = torch.empty((points, len(m)), dtype=torch.complex64, device="cuda")
    step = max(1, int(2e7) // (231 * n))
    for p0 in range(0, points, step):
        k = min(step, points - p0)
        looks = torch.randint(50, 232, (k, 1), generator=gen, device="cuda")
        w = torch.randn((k, 231, n, 2), generator=gen, device="cuda", dtype=torch.float32)
        z = torch.view_as_complex(w).to(torch.complex128) @ chol.T
        z = z * (torch.arange(231, device="cuda")[None] < looks)[:, :, None]
        rate = torch.rand((k, 1, 1), generator=gen, device="cuda", dtype=torch.float64)
        z = z * torch.exp(-1j * rate * torch.from_numpy(t).cuda() * (4 * math.pi * 50 / 56 / 365.25))
        gram = z.transpose(1, 2) @ z.conj()
        amp = gram.diagonal(dim1=1, dim2=2).real.sqrt()
        out[p0:p0 + k] = (gram / (amp[:, :, None] * amp[:, None, :]))[:, m, j].to(torch.complex64)
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "chain":
        rslc = _stack(case, seed)
        plan = DsChain(case["lines"], case["pixels"], case["images"], case["az"], case["r"], P_MAX, case["min_shp"],
                       precision="fp64", emi_precision=case["emi"])
        # where the program gathers the DS points' results (the plan reuses its own buffers)
        npix, n = case["lines"] * case["pixels"], case["images"]
        got = {"idx": torch.zeros((npix, 2), dtype=torch.int32, device="cuda"),
               "ph": torch.zeros((npix, n), dtype=torch.complex64, device="cuda"),
               "quality": torch.zeros((npix,), device="cuda"), "t_coh": torch.zeros((npix,), device="cuda")}
        return {"kind": kind, "rslc": rslc, "plan": plan, "got": got}
    if kind == "ks":
        rmli = _intensity(_stack(case, seed))
        rmli[:case["nodata"]] = math.nan
        return {"kind": kind, "rmli": rmli, "az": case["az"], "r": case["r"]}
    if kind == "coh":
        rslc = _stack(case, seed)
        is_shp, shp_num = _shps(case, rslc)
        idx, pc_is_shp = _candidates(shp_num, is_shp, 50)
        pick = torch.arange(case["points"], device="cuda") * idx.shape[0] // case["points"]  # evenly over the scene
        return {"kind": kind, "rslc": rslc, "idx": idx[pick], "pc_is_shp": pc_is_shp[pick],
                "precision": case["precision"]}
    if kind == "raster":
        rslc = _stack(case, seed)
        return {"kind": kind, "rslc": rslc, "is_shp": _shps(case, rslc)[0]}
    if kind == "emi":
        return {"kind": kind, "coh": _coherence_points(case, seed), "precision": case["precision"]}
    if kind == "tcoh":
        coh = _coherence_points(case, seed)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed + 1)
        ang = torch.rand((case["points"], case["images"]), generator=gen, device="cuda") * (2 * math.pi)
        return {"kind": kind, "coh": coh, "ph": torch.polar(torch.ones_like(ang), ang)}
    return {"kind": kind, "rslc": _stack(case, seed)}


def _candidates(shp_num, is_shp, min_shp):
    """DS points as the notebooks write them: indices and their masks."""
    sel = shp_num >= min_shp
    return torch.nonzero(sel).to(torch.int32), is_shp[sel]


def run(state):
    kind = state["kind"]
    if kind == "chain":
        res, got = state["plan"].run(state["rslc"]), state["got"]
        for key, to in got.items():
            to[:res.n_ds].copy_(getattr(res, key))
        return {**got, "shp_num": res.shp_num, "is_shp": res.is_shp}
    if kind == "ks":
        p = mb.ks_test(state["rmli"], state["az"], state["r"])
        is_shp, shp_num = mb.select_shp(p, P_MAX)
        return {"p": p, "is_shp": is_shp, "shp_num": shp_num}
    if kind == "coh":
        return {"coh": mb.emperical_co_pc(state["rslc"], state["idx"], state["pc_is_shp"],
                                          precision=state["precision"])}
    if kind == "raster":
        cov, coh = mb.emperical_co(state["rslc"], state["is_shp"])
        return {"cov": cov, "coh": coh}
    if kind == "emi":
        ph, quality = mb.emi(state["coh"], precision=state["precision"])
        return {"ph": ph, "quality": quality}
    if kind == "tcoh":
        return {"t_coh": mb.ds_temp_coh(state["coh"], state["ph"])}
    return {"amp_disp": mb.amp_disp(state["rslc"])}


# ------------------------------------------------------------------ what a pass cannot do without
# Share of the pixels that become DS points and the mean SHP share of their windows, as measured
# on the scene models (min_shp 50; 20 gives about 0.5).
DS_SHARE = {"c0": 0.13, "c1": 0.75, "c2": 0.27, "c3": 0.75}
SHP_SHARE = 0.4


def work(case):
    kind, n = case["kind"], case["images"]
    q = n * (n - 1) // 2
    emi_flops = 2.7 * n ** 3 + 80 * n ** 2  # factorisations of |Gamma| and M, solves, per point
    if kind == "emi":
        return {"bytes": case["points"] * (8 * q + 8 * n + 4), "flops": case["points"] * emi_flops}
    if kind == "tcoh":
        return {"bytes": case["points"] * (8 * q + 8 * n + 4), "flops": case["points"] * 20 * q}
    npix = case["lines"] * case["pixels"]
    if kind == "ampdisp":
        return {"bytes": npix * (8 * n + 4), "flops": npix * 6 * n}
    win = (2 * case["az"] + 1) * (2 * case["r"] + 1)
    if kind == "ks":
        return {"bytes": npix * (4 * n + 5 * win + 4), "flops": 0}
    looks = SHP_SHARE * win
    if kind == "raster":
        return {"bytes": npix * (8 * n + win + 16 * n * n), "flops": npix * 4 * looks * n * n}
    if kind == "coh":
        points = case["points"]
        return {"bytes": npix * 8 * n + points * (win + 8 + 8 * q), "flops": points * 8 * looks * q}
    ds = npix * (0.5 if case["min_shp"] < 50 else DS_SHARE[case["scene"]])
    return {"bytes": npix * (8 * n + win + 4) + ds * (8 * n + 16), "flops": ds * (8 * looks * q + emi_flops)}


# ------------------------------------------------------------------ the same in 64 bits
def _few(points, n):
    """Whether eigh of this many points stays within seconds (above 32 images it goes matrix by matrix)."""
    return points <= (50000 if n <= 32 else 5000 if n <= 128 else 3000)


def exact(case, seed):
    kind = case["kind"]
    if kind == "emi" and not _few(case["points"], case["images"]):
        return None
    if kind == "chain" and not _few(case["lines"] * case["pixels"] // 2, case["images"]):
        return None
    state = prepare(case, seed)
    if kind == "emi":
        ph, quality = _emi64(state["coh"])
        return {"ph": ph, "quality": quality}
    if kind == "tcoh":
        return {"t_coh": _tcoh64(state["coh"], state["ph"].to(torch.complex128))}
    if kind == "ampdisp":
        amp = state["rslc"].to(torch.complex128).abs()
        return {"amp_disp": amp.std(-1, correction=0) / amp.mean(-1)}
    if kind == "ks":
        return {"p": _ks64(state["rmli"], state["az"], state["r"]), "is_shp": None, "shp_num": None}
    if kind == "coh":
        return {"coh": _coherence64(state["rslc"], state["idx"], state["pc_is_shp"])[0]}
    if kind == "raster":
        lines, pixels, n = state["rslc"].shape
        at = torch.cartesian_prod(torch.arange(lines), torch.arange(pixels)).cuda()
        full, cov = _coherence64(state["rslc"], at, state["is_shp"].flatten(0, 1), full=True)
        return {"cov": cov.reshape(lines, pixels, n, n), "coh": full.reshape(lines, pixels, n, n)}
    rslc = state["rslc"]
    is_shp = _ks64(_intensity(rslc), case["az"], case["r"]).to(torch.float32).double() < P_MAX
    coh = _coherence64(rslc, *_candidates(is_shp.sum((-2, -1)), is_shp, case["min_shp"]))[0]
    coh = coh.to(torch.complex64)  # the type that coherence has between the steps
    got = {"idx": None, "shp_num": None, "is_shp": None}
    ph, quality = _emi64(coh)
    for key, v in (("ph", ph), ("quality", quality), ("t_coh", _tcoh64(coh, ph))):
        got[key] = v.new_zeros((case["lines"] * case["pixels"],) + v.shape[1:])
        got[key][:len(v)] = v
    return got


def _ks64(x, az, r):
    """The KS test's p of every pixel against its window, NaN outside the image and at no data."""
    lines, pixels, n = x.shape
    x = x.sort(-1).values
    en = math.sqrt(n / 2)
    table = torch.tensor([_ks_p((en + 0.12 + 0.11 / en) * k / n) for k in range(n + 1)], dtype=torch.float64).cuda()
    p = torch.full((lines, pixels, 2 * az + 1, 2 * r + 1), math.nan, dtype=torch.float64, device="cuda")
    for da in range(-az, az + 1):
        for dr in range(-r, r + 1):
            a0, a1, r0, r1 = max(0, -da), min(lines, lines - da), max(0, -dr), min(pixels, pixels - dr)
            if a0 >= a1 or r0 >= r1:
                continue
            a = x[a0:a1, r0:r1].contiguous()
            b = x[a0 + da:a1 + da, r0 + dr:r1 + dr].contiguous()
            k = torch.zeros(a.shape[:2], dtype=torch.int64, device="cuda")
            for v in (a, b):
                gap = torch.searchsorted(a, v, right=True) - torch.searchsorted(b, v, right=True)
                k = torch.maximum(k, gap.abs().amax(-1))
            ok = ~(a[..., -1].isnan() | b[..., -1].isnan())
            p[a0:a1, r0:r1, da + az, dr + r] = torch.where(ok, table[k.clamp(max=n)], math.nan)
    return p


def _ks_p(x):
    p = before = 0.0
    sign = 1
    for i in range(1, 101):
        p += sign * 2 * math.exp(-2 * x * x * i * i)
        if p == before:
            break
        sign, before = -sign, p
    return p


def _coherence64(rslc, idx, mask, full=False):
    """(points, pairs) coherence; with `full` (points, N, N) coherence and covariance."""
    lines, pixels, n = rslc.shape
    az_win, r_win = mask.shape[-2:]
    idx = idx.long()
    m, j = np.triu_indices(n, 1)
    m, j = torch.from_numpy(m).cuda(), torch.from_numpy(j).cuda()
    coh, cov = [], []
    step = max(1, int(3e7) // (az_win * r_win * n + n * n))
    for p0 in range(0, idx.shape[0], step):
        at = idx[p0:p0 + step]
        la = at[:, 0, None, None] + (torch.arange(az_win) - az_win // 2).cuda()[:, None]
        lr = at[:, 1, None, None] + (torch.arange(r_win) - r_win // 2).cuda()
        ok = mask[p0:p0 + step].bool() & (la >= 0) & (la < lines) & (lr >= 0) & (lr < pixels)
        z = rslc[la.clamp(0, lines - 1), lr.clamp(0, pixels - 1)].to(torch.complex128) * ok[..., None]
        z = z.flatten(1, 2)
        gram = z.transpose(1, 2) @ z.conj()
        amp = gram.diagonal(dim1=1, dim2=2).real.sqrt()
        gamma = gram / (amp[:, :, None] * amp[:, None, :])
        coh.append(gamma if full else gamma[:, m, j])
        if full:
            cov.append(gram / ok.sum((1, 2))[:, None, None])
    return torch.cat(coh), torch.cat(cov) if full else None


def _emi64(coh):
    points, q = coh.shape
    n = (1 + math.isqrt(1 + 8 * q)) // 2
    m, j = np.triu_indices(n, 1)
    m, j = torch.from_numpy(m).cuda(), torch.from_numpy(j).cuda()
    ph = torch.empty((points, n), dtype=torch.complex128, device="cuda")
    quality = torch.empty((points,), dtype=torch.float64, device="cuda")
    step = max(1, int(2e7) // (n * n))
    for p0 in range(0, points, step):
        c = coh[p0:p0 + step].to(torch.complex128)
        g = torch.eye(n, dtype=torch.complex128, device="cuda").repeat(c.shape[0], 1, 1)
        g[:, m, j] = c
        g[:, j, m] = c.conj()
        lam, v = torch.linalg.eigh(torch.linalg.inv(g.abs()) * g)
        v = v[:, :, 0] * v[:, :1, 0].conj()
        ph[p0:p0 + step] = v / v.abs()
        quality[p0:p0 + step] = lam[:, 0]
    return ph, quality


def _tcoh64(coh, ph):
    n = ph.shape[1]
    m, j = np.triu_indices(n, 1)
    m, j = torch.from_numpy(m).cuda(), torch.from_numpy(j).cuda()
    out = []
    step = max(1, int(3e7) // len(m))
    for p0 in range(0, coh.shape[0], step):
        c, p = coh[p0:p0 + step].to(torch.complex128), ph[p0:p0 + step]
        out.append((c / c.abs() * p[:, m].conj() * p[:, j]).sum(-1).abs() / len(m))
    return torch.cat(out)
