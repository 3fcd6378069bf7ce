"""What a user of this library has it do, as timed cases.

Each case is one call sequence through the public classes (FBP3D, FBP2D) on
data that is resident on the GPU: reconstruct a 2D slice from a parallel-beam
or fan-beam sinogram, rebin a fan-beam sinogram first, reconstruct a volume
from cone-beam projections or from parallel-beam sinograms, forward project a
volume. Inputs are projections of random ellipsoids, with photon noise where
the scan is a measured one. `exact` restates every path with torch in FP64.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "3dfilteredbackprojection-public_b200"))
import fbp_b200 as F  # noqa: E402

DEV = "cuda"
PRECISIONS = {"fp32": F.Precision.FP32, "mixed": F.Precision.MIXED, "mixed24": F.Precision.MIXED24}
RAM_LAK, SHEPP_LOGAN, COSINE, HANN = 0, 1, 2, 3


def slice2d(kind, edge, views, bins, filt, precision, det_width, vol_width, turns=1.0, sod=0.0, odd=0.0, i0=0.0,
            offset=0.0):
    return {"op": "slice2d", "kind": kind, "edge": edge, "views": views, "bins": bins, "filter": filt,
            "precision": precision, "det_width": float(det_width), "vol_width": float(vol_width),
            "turns": float(turns), "sod": float(sod), "odd": float(odd), "i0": float(i0), "offset": float(offset)}


def cone(edge, height, views, cols, rows, filt, precision, det_width, vol_width, sod, odd, i0=0.0, counts=False,
         offset=0.0):
    return {"op": "cone", "edge": edge, "height": height, "views": views, "cols": cols, "rows": rows, "filter": filt,
            "precision": precision, "det_width": float(det_width), "vol_width": float(vol_width),
            "sod": float(sod), "odd": float(odd), "i0": float(i0), "counts": counts, "offset": float(offset),
            "turns": 1.0}


def parallel3d(edge, height, views, cols, rows, filt, precision, turns=0.5):
    return {"op": "parallel3d", "edge": edge, "height": height, "views": views, "cols": cols, "rows": rows,
            "filter": filt, "precision": precision, "turns": float(turns), "offset": 0.0}


def forward(edge, height, views, det_width, vol_width, sod, odd):
    return {"op": "forward", "edge": edge, "height": height, "views": views, "det_width": float(det_width),
            "vol_width": float(vol_width), "sod": float(sod), "odd": float(odd), "turns": 1.0, "offset": 0.0}


def serving_cone(edge, views, precision):
    """A cone-beam request of the mixed serving stream: 1 mm voxels, magnification 1.5, detector 1.5 x edge."""
    det = edge * 3 // 2
    return cone(edge, edge, views, det, det, RAM_LAK, precision, 1.5 * det, edge, 3.0 * edge, 1.5 * edge)


def listed():
    out = {
        # one slice of a parallel-beam scan at the benchmark's smallest size: launches and latency count
        "parallel2d_256_fp32": slice2d("parallel", 256, 360, 367, RAM_LAK, "fp32", 367, 256, turns=0.5),
        # the benchmark's fan-beam slice with photon noise
        "fan2d_512_fp32": slice2d("fan", 512, 720, 768, SHEPP_LOGAN, "fp32", 768, 256, sod=500, odd=500, i0=1e5),
        # the largest slice of the serving stream, filtered on the tensor cores
        "fan2d_1024_mixed": slice2d("fan", 1024, 1440, 1536, SHEPP_LOGAN, "mixed", 768, 256, sod=500, odd=500,
                                    i0=1e5),
        # the reference's fan-beam program: rebin to parallel beam, filter, backproject
        "fan_rebin_512_fp32": dict(slice2d("fan", 512, 720, 768, SHEPP_LOGAN, "fp32", 768, 256, sod=500, odd=500),
                                   op="rebin"),
        # simulated scan: cone-beam projections of a volume
        "forward_cone_256": forward(256, 256, 360, 256 * 1.75, 256, 750, 450),
        # the smallest volume of the serving stream
        "cone_128_mixed": serving_cone(128, 360, "mixed"),
        # the benchmark's 256^3 scan in the plain FP32 form
        "cone_256_fp32": cone(256, 256, 360, 384, 384, RAM_LAK, "fp32", 384 * 1.6, 256, 750, 450),
        # a measured scan as it comes: photon counts, sizes that are multiples of nothing, a start angle
        "cone_ragged_fp32": cone(300, 251, 450, 421, 371, COSINE, "fp32", 421 * 1.2, 300, 640, 310, i0=2e4,
                                 counts=True, offset=0.35),
        # a mid-size scan in the 24-bit form
        "cone_512_mixed24": serving_cone(512, 720, "mixed24"),
        # the volume that takes most of the serving stream's time
        "cone_768_mixed": serving_cone(768, 1024, "mixed"),
        # the headline geometry at 2/3 scale (the detector does not see the whole volume), noisy, plain FP32 form
        "cone_960_fp32": cone(960, 980, 960, 1024, 1024, HANN, "fp32", 1024 * 0.381, 288, 400, 400, i0=5e4),
        # synchrotron-style stack of parallel-beam sinograms over half a turn
        "parallel3d_256_mixed": parallel3d(256, 256, 360, 367, 256, SHEPP_LOGAN, "mixed"),
    }
    return [dict(case, name=name) for name, case in out.items()]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges; a cone-beam case costs at most the largest listed one."""
    op = rng.choice(["slice2d", "slice2d", "rebin", "forward", "cone", "cone", "cone", "parallel3d"])
    precision = rng.choice(["fp32", "mixed", "mixed24"])
    filt = rng.randrange(4)
    if op in ("slice2d", "rebin"):
        edge, views, bins = log_int(rng, 200, 1024), rng.randrange(300, 1441), rng.randrange(300, 1537)
        if op == "slice2d" and rng.random() < 0.4:
            width = float(edge)
            return slice2d("parallel", edge, views, bins, filt, precision, 1.42 * width, width,
                           turns=rng.choice([0.5, 1.0]), offset=rng.uniform(0, 1))
        case = slice2d("fan", edge, views, bins, filt, precision, 768, 256, sod=rng.randrange(400, 700), odd=500,
                       i0=rng.choice([0.0, 1e5]), offset=rng.uniform(0, 1))
        return dict(case, op=op)
    if op == "forward":
        edge = log_int(rng, 64, 288)
        return forward(edge, max(1, int(edge * rng.uniform(0.5, 1.1))), rng.randrange(90, 361), 1.7 * edge, edge,
                       rng.uniform(2.0, 4.0) * edge, rng.uniform(1.0, 2.0) * edge)
    if op == "parallel3d":
        edge = log_int(rng, 96, 400)
        return parallel3d(edge, max(1, int(edge * rng.uniform(0.5, 1.1))), rng.randrange(180, 721),
                          int(edge * rng.uniform(1.0, 1.45)), edge, filt, precision, rng.choice([0.5, 1.0]))
    edge = log_int(rng, 96, 640)
    height, views = max(1, int(edge * rng.uniform(0.6, 1.1))), log_int(rng, 240, 900)
    if rng.random() < 0.6:  # the usual case: sizes of whole tiles, views in quarters of a turn
        edge, views = max(96, edge // 32 * 32), views // 4 * 4
    cols = int(edge * rng.uniform(1.0, 1.6))
    rows = int(cols * rng.uniform(0.8, 1.0))
    sod, odd = rng.uniform(1.6, 3.5) * edge, rng.uniform(0.4, 2.0) * edge
    width = 1.45 * edge * (sod + odd) / sod * rng.choice([1.0, 1.0, 0.7])
    return cone(edge, height, views, cols, rows, filt, precision, width, edge, sod, odd,
                i0=rng.choice([0.0, 5e4]), counts=rng.random() < 0.3, offset=rng.choice([0.0, rng.uniform(0, 6)]))


# ------------------------------------------------------------------------------------------------- inputs
def f32(x):
    """A length as the library gets it (C float)."""
    return float(np.float32(x))


def geometry_of(case):
    """Lengths, pitches and view angles in FP64, as the library forms them from its float arguments."""
    g = {"K": case["views"], "angles": f32(case["offset"]) + 2.0 * math.pi * f32(case["turns"]) *
         np.arange(case["views"]) / case["views"]}
    op = case["op"]
    g["cone"] = op in ("cone", "forward", "rebin") or case.get("kind") == "fan"
    if op in ("slice2d", "rebin"):
        g.update(nu=case["bins"], nv=1, nx=case["edge"], ny=1)
    elif op == "forward":
        g.update(nu=case["edge"], nv=case["height"], nx=case["edge"], ny=case["height"])
    else:
        g.update(nu=case["cols"], nv=case["rows"], nx=case["edge"], ny=case["height"])
    if op == "parallel3d":  # the detector spans the volume
        g.update(vox=1.0, du=case["edge"] / case["cols"], dv=case["height"] / case["rows"])
    else:
        g["du"] = g["dv"] = f32(case["det_width"]) / g["nu"]
        g["vox"] = f32(case["vol_width"]) / g["nx"]
    if g["cone"]:
        g.update(sod=f32(case["sod"]), sdd=f32(case["sod"]) + f32(case["odd"]))
    return g


def ellipsoids(rng, count):
    """Random ellipsoids in a ball of radius 1: (density, axes, centre, rotation)."""
    out = []
    for _ in range(count):
        c = rng.standard_normal(3)
        c *= 0.65 * rng.random() ** (1 / 3) / np.linalg.norm(c)
        q, r = np.linalg.qr(rng.standard_normal((3, 3)))
        out.append((rng.uniform(-0.2, 1.0), rng.uniform(0.08, 0.35, 3), c, q * np.sign(np.diag(r))))
    return out


def project(case, seed):
    """Line integrals [view][v][u] (FP32) of 12 random ellipsoids that fill the volume's cross-section.

    For one view and ellipsoid the discriminant of the ray-ellipsoid equation is a quadratic polynomial in the
    detector coordinates; it is evaluated about the centre of the ellipsoid's shadow. Lengths are in units of half
    the volume's width.
    """
    g = geometry_of(case)
    rng = np.random.default_rng(seed)
    R = 0.5 * g["nx"] * g["vox"]
    flat = g["nv"] == 1
    shapes = ellipsoids(rng, 12)
    u = torch.tensor((np.arange(g["nu"]) + 0.5 - 0.5 * g["nu"]) * g["du"] / R, device=DEV)
    v = torch.tensor((np.arange(g["nv"]) + 0.5 - 0.5 * g["nv"]) * g["dv"] / R, device=DEV)
    out = torch.empty((g["K"], g["nv"], g["nu"]), dtype=torch.float32, device=DEV)
    step = max(1, min(g["K"], (1 << 25) // (g["nu"] * g["nv"])))
    for k0 in range(0, g["K"], step):
        t = g["angles"][k0:k0 + step]
        co, si, ze = np.cos(t), np.sin(t), np.zeros_like(t)
        d, eu, ey = np.stack([co, ze, si], 1), np.stack([-si, ze, co], 1), np.stack([ze, ze + 1, ze], 1)
        p = out[k0:k0 + step]
        p.zero_()
        for rho, axes, centre, rot in shapes:
            if flat:
                centre = centre * np.array([1, 0, 1])  # a slice through the middle
            M = (rot / axes).T  # world -> unit ball
            to = lambda w: w @ M.T  # noqa: E731
            if g["cone"]:  # ray o + s w, o = the source, w = w0 + u eu + v ey
                q0, qu, qv = to(-d * (g["sod"] / R) - centre), 0 * d, 0 * d
                w0, wu, wv = to(d * (g["sdd"] / R)), to(eu), to(ey)
            else:  # o = u eu + v ey, w = d
                q0, qu, qv = to(0 * d - centre), to(eu), to(ey)
                w0, wu, wv = to(d), 0 * d, 0 * d
            dot = lambda x, y: (x * y).sum(1)  # noqa: E731
            # A = |w|^2; B = q.w and C = |q|^2 - 1 are at most linear and constant (cone) or linear and quadratic
            a = [dot(w0, w0), 2 * dot(w0, wu), 2 * dot(w0, wv), dot(wu, wu), 2 * dot(wu, wv), dot(wv, wv)]
            b0, bu, bv = dot(q0, w0), dot(q0, wu) + dot(qu, w0), dot(q0, wv) + dot(qv, w0)
            c = [dot(q0, q0) - 1, 2 * dot(q0, qu), 2 * dot(q0, qv), dot(qu, qu), 2 * dot(qu, qv), dot(qv, qv)]
            bb = [b0 * b0, 2 * b0 * bu, 2 * b0 * bv, bu * bu, 2 * bu * bv, bv * bv]
            # disc = B^2 - A C, one of A and C being constant
            e = [x - (a[i] * c[0] if g["cone"] else a[0] * c[i]) for i, x in enumerate(bb)]
            det = 4 * e[3] * e[5] - e[4] * e[4]
            uc, vc = (e[4] * e[2] - 2 * e[5] * e[1]) / det, (e[4] * e[1] - 2 * e[3] * e[2]) / det
            top = e[0] + 0.5 * (e[1] * uc + e[2] * vc)
            T = lambda x: torch.tensor(x, device=DEV)[:, None]  # noqa: E731
            U, V = u[None] - T(uc), v[None] - T(vc)
            disc = ((T(top) + T(e[3]) * U * U).float()[:, None, :] + (T(e[5]) * V * V).float()[:, :, None])
            disc.addcmul_((T(e[4]) * V).float()[:, :, None], U.float()[:, None, :])
            disc.clamp_(min=0).sqrt_()
            A = ((T(a[0]) + T(a[1]) * u + T(a[3]) * u * u).float()[:, None, :] +
                 (T(a[2]) * v + T(a[5]) * v * v).float()[:, :, None])
            A.addcmul_((T(a[4]) * v).float()[:, :, None], u.float()[None, None, :])
            p.addcdiv_(disc, A, value=2 * rho)
        if g["cone"]:
            p.mul_(((g["sdd"] / R) ** 2 + (u * u)[None, :] + (v * v)[:, None]).sqrt().float())
    if case.get("i0"):
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed)
        for k0 in range(0, g["K"], step):
            p = out[k0:k0 + step]
            mean = torch.exp(-p).mul_(case["i0"])
            p.copy_(mean.add_(mean.sqrt().mul_(torch.randn(p.shape, generator=gen, device=DEV))).round_().clamp_(min=1))
            if not case.get("counts"):
                p.div_(case["i0"]).log_().neg_()
    elif case.get("counts"):
        out.neg_().exp_().mul_(1000.0)
    return out


def base_of(case):
    return case["i0"] or 1000.0


def volume(case, seed):
    """A volume [z][y][x] of random ellipsoids with smooth texture."""
    rng = np.random.default_rng(seed)
    n, h = case["edge"], case["height"]
    x = torch.tensor((np.arange(n) + 0.5) / (0.5 * n) - 1, dtype=torch.float32, device=DEV)
    y = torch.tensor((np.arange(h) + 0.5 - 0.5 * h) / (0.5 * n), dtype=torch.float32, device=DEV)
    vol = torch.zeros((n, h, n), dtype=torch.float32, device=DEV)
    for rho, axes, c, rot in ellipsoids(rng, 12):
        M = (rot / axes).T
        r2 = 0
        for i in range(3):
            q = (float(M[i, 2]) * (x - c[2]))[:, None, None] + (float(M[i, 1]) * (y - c[1]))[None, :, None] + \
                (float(M[i, 0]) * (x - c[0]))[None, None, :]
            r2 = r2 + q * q
        vol += torch.where(r2 < 1, rho * (1 - 0.1 * r2), 0.0)
    return vol


def inputs(case, seed):
    if case["op"] == "forward":
        return volume(case, seed)
    p = project(case, seed)
    if case["op"] in ("slice2d", "rebin"):
        return p[:, 0].contiguous()
    return p.transpose(0, 1).contiguous() if case["op"] == "parallel3d" else p


# ------------------------------------------------------------------------------------------------- the calls
def prepare(case, seed):
    s = {"case": case, "raw": inputs(case, seed), "stream": torch.cuda.Stream()}
    s["stream"].wait_stream(torch.cuda.current_stream())
    s["fbp"] = F.FBP3D(0)
    s["fbp"].set_stream(s["stream"])
    op, n = case["op"], case["edge"]
    if op != "forward":
        s["fbp"].set_precision(PRECISIONS[case["precision"]])
    if op in ("slice2d", "rebin"):
        s["fbp2d"] = F.FBP2D(0, context=s["fbp"].ctx)
        s["work"] = torch.empty_like(s["raw"])
        s["out"] = torch.empty((n, n), dtype=torch.float32, device=DEV)
        if case["kind"] == "fan":
            s["geom"] = F.Geometry.cone(case["sod"], case["odd"], case["det_width"], case["vol_width"],
                                        case["turns"], case["offset"])
        else:
            s["geom"] = F.Geometry.parallel(case["det_width"], case["vol_width"], case["turns"], case["offset"])
        if op == "rebin":  # the same pitch at the isocentre
            s["width"] = case["det_width"] * case["sod"] / (case["sod"] + case["odd"])
            s["parallel"] = F.Geometry.parallel(s["width"], case["vol_width"], case["turns"], case["offset"])
    elif op == "forward":
        s["fbp"].generate_blank_volume(n, case["height"], n)
        s["fbp"].write_volume_data(s["raw"])
        s["out"] = torch.empty((case["views"], case["height"], n), dtype=torch.float32, device=DEV)
    else:
        s["out"] = torch.empty((n, case["height"], n), dtype=torch.float32, device=DEV)
    return s


def run(s):
    case, fbp = s["case"], s["fbp"]
    op = case["op"]
    if op == "slice2d":
        with torch.cuda.stream(s["stream"]):
            sino = s["work"].copy_(s["raw"])  # the filter works in place
        fan = case["kind"] == "fan"
        f = s["fbp2d"].apply_filter(sino, case["filter"], case["sod"] + case["odd"] if fan else 0.0,
                                    case["det_width"] if fan else 0.0)
        return s["fbp2d"].project_backward(f, s["geom"], (case["edge"], case["edge"]), out=s["out"])
    if op == "rebin":
        with torch.cuda.stream(s["stream"]):
            sino = s["fbp2d"].parallelize_fan_beam_sinogram(s["raw"], s["geom"], case["bins"], s["width"])
        f = s["fbp2d"].apply_filter(sino, case["filter"])
        return s["fbp2d"].project_backward(f, s["parallel"], (case["edge"], case["edge"]), out=s["out"])
    if op == "forward":
        fbp.project_forward_cone_to_projections(case["sod"], case["odd"], case["det_width"], case["vol_width"],
                                                case["turns"], case["views"], case["offset"])
        return fbp.download_projections(s["out"])
    if op == "parallel3d":
        fbp.upload_sinograms(s["raw"])
        fbp.apply_filter_to_sinograms(case["filter"])
        fbp.project_backward_parallel_from_sinograms(case["turns"], case["edge"], case["height"], case["offset"])
        return fbp.read_volume(s["out"])
    fbp.upload_projections(s["raw"])
    if case["counts"]:
        fbp.log_normalize_projections(base_of(case))
    fbp.apply_fdk_weights_to_projections(case["sod"], case["odd"], case["det_width"])
    fbp.apply_filter_to_projections(case["filter"])
    fbp.project_backward_cone_fdk_from_projections(case["sod"], case["odd"], case["det_width"], case["vol_width"],
                                                   case["turns"], case["edge"], case["height"], case["offset"])
    return fbp.read_volume(s["out"])


def work(case):
    """Inputs read and results written once; a bilinear tap and its weighted sum are 10 operations, a trilinear
    sample 22, a row filter two transforms of the padded row."""
    g = geometry_of(case)
    rows, voxels = g["K"] * g["nv"], g["nx"] * g["nx"] * g["ny"]
    if case["op"] == "forward":
        # half a voxel per step over a mean chord of about three quarters of the width
        return {"bytes": 4 * (voxels + rows * g["nu"]), "flops": 22 * rows * g["nu"] * 1.5 * g["nx"]}
    n = padded(g["nu"])
    return {"bytes": 4 * (voxels + rows * g["nu"]),
            "flops": 10.0 * voxels * g["K"] + rows * 2 * 2.5 * n * math.log2(n)}


# ------------------------------------------------------------------------------------------------- FP64
def padded(m):
    return 1 << (m - 1).bit_length() if m > 1 else 1


def filter_rows(x, filt):
    """Band-limited ramp (Kak & Slaney eq. 3.61) times the window, on rows padded to the next power of two."""
    m = x.shape[-1]
    n = padded(m)
    k = torch.arange(n, dtype=torch.float64, device=x.device)
    k = torch.where(k <= n // 2, k, k - n)
    h = torch.where(k % 2 != 0, -1.0 / (math.pi * torch.where(k == 0, 1.0, k)) ** 2, 0.0)
    h[0] = 0.25
    H = torch.fft.rfft(h).real
    f = torch.arange(n // 2 + 1, dtype=torch.float64, device=x.device) / n
    if filt == SHEPP_LOGAN:
        H = H * torch.sinc(f)
    elif filt == COSINE:
        H = H * torch.cos(math.pi * f)
    elif filt == HANN:
        H = H * 0.5 * (1 + torch.cos(2 * math.pi * f))
    return torch.fft.irfft(torch.fft.rfft(x, n=n) * H, n=n)[..., :m]


def backproject(views_of, g):
    """Sum over views of the distance-weighted bilinear taps, [z][y][x] in FP64; views_of(k) = filtered [v][u]."""
    nx, ny, nu, nv = g["nx"], g["ny"], g["nu"], g["nv"]
    x = (torch.arange(nx, dtype=torch.float64, device=DEV) + 0.5 - 0.5 * nx) * g["vox"]
    y = (torch.arange(ny, dtype=torch.float64, device=DEV) + 0.5 - 0.5 * ny) * g["vox"]
    vol = torch.zeros((nx, ny, nx), dtype=torch.float64, device=DEV)
    zs = max(1, (1 << 25) // (ny * nx))
    for k in range(g["K"]):
        q = torch.nn.functional.pad(views_of(k), (1, 2, 1, 2))  # zeros outside the detector
        c, s = math.cos(g["angles"][k]), math.sin(g["angles"][k])
        for z0 in range(0, nx, zs):
            z = x[z0:z0 + zs, None]
            t = z * c - x[None] * s
            if g["cone"]:
                rD = g["sod"] / (g["sod"] + x[None] * c + z * s)
                u = t * rD * (g["sdd"] / (g["sod"] * g["du"]))
                G = rD * (g["sdd"] / (g["sod"] * g["dv"]))
                W = rD * rD
            else:
                u, G, W = t / g["du"], torch.full_like(t, 1 / g["dv"]), torch.ones_like(t)
            u = (u + 0.5 * nu + 0.5).clamp(0, nu + 1.5)  # in the padded view
            iu = u.floor()
            fu = (u - iu).view(1, -1)
            iu = iu.long().view(-1)
            cols = (q[:, iu] * (1 - fu) + q[:, iu + 1] * fu) * W.view(1, -1)  # [v][z x]
            if ny == 1:
                vol[z0:z0 + zs, 0] += cols[1].view(-1, nx)
                continue
            v = (G[:, None, :] * y[None, :, None]).add_(0.5 * nv + 0.5).clamp_(0, nv + 1.5)
            iv = v.floor()
            v -= iv
            at = iv.long().mul_(cols.shape[1]).add_(torch.arange(cols.shape[1], device=DEV).view(-1, 1, nx))
            cols = cols.reshape(-1)
            lo = cols[at]
            hi = cols[at.add_(iu.numel())]
            vol[z0:z0 + zs] += lo.add_(hi.sub_(lo).mul_(v))
    scale = math.pi / g["K"] / g["du"]
    if g["cone"]:
        scale *= g["sdd"] / g["sod"]
    return vol.mul_(scale)


def rebin(fan, g, width):
    """Fan beam (flat detector, full turn) to parallel beam by bilinear interpolation in view and detector."""
    K, nu = fan.shape
    s = (torch.arange(nu, dtype=torch.float64, device=DEV) + 0.5 - 0.5 * nu) * (f32(width) / nu)
    ok = s.abs() < g["sod"]
    gam = torch.asin((s / g["sod"]).clamp(-1, 1))
    u = g["sdd"] * torch.tan(gam) / g["du"] + 0.5 * nu - 0.5
    b = torch.arange(K, dtype=torch.float64, device=DEV)[:, None] - gam[None] * (K / (2 * math.pi))
    fu, fb = u.floor(), b.floor()
    au, ab = (u - fu)[None], b - fb
    q = torch.nn.functional.pad(fan, (1, 1))
    iu = fu.clamp(-1, nu - 1).long() + 1
    inside = (ok & (fu >= -1) & (fu < nu))[None]
    ib = fb.long()
    r = [q[(ib + t) % K, iu[None]] * (1 - au) + q[(ib + t) % K, iu[None] + 1] * au for t in (0, 1)]
    return torch.where(inside, r[0] * (1 - ab) + r[1] * ab, 0.0)


def forward_exact(vol, g):
    """Trilinear samples at the midpoints of ceil(chord / (voxel / 2)) equal steps through the volume's box."""
    n, h, nu, nv = g["nx"], g["ny"], g["nu"], g["nv"]
    box = torch.tensor([0.5 * n, 0.5 * h, 0.5 * n], dtype=torch.float64, device=DEV) * g["vox"]
    src = vol.double()[None, None]
    u = ((torch.arange(nu, dtype=torch.float64, device=DEV) + 0.5 - 0.5 * nu) * g["du"])[None, :].expand(nv, nu)
    v = ((torch.arange(nv, dtype=torch.float64, device=DEV) + 0.5 - 0.5 * nv) * g["dv"])[:, None].expand(nv, nu)
    out = torch.empty((g["K"], nv, nu), dtype=torch.float64, device=DEV)
    for k in range(g["K"]):
        c, s = math.cos(g["angles"][k]), math.sin(g["angles"][k])
        o = torch.tensor([-g["sod"] * c, 0.0, -g["sod"] * s], dtype=torch.float64, device=DEV)
        w = torch.stack([(g["sdd"] - g["sod"]) * c - u * s, v, (g["sdd"] - g["sod"]) * s + u * c], -1) - o
        w = w / w.norm(dim=-1, keepdim=True)
        ta, tb = (-box - o) / w, (box - o) / w
        t0, t1 = torch.minimum(ta, tb).amax(-1), torch.maximum(ta, tb).amin(-1)
        hit = t1 > t0
        count = torch.where(hit, torch.ceil((t1 - t0) / (0.5 * g["vox"])), 1.0)
        step = torch.where(hit, (t1 - t0) / count, 0.0)
        most, acc = int(count.max()), torch.zeros_like(t0)
        chunk = max(1, (1 << 23) // (nu * nv))
        for q0 in range(0, most, chunk):
            q = torch.arange(q0, min(most, q0 + chunk), dtype=torch.float64, device=DEV)[:, None, None]
            at = (o + (t0 + (q + 0.5) * step)[..., None] * w) / box  # [-1, 1] over the box, (x, y, z)
            got = torch.nn.functional.grid_sample(src, at[None], mode="bilinear", padding_mode="zeros",
                                                  align_corners=False)[0, 0]
            acc += torch.where(q < count, got, 0.0).sum(0)
        out[k] = torch.where(hit, acc * step, 0.0)
    return out


def exact(case, seed):
    g = geometry_of(case)
    if g["nx"] * g["nx"] * g["ny"] * g["K"] > 1.2e11:
        return None  # minutes in FP64
    raw = inputs(case, seed)
    op = case["op"]
    if op == "forward":
        return forward_exact(raw, g)
    if op == "rebin":
        sdd = g["sdd"]
        width = case["det_width"] * case["sod"] / (case["sod"] + case["odd"])
        rows = filter_rows(rebin(raw.double(), g, width), case["filter"])
        g = dict(g, cone=False, du=f32(width) / g["nu"])
        return backproject(lambda k: rows[k:k + 1], g)[:, 0]
    if op == "slice2d":
        rows = raw.double()
        if g["cone"]:
            u = (torch.arange(g["nu"], dtype=torch.float64, device=DEV) + 0.5 - 0.5 * g["nu"]) * g["du"]
            rows = rows * (g["sdd"] / (g["sdd"] ** 2 + u * u).sqrt())
        rows = filter_rows(rows, case["filter"])
        return backproject(lambda k: rows[k:k + 1], g)[:, 0]

    u = (torch.arange(g["nu"], dtype=torch.float64, device=DEV) + 0.5 - 0.5 * g["nu"]) * g["du"]
    v = (torch.arange(g["nv"], dtype=torch.float64, device=DEV) + 0.5 - 0.5 * g["nv"]) * g["dv"]

    def view(k):
        q = (raw[:, k] if op == "parallel3d" else raw[k]).double()
        if case.get("counts"):
            q = -torch.log(q / base_of(case))
        if g["cone"]:
            q = q * (g["sdd"] / (g["sdd"] ** 2 + (u * u)[None] + (v * v)[:, None]).sqrt())
        return filter_rows(q, case["filter"])

    vol = backproject(view, g)
    vol[:, :g["nx"]].clamp_(min=0)  # the library clips negatives of the y-slices below the volume's z size
    return vol
