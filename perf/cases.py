"""The work users of this framework have it do, as cases that can be timed.

Four kinds of call, each through a public entry point:

  proj, back  device.Plan.proj / Plan.back: one projector or backprojector call
              on device tensors (what AAPM_script/DD2MutiSlices.m calls the mex
              functions for), from one slice of one subset to a whole scan
  solve       device.OSSART: a new sinogram and start image into a kept solver,
              some OS-SART iterations, the image out
  recon       dd2.OSSART_AAPM: the reference's own call, host arrays in and out,
              solver set-up included
  rebin       ddfan_helical_to_fan_dev: raw helical views to the fan-beam
              sinogram and the per-slice angle lists that a solve takes

A case is a dict of plain values; sizes follow configs.py (c1 to c4).  Images are
sums of ellipsoids in attenuation per mm, sinograms their line integrals in
closed form, with Poisson noise where a solve starts from them.
"""
import ctypes
import math

import numpy as np
import torch

from aapm_lowdosectimagerecon_competition_b200 import dd2, device
from aapm_lowdosectimagerecon_competition_b200._lib import call

SID, SDD = 595.0, 1085.6  # the c2 scanner (mm)
TWOPI = 6.283185307179586


def _case(kind, N, Z, PN, DNU, name=None, **more):
    c = {"kind": kind, "N": N, "Z": Z, "PN": PN, "DNU": DNU, "sat": "hilo", "back": "adj", "masked": False, "spacing": 0.0}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one slice, one of c1's 8 subsets, the default precision: the smallest
        # calls, where launches and latency count
        _case("back", 256, 1, 123, 888, name="back_one_slice"),
        _case("proj", 256, 1, 123, 888, name="proj_one_slice"),
        # a c3 subset (96 views of 512^2 x 128): what a hand-written OS-SART loop
        # does at every step, projector and the reference's backprojector
        _case("proj", 512, 128, 96, 736, name="proj_subset", sat="direct"),
        _case("back", 512, 128, 96, 736, name="back_subset", sat="direct", back="ref"),
        # c2: a whole scan's projection in one call, the default precision, with the disk mask
        _case("proj", 512, 64, 2304, 736, name="proj_scan", masked=True),
        # a whole scan's exact adjoint at ragged sizes (slices no multiple of 4, odd view count)
        _case("back", 384, 45, 1111, 701, name="back_scan_ragged", sat="direct", masked=True),
        # c1 as the reference runs it: one call from host arrays, set-up included
        _case("recon", 256, 1, 984, 888, name="recon_call", back="ref", masked=True, subsets=8, iters=5),
        # c3, one iteration of the flagship solve: the largest
        _case("solve", 512, 128, 2304, 736, name="solve_large", sat="direct", back="ref", masked=True, subsets=24, iters=1),
        # the smallest of the serving mix (c4): few slices, many small subset steps
        _case("solve", 256, 16, 720, 736, name="solve_small", sat="direct", back="ref", masked=True, subsets=24, iters=2),
        # the solver's defaults (hi/lo precision, exact adjoint) at ragged sizes
        _case("solve", 384, 37, 1111, 736, name="solve_default_ragged", masked=True, subsets=10, iters=1),
        # rebinned data: every slice its own angle list, 5 subsets as reconscript.m
        _case("solve", 384, 24, 720, 736, name="solve_per_slice", back="ref", masked=True, subsets=5, iters=1, spacing=27.07),
        # helical-to-fan rebinning of a Siemens-like scan, ahead of such a solve
        _case("rebin", 64, 96, 2304, 736, name="rebin_scan"),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    while True:
        kind = rng.choice(["proj", "proj", "back", "back", "solve", "solve", "solve", "recon", "rebin"])
        if kind == "rebin":
            c = _case("rebin", 4 * rng.randint(8, 16), rng.randint(8, 128), rng.randint(720, 2304), rng.randint(500, 900))
            if c["PN"] * c["DNU"] * c["Z"] <= 2304 * 736 * 128:
                return c
            continue
        N, Z, DNU = _log(rng, 160, 768), _log(rng, 1, 128), rng.randint(500, 900)
        c = _case(kind, N, Z, _log(rng, 90, 2304), DNU, sat=rng.choice(["direct", "hilo"]), back=rng.choice(["ref", "adj"]),
                  masked=rng.random() < 0.5)
        if kind in ("solve", "recon"):
            c["PN"] = _log(rng, 360, 2304)
            c["masked"] = True
            c["subsets"] = rng.choice([5, 8, 10, 12, 24])
            c["iters"] = rng.randint(1, 3)
            if kind == "recon":
                c["Z"] = min(Z, 24)
            elif rng.random() < 0.2:
                c["spacing"] = round(rng.uniform(10.0, 40.0), 2)
                c["Z"], c["N"], c["iters"], c["subsets"] = max(2, min(Z, 32)), min(N, 512), 1, 5
        # at most a quarter of the largest listed case's work
        if c["PN"] * c["N"] ** 2 * c["Z"] * c.get("iters", 1) <= 2304 * 512 ** 2 * 128 // 4:
            return c


def work(case):
    N, Z, P, U = case["N"], case["Z"], case["PN"], case["DNU"]
    if case["kind"] == "rebin":
        # the raw views the slices read once, the fan-beam rows written once;
        # two products and a sum per row sample, its weight and its position
        return {"bytes": 4.0 * (_rebin_geometry(case)["TV"] * U * N + P * U * Z + P * Z), "flops": 12.0 * P * U * Z}
    img, sino = 4.0 * N * N * Z, 4.0 * P * U * Z
    pix = 4.0 * P * N * N * Z  # per view and pixel: two overlap-weighted sums, one for each channel it meets
    if case["kind"] in ("proj", "back"):
        return {"bytes": img + sino, "flops": pix}
    # a solve: each iteration projects every view once and backprojects it once;
    # the image is read and written per subset, the sinogram read per iteration
    n = case["iters"]
    return {"bytes": n * (2.0 * img * case["subsets"] + sino), "flops": n * 2.0 * pix}


# ---------------------------------------------------------------- inputs


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _scan(case):
    """Geometry of a case: the c2 field of view on its image grid and detector."""
    N, U = case["N"], case["DNU"]
    f = np.float32
    g = {"dx": f(0.7 * 512.0 / N), "cell": f(1.2858 * 736.0 / U), "cnt": f((U + 1) / 2.0), "sid": f(SID), "sdd": f(SDD)}
    # arc detector in single precision (AAPM_script/DD2MutiSlices.m:55-76)
    step = f(math.atan(float(g["cell"] / f(2) / g["sdd"]))) * f(2)
    beta = ((np.arange(1, U + 1, dtype=np.float32) - g["cnt"]) * step).astype(np.float64)
    g["xds"] = (np.sin(beta).astype(f) * g["sdd"]).astype(f)
    g["yds"] = (g["sid"] - np.cos(beta).astype(f) * g["sdd"]).astype(f)
    ii = np.arange(1, N + 1) - 0.5 - N / 2.0
    r = np.sqrt((ii[None, :] ** 2 + ii[:, None] ** 2)) / (N / 2.0)
    g["mask"] = (r < 1.3).astype(np.uint8) if case["masked"] else None
    return g


def _angles(case):
    """float32 (PN,), or (PN, Z) as rebinning leaves them: slice z starts
    floor(spacing z) raw views after slice 0."""
    P, Z = case["PN"], case["Z"]
    if not case["spacing"]:
        return (np.arange(P) * (2.0 * math.pi / P)).astype(np.float32)
    i = np.arange(P)[:, None] + np.floor(case["spacing"] * np.arange(Z)).astype(np.int64)[None, :]
    return np.fmod(i.astype(np.float32) * np.float32(2.0 * math.pi / P), np.float32(2.0 * math.pi)).astype(np.float32)


def _ellipsoids(case, seed):
    """A water cylinder and nine ellipsoids: (cx, cy, a, b, angle, mu, cz, c), lengths in mm."""
    rng = np.random.default_rng(seed)
    N, Z = case["N"], case["Z"]
    dx = 0.7 * 512.0 / N
    R, H = 0.43 * N * dx, Z * dx
    out = [(0.0, 0.0, R, R, 0.0, 0.02, 0.0, 1e6)]
    for _ in range(9):
        cx, cy = rng.uniform(-0.5, 0.5, 2) * R
        a, b = rng.uniform(0.05, 0.3, 2) * R
        out.append((cx, cy, a, b, rng.uniform(0, math.pi), rng.uniform(-0.008, 0.012), rng.uniform(-0.5, 0.5) * H, rng.uniform(0.4, 1.0) * H))
    return out


def _z_scale(case, cz, c, dev):
    z = (torch.arange(case["Z"], device=dev, dtype=torch.float64) - (case["Z"] - 1) / 2.0) * (0.7 * 512.0 / case["N"])
    return (1.0 - ((z - cz) / c) ** 2).clamp(min=0.0).float()


def _image(case, seed, dev):
    """The phantom on the grid with a little texture, float32 (N, N, Z)."""
    N, Z = case["N"], case["Z"]
    x = ((torch.arange(N, device=dev, dtype=torch.float64) - (N - 1) / 2.0) * (0.7 * 512.0 / N)).float()
    img = torch.zeros((N, N, Z), device=dev)
    for cx, cy, a, b, th, mu, cz, c in _ellipsoids(case, seed):
        X, Y = x[None, :] - cx, x[:, None] - cy
        q = ((X * math.cos(th) + Y * math.sin(th)) / a) ** 2 + ((Y * math.cos(th) - X * math.sin(th)) / b) ** 2
        img += mu * (q[:, :, None] <= _z_scale(case, cz, c, dev)[None, None, :])
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    return img * (1.0 + 0.02 * torch.randn(img.shape, device=dev, generator=g))


def _sinogram(case, seed, dev):
    """Line integrals of the phantom over the pixel pitch (the projector's unit), float32 (PN, DNU, Z)."""
    g, P, U, Z = _scan(case), case["PN"], case["DNU"], case["Z"]
    ang = torch.from_numpy(_angles(case)).to(dev).double()
    ang = ang[:, None] if ang.dim() == 1 else ang
    cs, sn = torch.cos(ang), torch.sin(ang)  # (P, 1 or Z)
    xd = torch.from_numpy(g["xds"]).to(dev).double()[None, :, None]
    yd = torch.from_numpy(g["yds"]).to(dev).double()[None, :, None]
    out = torch.empty((P, U, Z), device=dev)
    part = max(1, (1 << 25) // (U * Z))
    for p0 in range(0, P, part):
        c, s = cs[p0:p0 + part, None, :], sn[p0:p0 + part, None, :]
        sx, sy = -SID * s, SID * c
        dx, dy = xd * c - yd * s - sx, xd * s + yd * c - sy
        ln = torch.sqrt(dx * dx + dy * dy)
        dx, dy = dx / ln, dy / ln
        acc = 0.0
        for cx, cy, a, b, th, mu, cz, cc in _ellipsoids(case, seed):
            k, m = math.cos(th), math.sin(th)
            px, py = ((sx - cx) * k + (sy - cy) * m) / a, ((sy - cy) * k - (sx - cx) * m) / b
            qx, qy = (dx * k + dy * m) / a, (dy * k - dx * m) / b
            pq, pp, qq = px * qx + py * qy, px * px + py * py, qx * qx + qy * qy
            base, slope = (pq * pq - qq * pp).float(), qq.float()
            z = _z_scale(case, cz, cc, dev)[None, None, :]
            acc = acc + torch.sqrt((base + slope * z).clamp(min=0.0)) * (2.0 * mu / slope)
        out[p0:p0 + part] = acc / float(g["dx"])
    return out


def _noisy(y, case, seed):
    """The log of Poisson counts at 1.5e5 photons a ray."""
    dx = 0.7 * 512.0 / case["N"]
    g = torch.Generator(device=y.device)
    g.manual_seed(seed + 1)
    for p in y.split(max(1, (1 << 25) // (y.shape[1] * y.shape[2]))):
        n = torch.poisson(1.5e5 * torch.exp(-p * dx), generator=g)
        p.copy_(-torch.log(n.clamp(min=1.0) / 1.5e5) / dx)
    return y


def _rebin_geometry(case):
    """A Siemens-like helical scan: N detector rows, pitch 0.8, Z slices over
    the range its views cover; slice starts fall between raw views."""
    f = np.float32
    T, H, Z = case["PN"], case["N"], case["Z"]
    g = {"SD": f(SDD), "SO": f(SID), "BV": f(0.3), "PW": f(1.2858 * 736.0 / case["DNU"]), "PH": f(1.0947), "cnt": f((case["DNU"] + 1) / 2.0), "pitch": f(0.8)}
    h = float(g["pitch"]) * float(g["PH"]) * H * SID / SDD
    dz = h / T
    spacing = T / 26.77  # raw views between slices: 86.07 of 2304, an AAPM-length scan's
    start = np.floor(spacing * np.arange(Z)) + 5.5
    g["TV"] = int(start[-1]) + T + 2
    g["z"] = (h * 0.5 + start * dz).astype(np.float32)
    return g


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    if case["kind"] == "rebin":
        s = _rebin_geometry(case)
        g = torch.Generator(device=dev)
        g.manual_seed(seed)
        s["raw"] = torch.rand((s["TV"], case["DNU"], case["N"]), device=dev, generator=g) * 8.0
        s["out"] = torch.empty((case["PN"], case["DNU"], case["Z"]), device=dev)
        s["views"] = torch.empty((case["PN"], case["Z"]), device=dev)
        s["case"] = case
        return s
    g, N, Z = _scan(case), case["N"], case["Z"]
    ang = _angles(case)
    s = {"case": case, "scan": g}
    if case["kind"] in ("proj", "back"):
        s["angs"] = torch.from_numpy(ang).to(dev)
        s["plan"] = device.Plan(0.0, g["sid"], case["DNU"], g["xds"], g["yds"], g["cnt"], N, N, Z, case["PN"], g["dx"],
                                mask=g["mask"], sat=case["sat"])
        if case["kind"] == "proj":
            s["in"] = _image(case, seed, dev)
            s["out"] = torch.empty((case["PN"], case["DNU"], Z), device=dev)
        else:
            s["in"] = _sinogram(case, seed, dev)
            s["out"] = torch.empty((N, N, Z), device=dev)
        return s
    y = _noisy(_sinogram(case, seed, dev), case, seed)
    hangs = ang if ang.ndim == 2 else np.repeat(ang[:, None], Z, axis=1)
    if case["kind"] == "recon":
        s["y"], s["hangs"], s["x0"] = y.cpu().numpy(), hangs, np.zeros((N, N, Z), np.float32)
        s["conf"] = {"recon": {"XN": N, "YN": N, "dx": float(g["dx"])}, "SLN": Z,
                     "acq": {"sid": float(g["sid"]), "sdd": float(g["sdd"]), "DNU": case["DNU"], "PN": case["PN"],
                             "detCellWidth": float(g["cell"]), "detCntIdx": float(g["cnt"])}}
        return s
    s["y"], s["x0"], s["out"] = y, torch.zeros((N, N, Z), device=dev), torch.empty((N, N, Z), device=dev)
    s["solver"] = device.OSSART(0.0, g["sid"], case["DNU"], g["xds"], g["yds"], g["cnt"], hangs, N, N, Z, g["dx"], mask=g["mask"],
                                numOfOS=case["subsets"], useFISTA=1, nonneg=1, sat=case["sat"], back=case["back"])
    return s


def run(state):
    c = state["case"]
    if c["kind"] == "proj":
        return state["plan"].proj(state["angs"], state["in"], out=state["out"])
    if c["kind"] == "back":
        return state["plan"].back(state["angs"], state["in"], out=state["out"], mode=c["back"])
    if c["kind"] == "solve":
        sv = state["solver"]
        sv.set_sinogram(state["y"])
        sv.set_image(state["x0"])
        sv.iterate(c["iters"])
        return sv.image(out=state["out"])
    if c["kind"] == "recon":
        return dd2.OSSART_AAPM(state["y"], state["hangs"], state["x0"], state["conf"], c["iters"], c["subsets"], state["scan"]["mask"],
                               useFISTA=1, nonneg=1, sat=c["sat"], back=c["back"])
    z = state["z"]
    call("ddfan_helical_to_fan_dev", _ptr(state["raw"]), state["TV"], z.ctypes.data_as(ctypes.c_void_p), c["Z"], state["SD"], state["SO"],
         state["BV"], c["DNU"], c["N"], state["PW"], state["PH"], c["PN"], state["cnt"], state["pitch"], 1, _ptr(state["out"]),
         _ptr(state["views"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return state["out"], state["views"]


# ---------------------------------------------------------------- the same in 64 bits


def _boundaries(c):
    """Channel boundaries, float32 as the reference keeps them (AAPM_script/utilities.cuh:268-287)."""
    c = c.astype(np.float64)
    b = np.concatenate([[1.5 * c[0] - 0.5 * c[1]], 0.5 * (c[:-1] + c[1:]), [1.5 * c[-1] - 0.5 * c[-2]]])
    return b.astype(np.float32).astype(np.float64)


class _Exact:
    """Projector, both backprojectors and OS-SART of a case in float64 torch."""

    def __init__(self, case, dev):
        g = _scan(case)
        self.N, self.U, self.dev, self.dx = case["N"], case["DNU"], dev, float(g["dx"])
        t = lambda v: torch.as_tensor(np.asarray(v, np.float64), device=dev)
        self.bx, self.by = t(_boundaries(g["xds"])), t(_boundaries(g["yds"]))
        self.xd, self.yd = t(g["xds"]), t(g["yds"])
        self.y0, self.cnt = float(g["sid"]), float(g["cnt"])
        self.mask = torch.ones((self.N, self.N), device=dev, dtype=torch.float64) if g["mask"] is None else t(g["mask"])
        S2D = math.hypot(float(g["xds"][0]), float(g["yds"][0]) - self.y0)
        e = np.diff(np.stack([g["xds"][:2], g["yds"][:2]]).astype(np.float64), axis=1)
        self.dbeta = 2.0 * math.atan(math.hypot(e[0, 0], e[1, 0]) / S2D * 0.5)
        self.oc = (self.N - 1) * 0.5

    def view(self, th):
        """(x-major?, positions of the boundary rays on every line, channel weights, source)."""
        th = math.fmod(float(th), TWOPI)
        cs, sn = math.cos(th), math.sin(th)
        sx, sy = -self.y0 * sn, self.y0 * cs
        Bx, By = self.bx * cs - self.by * sn, self.bx * sn + self.by * cs
        Dx, Dy = self.xd * cs - self.yd * sn - sx, self.xd * sn + self.yd * cs - sy
        xm = abs(cs) <= abs(sn)
        if not xm:
            Bx, By, ux, uy, Dm = By, Bx, sy, sx, Dy
        else:
            ux, uy, Dm = sx, sy, Dx
        F = (By - uy) / (Bx - ux)
        C = ((-self.oc * self.dx - Bx) * F + By) / self.dx + self.oc + 0.5
        ii = torch.arange(self.N, device=self.dev, dtype=torch.float64)[:, None]
        return xm, ii * F + C, torch.sqrt(Dx * Dx + Dy * Dy) / Dm.abs(), (sx, sy)

    def _sums(self, img):
        x = img * self.mask[:, :, None]
        pad = lambda v: torch.cat([torch.zeros_like(v[:, :1]), torch.cumsum(v, 1)], 1).reshape(-1, img.shape[2])
        return pad(x), pad(x.transpose(0, 1))

    def proj(self, img, angs):
        N, U = self.N, self.U
        rows, cols = self._sums(img)
        out = torch.empty((len(angs), U, img.shape[2]), device=self.dev, dtype=torch.float64)
        base = torch.arange(N, device=self.dev)[:, None] * (N + 1)
        for p, th in enumerate(angs):
            xm, c, w, _ = self.view(th)
            S = cols if xm else rows
            cc = c.clamp(0, N)
            k = cc.floor().long().clamp(max=N - 1)
            f = (cc - k)[:, :, None]
            at = (base + k)
            phi = S[at] * (1.0 - f) + S[at + 1] * f
            out[p] = ((phi[:, 1:] - phi[:, :-1]) / (c[:, 1:] - c[:, :-1])[:, :, None]).sum(0) * w[:, None]
        return out

    def back(self, prj, angs, mode):
        N, U = self.N, self.U
        out = torch.zeros((N, N, prj.shape[2]), device=self.dev, dtype=torch.float64)
        v = (torch.arange(N, device=self.dev, dtype=torch.float64) - self.oc) * self.dx
        edge = torch.arange(N + 1, device=self.dev, dtype=torch.float64)[None, :].expand(N, N + 1)
        for p, th in enumerate(angs):
            xm, c, w, (sx, sy) = self.view(th)
            q = prj[p] * w[:, None] if mode == "adj" else prj[p]
            Q = torch.cat([torch.zeros_like(q[:1]), torch.cumsum(q, 0)], 0)
            if mode == "adj":
                s = 1.0 if float(c[N // 2, U] - c[N // 2, 0]) >= 0 else -1.0
                c, e = (s * c).contiguous(), (s * edge).contiguous()
                b = (torch.searchsorted(c, e, right=True) - 1).clamp(0, U - 1)
                c0, c1 = torch.gather(c, 1, b), torch.gather(c, 1, b + 1)
                f = ((e - c0) / (c1 - c0)).clamp(0, 1)[:, :, None]
                h = Q[b] * (1.0 - f) + Q[b + 1] * f
                d = s * (h[:, 1:] - h[:, :-1])
                out += d.transpose(0, 1) if xm else d
                continue
            dx, dy = (v - sx)[None, :], (v - sy)[:, None]
            l2 = dx * dx + dy * dy
            alpha = torch.asin((sy * dx - sx * dy) / math.hypot(0.0, self.y0) / torch.sqrt(l2))
            dv = (dx if abs(sx) > abs(sy) else dy).expand(N, N)
            da = dv / l2 * self.dx * 0.5
            h = []
            for a in (alpha - da, alpha + da):
                t = (a / self.dbeta + self.cnt + 0.5).clamp(0, U)
                k = t.floor().long().clamp(max=U - 1)
                f = (t - k)[:, :, None]
                h.append(Q[k] * (1.0 - f) + Q[k + 1] * f)
            out += (h[1] - h[0]) * (self.dx / dv * torch.sqrt(l2))[:, :, None]
        return out * self.mask[:, :, None]

    def solve(self, y, angs, slice0, case, nonneg=True):
        """OS-SART with FISTA momentum (AAPM_script/OSSART_AAPM.m:57-115) of slices that share angs; sums from slice0's list."""
        n, one = case["subsets"], torch.ones((self.N, self.N, 1), device=self.dev, dtype=torch.float64)
        subs = [list(range(k, len(angs), n)) for k in range(n)]
        if not hasattr(self, "weights"):
            self.weights = [(self.proj(one, slice0[v]), self.back(torch.ones((len(v), self.U, 1), device=self.dev, dtype=torch.float64), slice0[v], case["back"]))
                            for v in subs]
        x = torch.zeros((self.N, self.N, y.shape[2]), device=self.dev, dtype=torch.float64)
        prev, t0 = x.clone(), 1.0
        for _ in range(case["iters"]):
            for v, (row, col) in zip(subs, self.weights):
                ax = self.proj(x, angs[v])
                r = torch.where(row != 0, (y[v] - ax) / torch.where(row != 0, row, torch.ones_like(row)), ax)
                t = self.back(r, angs[v], case["back"])
                x = x + t / torch.where(col != 0, col, torch.ones_like(col))
                x = x.clamp(min=0) if nonneg else x
            t1 = (1.0 + math.sqrt(1.0 + 4.0 * t0 * t0)) / 2.0
            x = x + (t0 - 1.0) / t1 * (x - prev)
            prev, t0 = x.clone(), t1
        return x


def _exact_rebin(case, seed, dev):
    """AAPM_script/HelicalToFanFunc_mex.cpp:41-139 in float64."""
    s = _rebin_geometry(case)
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    W, H, T, Z = case["DNU"], case["N"], case["PN"], case["Z"]
    raw = torch.rand((s["TV"], W, H), device=dev, generator=g) * 8.0
    SD, SO, PH = float(s["SD"]), float(s["SO"]), float(s["PH"])
    h = float(s["pitch"]) * PH * H * SO / SD
    dz = h / T
    j = torch.arange(1, W + 1, device=dev, dtype=torch.float64)
    sm = SO * torch.cos((j - float(s["cnt"])) * 2.0 * math.atan(float(s["PW"]) / SD * 0.5))
    out = torch.zeros((T, W, Z), device=dev, dtype=torch.float64)
    views = torch.zeros((T, Z), device=dev, dtype=torch.float64)
    for z in range(Z):
        zp = float(s["z"][z])
        i = int(math.floor((zp - h * 0.5) / dz)) + torch.arange(T, device=dev)
        v = SD * (zp - (i - 1).double() * dz)[:, None] / sm[None, :]
        dv = ((H - 1.0) * 0.5 / PH + v) / PH + 1.0
        k = dv.floor().long()
        ok = ((k >= 1) & (k <= H - 1)).all(1)
        k = k.clamp(1, H - 1)
        t, d = dv - k, raw[i - 1]
        lo, hi = torch.gather(d, 2, (k - 1)[:, :, None])[:, :, 0].double(), torch.gather(d, 2, k[:, :, None])[:, :, 0].double()
        out[:, :, z] = torch.where(ok[:, None], SD / torch.sqrt(SD * SD + v * v) * (lo * (1.0 - t) + hi * t), torch.zeros_like(lo))
        lam = (i - 1).double() * (TWOPI / T) + float(s["BV"])
        views[:, z] = lam - TWOPI * (torch.ceil(lam / TWOPI) - 1).clamp(min=0)
    return out, views


def exact(case, seed):
    dev = _device()
    if case["kind"] == "rebin":
        return _exact_rebin(case, seed, dev)
    Z, n = case["Z"], case.get("iters", 1)
    # samples gathered in 64 bits, and views walked one by one
    if case["PN"] * case["N"] * case["DNU"] * Z * n > 1.2e11 or case["PN"] * n * (Z if case["spacing"] else 1) > 20000:
        return None
    E, angs = _Exact(case, dev), _angles(case)
    if case["kind"] == "proj":
        return E.proj(_image(case, seed, dev).double(), angs)
    y = _sinogram(case, seed, dev)
    if case["kind"] == "back":
        return E.back(y.double(), angs, case["back"])
    y = _noisy(y, case, seed)
    if not case["spacing"]:
        x = E.solve(y.double(), angs, angs, case)
    else:
        a0 = np.ascontiguousarray(angs[:, 0])
        x = torch.cat([E.solve(y[:, :, z:z + 1].double(), np.ascontiguousarray(angs[:, z]), a0, case) for z in range(Z)], 2)
    return x.cpu().numpy() if case["kind"] == "recon" else x
