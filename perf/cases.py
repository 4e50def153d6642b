"""The work that programs built on this framework spend their time in, as cases
that can be timed: projector layers in both directions and under autograd, the
reference's drop-in call, the iterative reconstructions, batches of them, the
filtered layer and a training step. Every case goes through the public entry
points of ``dtvb200`` (or the drop-in module) on inputs made from a seed:
ellipsoid phantoms, and their analytic line integrals with Poisson noise.

A case is a dict of plain values. ``prepare`` makes what a program holds before
the call, ``run`` is one pass, ``work`` the bytes and operations a pass cannot
do without, and ``exact`` the same outputs in 64-bit torch arithmetic.
"""
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "dtv-net_b200"))

import dtvb200  # noqa: E402
import dtvb200.nets  # noqa: E402
import dtvb200.phantom  # noqa: E402
import JITStandardGeometry as dropin  # noqa: E402

DEV = "cuda"
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def _case(name, kind, size, views, det, pitch=1.0, geometry="circular", sampler="soft", batch=1,
          iters=0, dtype="f32", planes=1):
    c = dict(kind=kind, geometry=geometry, nx=size[0], ny=size[1], nz=size[2], views=views,
             nu=det[0], nv=det[1], pitch=pitch, sampler=sampler, batch=batch, iters=iters,
             dtype=dtype, planes=planes)
    return dict(c, name=name) if name else c


def listed():
    return [
        # The reference's own module interface (JITStandardGeometry.forward and
        # .backward) on the smallest scan anyone tries first: launch latency.
        _case("dropin_small", "dropin", (24, 20, 12), 16, (32, 20), geometry="standard"),
        # The reference's default layer, x - BP(FP(x) - p), on its flat slab:
        # 48 views of a wide, low detector, software sampler.
        _case("layer_slab", "layer", (256, 256, 64), 48, (288, 28), geometry="standard"),
        # Forward projection of a large BF16-stored volume (texture sampler): the
        # full-resolution scans, a sparse subset of their views.
        _case("forward_512", "forward", (512, 512, 512), 24, (1024, 768), 0.8, sampler="pairs",
              dtype="bf16"),
        # FDK backprojection alone at the sparse-view size: FBP-like use and half
        # of every iteration of an iterative method.
        _case("backward_256", "backward", (256, 256, 256), 64, (384, 384), 1.2, sampler="pairs"),
        # A differentiable data step through the matched pair with its gradient:
        # what an unrolled network pays per stage besides its convolutions.
        _case("layer_grad", "grad", (128, 128, 128), 48, (192, 192), 1.5, batch=2),
        # The sparse-view DTV reconstruction as shipped: texture operators corrected
        # by the exact ones, FP16-stored extrapolation, one captured graph.
        _case("dtv_corrected", "dtv", (256, 256, 256), 64, (384, 384), 1.2, sampler="pairs",
              iters=12, dtype="f16"),
        # DTV through the exact-weight operators alone, eager, on an odd-sized
        # volume and detector: reconstructions of cropped real scans.
        _case("dtv_exact_odd", "dtv", (151, 163, 97), 45, (231, 149), 1.2, sampler="exact", iters=6),
        # FISTA-TV on a small scan, graph-captured: latency of an iteration.
        _case("fista_tv_64", "fista_tv", (64, 64, 64), 60, (128, 128), 1.0, sampler="pairs",
              iters=20),
        # Heterogeneous FISTA reconstructions in one graph (sizes derived from
        # the first one's: half and three quarters of its edge beside it).
        _case("batch_fista", "batch", (192, 192, 192), 60, (288, 288), 1.5, sampler="pairs", batch=4,
              iters=6),
        # ASD-POCS with its ten TV descent steps per data step, odd sizes.
        _case("asd_pocs", "asd", (143, 129, 77), 36, (217, 121), 1.2, iters=4),
        # The filtered layer on the many-view module geometry (21 detector modules
        # per angle, tilted rows: no circular symmetry to use).
        _case("fbp_modules", "fbp", (256, 256, 64), 1008, (80, 128), geometry="vector", planes=21),
        # One training step (loss, gradients, Adam's update of weights and step sizes)
        # of the unrolled network with checkpointed stages and BF16 convolutions.
        _case("train_step", "train", (128, 128, 128), 48, (192, 192), 1.5, batch=2, iters=2,
              dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds: sizes log-uniform over their ranges, odd
    ones among them, within the cost of the largest listed case."""
    kind = rng.choice(["dropin", "layer", "forward", "backward", "grad", "dtv", "fista_tv", "batch",
                       "asd", "fbp", "train"])
    if kind == "fbp":
        planes = rng.choice([3, 7, 21])
        nx = 2 * _log(rng, 24, 112)
        return _case(None, kind, (nx, nx + rng.choice([0, 1, -3]), _log(rng, 12, 64)),
                     planes * rng.randint(7, 1 + 600 // planes), (4 * rng.randint(8, 20), rng.randint(33, 128)),
                     geometry="vector", planes=planes)
    top = {"dropin": 128, "layer": 224, "forward": 384, "backward": 256, "grad": 144, "dtv": 200,
           "fista_tv": 128, "batch": 160, "asd": 160, "train": 112}[kind]
    n = _log(rng, 16 if kind == "dropin" else 48, top)
    if kind in ("train", "batch"):
        n = 8 * (n // 8)
    elif rng.random() < 0.5:
        n = 4 * (n // 4)
    ny = n if rng.random() < 0.5 else max(9, n - rng.randint(1, n // 4))
    nz = n if rng.random() < 0.4 else max(9, _log(rng, max(9, n // 4), n))
    if kind in ("train", "batch"):
        ny = nz = n
    views = rng.randint(16, 72)
    pitch = rng.choice([1.0, 1.2, 1.5])
    det = (max(17, int(1.9 * n / pitch) + rng.randint(0, 5)), max(11, int(2.0 * nz / pitch) + rng.randint(0, 5)))
    geometry = "standard" if kind in ("dropin", "layer") else "circular"
    sampler = {"forward": rng.choice(["pairs", "soft", "exact", "tex"]),
               "backward": rng.choice(["pairs", "soft", "exact"]),
               "dtv": rng.choice(["pairs", "exact", "soft"]), "fista_tv": "pairs",
               "batch": "pairs"}.get(kind, "soft")
    iters = {"dtv": rng.randint(4, 10), "fista_tv": rng.randint(5, 20), "batch": rng.randint(3, 6),
             "asd": rng.randint(2, 4), "train": 2}.get(kind, 0)
    batch = {"grad": rng.choice([1, 2]), "batch": rng.choice([3, 4]),
             "forward": rng.choice([1, 1, 2])}.get(kind, 1)
    if n > 256:
        batch, views = 1, min(views, 40)
    dtype = {"forward": rng.choice(["f32", "f16", "bf16"]),
             "dtv": rng.choice(["f32", "f16", "bf16"]), "train": "bf16"}.get(kind, "f32")
    return _case(None, kind, (n, ny, nz), views, det, pitch, geometry, sampler, batch, iters, dtype)


# ---- geometry ------------------------------------------------------------------------------
SOD, SDD = 500.0, 1000.0          # circular orbits
SID_STD, SDD_STD = 1000.0, 2000.0  # the Standard layer


def _angles(c):
    return np.linspace(0, 360, c["views"], endpoint=False)


def _module_views(c):
    """[n,12] float32 projection vectors of the module scanner: per angle,
    `planes` flat modules side by side on an arc about the source, rows tilted
    towards it (source, detector, v, u; z of source and detector negated)."""
    P, W, H = c["planes"], c["nu"], c["nv"]
    sod, sdd = 1.6 * max(c["nx"], c["ny"]), 2.8 * max(c["nx"], c["ny"])
    fan = 2 * math.asin(min(0.9, 0.72 * max(c["nx"], c["ny"]) / sod))
    du = 2 * sdd * math.tan(fan / P / 2) / W
    dv = 1.15 * c["nz"] * sdd / sod / H
    A = c["views"] // P
    pv = np.zeros((A, P, 12))
    for a in range(A):
        t = 2 * math.pi * a / A
        src = -sod * np.array([math.cos(t), math.sin(t), 0.0])
        for j in range(P):
            g = t + fan * ((j + 0.5) / P - 0.5)
            ex, ey = np.array([math.cos(g), math.sin(g), 0.0]), np.array([-math.sin(g), math.cos(g), 0.0])
            det = src + sdd * ex
            pv[a, j] = np.concatenate([src, det, dv * (np.array([0, 0, 1.0]) + 0.05 * ex), du * ey])
    return pv.reshape(A * P, 12).astype(np.float32)


def _geometry(c):
    size, det = (c["nx"], c["ny"], c["nz"]), (c["nu"], c["nv"])
    if c["geometry"] == "standard":
        return dtvb200.standard(_angles(c).astype(np.float32), size, det, SID_STD, SDD_STD)
    if c["geometry"] == "vector":
        return dtvb200.vector(_module_views(c), size, det)
    return dtvb200.circular(_angles(c), size, (1.0,) * 3, det, (c["pitch"],) * 2, SOD, SDD)


class _Scan:
    """The geometry in 64 bits, from the conventions of the layers alone."""

    def __init__(self, c):
        self.n = (c["nx"], c["ny"], c["nz"])
        self.nu, self.nv = c["nu"], c["nv"]
        t64 = lambda a: torch.tensor(np.asarray(a, dtype=np.float64), device=DEV)  # noqa: E731
        if c["geometry"] == "vector":
            pv = _module_views(c).astype(np.float64)
            flip = np.array([1.0, 1.0, -1.0])
            S, D, U, V = pv[:, 0:3] * flip, pv[:, 3:6] * flip, pv[:, 9:12], pv[:, 6:9]
            self.vox, off, det_off, self.phase, self.power = 1.0, 0.0, 0.5, "vector", 1
            n = pv.shape[0]
            self.bp_scale = 2 * 3.14159265359 / (n // 21) if n >= 21 else 0.0
        else:
            std = c["geometry"] == "standard"
            pi = 3.14159265359 if std else math.pi
            ang = _angles(c)
            ang = ang.astype(np.float32).astype(np.float64) if std else ang
            sod, sdd = (SID_STD, SDD_STD) if std else (SOD, SDD)
            p = 1.0 if std else c["pitch"]
            b = ang / 180.0 * pi - pi / 2
            e = np.stack([np.cos(b), np.sin(b), 0 * b], 1)
            S, D = -sod * e, (sdd - sod) * e
            U = p * np.stack([-np.sin(b), np.cos(b), 0 * b], 1)
            V = np.zeros_like(U)
            V[:, 2] = p
            self.vox = sod / sdd if std else 1.0
            off, det_off, self.phase = (0.0, 0.0, "standard") if std else (0.5, 0.5, "box")
            self.power, self.bp_scale = 2, pi / len(b)
        self.views = S.shape[0]
        self.S, self.D, self.U, self.V = t64(S), t64(D), t64(U), t64(V)
        self.n3 = t64(self.n)
        self.O = (-self.n3 / 2 + off) * self.vox  # centre of voxel (0, 0, 0)
        self.cu, self.cv = -self.nu / 2 + det_off, -self.nv / 2 + det_off

    def rays(self, k):
        """Directions source -> pixel of view k, world units, [nv*nu, 3]."""
        u = torch.arange(self.nu, device=DEV, dtype=torch.float64) + self.cu
        v = torch.arange(self.nv, device=DEV, dtype=torch.float64) + self.cv
        P = self.D[k] + u[None, :, None] * self.U[k] + v[:, None, None] * self.V[k]
        return (P - self.S[k]).reshape(-1, 3)

    def alphas(self, k, r):
        """First sample's distance from the source and the sample count, per ray."""
        d = r / r.norm(dim=1, keepdim=True)
        if self.phase == "box":
            lo_c, hi_c = self.O - 0.5 * self.vox, self.O + (self.n3 - 0.5) * self.vox
            t0, t1 = (lo_c - self.S[k]) / d, (hi_c - self.S[k]) / d
            lo, hi = torch.minimum(t0, t1).amax(1), torch.maximum(t0, t1).amin(1)
            return d, lo + 0.5 * self.vox, torch.ceil((hi - lo).clamp_min(0) / self.vox)
        a = d.abs()
        ax = (a[:, 1] > a[:, 0]).long() if self.phase == "standard" else a.argmax(1)
        da, sa, ea = d.gather(1, ax[:, None])[:, 0], self.S[k][ax], self.n3[ax] / 2
        t0, t1 = (-ea - sa) / da, (ea - sa) / da
        lo, hi = torch.minimum(t0, t1) - 3, torch.maximum(t0, t1) + 3
        return d, lo, torch.ceil((hi - lo) / self.vox)

    def forward(self, x):
        """[B,1,Z,Y,X] float64 -> [B,1,N,nv,nu]."""
        B = x.shape[0]
        out = torch.zeros((B, self.views, self.nv * self.nu), dtype=torch.float64, device=DEV)
        vol = F.pad(x, (1, 1, 1, 1, 1, 1))
        span = (self.n3 + 1) / 2  # padded grid's half extent in voxels
        for k in range(self.views):
            r = self.rays(k)
            d, a0, count = self.alphas(k, r)
            # only samples inside (-1, n) on every axis can be non-zero
            base = (self.S[k] + a0[:, None] * d - self.O) / self.vox
            t0, t1 = (-1 - base) / d, (self.n3 - base) / d
            k0 = torch.minimum(t0, t1).amax(1).clamp_min(0).floor()
            k1 = torch.minimum(torch.maximum(t0, t1).amin(1).ceil() + 1, count)
            live = torch.nonzero(k1 > k0)[:, 0]
            if not live.numel():
                continue
            K = int((k1 - k0)[live].max())
            step = max(1, 60_000_000 // K)
            for i in range(0, live.numel(), step):
                s = live[i:i + step]
                kk = k0[s, None] + torch.arange(K, device=DEV, dtype=torch.float64)
                pos = base[s, None, :] + kk[:, :, None] * d[s, None, :]
                pos = (pos + 1) / span - 1
                val = F.grid_sample(vol, pos[None, :, :, None, :].expand(B, -1, -1, -1, -1),
                                    mode="bilinear", padding_mode="zeros", align_corners=True)
                val = val[:, 0, :, :, 0] * (kk < count[s, None])
                out[:, k, s] = val.sum(2) * self.vox
        return out.reshape(B, 1, self.views, self.nv, self.nu)

    def adjoint(self, y):
        """The transpose of forward, [B,1,N,nv,nu] -> [B,1,Z,Y,X]."""
        x = torch.zeros((y.shape[0], 1) + self.n[::-1], dtype=torch.float64, device=DEV)
        for k in range(self.views):
            one = _one_view(self, k)
            with torch.enable_grad():
                z = torch.zeros_like(x).requires_grad_()
                x += torch.autograd.grad(one.forward(z), z, y[:, :, k:k + 1])[0]
        return x

    def backward(self, y):
        """FDK-weighted backprojection, [B,1,N,nv,nu] -> [B,1,Z,Y,X]."""
        X, Y, Z = self.n
        B = y.shape[0]
        ax = [torch.arange(n, device=DEV, dtype=torch.float64) * self.vox + self.O[i]
              for i, n in enumerate(self.n)]
        out = torch.zeros((B, Z, Y, X), dtype=torch.float64, device=DEV)
        zstep = max(1, 40_000_000 // (X * Y))
        for k in range(self.views):
            S, D, U, V = self.S[k], self.D[k], self.U[k], self.V[k]
            nr = torch.linalg.cross(U, V)
            sdd = torch.dot(D - S, nr)
            vn, nu_ = torch.linalg.cross(V, nr), torch.linalg.cross(nr, U)
            Ut, Vt = vn / torch.dot(U, vn), nu_ / torch.dot(V, nu_)
            img = F.pad(y[:, :, k], (1, 1, 1, 1))
            for z0 in range(0, Z, zstep):
                lin = lambda w: ((ax[2][z0:z0 + zstep, None, None] - S[2]) * w[2]  # noqa: E731
                                 + (ax[1][:, None] - S[1]) * w[1] + (ax[0] - S[0]) * w[0])
                h = lin(nr) / sdd
                u = lin(Ut) / h + torch.dot(Ut, S - D) - self.cu
                v = lin(Vt) / h + torch.dot(Vt, S - D) - self.cv
                g = torch.stack([(u + 1) * 2 / (self.nu + 1) - 1, (v + 1) * 2 / (self.nv + 1) - 1], -1)
                w = self.bp_scale / h ** self.power
                if self.phase == "vector":  # the reference's extent test on the volume size
                    w = w * ((u + 0.5 >= -1) & (u + 0.5 <= X + 1) & (v + 0.5 >= -1) & (v + 0.5 <= Y + 1))
                zz = g.shape[0]
                val = F.grid_sample(img, g.reshape(1, zz * Y, X, 2).expand(B, -1, -1, -1),
                                    mode="bilinear", padding_mode="zeros", align_corners=True)
                out[:, z0:z0 + zz] += val.reshape(B, zz, Y, X) * w
        return out[:, None]

    def samples(self):
        """Ray samples of one volume, from the rays' density at the volume."""
        rays = (self.D - self.S).norm(dim=1) / self.S.norm(dim=1) * self.vox
        area = torch.linalg.cross(self.U, self.V).norm(dim=1)
        per = float((rays ** 2 / area).sum())
        dense = per * self.n[0] * self.n[1] * self.n[2]
        return min(dense, self.views * self.nu * self.nv * 1.2 * max(self.n))


def _one_view(scan, k):
    one = object.__new__(_Scan)
    one.__dict__.update(scan.__dict__)
    one.views = 1
    for a in ("S", "D", "U", "V"):
        setattr(one, a, getattr(scan, a)[k:k + 1])
    return one


# ---- inputs --------------------------------------------------------------------------------
def _phantom(c, seed):
    vol = dtvb200.phantom.ellipsoids((c["nz"], c["ny"], c["nx"]), seed=seed, device=DEV)
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    return vol + 0.01 * torch.randn(vol.shape, generator=g, device=DEV)  # a reconstruction's noise


def _sinogram(c, seed):
    """Line integrals of the seed's phantom over every ray, with Poisson noise."""
    scan = _Scan(c)
    cen, axs, R, val = dtvb200.phantom.ellipsoid_params(seed)
    edge = max(scan.n)
    out = torch.zeros((scan.views, scan.nv * scan.nu), dtype=torch.float64, device=DEV)
    mid = (scan.n3 - 1) / 2
    # rays in each ellipsoid's unit-ball coordinates
    maps = [torch.tensor(R[e].T / (2.0 * axs[e])[:, None], device=DEV) * (2.0 / edge / scan.vox)
            for e in range(len(val))]
    for k in range(scan.views):
        r = scan.rays(k)
        length = r.norm(dim=1)
        q0 = scan.S[k] - scan.O - mid * scan.vox
        for e in range(len(val)):
            c0 = torch.tensor(cen[e], device=DEV) * (edge * scan.vox / 2)
            o, d = maps[e] @ (q0 - c0), r @ maps[e].T
            A, Bq, Cq = (d * d).sum(1), d @ o, torch.dot(o, o) - 1
            out[k] += float(val[e]) * 2 * torch.sqrt((Bq * Bq - A * Cq).clamp_min(0)) / A * length
    sino = out.reshape(1, 1, scan.views, scan.nv, scan.nu).clamp_min(0)
    return dtvb200.phantom.poisson_noise(sino, seed=seed).to(torch.float32)


def _step(c):
    """A stable gradient step for BP(FP): the inverse of about its norm."""
    mag = SDD / SOD
    return 0.6 / (math.pi * mag * mag * max(c["nx"], c["ny"]))


def _members(c):
    """The reconstructions of a batch: edges 1, 1/2, 3/4 of the first one's."""
    out = []
    for i in range(c["batch"]):
        k = (1.0, 0.5, 0.75, 0.5)[i]
        e = lambda n: max(8, int(n * k))  # noqa: E731
        out.append(dict(c, nx=e(c["nx"]), ny=e(c["ny"]), nz=e(c["nz"]), nu=e(c["nu"]), nv=e(c["nv"]),
                        views=max(8, c["views"] - 9 * i), batch=1))
    return out


def _net(c, projector):
    torch.manual_seed(7)
    return dtvb200.nets.UnrolledPDHG(projector, stages=c["iters"], features=32, lamb=_step(c) / 10,
                                     tau=1e-2).to(DEV)


def _inputs(c, seed):
    """The tensors of a pass, by name."""
    kind = c["kind"]
    if kind == "batch":
        return {"sino": [_sinogram(m, seed + i) for i, m in enumerate(_members(c))]}
    t = {}
    if kind in ("dropin", "layer", "forward", "grad", "fbp"):
        t["vol"] = torch.cat([_phantom(c, seed + b) for b in range(c["batch"])]).to(DTYPES[c["dtype"]])
    if kind != "forward":
        t["sino"] = torch.cat([_sinogram(c, seed + b) for b in range(c["batch"])])
    if kind == "train":
        t["truth"] = torch.cat([dtvb200.phantom.ellipsoids((c["nz"], c["ny"], c["nx"]), seed=seed + b,
                                                           device=DEV) for b in range(c["batch"])])
    if kind == "grad":
        g = torch.Generator(device=DEV).manual_seed(seed + 5)
        t["out_grad"] = torch.randn(t["vol"].shape, generator=g, device=DEV)
    if kind == "fbp":  # the layers hand sinograms round as (angle, row, plane, column)
        t["sino"] = _to_layer(c, t["sino"])
    return t


def _to_layer(c, s):
    P, H, W = c["planes"], c["nv"], c["nu"]
    return s.reshape(-1, c["views"] // P, P, H, W).permute(0, 1, 3, 2, 4).reshape(s.shape).contiguous()


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = dict(_inputs(c, seed), kind=kind)
    size, det = (c["nx"], c["ny"], c["nz"]), (c["nu"], c["nv"])
    if kind == "dropin":
        st["angles"] = torch.tensor(_angles(c), device=DEV)
        st["size"], st["det"] = torch.tensor(size, device=DEV), torch.tensor(det, device=DEV)
        return st
    if kind == "batch":
        plans = [dtvb200.Plan(_geometry(m), sampler=c["sampler"], device=DEV) for m in _members(c)]
        st["alg"] = dtvb200.Batched([dtvb200.FISTA(p, c["iters"], lamb=0.05, L=_step(m))
                                     for p, m in zip(plans, _members(c))], use_graph=True)
        st["image"] = [torch.zeros(p.vol_shape(1), device=DEV) for p in plans]
        return st
    geo = _geometry(c)
    if kind in ("layer", "grad", "fbp", "train"):
        proj = dtvb200.Projector(geo, sampler=c["sampler"], max_batch=c["batch"])
        if kind == "fbp":
            st["layer"] = dtvb200.BeijingGeometryWithFBP(
                proj, 2.8 * max(c["nx"], c["ny"]), c["planes"]).to(DEV)
        elif kind == "train":
            st["net"] = _net(c, proj)
            st["opt"] = torch.optim.Adam(st["net"].parameters(), lr=1e-4)
            st["image"] = torch.zeros_like(st["truth"])
        else:
            st["layer"] = dtvb200.StandardGeometry(proj, matched=kind == "grad", lamb=_step(c))
        proj.plan(torch.device(DEV, torch.cuda.current_device()), c["batch"])
        return st
    plan = st["plan"] = dtvb200.Plan(geo, c["batch"], sampler=c["sampler"], device=DEV)
    if kind in ("dtv", "fista_tv", "asd"):
        st["image"] = torch.zeros(plan.vol_shape(1), device=DEV)
    if kind == "dtv":
        fast = c["sampler"] == "pairs"
        exact = dtvb200.Plan(geo, sampler="exact", device=DEV) if fast else None
        st["alg"] = dtvb200.DTVCP(plan, c["iters"], sigma=_step(c), tau=_step(c), mu=1.0, v=(0.5,) * 3,
                                  quirk=False, f_dtype=DTYPES[c["dtype"]], use_graph=fast, exact=exact)
    elif kind == "fista_tv":
        st["alg"] = dtvb200.DTVFISTA(plan, c["iters"], sigma=_step(c), v=(0.02,) * 3, t=(1e-3,) * 3,
                                     quirk=False, use_graph=True)
    elif kind == "asd":
        st["alg"] = dtvb200.ASDPOCS(plan, c["iters"], beta=_step(c), alpha=0.2, quirk=False)
    return st


def run(st):
    kind = st["kind"]
    if kind == "dropin":
        a = (st["angles"], st["size"], st["det"], SID_STD, SDD_STD, torch.cuda.current_device())
        return dropin.forward(st["vol"], *a), dropin.backward(st["sino"], *a)
    if kind == "forward":
        return st["plan"].forward(st["vol"])
    if kind == "backward":
        return st["plan"].backward(st["sino"])
    if kind in ("layer", "fbp"):
        with torch.no_grad():
            return st["layer"](st["vol"], st["sino"])
    if kind == "grad":
        x = st["vol"].detach().requires_grad_()
        y = st["layer"](x, st["sino"])
        y.backward(st["out_grad"])
        return y.detach(), x.grad
    if kind == "train":
        net = st["net"]
        st["opt"].zero_grad(set_to_none=True)
        out = net(st["image"], st["sino"])
        torch.mean((out - st["truth"]) ** 2).backward()
        st["opt"].step()
        return [out.detach()] + [p.detach() for p in net.parameters()]
    return st["alg"].run(st["image"], st["sino"])


def work(case):
    c, kind = case, case["kind"]
    if kind == "batch":
        parts = [work(dict(m, kind="fista")) for m in _members(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    vox, pix = c["nx"] * c["ny"] * c["nz"], c["views"] * c["nu"] * c["nv"]
    B = c["batch"]
    fp, bp = 25.0 * _Scan(c).samples(), 16.0 * vox * c["views"]
    pairs = {"dropin": 1, "layer": 1, "fbp": 1, "grad": 2, "train": 2 * c["iters"]}.get(kind, c["iters"])
    adj = fp if kind in ("grad", "train") else bp
    if kind in ("forward", "backward"):
        esz = {"f32": 4}.get(c["dtype"], 2) if kind == "forward" else 4
        return {"bytes": B * (esz * vox + 4.0 * pix), "flops": B * (fp if kind == "forward" else bp)}
    extra = 0.0
    if kind == "train":  # three convolutions, forward and both gradients
        extra = 3 * c["iters"] * 2.0 * 27 * (32 * 32 + 2 * 32) * vox
    vols = {"dropin": 2, "grad": 4, "dtv": 2, "train": 3}.get(kind, 2)
    sinos = {"dropin": 2}.get(kind, 1)
    return {"bytes": B * 4.0 * (vols * vox + sinos * pix), "flops": B * (pairs * (fp + adj) + extra)}


# ---- the same in 64 bits --------------------------------------------------------------------
def _d(x, axis, transpose=False):
    """D = shift - I along x, y, z (clean borders), or its transpose."""
    dim = -1 - axis
    n = x.shape[dim]
    out = -x.clone()
    if transpose:
        out.narrow(dim, 1, n - 1).add_(x.narrow(dim, 0, n - 1))
    else:
        out.narrow(dim, 0, n - 1).add_(x.narrow(dim, 1, n - 1))
    return out


def _soft(x, t):
    return torch.sign(x) * (x.abs() - t).clamp_min(0)


def _l1_threshold(a, radius):
    u = a.abs().reshape(-1)
    if float(u.sum()) < radius:
        return 0.0
    if radius <= 0:
        return float(u.max())
    u = torch.sort(u, descending=True)[0]
    cs = torch.cumsum(u, 0)
    j = torch.arange(1, u.numel() + 1, device=u.device, dtype=torch.float64)
    rho = int(torch.nonzero(u - (cs - radius) / j > 0)[-1])
    return float((cs[rho] - radius) / (rho + 1))


def _exact_dtv(c, scan, g):
    sg, mu, v = _step(c), 1.0, 0.5
    f = torch.zeros((1, 1) + scan.n[::-1], dtype=torch.float64, device=DEV)
    fbar, w, cc = f.clone(), torch.zeros_like(g), torch.zeros_like(f)
    duals, t = [torch.zeros_like(f) for _ in range(3)], [0.0] * 3
    for it in range(c["iters"]):
        if it % 10 == 0:
            t = [float(_d(f, a).abs().sum()) for a in range(3)]
        w = (w + sg * (scan.forward(fbar) - g)) / (1 + sg)
        recon = scan.backward(w)
        for a in range(3):
            y = duals[a] + v * sg * _d(fbar, a)
            lam = _l1_threshold(y, sg * v * t[a])
            duals[a] = y.clamp(-lam, lam)
        cc = -(-cc - sg * mu * fbar).clamp_min(0)
        reg = mu * cc + sum(v * _d(duals[a], a, True) for a in range(3))
        fn = f - recon - sg * reg
        fbar, f = 2 * fn - f, fn
    return f


def _exact_fista(c, scan, g, tv):
    L = _step(c)
    x = torch.zeros((1, 1) + scan.n[::-1], dtype=torch.float64, device=DEV)
    y, t = x.clone(), 1.0
    for _ in range(c["iters"]):
        tp = (1 + math.sqrt(1 + 4 * t * t)) / 2
        z = y - L * scan.backward(scan.forward(y) - g)
        if tv:
            z = z.clamp_min(0)
            n = z + sum(1e-3 * _d(_soft(_d(z, a), 0.02), a, True) for a in range(3))
            y = n + (t - 1) / tp * (n - y)
        else:
            n = _soft(z, 0.05 * L)
            y, x = n + (t - 1) / tp * (n - x), n
        t = tp
    return y if tv else x


def _exact_asd(c, scan, g):
    beta, alpha, rmax, davg = _step(c), 0.2, 0.95, 1.0
    f = torch.zeros((1, 1) + scan.n[::-1], dtype=torch.float64, device=DEV)
    for i in range(c["iters"]):
        f0 = f
        f = f0 - beta * scan.backward(scan.forward(f0) - g)
        dp = float((f0 - f).abs().mean())
        davg = alpha * dp if i == 0 else davg
        data = f
        for _ in range(10):
            ds = [_d(f, a) for a in range(3)]
            nrm = torch.sqrt(sum(x * x for x in ds)) + 1
            f = f - davg * sum(_d(ds[a] / nrm, a, True) for a in range(3))
        if float((f - data).abs().mean()) > rmax * dp:
            davg *= alpha
        beta *= 0.9999
    return f.clamp_min(0)


def _exact_fbp(c, scan, x, p):
    P, W, H, A = c["planes"], c["nu"], c["nv"], c["views"] // c["planes"]
    row, sdd = W * P, 2.8 * max(c["nx"], c["ny"])
    r = _to_layer(c, scan.forward(x)) - p
    i = torch.arange(H, device=DEV, dtype=torch.float64)[:, None] - row / 2
    j = torch.arange(row, device=DEV, dtype=torch.float64)[None, :] - H / 2
    r = r.reshape(1, A, H, row) * (sdd / torch.sqrt(sdd ** 2 + i ** 2 + j ** 2))
    k = np.arange(row + 1) - row // 2
    with np.errstate(divide="ignore"):
        taps = np.where(k % 2 == 0, 0.0, -0.5 / (np.pi ** 2 * k.astype(np.float64) ** 2))
    taps[row // 2] = 0.125
    full = 2 * row + 1  # correlation with zero padding by the FFT
    k64 = torch.tensor(taps, device=DEV)
    spec = torch.fft.rfft(F.pad(r, (row // 2, row // 2)), full) * torch.fft.rfft(k64, full).conj()
    r = torch.fft.irfft(spec, full)[..., :row]
    r = r.reshape(1, A, H, P, W).permute(0, 1, 3, 2, 4).reshape(1, 1, c["views"], H, W)
    return x - scan.backward(r)


def _exact_train(c, scan, t):
    proj = dtvb200.Projector(_geometry(c), max_batch=c["batch"])  # holds no numbers of the net
    net = _net(c, proj).double()
    opt = torch.optim.Adam(net.parameters(), lr=1e-4)

    class Fwd(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            return scan.forward(x)

        @staticmethod
        def backward(ctx, g):
            return scan.adjoint(g)

    class Adj(torch.autograd.Function):
        @staticmethod
        def forward(ctx, y):
            return scan.adjoint(y)

        @staticmethod
        def backward(ctx, g):
            return scan.forward(g)

    x = torch.zeros_like(t["truth"], dtype=torch.float64)
    for s in range(c["iters"]):
        x = x - net.lamb[s] * Adj.apply(Fwd.apply(x) - t["sino"].double()) - net.tau[s] * net.blocks[s](x)
    torch.mean((x - t["truth"].double()) ** 2).backward()
    opt.step()
    return [x.detach()] + [p.detach() for p in net.parameters()]


def exact(case, seed):
    c, kind = case, case["kind"]
    with torch.no_grad():
        t = _inputs(c, seed)
        if kind == "batch":
            return [_exact_fista(m, _Scan(m), s.double(), False) for m, s in zip(_members(c), t["sino"])]
        scan = _Scan(c)
        vol, sino = (t[k].double() if k in t else None for k in ("vol", "sino"))
        if kind == "dropin":
            return scan.forward(vol), scan.backward(sino)
        if kind == "forward":
            return scan.forward(vol)
        if kind == "backward":
            return scan.backward(sino)
        if kind == "layer":
            return vol - _step(c) * scan.backward(scan.forward(vol) - sino)
        if kind == "grad":
            y = vol - _step(c) * scan.adjoint(scan.forward(vol) - sino)
            g = t["out_grad"].double()
            return y, g - _step(c) * scan.adjoint(scan.forward(g))
        if kind == "fbp":
            return _exact_fbp(c, scan, vol, sino)
        if kind == "dtv":
            return _exact_dtv(c, scan, sino)
        if kind == "asd":
            return _exact_asd(c, scan, sino)
        if kind == "fista_tv":
            return _exact_fista(c, scan, sino, True)
    return _exact_train(c, scan, t)
