"""The workloads whose speed is tracked: the framework's main path through its
public entry points, over the sizes, storage types and scanners it is used with.

``listed()`` names them, ``draw(rng)`` makes one more of the same ranges,
``prepare`` builds what a program holds before the call (geometry handle,
volume, measured data), ``run`` is one pass, ``work`` the bytes and operations a
pass cannot do without, and ``exact`` the pass's outputs in 64 bits from plain
torch.  Lengths are millimetres.
"""
import math

import numpy as np
import torch

import gpu_b200
from gpu_b200 import autograd

DT = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
CODE = {"f32": gpu_b200.F32, "bf16": gpu_b200.BF16, "f16": gpu_b200.F16}
TETRA = 3  # ct_style of the tetrahedron beam

# The working-size scan: 512^3 voxels, 1024 views of a 1024 x 768 detector.
SCAN512 = dict(nx=512, ny=512, nz=512, nu=1024, nv=768, n_views=1024, vx=0.5, du=0.4, dso=1000.0, dod=-500.0, style=0,
               n_sources=0)
# The plain method's small scan: 128^3, 180 views, 128^2 detector.
SCAN128 = dict(nx=128, ny=128, nz=128, nu=128, nv=128, n_views=180, vx=1.0, du=1.6, dso=1000.0, dod=-500.0, style=0,
               n_sources=0)
# The gradient-based reconstruction's scan: 256^3, 360 views, 384^2 detector.
SCAN256 = dict(nx=256, ny=256, nz=256, nu=384, nv=384, n_views=360, vx=0.5, du=204.8 / 384, dso=1000.0, dod=-500.0,
               style=0, n_sources=0)
# The tetrahedron-beam scan: 512^3, 64 sources of 16 detector rows, 360 views.
SCAN_TETRA = dict(nx=512, ny=512, nz=512, nu=1024, nv=16, n_views=360, vx=0.1, du=0.12, dso=200.0, dod=-200.0,
                  style=TETRA, n_sources=64)


def listed():
    return [
        # one view of a small volume: an interactive re-projection, all latency
        dict(SCAN128, name="project_one_view", kind="project", views=1, dtype="f32", fast=False),
        # simulating or re-projecting a chunk of views at the working size, the default arithmetic
        dict(SCAN512, name="project_chunk", kind="project", views=32, dtype="f32", fast=False),
        # a reduced-precision volume of odd sizes, fused ray sums
        dict(SCAN128, name="project_ragged_mixed", kind="project", nx=301, ny=259, nz=211, nu=413, nv=301, vx=0.8,
             du=0.9, views=60, dtype="bf16", fast=True),
        # one step of gradient-based reconstruction: the loss and its gradient (projector forward, adjoint backward)
        dict(SCAN256, name="gradient_step", kind="gradient", chunk=64),
        # the reference's host call on host arrays: one SART pass of the small plain scan
        dict(SCAN128, name="dropin_small", kind="dropin", beta=0.8),
        # SART views of the working-size scan in FP32
        dict(SCAN512, name="sart_working_size", kind="sart", views=16, dtype="f32", beta=0.8),
        # SART views of the tetrahedron-beam scanner on FP16 storage
        dict(SCAN_TETRA, name="sart_tetrahedron", kind="sart", views=10, dtype="f16", beta=0.8),
        # whole iterations of the mixed-precision solver (SART + FISTA + FGP-TV): the headline engine at medium size
        dict(SCAN256, name="solver_mixed", kind="solver", dtype="f16", fast=True, beta=0.0625, lam=2e-4, iters=2),
        # the TV prox alone at the working size
        dict(name="denoise_working_size", kind="denoise", nx=512, ny=512, nz=512, dtype="f32", lam=1.25e-5, iters=20),
        # the TV prox of an odd-sized BF16 volume
        dict(name="denoise_ragged_bf16", kind="denoise", nx=333, ny=257, nz=190, dtype="bf16", lam=1.25e-5, iters=20),
        # a full analytic reconstruction of the working-size scan: the largest call
        dict(SCAN512, name="fdk_working_size", kind="fdk"),
        # many small scans of uneven sizes iterated together
        dict(name="batch_uneven", kind="batch", scans=12, shapes=4, dtype="bf16", beta=0.0625, lam=2e-4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_scan(rng, most):
    """A cone-beam scan of a drawn size: the voxel pitch and the detector follow the volume as the listed ones do.
    nx + ny is even: with an odd sum the backprojectors of the version these cases were first timed on read a
    misaligned shared-memory table."""
    n = _log_int(rng, 64, most)
    nx, ny = n, n + 2 * int(0.5 * n * rng.uniform(-0.2, 0.15))
    nz = max(16, int(n * rng.uniform(0.6, 1.05)))
    vx = rng.choice([0.25, 0.5, 0.8, 1.0]) if n > 160 else rng.choice([0.5, 1.0, 1.3])
    vx = min(vx, 260.0 / n)
    nu, nv = int(n * rng.uniform(1.0, 2.0)), int(n * rng.uniform(0.9, 1.5))
    du = 1.5 * vx * max(nx, ny) / nu * rng.uniform(0.85, 1.2)
    return dict(nx=nx, ny=ny, nz=nz, nu=nu, nv=nv, n_views=_log_int(rng, 90, 720), vx=vx, du=du, dso=1000.0,
                dod=-500.0, style=0, n_sources=0)


def draw(rng):
    kind = rng.choice(["project", "project", "gradient", "sart", "sart", "solver", "denoise", "denoise", "fdk", "dropin",
                       "batch"])
    if kind == "denoise":
        return dict(kind=kind, nx=_log_int(rng, 48, 512), ny=_log_int(rng, 48, 512), nz=_log_int(rng, 48, 512),
                    dtype=rng.choice(["f32", "bf16", "f16"]), lam=rng.choice([1.25e-5, 1e-4]), iters=20)
    if kind == "batch":
        return dict(kind=kind, scans=rng.randint(4, 12), shapes=rng.randint(1, 999), dtype="bf16", beta=0.0625, lam=2e-4)
    if kind == "project":
        s = _draw_scan(rng, 512)
        s["style"] = rng.choice([0, 0, 0, 1, 2])
        return dict(s, kind=kind, views=min(_log_int(rng, 1, 48), s["n_views"]), dtype=rng.choice(["f32", "bf16", "f16"]),
                    fast=rng.random() < 0.5)
    if kind == "sart":
        if rng.random() < 0.3:  # the tetrahedron beam, its detector band shorter than the magnified volume
            n = _log_int(rng, 96, 512)
            s = dict(SCAN_TETRA, nx=n, ny=n, nz=n, vx=51.2 / n, nu=2 * n, du=61.44 / n, nv=rng.choice([6, 8, 12]),
                     n_sources=rng.choice([24, 32, 48]))
        else:
            s = _draw_scan(rng, 512)
        return dict(s, kind=kind, views=rng.randint(4, 16), dtype=rng.choice(["f32", "f16"]), beta=0.8)
    if kind == "fdk":
        return dict(_draw_scan(rng, 400), kind=kind)
    s = _draw_scan(rng, 224)
    s["n_views"] = min(s["n_views"], 360)
    if kind == "gradient":
        return dict(s, kind=kind, chunk=rng.choice([32, 64]))
    if kind == "dropin":
        return dict(s, kind=kind, beta=0.8)
    return dict(s, kind="solver", dtype=rng.choice(["f32", "f16", "bf16"]), fast=rng.random() < 0.5, beta=0.0625, lam=2e-4,
                iters=2)


# ------------------------------------------------------------------ inputs

def _batch_scans(case):
    """The scans of a batch case: cubes of 48 to 192 voxels, each with its own views, detector and distance."""
    rng = np.random.default_rng(case["shapes"])
    out = []
    for _ in range(case["scans"]):
        n = int(rng.choice([48, 64, 96, 128, 192]))
        nv = int(rng.integers(96, 257))
        dso = float(rng.uniform(600.0, 1200.0))
        out.append(dict(nx=n, ny=n, nz=n, nu=nv, nv=nv, n_views=int(rng.integers(90, 200)), vx=128.0 / n, du=204.8 / nv,
                        dso=dso, dod=-0.5 * dso, style=0, n_sources=0))
    return out


def _vz(s):
    return s["du"] if s["style"] in (1, 2) else s["vx"]


def _desc(s, fast=False):
    return gpu_b200.make_desc(s["nx"], s["ny"], s["nz"], s["vx"], s["nu"], s["nv"], s["du"], s["dso"], s["dod"],
                              s["n_views"], ct_style=s["style"], n_sources=s["n_sources"], fast_sums=fast)


def _rows(s):
    return s["nv"] * (s["n_sources"] if s["style"] == TETRA else 1)


def _ellipsoids(s, seed, n=6):
    """n random ellipsoids inside the field of view: centres, rotation/semi-axis matrices, attenuations (per mm)."""
    r = np.random.default_rng(seed)
    ext = 0.5 * np.array([s["nx"] * s["vx"], s["ny"] * s["vx"], s["nz"] * _vz(s)])
    c = r.uniform(-0.45, 0.45, (n, 3)) * ext
    ax = r.uniform(0.05, 0.45, (n, 3)) * ext.min()
    q, _ = np.linalg.qr(r.standard_normal((n, 3, 3)))
    w = q / ax[:, :, None]
    return [torch.tensor(a, dtype=torch.float32, device="cuda") for a in (c, w, r.uniform(0.005, 0.03, n))]


def _centres(n, pitch, dtype=torch.float32):
    return (torch.arange(n, device="cuda", dtype=dtype) + 0.5 - 0.5 * n) * pitch


def _phantom(s, seed):
    """The ellipsoids on the voxel grid, with the texture of a reconstruction (3 % noise), FP32."""
    c, w, mu = _ellipsoids(s, seed)
    x, y, z = (_centres(n, p) for n, p in ((s["nx"], s["vx"]), (s["ny"], s["vx"]), (s["nz"], _vz(s))))
    vol = torch.zeros((s["nz"], s["ny"], s["nx"]), device="cuda")
    for a in range(len(mu)):
        r2 = 0.0
        for b in range(3):
            r2 = r2 + (w[a, b, 2] * (z - c[a, 2])[:, None, None] + w[a, b, 1] * (y - c[a, 1])[None, :, None]
                       + w[a, b, 0] * (x - c[a, 0])[None, None, :]) ** 2
        vol += mu[a] * (r2 <= 1.0)
    g = torch.Generator(device="cuda").manual_seed(seed)
    return vol.add_(torch.rand(vol.shape, device="cuda", generator=g), alpha=9e-4)


def _rays(s, views, dtype):
    """Source and detector-pixel positions (x, y, z, broadcastable to (views, rows, nu)) of a range of views."""
    kw = dict(device="cuda", dtype=dtype)
    th = torch.tensor([-j * (360.0 / s["n_views"]) * math.pi / 180.0 for j in views], dtype=torch.float64)[:, None, None]
    sn, cs = torch.sin(th).to(**kw), torch.cos(th).to(**kw)
    pu = (torch.arange(s["nu"], **kw) + 0.5 - 0.5 * s["nu"])[None, None, :] * s["du"]
    v = torch.arange(_rows(s), **kw)[None, :, None]
    src = torch.div(v, s["nv"], rounding_mode="floor") if s["style"] == TETRA else torch.zeros_like(v)
    dz = (v - src * s["nv"] + 0.5 - 0.5 * s["nv"]) * s["du"]
    sy = pu if s["style"] == 2 else torch.zeros_like(pu)
    if s["style"] in (1, 2):
        sz = dz
    elif s["style"] == TETRA:  # the first source sees the volume's bottom face from the bottom row, the last its top face
        top, zm = 0.5 * s["nz"] * s["vx"], (0.5 * s["nv"] - 0.5) * s["du"]
        z0 = (zm - top) * (s["dso"] - s["dod"]) / s["dso"] - zm
        sz = z0 + src * (-2.0 * z0 / (s["n_sources"] - 1))
    else:
        sz = torch.zeros_like(dz)
    return ((s["dso"] * cs - sy * sn, s["dso"] * sn + sy * cs, sz), (s["dod"] * cs - pu * sn, s["dod"] * sn + pu * cs, dz))


def _measured(s, seed, views):
    """Line integrals of the ellipsoids for views [0, views), with 0.5 % noise, FP32."""
    c, w, mu = _ellipsoids(s, seed)
    out = torch.zeros((views, _rows(s), s["nu"]), device="cuda")
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    group = max(1, 2000000 // (_rows(s) * s["nu"]))
    for j in range(0, views, group):
        acc = out[j:j + group]
        p, q = _rays(s, range(j, j + acc.shape[0]), torch.float32)
        d = [b - a for a, b in zip(p, q)]
        norm = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
        for e in range(len(mu)):
            o = [a - c[e, k] for k, a in enumerate(p)]
            aa = bb = cc = 0.0
            for k in range(3):  # the in-plane terms do not depend on the row: summed before they meet the z terms
                dk = (w[e, k, 0] * d[0] + w[e, k, 1] * d[1]) + w[e, k, 2] * d[2]
                ok = (w[e, k, 0] * o[0] + w[e, k, 1] * o[1]) + w[e, k, 2] * o[2]
                aa, bb, cc = aa + dk * dk, bb + dk * ok, cc + ok * ok
            disc = torch.clamp(bb * bb - aa * (cc - 1.0), min=0.0)
            acc += 2.0 * mu[e] * norm * torch.sqrt(disc) / aa
        noise = torch.randn(acc.shape, device="cuda", generator=g)
        acc.add_(noise, alpha=0.005 * 0.1 * 0.25 * s["nx"] * s["vx"])
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "denoise":
        s = dict(case, vx=0.5, style=0)
        geom = gpu_b200.Geometry(gpu_b200.make_desc(s["nx"], s["ny"], s["nz"], 0.5, 64, 64, 1.0, 1000.0, -1000.0, 8))
        return dict(case=case, geom=geom, noisy=_phantom(s, seed).to(DT[case["dtype"]]),
                    out=torch.empty((s["nz"], s["ny"], s["nx"]), device="cuda", dtype=DT[case["dtype"]]))
    if kind == "batch":
        scans = _batch_scans(case)
        geoms = [gpu_b200.Geometry(_desc(s)) for s in scans]
        b = gpu_b200.Batch(geoms, CODE[case["dtype"]], beta=case["beta"], lambda_tv=case["lam"], fgp_iters=20, refine=2)
        for i, s in enumerate(scans):
            b.set_sinogram(i, _measured(s, seed + i, s["n_views"]))
        return dict(case=case, batch=b, out=[torch.empty(g.vol_shape, device="cuda") for g in geoms])
    if kind == "dropin":
        gpu_b200.set_default_geometry(_desc(case))
        return dict(case=case, vol=np.zeros((case["nz"], case["ny"], case["nx"]), np.float32),
                    sino=_measured(case, seed, case["n_views"]).cpu().numpy())
    geom = gpu_b200.Geometry(_desc(case, case.get("fast", False)))
    state = dict(case=case, geom=geom)
    if kind == "project":
        state.update(vol=_phantom(case, seed).to(DT[case["dtype"]]),
                     out=torch.empty((case["views"],) + geom.view_shape, device="cuda"))
    elif kind == "gradient":
        state.update(vol=_phantom(case, seed + 7).requires_grad_(True), sino=_measured(case, seed, case["n_views"]))
    elif kind == "sart":
        state.update(start=(0.5 * _phantom(case, seed)).to(DT[case["dtype"]]), sino=_measured(case, seed, case["views"]))
        state["vol"] = torch.empty_like(state["start"])
        full = torch.zeros((case["n_views"],) + geom.view_shape, device="cuda")
        full[: case["views"]] = state["sino"]
        state["sino"] = full
    elif kind == "solver":
        state.update(sino=_measured(case, seed, case["n_views"]).to(DT[case["dtype"]]),
                     out=torch.empty(geom.vol_shape, device="cuda"))
        state["solver"] = gpu_b200.Solver(geom, CODE[case["dtype"]], beta=case["beta"], lambda_tv=case["lam"],
                                          fgp_iters=20, refine=0 if case["dtype"] == "f32" else 2)
        state["solver"].set_sinogram(state["sino"])
    else:
        state.update(sino=_measured(case, seed, case["n_views"]), out=torch.empty(geom.vol_shape, device="cuda"))
    return state


# ------------------------------------------------------------------ one pass

def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "project":
        return state["geom"].forward(state["vol"], state["out"], 0, case["views"])
    if kind == "gradient":
        loss = autograd.data_fidelity_loss(state["vol"], state["sino"], state["geom"], case["chunk"])
        grad, = torch.autograd.grad(loss, state["vol"])
        return {"loss": loss.detach(), "grad": grad}
    if kind == "dropin":
        state["vol"][...] = 0.0
        gpu_b200.reconstruction_3d_ray_driven_cbct(state["vol"], state["sino"], case["beta"])
        return state["vol"]
    if kind == "sart":
        state["vol"].copy_(state["start"])
        state["geom"].sart_views(state["vol"], state["sino"], case["beta"], 0, case["views"], flags=gpu_b200.SART_TILED)
        return state["vol"]
    if kind == "solver":
        state["solver"].set_volume(None)
        state["solver"].iterate(case["iters"], objectives=False)
        return state["solver"].get_volume_f32(state["out"])
    if kind == "denoise":
        state["out"].copy_(state["noisy"])
        return state["geom"].fgp_tv(state["out"], case["lam"], case["iters"])
    if kind == "fdk":
        return state["geom"].fdk(state["sino"], state["out"].zero_())
    state["batch"].reset()
    state["batch"].iterate(1)
    return [state["batch"].get_volume_f32(i, out) for i, out in enumerate(state["out"])]


# ------------------------------------------------------------------ the work of a pass

def _pairs(s):
    """(Voxel, ray) intersections of one view: each voxel's mean projected area over a detector pixel's."""
    mag = 1.0 if s["style"] == 2 else (s["dso"] - s["dod"]) / s["dso"]
    fan = 1.0 if s["style"] in (1, 2) else mag
    per = 1.27 * (s["vx"] * mag / s["du"]) * (_vz(s) * fan / s["du"])
    if s["style"] == TETRA:  # the sources' bands overlap: the rows of all sources over the volume's height
        per = 1.27 * (s["vx"] * mag / s["du"]) * _rows(s) / s["nz"]
    return s["nx"] * s["ny"] * s["nz"] * per


def work(case):
    """Bytes: inputs read once, outputs written once.  Operations: 4 per intersection of a projection (alpha step, chord,
    product, sum), 6 of a SART update (overlap, chord, two products and sums), 40 per voxel of a TV step, 20 per
    (voxel, view) of an FDK backprojection."""
    kind = case["kind"]
    if kind == "batch":
        scans = _batch_scans(case)
        parts = [work(dict(s, kind="solver", dtype=case["dtype"], iters=1)) for s in scans]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    V = case["nx"] * case["ny"] * case["nz"]
    es = 4 if case.get("dtype", "f32") == "f32" else 2
    if kind == "denoise":
        return {"bytes": 2 * V * es, "flops": 40 * V * case["iters"]}
    P, n = _rows(case) * case["nu"], case["n_views"]
    if kind == "project":
        return {"bytes": V * es + case["views"] * P * 4, "flops": 4 * case["views"] * _pairs(case)}
    if kind == "gradient":
        return {"bytes": 2 * V * 4 + n * P * 4, "flops": 8 * n * _pairs(case)}
    if kind in ("sart", "dropin"):
        v = case["views"] if kind == "sart" else n
        return {"bytes": 2 * V * es + v * P * 4, "flops": 10 * v * _pairs(case)}
    if kind == "solver":
        return {"bytes": V * 4 + n * P * es, "flops": case["iters"] * (10 * n * _pairs(case) + 800 * V)}
    return {"bytes": 2 * V * 4 + n * P * 4, "flops": 20 * n * V}


# ------------------------------------------------------------------ the outputs in 64 bits

def _trace(s, views, visit):
    """Siddon's traversal of every ray of `views` in FP64, all rays in step: visit(voxel index, chord) once per step
    (chord 0 once a ray has left the volume), rays laid out (views, rows, nu)."""
    p, q = _rays(s, views, torch.float64)
    full = (len(views), _rows(s), s["nu"])
    x1 = torch.stack([b.expand(full) for b in q]).flatten(1)
    dr = torch.stack([(a - b).expand(full) for a, b in zip(p, q)]).flatten(1)
    n = torch.tensor([s["nx"], s["ny"], s["nz"]], device="cuda")[:, None]
    pitch = torch.tensor([s["vx"], s["vx"], _vz(s)], device="cuda", dtype=torch.float64)[:, None]
    low = -0.5 * n * pitch
    d12 = dr.square().sum(0).sqrt()
    still = dr.abs() < 1e-6 * pitch
    safe = torch.where(still, torch.ones_like(dr), dr)
    a0, a1 = (low - x1) / safe, (low + n * pitch - x1) / safe
    inside = (x1 >= low) & (x1 <= low + n * pitch)
    inf = torch.tensor(math.inf, device="cuda", dtype=torch.float64)
    lo = torch.where(still, torch.where(inside, -inf, inf), torch.minimum(a0, a1)).amax(0)
    hi = torch.where(still, torch.where(inside, inf, -inf), torch.maximum(a0, a1)).amin(0)
    hi = torch.maximum(hi, lo)
    lo, hi = torch.where(torch.isfinite(lo), lo, 0.0), torch.where(torch.isfinite(hi) & torch.isfinite(lo), hi, 0.0)
    up = dr > 0
    at = (x1 + lo * dr - low) / pitch
    plane = torch.where(up, torch.floor(at + 1e-9) + 1, torch.ceil(at - 1e-9) - 1)
    nxt = torch.where(still, inf, (low + plane * pitch - x1) / safe)
    step = torch.where(still, inf, (pitch / safe).abs())
    for k in range(int(n.sum()) + 3):
        m = torch.minimum(nxt.amin(0), hi)
        mid = 0.5 * (lo + m)
        ijk = torch.minimum(torch.floor((x1 + mid * dr - low) / pitch).long().clamp_(min=0), n - 1)
        visit((ijk[2] * s["ny"] + ijk[1]) * s["nx"] + ijk[0], (m - lo) * d12)
        nxt = torch.where(nxt <= m, nxt + step, nxt)
        lo = m
        if k % 32 == 31 and not bool((lo < hi).any()):
            break


def _project64(s, vol, views):
    """(Ray sums, chord sums) of `views` in FP64."""
    rays = len(views) * _rows(s) * s["nu"]
    out = torch.zeros((2, rays), device="cuda", dtype=torch.float64)
    flat = vol.double().flatten()

    def visit(idx, chord):
        out[0].addcmul_(flat[idx], chord)
        out[1].add_(chord)

    _trace(s, views, visit)
    return out.view(2, len(views), _rows(s), s["nu"])


def _chunks(s, views):
    per = max(1, int(8e6) // (_rows(s) * s["nu"]))
    return [list(range(a, min(views, a + per))) for a in range(0, views, per)]


def _sart64(s, vol, sino, beta, views):
    f = vol.double().flatten().clone()
    ex = (torch.arange(s["nx"], device="cuda") - (0.5 * s["nx"] - 0.5)) * s["vx"]
    ey = (torch.arange(s["ny"], device="cuda") - (0.5 * s["ny"] - 0.5)) * s["vx"]
    r2 = (0.5 * s["nx"] - 0.5) * (0.5 * s["ny"] - 0.5) * s["vx"] ** 2
    fov = ((ex ** 2)[None, :] + (ey ** 2)[:, None] < r2).expand(s["nz"], -1, -1).flatten()
    least = 1e-3 if s["style"] == TETRA else 1e-6
    for j in range(views):
        ax, ln = _project64(s, f, [j]).flatten(2)[:, 0]
        c = torch.where(ln < 1e-6 * _vz(s), torch.zeros_like(ax), (sino[j].double().flatten() - ax) / ln.clamp(min=1e-30))
        num, den = torch.zeros_like(f), torch.zeros_like(f)

        def visit(idx, chord):
            num.index_add_(0, idx, chord * c)
            den.index_add_(0, idx, chord)

        _trace(s, [j], visit)
        f += torch.where(fov & (den > least * s["vx"]), beta * num / den.clamp(min=1e-30), torch.zeros_like(f))
    return f.view(s["nz"], s["ny"], s["nx"])


def _denoise64(vol, lam, iters):
    f = vol.double()

    def div(r, s, t):
        out = r + s + t
        out[:, :, 1:] -= r[:, :, :-1]
        out[:, 1:] -= s[:, :-1]
        out[1:] -= t[:-1]
        return out

    old = [torch.zeros_like(f) for _ in range(3)]
    cur = [torch.zeros_like(f) for _ in range(3)]
    t0 = 1.0
    for _ in range(iters):
        L = f - lam * div(*cur)
        cur[0][:, :, :-1] += (L[:, :, :-1] - L[:, :, 1:]) / (12.0 * lam)
        cur[1][:, :-1] += (L[:, :-1] - L[:, 1:]) / (12.0 * lam)
        cur[2][:-1] += (L[:-1] - L[1:]) / (12.0 * lam)
        size = torch.sqrt(cur[0] ** 2 + cur[1] ** 2 + cur[2] ** 2).clamp_(min=1.0)
        t1 = 0.5 * (1.0 + math.sqrt(1.0 + 4.0 * t0 * t0))
        for k in range(3):
            cur[k] /= size
            new = cur[k].clone()
            cur[k] += (t0 - 1.0) / t1 * (new - old[k])
            old[k] = new
        t0 = t1
    return f - lam * div(*old)


def _fdk64(s, sino):
    """FDK in the +theta frame: cosine weight, ramp filter on a doubled row, bilinear voxel-driven backprojection."""
    R, ZP, n = s["nu"], s["nv"], s["n_views"]
    dso, sdd = s["dso"], s["dso"] - s["dod"]
    kw = dict(device="cuda", dtype=torch.float64)
    pu = (torch.arange(R, **kw) + 0.5 - 0.5 * R) * s["du"] * dso / sdd
    pv = (torch.arange(ZP, **kw) + 0.5 - 0.5 * ZP) * s["du"] * dso / sdd
    weight = dso / torch.sqrt(dso ** 2 + (pu ** 2)[None, :] + (pv ** 2)[:, None])
    ramp = torch.arange(R + 1, **kw) * (0.5 / (s["du"] * dso / sdd) / R * 0.5)
    x, y, z = (_centres(m, s["vx"], torch.float64) for m in (s["nx"], s["ny"], s["nz"]))
    vol = torch.zeros((s["nz"], s["ny"], s["nx"]), **kw)
    for j in range(n):
        g = torch.fft.irfft(torch.fft.rfft(sino[j].double() * weight, n=2 * R) * ramp, n=2 * R)[:, :R].contiguous()
        th = j * (360.0 / n) * math.pi / 180.0
        sn, cs = math.sin(th), math.cos(th)
        t = x[None, :] * cs + y[:, None] * sn
        ds = dso - (y[:, None] * cs - x[None, :] * sn)
        p = t * (sdd / s["du"]) / ds + (0.5 * R - 0.5)
        bn = torch.floor(p).clamp_(0, R - 2)
        b0 = p - bn
        ok = (p >= 0) & (p + 1 < R)
        scale = torch.where(ok, dso * dso / (ds * ds) * (2.0 * math.pi / n), torch.zeros_like(p))
        bi, row = bn.long(), sdd / s["du"] / ds
        for k0 in range(0, s["nz"], 64):
            ksi = z[k0:k0 + 64, None, None] * row + (0.5 * ZP - 0.5)
            an = torch.floor(ksi).clamp_(0, ZP - 2)
            a0 = ksi - an
            q = an.long() * R + bi
            flat = g.flatten()
            val = (1 - a0) * ((1 - b0) * flat[q] + b0 * flat[q + 1]) + a0 * ((1 - b0) * flat[q + R] + b0 * flat[q + R + 1])
            vol[k0:k0 + 64] += torch.where((ksi >= 0) & (ksi + 1 < ZP), val, torch.zeros_like(val)) * scale
    return vol


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solver", "batch"):  # whole engines: minutes in 64 bits
        return None
    if kind == "denoise":
        return _denoise64(_phantom(dict(case, vx=0.5, style=0), seed).to(DT[case["dtype"]]), case["lam"], case["iters"])
    if kind == "project":
        vol = _phantom(case, seed).to(DT[case["dtype"]])
        return torch.cat([_project64(case, vol, v)[0] for v in _chunks(case, case["views"])])
    if kind == "gradient":
        vol, b = _phantom(case, seed + 7), _measured(case, seed, case["n_views"])
        loss, grad = 0.0, torch.zeros(vol.numel(), device="cuda", dtype=torch.float64)
        for v in _chunks(case, case["n_views"]):
            r = _project64(case, vol, v)[0] - b[v[0]:v[-1] + 1].double()
            loss += 0.5 * float((r * r).sum())
            r = r.flatten()
            _trace(case, v, lambda idx, chord: grad.index_add_(0, idx, chord * r))
        return {"loss": torch.tensor(loss, dtype=torch.float64), "grad": grad.view(vol.shape)}
    if kind == "dropin":
        b = _measured(case, seed, case["n_views"])
        return _sart64(case, torch.zeros((case["nz"], case["ny"], case["nx"]), device="cuda"), b, case["beta"],
                       case["n_views"]).cpu().numpy()
    if kind == "sart":
        start = (0.5 * _phantom(case, seed)).to(DT[case["dtype"]])
        return _sart64(case, start, _measured(case, seed, case["views"]), case["beta"], case["views"])
    if case["nx"] * case["ny"] * case["nz"] * case["n_views"] > 2e10:  # over 20 seconds
        return None
    return _fdk64(case, _measured(case, seed, case["n_views"]))
