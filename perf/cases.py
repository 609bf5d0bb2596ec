"""The work this framework is used for, as measurable cases over the whole range of its sizes.

listed() names the cases, draw() gives more of the same ranges, prepare() makes what a program
holds before the call (plans, handles and seeded inputs on the GPU or in pinned host memory),
run() is one pass through the public entry points, work() the bytes and operations a pass cannot
do without, and exact() the same result in 64-bit torch arithmetic.

Kinds of case:
  recon      Reconstruction.run, fan views and volume on the device
  stream     Reconstruction.run from a pinned host fan to a pinned host volume
  batch      Batch.run of several uneven scans, fan views and volumes on the device
  views      one block or scan of views: lct_rebin_fan2par[_scan], then lct_filter_rows in place
  bp         lct_backproject_par of one block of filtered views
  cnn_infer  CNN.infer_volume, the learned correction of a volume
  cnn_grad   CNN.forward and CNN.backward on a batch of slices, and the gradients
  simulate   simulate_gpu, the fan views of a seeded phantom
"""
from __future__ import annotations

import ctypes as C
import math
import random
from pathlib import Path

import numpy as np
import torch

from listctrecons_b200 import capi, learn
from listctrecons_b200.recon import BLOCK_SLICES, Batch, Plan, Reconstruction
from listctrecons_b200.scan import MU_WATER, Phantom, ScanGeometry, simulate_gpu

ROOT = Path(__file__).resolve().parent.parent
WEIGHTS = ROOT / "listctrecons_b200" / "weights" / "cnn_cfg4.npz"

INTERP = {"tex8": capi.INTERP_TEX8, "exact": capi.INTERP_EXACT}
FILTER = {"fp32": capi.FILTER_FP32, "bf16x3": capi.FILTER_BF16X3, "bf16x6": capi.FILTER_BF16X6}
KIND = {"ramlak": capi.FILTER_RAMLAK, "shepp_logan": capi.FILTER_SHEPP_LOGAN}
PI = math.pi


def listed():
    return [
        # the smallest reconstruction anyone runs (a geometry check), with the library's defaults:
        # launches and the gaps between them
        dict(name="recon_tiny", kind="recon", ns=96, nt=8, ds=1.0, npt=120, pitch=1.0, nx=32, dx=1.0,
             dz=1.0, blocks=1, interp="tex8", filter="fp32", taps="ramlak", mode="scan"),
        # a small 16-row scan with the library's defaults (the reference's own sampling)
        dict(name="recon_small", kind="recon", ns=672, nt=16, ds=1.0, npt=1160, pitch=1.0, nx=256,
             dx=1.0, dz=1.0, blocks=1, interp="tex8", filter="fp32", taps="ramlak", mode="scan"),
        # the benchmark's volume in the mixed-precision path: the largest call
        dict(name="recon_large", kind="recon", ns=736, nt=64, ds=0.6, npt=1152, pitch=0.8, nx=512,
             dx=0.5, dz=0.5, blocks=8, interp="exact", filter="bf16x6", taps="shepp_logan", mode="scan"),
        # the PI-original chain (the reference's alternate configuration), per block
        dict(name="recon_pi", kind="recon", ns=736, nt=64, ds=0.6, npt=1152, pitch=0.8, nx=256,
             dx=1.0, dz=1.0, blocks=1, interp="exact", filter="bf16x6", taps="ramlak", mode="pi"),
        # a scanner's buffer in, a volume out: uploads, compute and downloads overlapped
        dict(name="stream_medium", kind="stream", ns=800, nt=32, ds=0.6, npt=1200, pitch=1.1, nx=384,
             dx=0.65, dz=0.75, blocks=3, interp="exact", filter="bf16x6", taps="ramlak", mode="scan"),
        # several uneven scans together (rows, columns, pitch and volume all differ)
        dict(name="batch_mixed", kind="batch", scans=4, mix=3, interp="exact", filter="bf16x6",
             taps="ramlak"),
        # the first two stages of the drop-in's per-block flow: reference rebin, FP32 ramp filter
        dict(name="views_block_fp32", kind="views", ns=672, nt=16, ds=1.0, npt=1160, pitch=1.0,
             views=3508, interp="tex8", filter="fp32", taps="ramlak", mode="block"),
        # the same stages as the mixed-precision path runs them, on a 64-row scan
        dict(name="views_scan_bf16x6", kind="views", ns=736, nt=64, ds=0.6, npt=1152, pitch=0.8,
             views=1833, interp="exact", filter="bf16x6", taps="shepp_logan", mode="scan"),
        # one block of the drop-in's backprojection stage, a detector and image of odd sizes
        dict(name="bp_block_ragged", kind="bp", ns=735, nt=31, ds=0.6, npt=1152, pitch=0.9, nx=307,
             dx=0.8, dz=0.6, interp="tex8", addr="border"),
        # the learned correction of a 512 x 512 volume
        dict(name="cnn_infer_512", kind="cnn_infer", nx=512, nz=64, max_slices=32),
        # a training batch of the learned correction: forward, backward, gradients
        dict(name="cnn_grad_256", kind="cnn_grad", nx=256, batch=16),
        # the views of one training scan: 40 ellipsoids, Poisson noise
        dict(name="simulate_scan", kind="simulate", ns=736, nt=64, ds=0.6, npt=1152, pitch=1.5,
             nx=256, dx=1.0, dz=1.0, views=600, ellipsoids=40, i0=1e5),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random):
    kind = rng.choice(["recon", "recon", "stream", "batch", "views", "views", "bp", "cnn_infer",
                       "cnn_grad", "simulate"])
    exact = rng.random() < 0.5
    prec = dict(interp="exact" if exact else "tex8", filter="bf16x6" if exact else "fp32",
                taps=rng.choice(["ramlak", "shepp_logan"]))
    nt = rng.choice([8, 16, 31, 32, 64])
    ns = int(_log(rng, 367, 896)) if rng.random() < 0.5 else 4 * int(_log(rng, 92, 224))
    geo = dict(ns=ns, nt=nt, ds=round(rng.uniform(0.5, 1.0), 2), npt=2 * rng.randint(400, 600),
               pitch=round(rng.uniform(0.5, 1.3), 3))
    nx = int(_log(rng, 96, 400))
    image = dict(nx=nx, dx=round(256.0 / nx, 3), dz=round(rng.uniform(0.5, 1.0), 2))
    if kind == "recon":
        mode = rng.choice(["scan", "scan", "scan", "block", "pi"])
        blocks = 1 if mode == "pi" else rng.randint(1, 3)
        if mode == "pi":
            image = dict(image, nx=min(nx, 256))
            prec = dict(prec, interp="exact", filter="bf16x6")
        return dict(kind=kind, **geo, **image, blocks=blocks, **prec, mode=mode)
    if kind == "stream":
        return dict(kind=kind, **geo, **image, blocks=rng.randint(1, 3), **prec, mode="scan")
    if kind == "batch":
        return dict(kind=kind, scans=rng.randint(2, 4), mix=rng.randint(0, 10 ** 6), interp="exact",
                    filter="bf16x6", taps=prec["taps"])
    if kind == "views":
        return dict(kind=kind, **geo, views=int(_log(rng, 64, 3000)), **prec,
                    mode=rng.choice(["block", "scan"]))
    if kind == "bp":
        return dict(kind=kind, **geo, **image, interp=prec["interp"],
                    addr=rng.choice(["border", "clamp"]))
    if kind == "cnn_infer":
        return dict(kind=kind, nx=int(_log(rng, 64, 512)), nz=rng.randint(8, 64),
                    max_slices=rng.choice([16, 32]))
    if kind == "cnn_grad":
        return dict(kind=kind, nx=int(_log(rng, 48, 256)), batch=rng.randint(4, 16))
    return dict(kind=kind, **geo, **image, views=int(_log(rng, 64, 800)),
                ellipsoids=rng.randint(10, 40), i0=1e5)


# ------------------------------------------------------------------------------------------
# geometry
# ------------------------------------------------------------------------------------------
def _geometry(c) -> ScanGeometry:
    return ScanGeometry(ns=c["ns"], nt=c["nt"], ds=c["ds"], dt=c["ds"], npt=c["npt"],
                        pitch=c["pitch"], nx=c.get("nx", 64), ny=c.get("nx", 64),
                        dx=c.get("dx", 1.0), dz=c.get("dz", 1.0))


def _plan(c) -> tuple[ScanGeometry, Plan]:
    geo = _geometry(c).with_blocks(c.get("blocks", 1))
    return geo, Plan(geo)


def _mixed_scans(c) -> list[dict]:
    """Uneven scans of the batched configuration's ranges."""
    r = random.Random(c["mix"])
    out = []
    for _ in range(c["scans"]):
        nt = r.choice([16, 32, 64])
        nx = r.choice([256, 384]) if nt < 64 else 256
        out.append(dict(ns=r.choice([672, 736, 800, 896]), nt=nt, ds=r.choice([0.5, 0.6]),
                        npt=r.choice([1000, 1152, 1200]), pitch=round(r.uniform(0.5, 1.5), 3), nx=nx,
                        dx=256.0 / nx, dz=r.choice([0.5, 0.75, 1.0]), blocks=r.choice([1, 2]),
                        interp=c["interp"], filter=c["filter"], taps=c["taps"], mode="scan"))
    return out


def _opts(c) -> dict:
    o = dict(interp=INTERP[c["interp"]], filter_mode=FILTER[c["filter"]], filter_kind=KIND[c["taps"]])
    if c["mode"] == "block":
        o.update(mode=capi.MODE_BLOCK)
    elif c["mode"] == "pi":
        o.update(mode=capi.MODE_BLOCK, rebinner=capi.REBIN_PI_ORI, preweight=capi.PW_PI_ORI,
                 backprojector=capi.BP_PI_ORI)
    return o


def _window(plan: Plan) -> tuple[int, int]:
    """Fan views [first, first + count) that the plan's blocks need."""
    i = plan.info
    starts = [b.block_proj_start for b in plan.blocks[i.first_block:i.first_block + i.n_blocks_run]]
    return min(starts), max(starts) + i.ctg.n_angle_add - min(starts)


# ------------------------------------------------------------------------------------------
# seeded inputs
# ------------------------------------------------------------------------------------------
def _fan(geo: ScanGeometry, seed: int, v0: int, n: int, i0: float = 1e5, out=None):
    """Noisy line integrals [n][nt][ns] of eight seeded ellipsoids along views [v0, v0 + n)."""
    dev = "cuda"
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=dev).manual_seed(seed)
    fov = 0.5 * geo.nx * geo.dx
    R = geo.dso
    j = torch.arange(v0, v0 + n, device=dev, dtype=torch.float64)
    beta = (geo.start_angle + j * (2 * PI / geo.npt)).float()[:, None]
    zs = (geo.z_start + geo.z_dir * j * (geo.feed / geo.npt)).float()
    al = ((torch.arange(geo.ns, device=dev) - (geo.ns - 1) / 2.0) * (geo.ds / R)).float()[None, :]
    t = ((torch.arange(geo.nt, device=dev) - (geo.nt - 1) / 2.0) * (geo.dt / R)).float()
    z_lo, z_hi = float(zs.min()), float(zs.max())
    ells = []
    for _ in range(8):
        a, b, h = rng.uniform(0.06, 0.45, size=3) * fov
        r, w = rng.uniform(0, 0.5) * fov, rng.uniform(0, 2 * PI)
        ells.append((r * math.cos(w), r * math.sin(w), rng.uniform(z_lo, z_hi), a, b,
                     max(h, 0.15 * (z_hi - z_lo)), rng.uniform(0, PI), rng.uniform(0.3, 1.5) * MU_WATER))
    if out is None:
        out = torch.empty((n, geo.nt, geo.ns), dtype=torch.float32, device=dev)
    step = max(1, (8 << 20) // (geo.nt * geo.ns))
    for s in range(0, n, step):
        bt, z, o = beta[s:s + step], zs[s:s + step], out[s:s + step]
        p = torch.zeros_like(o)
        for cx, cy, cz, a, b, h, phi, mu in ells:
            sx, sy = -R * torch.sin(bt) - cx, R * torch.cos(bt) - cy
            qx, qy = math.cos(phi) * sx + math.sin(phi) * sy, -math.sin(phi) * sx + math.cos(phi) * sy
            ang = bt - al - phi
            ux, uy = torch.sin(ang) / a, -torch.cos(ang) / b
            qx, qy, qz = qx / a, qy / b, (z[:, None] - cz) / h
            A = (ux * ux + uy * uy)[:, None, :] + ((t / h) ** 2 * 1.0)[None, :, None]
            B = (qx * ux + qy * uy)[:, None, :] + (qz * (t / h)[None, :])[:, :, None]
            cc = (qx * qx + qy * qy + qz * qz - 1.0)[:, :, None]
            p += (2 * mu) * (B * B - A * cc).clamp_(min=0).sqrt_() / A
        noise = torch.randn(o.shape, device=dev, generator=gen)
        o.copy_((p + noise * ((p * 0.5).exp_() / math.sqrt(i0))).clamp_(max=math.log(i0)))
    return out


def _taps(kind: str, ns: int, ds: float):
    h = np.zeros(2 * ns, dtype=np.float32)
    capi.check(capi.load().lct_filter_taps(KIND[kind], capi.WINDOW_NONE, ns, np.float32(ds), h.ctypes.data))
    return torch.from_numpy(h).cuda()


def _block_geom(c) -> tuple[capi.Geom, capi.Img, ScanGeometry, Plan]:
    geo, plan = _plan(c)
    g, ig = capi.Geom.from_buffer_copy(plan.info.ctg), capi.Img.from_buffer_copy(plan.info.ig)
    return g, ig, geo, plan


def _views_geom(c):
    g, _, geo, _ = _block_geom(c)
    g.n_angle = c["views"]
    g.n_angle_add = c["views"] + 2 * g.add_projections
    return g, geo


def _cnn_volume(seed: int, nz: int, n: int, calib: float):
    """An FDK-like volume: smooth random ellipsoids with noise, in raw FDK units."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    y = torch.linspace(-1, 1, n, device="cuda")[None, :, None]
    x = torch.linspace(-1, 1, n, device="cuda")[None, None, :]
    z = torch.linspace(-1, 1, nz, device="cuda")[:, None, None]
    v = torch.zeros((nz, n, n), device="cuda")
    for _ in range(10):
        cx, cy, cz = rng.uniform(-0.6, 0.6, size=3)
        a, b, h = rng.uniform(0.1, 0.5, size=3)
        d = ((x - cx) / a) ** 2 + ((y - cy) / b) ** 2 + ((z - cz) / h) ** 2
        v += rng.uniform(0.2, 1.5) * MU_WATER * torch.sigmoid((1.0 - d) * 12.0)
    v += 0.15 * MU_WATER * torch.randn(v.shape, device="cuda", generator=gen)
    return v / calib


def _cnn_pair(c, seed: int, calib: float):
    """5-slice inputs [batch][5][n][n] and targets [batch][n][n]."""
    vol = _cnn_volume(seed, c["batch"] + 4, c["nx"], calib)
    in5 = torch.stack([vol[k:k + c["batch"]] for k in range(5)], dim=1).contiguous()
    gen = torch.Generator(device="cuda").manual_seed(seed + 77)
    err = torch.randn(vol[2:-2].shape, device="cuda", generator=gen)
    return in5, (calib * vol[2:-2] + 0.1 * MU_WATER * err).contiguous()


def _he_params(seed: int) -> np.ndarray:
    """Starting weights of a training run (He-normal, the last layer a tenth of it, zero biases)."""
    rng = np.random.default_rng(seed)
    p = np.zeros(learn.N_PARAMS, dtype=np.float32)
    for l, (ws, _, shape) in enumerate(learn.layer_slices()):
        sd = math.sqrt(2.0 / (9 * shape[1])) * (0.1 if l == 7 else 1.0)
        p[ws] = rng.normal(0.0, sd, size=ws.stop - ws.start)
    return p


def _phantom(c, geo: ScanGeometry, seed: int) -> Phantom:
    z = geo.zpos64()
    return Phantom.random(c["ellipsoids"], seed=seed, fov_radius=0.5 * geo.nx * geo.dx,
                          z_lo=float(z.min()), z_hi=float(z.max()))


# ------------------------------------------------------------------------------------------
# prepare / run
# ------------------------------------------------------------------------------------------
def prepare(case, seed):
    c, k = case, case["kind"]
    if k in ("recon", "stream"):
        geo, plan = _plan(c)
        rec = Reconstruction(plan, **_opts(c))
        v0, n = _window(plan)
        fan = _fan(geo, seed, v0, n)
        if k == "recon":
            image = torch.empty(rec.image_shape, device="cuda")
        else:
            host = torch.empty(fan.shape, pin_memory=True)
            host.copy_(fan)
            fan, image = host, torch.empty(rec.image_shape, pin_memory=True)
        return dict(kind=k, rec=rec, fan=fan, view0=v0, image=image)
    if k == "batch":
        scans = [_plan(s) for s in _mixed_scans(c)]
        o = _opts(dict(c, mode="scan"))
        batch = Batch([p for _, p in scans], **o)
        wins = [_window(p) for _, p in scans]
        fans = [_fan(g, seed + 1000 * i, *w) for i, ((g, _), w) in enumerate(zip(scans, wins))]
        images = [torch.empty(s, device="cuda") for s in batch.image_shapes]
        return dict(kind=k, batch=batch, fans=fans, view0=[w[0] for w in wins], images=images)
    if k == "views":
        g, geo = _views_geom(c)
        return dict(kind=k, case=c, g=g, fan=_fan(geo, seed, 0, g.n_angle_add), h=_taps(c["taps"], g.ns, g.ds),
                    par=torch.empty((g.n_angle, g.nt, g.ns), device="cuda"))
    if k == "bp":
        g, ig, betas, views = _bp_inputs(c, seed)
        return dict(kind=k, case=c, g=g, ig=ig, betas=betas, views=views,
                    image=torch.empty((ig.nz, ig.ny, ig.nx), device="cuda"))
    if k == "cnn_infer":
        w = learn.load_weights(WEIGHTS)
        cnn = learn.cnn_from_weights(WEIGHTS, c["max_slices"], c["nx"], c["nx"])
        vol = _cnn_volume(seed, c["nz"], c["nx"], w["calib"])
        return dict(kind=k, cnn=cnn, vol=vol, out=torch.empty_like(vol), bound=w["bound"])
    if k == "cnn_grad":
        cnn = learn.CNN(c["batch"], c["nx"], c["nx"], train=True)
        cnn.set_params(_he_params(seed))
        cnn.set_scales(0.5, 1.0 / MU_WATER)
        in5, target = _cnn_pair(c, seed, 0.5)
        return dict(kind=k, cnn=cnn, in5=in5, target=target, resid=torch.empty_like(target),
                    grads=torch.empty(learn.N_PARAMS, device="cuda"))
    geo, _ = _plan(c)
    return dict(kind=k, geo=geo, phantom=_phantom(c, geo, seed), i0=c["i0"], seed=seed, views=c["views"],
                out=torch.empty((c["views"], geo.nt, geo.ns), device="cuda"))


def _bp_inputs(c, seed):
    """One block of filtered views: zero-mean rows with the scan's edges and noise."""
    g, ig, geo, plan = _block_geom(c)
    first = plan.blocks[0].block_proj_start + g.add_projections
    fan = _fan(geo, seed, first, g.n_angle)
    views = fan.clone()
    views[:, :, 1:-1] -= 0.5 * (fan[:, :, :-2] + fan[:, :, 2:])
    views = (views * (0.25 / g.ds)).contiguous()
    betas = torch.from_numpy(geo.angles32()[first:first + g.n_angle]).cuda()
    return g, ig, betas, views


def _stream():
    return torch.cuda.current_stream().cuda_stream


def run(state):
    s, k = state, state["kind"]
    if k in ("recon", "stream"):
        return s["rec"].run(s["fan"], s["image"], fan_view0=s["view0"])
    if k == "batch":
        return s["batch"].run(s["fans"], s["images"], fan_view0=s["view0"])
    if k == "views":
        c, g, lib = s["case"], s["g"], capi.load()
        if c["mode"] == "block":
            capi.check(lib.lct_rebin_fan2par(C.byref(g), s["fan"].data_ptr(), s["par"].data_ptr(),
                                             INTERP[c["interp"]], capi.ADDR_BORDER, _stream()))
        else:
            capi.check(lib.lct_rebin_fan2par_scan(C.byref(g), s["fan"].data_ptr(), 0, g.n_angle_add,
                                                  s["par"].data_ptr(), g.add_projections, g.n_angle,
                                                  INTERP[c["interp"]], capi.ADDR_BORDER, 0, _stream()))
        capi.check(lib.lct_filter_rows(g.ns, s["h"].data_ptr(), s["par"].data_ptr(), g.n_angle * g.nt,
                                       FILTER[c["filter"]], _stream()))
        return s["par"]
    if k == "bp":
        c = s["case"]
        addr = capi.ADDR_CLAMP if c["addr"] == "clamp" else capi.ADDR_BORDER
        capi.check(capi.load().lct_backproject_par(
            C.byref(s["g"]), C.byref(s["ig"]), s["betas"].data_ptr(), s["views"].data_ptr(),
            s["image"].data_ptr(), INTERP[c["interp"]], addr, _stream()))
        return s["image"]
    if k == "cnn_infer":
        return s["cnn"].infer_volume(s["vol"], s["bound"], out=s["out"], count=False)[0]
    if k == "cnn_grad":
        cnn = s["cnn"]
        resid = cnn.forward(s["in5"], s["resid"])
        cnn.backward(s["in5"], s["target"])
        capi.check(capi.load().lct_cnn_get_grads(cnn._h, s["grads"].data_ptr(), 1))
        return resid, s["grads"]
    return simulate_gpu(s["geo"], s["phantom"], i0=s["i0"], seed=s["seed"], v0=0, v1=s["views"],
                        out=s["out"])


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def _recon_work(c):
    geo, plan = _plan(c)
    g, ig = plan.info.ctg, plan.info.ig
    nb = plan.info.n_blocks_run
    _, n = _window(plan)
    voxels = nb * BLOCK_SLICES * ig.nx * ig.ny
    half = g.n_proj_turn // 2
    samples = (half + 1) if c["mode"] == "pi" else 2 * half  # per voxel, a conjugate pair once
    rows = (n - 2 * g.add_projections) * g.nt
    return {"bytes": 4.0 * (n * g.nt * g.ns + voxels),
            "flops": 10.0 * voxels * samples + 2.0 * g.ns * g.ns * rows + 3.0 * g.ns * rows}


def work(case):
    c, k = case, case["kind"]
    if k in ("recon", "stream"):
        return _recon_work(c)
    if k == "batch":
        w = [_recon_work(s) for s in _mixed_scans(c)]
        return {key: sum(x[key] for x in w) for key in ("bytes", "flops")}
    if k == "views":
        g, _ = _views_geom(c)
        rows = g.n_angle * g.nt
        return {"bytes": 4.0 * g.ns * g.nt * (g.n_angle + g.n_angle_add), "flops": (2.0 * g.ns + 3.0) * g.ns * rows}
    if k == "bp":
        g, ig, _, _ = _block_geom(c)
        voxels = ig.nx * ig.ny * ig.nz
        return {"bytes": 4.0 * (g.n_angle * g.nt * g.ns + voxels),
                "flops": 10.0 * voxels * 2 * (g.n_proj_turn // 2)}
    if k == "cnn_infer":
        v = c["nz"] * c["nx"] ** 2
        return {"bytes": 8.0 * v, "flops": 2.0 * 9 * (5 * 32 + 6 * 32 * 32 + 32) * v}
    if k == "cnn_grad":
        v = c["batch"] * c["nx"] ** 2
        fwd = 2.0 * 9 * (5 * 32 + 6 * 32 * 32 + 32)
        return {"bytes": 4.0 * 7 * v, "flops": (2 * fwd + fwd - 2.0 * 9 * 5 * 32) * v}
    rays = c["views"] * c["nt"] * c["ns"]
    return {"bytes": 4.0 * rays, "flops": rays * (30.0 * c["ellipsoids"] + 60.0)}


# ------------------------------------------------------------------------------------------
# the same results in 64 bits
# ------------------------------------------------------------------------------------------
F64 = torch.float64


def _ar(n):
    return torch.arange(n, device="cuda", dtype=F64)


def _q8(a):
    return torch.floor(a * 256.0 + 0.5) / 256.0


def _filter64(rows, kind, ds):
    """rows [..., ns] FP64 -> sum_k h[is - k] row[k], by FFT."""
    ns = rows.shape[-1]
    n = torch.arange(-ns, ns, device="cuda", dtype=F64)
    if kind == "ramlak":
        h = torch.where(n.long() % 2 != 0, -1.0 / (PI * PI * n * n * ds), torch.zeros_like(n))
        h[ns] = 0.25 / ds
    else:
        h = -2.0 / (PI * PI * ds * (4.0 * n * n - 1.0))
    L = 1 << (3 * ns).bit_length()
    H = torch.fft.rfft(h, L)
    out = torch.empty_like(rows)
    flat, o = rows.view(-1, ns), out.view(-1, ns)
    step = max(1, (64 << 20) // L)
    for s in range(0, flat.shape[0], step):
        y = torch.fft.irfft(torch.fft.rfft(flat[s:s + step], L) * H, L)
        o[s:s + step] = y[:, ns:2 * ns]
    return out


def _lerp_views(fan, v0, w):
    """fan [n][nt][ns]; v0 [m][ns] view of the first tap, w [m][ns] weight of the second -> [m][nt][ns]."""
    n, nt, ns = fan.shape
    pad = torch.cat([torch.zeros_like(fan[:1]), fan, torch.zeros_like(fan[:1])])
    cols = torch.arange(ns, device="cuda")[None, :].expand_as(v0)
    take = lambda v: pad[(v + 1).clamp(0, n + 1), :, cols].permute(0, 2, 1).double()  # noqa: E731
    out = torch.empty((v0.shape[0], nt, ns), device="cuda", dtype=F64)
    for s in range(0, v0.shape[0], 256):
        e = slice(s, s + 256)
        v, ww = v0[e], w[e][:, None, :]
        cols = torch.arange(ns, device="cuda")[None, :].expand_as(v)
        out[e] = (1.0 - ww) * take(v) + ww * take(v + 1)
    return out


def _rebin64_scan(g, fan, shift0, m, interp):
    """m parallel views; view k reads fan coordinate k + shift0 + alpha(is) / orbit."""
    s = ((_ar(g.ns) - g.ws) * g.ds / g.dso) / g.orbit
    fs = torch.floor(s)
    w = s - fs
    if interp == "tex8":
        w = _q8(w)
    v0 = torch.arange(m, device="cuda")[:, None] + fs.long()[None, :] + shift0
    return _lerp_views(fan, v0, w[None, :].expand(m, -1))


def _rebin64_block(g, fan, interp):
    """Block coordinate: the index rule is defined in FP32 for the texture sampling."""
    if interp == "exact":
        return _rebin64_scan(g, fan, g.add_projections, g.n_angle, "exact")
    f = torch.float32
    ss = (torch.arange(g.ns, device="cuda", dtype=f) - g.ws) * torch.tensor(g.ds, dtype=f, device="cuda")
    turn = (ss / torch.tensor(g.dso, dtype=f, device="cuda")) / torch.tensor(g.orbit, dtype=f, device="cuda")
    cz = torch.arange(g.n_angle, device="cuda", dtype=f)[:, None] + turn[None, :]
    xb = ((cz + float(g.add_projections)) + 0.5) - 0.5
    fl = torch.floor(xb)
    return _lerp_views(fan, fl.long(), _q8((xb - fl).double()))


def _windows(g, ig):
    f = np.float32
    dzv = f(f(g.pitch) / f(g.n_proj_turn))
    half = g.n_proj_turn // 2
    out = []
    for z in range(ig.nz):
        zc = f(f(f(z) - f(ig.wz)) * f(ig.dz))
        q = float(f(f(zc - f(g.source_z0)) / dzv))
        mid = int(math.floor(abs(q) + 0.5) * (1 if q >= 0 else -1))
        mid = min(max(mid, 0), g.n_angle - 1)
        out.append((max(mid - half, 0), mid, mid + half if mid + half < g.n_angle else g.n_angle - 1))
    return out


class _View:
    """Bilinear samples of one view with its border rule (a frame of two texels around it)."""

    def __init__(self, view, clamp):
        v = view.double()[None, None]
        p = torch.nn.functional.pad(v, (2, 3, 2, 3), mode="replicate" if clamp else "constant")
        self.p = p[0, 0].contiguous()
        self.nt, self.ns = view.shape

    def column(self, x, tex):
        i = torch.floor(x)
        a = x - i
        return i.long().clamp_(-2, self.ns) + 2, (_q8(a) if tex else a)

    def sample(self, col, a, y, tex):
        j = torch.floor(y)
        b = y - j
        at = (j.long().clamp_(-2, self.nt) + 2) * self.p.shape[1] + col
        flat = self.p.view(-1)
        t00, t01 = flat[at], flat[at + 1]
        t10, t11 = flat[at + self.p.shape[1]], flat[at + self.p.shape[1] + 1]
        if tex:
            b = _q8(b)
            w11 = torch.floor(a * b * 256.0 + 0.5) / 256.0
            return t00 + a * (t01 - t00) + b * (t10 - t00) + w11 * ((t11 - t10) - (t01 - t00))
        top, bot = t00 + a * (t01 - t00), t10 + a * (t11 - t10)
        return top + b * (bot - top)


def _grid(ig):
    x = ((_ar(ig.nx) - ig.wx) * ig.dx)[None, :]
    y = ((_ar(ig.ny) - ig.wy) * ig.dy)[:, None]
    return x, y


def _bp64(g, ig, betas, views, interp, clamp=False):
    """The helical backprojection over full view windows, conjugate pairs once."""
    tex = interp == "tex8"
    win = _windows(g, ig)
    half = g.n_proj_turn // 2
    dzv = g.pitch / g.n_proj_turn
    x, y = _grid(ig)
    zc = ((_ar(ig.nz) - ig.wz) * ig.dz)
    acc = torch.zeros((ig.nz, ig.ny, ig.nx), device="cuda", dtype=F64)
    ang = betas.double().cpu().numpy()
    kq = g.dso * g.z_dir / g.dt
    for ia in range(min(w[0] for w in win), max(w[1] for w in win)):
        zs = [z for z, w in enumerate(win) if w[0] <= ia < w[1]]
        if not zs:
            continue
        lo, hi = zs[0], zs[-1] + 1
        s = []
        for v, sign in ((ia, 1.0), (ia + half, -1.0)):
            cb, sb = math.cos(ang[v]), math.sin(ang[v])
            if sign > 0:
                phat = -x * cb - y * sb
                theta = torch.asin(phat / g.dso)
                sq = torch.sqrt(g.dso * g.dso - phat * phat)
            lhat = sq + x * sb - y * cb
            zr = g.source_z0 + (v + sign * theta / g.orbit) * dzv
            q = (zc[lo:hi, None, None] - zr) * (kq / lhat)
            view = _View(views[v], clamp)
            col, a = view.column(sign * theta * (g.dso / g.ds) + g.ws, tex)
            s.append((q, view.sample(col, a, q + g.wt, tex)))
        (q1, s1), (q2, s2) = s
        o1, o2 = q1.abs() > g.wt, q2.abs() > g.wt
        w1 = -2.0 * q2 / (q1 - q2)
        w1 = torch.where(o1, torch.where(o2, 1.0, 0.0), torch.where(o2, 2.0, w1))
        acc[lo:hi] += s2 * 2.0 + w1 * (s1 - s2)
    for z, (a0, _, a1) in enumerate(win):
        acc[z] *= 2.0 * PI / (a1 - a0)
    return acc


def _pi64(g, ig, fan, betas, kind):
    """The PI-original chain of one block: rebin, pre-weight, filter, PI-window backprojection."""
    n, nt, ns = fan.shape
    s = (_ar(ns) - g.ws) * g.ds
    gamma = torch.asin(s / g.dso)
    it = _ar(nt)[:, None]
    px = gamma * g.dso / g.ds + g.ws
    q = ((it - g.wt) * g.pitch / (2.0 * (nt - 1)) - gamma * g.pitch / (2 * PI)) / torch.cos(gamma)
    qi = q / g.dt + g.wt
    shift = gamma / g.orbit + g.add_projections
    i, j, k = torch.floor(px), torch.floor(qi), torch.floor(shift)
    a, b, c = px - i, qi - j, shift - k
    pad = torch.nn.functional.pad(fan, (1, 2, 1, 2, 1, 2))
    ic, jc = i.long().clamp(-1, ns) + 1, j.long().clamp(-1, nt) + 1
    t = (it - g.wt) * g.pitch / (2.0 * nt)
    w = g.dso * g.dso - s * s
    w = torch.sqrt(w) / torch.sqrt(w + (t - gamma * g.pitch / (2 * PI)) ** 2)
    par = torch.empty((g.n_angle, nt, ns), device="cuda", dtype=F64)
    for ia in range(g.n_angle):
        o = torch.zeros((nt, ns), device="cuda", dtype=F64)
        for dk, wk in ((0, 1 - c), (1, c)):
            kc = ((ia + k).long() + dk).clamp(-1, n) + 1
            for dj, wj in ((0, 1 - b), (1, b)):
                for di, wi in ((0, 1 - a), (1, a)):
                    o += wk * wj * wi * pad[kc[None, :].expand(nt, -1), jc + dj, (ic + di)[None, :].expand(nt, -1)]
        par[ia] = o * w
    par = _filter64(par, kind, g.ds)
    half = g.n_proj_turn // 2
    dzv = g.pitch / g.n_proj_turn
    x, y = _grid(ig)
    win = _windows(g, ig)
    zc = (_ar(ig.nz) - ig.wz) * ig.dz
    acc = torch.zeros((ig.nz, ig.ny, ig.nx), device="cuda", dtype=F64)
    amin = torch.full(acc.shape, -1, device="cuda", dtype=torch.int32)
    walking = torch.ones(acc.shape, device="cuda", dtype=torch.bool)
    mid = torch.tensor([m for _, m, _ in win], device="cuda")[:, None, None]
    ang = betas.double().cpu().numpy()

    def at(v):
        cb, sb = math.cos(ang[v]), math.sin(ang[v])
        sv = -x * cb - y * sb
        gm = torch.asin(sv / g.dso)
        temp1 = torch.sqrt(g.dso * g.dso - sv * sv)
        gt2 = gm * (g.pitch / (2 * PI))
        den = temp1 + x * sb - y * cb
        tv = (temp1 * (zc[:, None, None] - (g.source_z0 + dzv * v) - gt2) / den + gt2) * g.z_dir
        view = _View(par[v], False)
        col, aa = view.column(sv / g.ds + g.ws, False)
        return tv, view.sample(col, aa, tv * 2 * (nt - 1) / g.pitch + g.wt, False)

    top = max(m for _, m, _ in win)
    for v in range(top, -1, -1):
        tv, smp = at(v)
        here = walking & (mid >= v)
        stop = here & (tv.abs() > g.pitch / 4)
        amin[stop] = v
        walking &= ~stop
        acc += torch.where(here & ~stop, smp, 0.0)
        if v < top - 32 and v % 16 == 0 and not bool(walking.any()):
            break
    for v in range(min(m for _, m, _ in win) + 1, g.n_angle):
        here = (v > mid) & (v <= amin + half)
        if v % 16 == 0 and not bool(((amin + half) >= v).any()):
            break
        acc += torch.where(here, at(v)[1], 0.0)
    return acc * (PI / half)


def _recon64(c, seed):
    geo, plan = _plan(c)
    g, ig = plan.info.ctg, plan.info.ig
    first, n = _window(plan)
    fan = _fan(geo, seed, first, n)
    add, nb = g.add_projections, plan.info.n_blocks_run
    blocks = plan.blocks[plan.info.first_block:plan.info.first_block + nb]
    betas = torch.from_numpy(geo.angles32()).cuda()
    out = torch.empty((nb * BLOCK_SLICES, ig.ny, ig.nx), device="cuda", dtype=F64)
    if c["mode"] == "scan":
        par = _rebin64_scan(g, fan, add, n - 2 * add, c["interp"])
        par = _filter64(par, c["taps"], g.ds)
    for b, bi in enumerate(blocks):
        off = bi.block_proj_start - first
        bt = betas[bi.block_proj_start + add:][:g.n_angle]
        block = fan[off:off + g.n_angle_add]
        o = out[b * BLOCK_SLICES:(b + 1) * BLOCK_SLICES]
        if c["mode"] == "pi":
            o.copy_(_pi64(g, ig, block, bt, c["taps"]))
            continue
        if c["mode"] == "scan":
            views = par[off:off + g.n_angle]
        else:
            views = _filter64(_rebin64_block(g, block, c["interp"]), c["taps"], g.ds)
        o.copy_(_bp64(g, ig, bt, views, c["interp"]))
    return out


def _net64(params, in5, k_in):
    """The network in FP64: in5 [n][5][h][w] raw slices -> residual [n][h][w]."""
    x = in5.double() * k_in
    for l, (ws, bs, shape) in enumerate(learn.layer_slices()):
        x = torch.nn.functional.conv2d(x, params[ws].view(shape), params[bs], padding=1)
        if l < 7:
            x = torch.relu(x)
    return x[:, 0]


def _mulhilo(a, b):
    p = a * b  # wraps modulo 2^64
    return (p >> 32) & 0xFFFFFFFF, p & 0xFFFFFFFF


def _philox(c, k0, k1):
    c0, c1, c2, c3 = c
    for _ in range(10):
        h0, l0 = _mulhilo(c0, 0xD2511F53)
        h1, l1 = _mulhilo(c2, 0xCD9E8D57)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def _noisy64(p, i0, seed, idx):
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    full = lambda v: torch.full_like(idx, v)  # noqa: E731
    c = _philox((idx & 0xFFFFFFFF, idx >> 32, full(0x4C435430), full(0)), k0, k1)
    u = [(v.double() + 0.5) / 4294967296.0 for v in c[:2]]
    lam = i0 * torch.exp(-p)
    n = torch.floor(lam + torch.sqrt(lam) * torch.sqrt(-2.0 * torch.log(u[0])) * torch.cos(2 * PI * u[1]) + 0.5)
    low = lam < 30.0
    if bool(low.any()):
        lim, prod = torch.exp(-lam[low]), u[0][low]
        cc = [c[2][low], c[3][low], torch.full_like(c[2][low], 0x4B4E5554), torch.zeros_like(c[2][low])]
        count, j = torch.zeros_like(prod), 0
        while True:
            go = prod > lim
            if not bool(go.any()):
                break
            if j == 4:
                cc, j = list(_philox(cc, k0, k1)), 0
            prod = torch.where(go, prod * ((cc[j].double() + 0.5) / 4294967296.0), prod)
            count += go
            j += 1
        n[low] = count
    return -torch.log(n.clamp(min=1.0) / i0)


def _simulate64(c, seed):
    geo, _ = _plan(c)
    rec = _phantom(c, geo, seed).records
    R, ws, wt = geo.dso, float(np.float32(geo.central_channel)), float(np.float32((geo.nt - 1) / 2.0))
    f32 = lambda v: float(np.float32(v))  # noqa: E731
    a = (_ar(geo.ns) - ws) * f32(geo.ds) / f32(R)
    t = (_ar(geo.nt) - wt) * f32(geo.dt)
    ang, zp = geo.angles64(), geo.zpos64()
    out = torch.empty((c["views"], geo.nt, geo.ns), device="cuda", dtype=F64)
    for v in range(c["views"]):
        b, z = float(ang[v]), float(zp[v])
        S = (-f32(R) * math.sin(b), f32(R) * math.cos(b), z)
        D = (torch.sin(b - a)[None, :], -torch.cos(b - a)[None, :], (t / f32(R))[:, None])
        dn = torch.sqrt(D[0] ** 2 + D[1] ** 2 + D[2] ** 2)
        p = torch.zeros((geo.nt, geo.ns), device="cuda", dtype=F64)
        for e in rec:
            A = B = 0.0
            cq = -1.0
            for r in range(3):
                m = [e[6 + 3 * k + r] / e[3 + r] for k in range(3)]
                sv = sum(m[k] * (S[k] - e[k]) for k in range(3))
                dv = m[0] * D[0] + m[1] * D[1] + m[2] * D[2]
                A, B, cq = A + dv * dv, B + sv * dv, cq + sv * sv
            p += 2.0 * e[15] * torch.sqrt((B * B - A * cq).clamp(min=0)) / A * dn
        idx = ((v * geo.nt + torch.arange(geo.nt, device="cuda"))[:, None] * geo.ns
               + torch.arange(geo.ns, device="cuda")[None, :])
        out[v] = _noisy64(p, c["i0"], int(seed), idx)
    return out


def exact(case, seed):
    c, k = case, case["kind"]
    if k in ("recon", "stream"):
        _, plan = _plan(c)
        win = _windows(plan.info.ctg, plan.info.ig)
        steps = c["blocks"] * (win[-1][1] - win[0][0])
        if steps * (4000 + c["nx"] ** 2 * 0.1) > 4e8:
            return None  # more than about 20 seconds
        return _recon64(c, seed)
    if k == "batch":
        scans = _mixed_scans(c)
        return [_recon64(s, seed + 1000 * i) if i == 0 else None for i, s in enumerate(scans)]
    if k == "views":
        g, geo = _views_geom(c)
        fan = _fan(geo, seed, 0, g.n_angle_add)
        par = (_rebin64_block(g, fan, c["interp"]) if c["mode"] == "block" else
               _rebin64_scan(g, fan, g.add_projections, g.n_angle, c["interp"]))
        return _filter64(par, c["taps"], g.ds)
    if k == "bp":
        g, ig, betas, views = _bp_inputs(c, seed)
        return _bp64(g, ig, betas, views, c["interp"], c["addr"] == "clamp")
    if k == "cnn_infer":
        w = learn.load_weights(WEIGHTS)
        vol = _cnn_volume(seed, c["nz"], c["nx"], w["calib"])
        params = torch.from_numpy(w["params"]).cuda().double()
        out = w["calib"] * vol.double()
        z = torch.arange(c["nz"], device="cuda")
        for s in range(0, c["nz"], 4):
            sl = [(z[s:s + 4] + d).clamp(0, c["nz"] - 1) for d in range(-2, 3)]
            in5 = torch.stack([vol[i] for i in sl], dim=1)
            d = _net64(params, in5, w["calib"] * w["in_scale"]) / w["in_scale"]
            out[s:s + 4] += torch.where(d.abs() <= w["bound"], d, 0.0)
        return out
    if k == "cnn_grad":
        in5, target = _cnn_pair(c, seed, 0.5)
        params = torch.from_numpy(_he_params(seed)).cuda().double().requires_grad_(True)
        res, grads = [], torch.zeros(learn.N_PARAMS, device="cuda", dtype=F64)
        for s in range(0, c["batch"], 2):
            r = _net64(params, in5[s:s + 2], 0.5 / MU_WATER)
            d = (0.5 * in5[s:s + 2, 2].double() - target[s:s + 2].double()) / MU_WATER + r
            loss = d.square().sum() / (c["batch"] * c["nx"] ** 2)
            grads += torch.autograd.grad(loss, params)[0]
            res.append(r.detach())
        return torch.cat(res), grads
    return _simulate64(c, seed)
