"""The performance cases of the engine: the calls a reconstruction program makes.

A program creates a context for a scan's geometry, uploads the sinogram, forms
a start image (FBP, or a coarser grid's reconstruction, or the warm-start
network's), runs ICD iterations, evaluates the MAP cost and takes the object
out.  Each case is one of those calls, through the Python binding
(timbir-python_b200/xtg.py) or, where that has none, the C ABI:

  icd       one ICD iteration over the resident object
  step      a scan from pinned host memory: upload, iteration, object back
  cost      the MAP cost in FP64
  fbp       the filtered-backprojection start
  multires  the coarse-to-fine start
  nhicd     the allocation-free NHICD thresholds on device maps
  net       the warm-start network's forward pass over a volume
  train     one training step of the network (gradients, then Adam)
  conv      one 3x3x3 convolution layer: forward, input or weight gradient

Sinograms are line integrals of seeded ellipsoids with Poisson counts at 1e4
photons per ray, 0.5 % of the entries zingers where that correction is on.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "timbir-python_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import xtg  # noqa: E402

WEIGHTS = os.path.join(PKG, "weights", "warmstart_plain3d.bin")
I0 = 1e4
# (cin, cout, level) of the network's 3x3x3 convolutions, level l at 1/2^l the resolution
LAYERS = [(2, 32, 0), (32, 32, 0), (32, 48, 1), (48, 48, 1), (48, 64, 2), (64, 64, 2), (64, 96, 3), (96, 96, 3),
          (160, 64, 2), (64, 64, 2), (112, 48, 1), (48, 48, 1), (80, 32, 0), (32, 32, 0)]
SCALE = 100.0
AMODES = {"auto": xtg.XTG_A_AUTO, "table32": xtg.XTG_A_TABLE32, "fp16": xtg.XTG_A_FP16, "fp32": xtg.XTG_A_FP32}


# ------------------------------------------------------------------ cases --
def scan(kind, n, nz, views, frames=1, a="auto", zinger=True, **more):
    return dict({"kind": kind, "n": n, "nz": nz, "views": views, "frames": frames, "a": a, "zinger": zinger}, **more)


def listed():
    return [
        # the smallest call: thresholds for four small maps inside an acquisition loop
        {"name": "nhicd_4x128", "kind": "nhicd", "maps": 4, "ny": 128, "nx": 128},
        # a few slices for a quick look (configuration 1: 128^2 x 4, 180 views)
        dict(scan("icd", 128, 4, 180, zinger=False), name="icd_128x4"),
        # a cropped detector: odd rows, bins no power of two, the FP16 table
        dict(scan("icd", 180, 27, 400, a="fp16"), name="icd_180x27_fp16"),
        # 4D: 16 interlaced frames of 64 views
        dict(scan("icd", 256, 16, 1024, frames=16, zinger=False), name="icd_4d_256x16x16"),
        # plain 3D at scale
        dict(scan("icd", 512, 64, 1024), name="icd_512x64"),
        # scans streaming through one context, host to host
        dict(scan("step", 256, 32, 512), name="step_256x32"),
        # the convergence check of the at-scale reconstruction
        dict(scan("cost", 512, 64, 1024), name="cost_512x64"),
        # its start image
        dict(scan("fbp", 512, 64, 1024), name="fbp_512x64"),
        # the coarse-to-fine start of a middle-sized one
        dict(scan("multires", 256, 32, 512, iters=30), name="multires_256x32"),
        # the learned start's inference over the at-scale volume
        {"name": "net_512x64", "kind": "net", "nb": 1, "y": 512, "x": 512, "z": 64},
        # a training step as train_warmstart.py runs it for the committed weights
        {"name": "train_8x32x128x32", "kind": "train", "nb": 8, "y": 32, "x": 128, "z": 32},
        # a level-1 layer's weight gradient in that step
        {"name": "conv_wgrad_48", "kind": "conv", "op": "wgrad", "nb": 8, "y": 16, "x": 64, "z": 16, "cin": 48,
         "cout": 48},
    ]


def logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["icd", "icd", "icd", "step", "cost", "fbp", "multires", "nhicd", "net", "train", "conv"])
    if kind in ("icd", "step", "cost", "fbp", "multires"):
        while True:
            frames = rng.choice([1, 1, 1, 4, 8]) if kind in ("icd", "cost", "fbp") else 1
            n = logint(rng, 64, 512)
            nz = logint(rng, 3, 96)
            if kind == "multires" or rng.random() < 0.5:
                n, nz = max(64, n // 4 * 4), max(4, nz // 4 * 4)
            if nz > 32:  # longer z-lines come in multiples of 8 rows (two z-blocks of whole 16-byte groups)
                nz = nz // 8 * 8
            views = frames * logint(rng, 32, 128) if frames > 1 else logint(rng, 90, 1024)
            if 1e7 < float(n) * n * nz * views <= 1.7e10 and frames * n * n * nz < 1 << 26:
                break
        c = scan(kind, n, nz, views, frames, rng.choice(["auto", "auto", "table32", "fp16", "fp32"]) if kind == "icd" else "auto",
                 rng.random() < 0.6)
        if kind == "multires":
            c["iters"] = rng.randint(20, 40)
        return c
    if kind == "nhicd":
        ny, nx = logint(rng, 48, 700), logint(rng, 48, 700)
        return {"kind": "nhicd", "maps": rng.randint(1, max(1, min(64, (1 << 20) // (ny * nx)))), "ny": ny, "nx": nx}
    if kind == "net":
        while True:
            c = {"kind": "net", "nb": rng.choice([1, 1, 2, 4]), "y": 8 * logint(rng, 6, 64), "x": 8 * logint(rng, 6, 64),
                 "z": 8 * rng.randint(1, 8)}
            if c["nb"] * c["y"] * c["x"] * c["z"] <= 1 << 24:
                return c
    if kind == "train":
        return {"kind": "train", "nb": rng.randint(1, 8), "y": 8 * rng.randint(2, 8), "x": rng.choice([32, 64, 64, 72, 128]),
                "z": 8 * rng.randint(1, 4)}
    cin, cout, lvl = rng.choice(LAYERS[1:])
    return {"kind": "conv", "op": rng.choice(["forward", "dgrad", "wgrad"]), "nb": rng.randint(1, 8),
            "y": rng.randint(32, 72) >> lvl, "x": rng.choice([128, rng.randint(32, 160)]) >> lvl, "z": 32 >> lvl,
            "cin": cin, "cout": cout}


# ----------------------------------------------------------------- inputs --
def gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + salt)


def views_of(c):
    """View times and angles (degrees): uniform over 180 degrees, or for
    several frames interlaced sub-frames in bit-reversed order."""
    n, f = c["views"], c["frames"]
    if f == 1:
        return np.arange(n, dtype=np.float64), 180.0 * np.arange(n) / n
    per = n // f  # views of a frame: two sub-frames where that divides
    k = 8
    i = np.arange(n)
    sub = (i // max(per // 2, 1)) % k
    rev = ((sub & 1) << 2) | (sub & 2) | ((sub >> 2) & 1)
    ang = (i % max(per // 2, 1)) * 180.0 / max(per // 2, 1) + rev * 180.0 / (k * max(per // 2, 1))
    return i.astype(np.float64), np.round(ang, 6)


def params_of(c):
    n, nz, f = c["n"], c["nz"], c["frames"]
    rdelta = float(c["views"] // f)
    sig = 200000.0
    slope = 1000.0 / (0.521225397034623 - 0.496372335005353 * 0.001205) / 0.0001
    chu = -slope * (0.496372335005353 * 0.001205 * 0.0001)
    # temporal prior at half the spatial one's weight
    sigt = chu + (sig - chu) / (rdelta * math.sqrt(0.5)) if f > 1 else sig
    return xtg.Params(
        p=1.2, sigma_s=sig, sigma_t=sigt, c_s=0.01, c_t=0.01, length_r=float(n), length_t=float(nz),
        rotation_center=n / 2.0, Rtime_delta=rdelta, radius_obj=float(n), zingerT=4.0 if c["zinger"] else 100000.0,
        zingerDel=0.5 if c["zinger"] else 0.0, iter=100, Rtime_num=f, num_projections=c["views"], N_r=n, N_t=nz,
        num_threads=1, positivity=1)


def ellipsoids(seed, count):
    """Rows (cx, cy, cz, a, b, c, phi, mu, vx, vy) in units of the half-widths."""
    r = np.random.default_rng(int(seed))
    rad, th = 0.6 * np.sqrt(r.random(count)), 2 * np.pi * r.random(count)
    ax = r.uniform(0.05, 0.35, (count, 2))
    return np.column_stack([rad * np.cos(th), rad * np.sin(th), r.uniform(-0.9, 0.9, count), ax,
                            r.uniform(0.3, 1.2, count), np.pi * r.random(count), r.uniform(0.0, 0.01, count),
                            r.uniform(-0.02, 0.02, (count, 2))])


def raster(ell, frames, n, nz):
    """The ellipsoids on the voxel grid, [frames][n][n][nz]."""
    g = (torch.arange(n, device="cuda") + 0.5) / (n / 2) - 1
    h = (torch.arange(nz, device="cuda") + 0.5) / (nz / 2) - 1
    y, x = g[:, None], g[None, :]
    out = torch.zeros((frames, n, n, nz), device="cuda")
    for f in range(frames):
        for cx, cy, cz, a, b, cc, phi, mu, vx, vy in ell:
            dx, dy = x - (cx + f * vx / frames), y - (cy + f * vy / frames)
            u, v = dx * math.cos(phi) + dy * math.sin(phi), -dx * math.sin(phi) + dy * math.cos(phi)
            q = (u / a) ** 2 + (v / b) ** 2
            out[f] += mu * (q[:, :, None] + ((h - cz) / cc) ** 2 < 1)
    return out


def sinogram(c, ell, seed):
    """y and w, [views][bins][rows], on the GPU."""
    n, nz = c["n"], c["nz"]
    _, ang = views_of(c)
    th = torch.from_numpy(ang).to("cuda", torch.float32) * (math.pi / 180)
    half = n / 2.0
    r = (torch.arange(n, device="cuda") + 0.5 - half) / half
    h = (torch.arange(nz, device="cuda") + 0.5) / (nz / 2) - 1
    fr = torch.arange(c["views"], device="cuda") // max(c["views"] // c["frames"], 1)
    ax = torch.zeros((c["views"], n, nz), device="cuda")
    for cx, cy, cz, a, b, cc, phi, mu, vx, vy in ell:
        # bins measure x cos - y sin; (cos, -sin) against the ellipse's own axes
        px, py = cx + fr * vx / c["frames"], cy + fr * vy / c["frames"]
        rc = px * torch.cos(th) - py * torch.sin(th)
        al = th + phi
        w2 = (a * torch.cos(al)) ** 2 + (b * torch.sin(al)) ** 2
        s2 = 1 - ((h - cz) / cc) ** 2
        d2 = (r[None, :] - rc[:, None]) ** 2
        q = (w2[:, None, None] * s2[None, None, :] - d2[:, :, None]).clamp_(min=0).sqrt_()
        ax += q * ((2 * mu * half * a * b) / w2)[:, None, None]
    g = gen(seed, 1)
    w = torch.poisson(I0 * torch.exp(-ax), generator=g).clamp_(min=1)
    y = torch.log(I0 / w)
    if c["zinger"]:
        hit = torch.rand(y.shape, device="cuda", generator=g) < 0.005
        y += hit * (2 + 3 * torch.rand(y.shape, device="cuda", generator=g))
    return y, w


def start_image(c, ell, seed):
    """The phantom with noise, not below 0, [frames][n][n][nz]."""
    x = raster(ell, c["frames"], c["n"], c["nz"])
    x += 2e-4 * torch.randn(x.shape, device="cuda", generator=gen(seed, 2))
    return x.clamp_(min=0)


def scan_state(c, seed):
    ell = ellipsoids(seed, 8 if c["frames"] > 1 else 30)
    t, a = views_of(c)
    ctx = xtg.Context(params_of(c), t, a)
    ctx.set_options(a_mode=AMODES[c["a"]])
    y, w = sinogram(c, ell, seed)
    s = {"ctx": ctx, "it": 6}
    if c["kind"] == "step":
        s["y"], s["w"] = y.cpu().pin_memory(), w.cpu().pin_memory()
        s["back"] = torch.empty(ctx.obj_shape, dtype=torch.float32).pin_memory()
    ctx.upload_sino(y.cpu().numpy(), w.cpu().numpy())
    if c["kind"] in ("icd", "step", "cost"):
        ctx.upload_object(start_image(c, ell, seed).permute(0, 3, 1, 2).contiguous().cpu().numpy())
        ctx.init_error_sino()
    if c["kind"] in ("icd", "step"):  # in the middle of a reconstruction: neither the first sweeps nor converged
        for it in range(1, s["it"]):
            ctx.iteration(it)
    s["x"] = torch.empty((ctx.N_time, ctx.N_y, ctx.N_x, ctx.N_z), device="cuda")
    torch.cuda.synchronize()
    return s


def images(c, seed):
    """FBP-like and start-like images and the object itself, [nb][y][x][z]."""
    shape = (c["nb"], c["y"], c["x"], c["z"])
    m = max(c["y"], c["x"])
    g = gen(seed, 3)
    true = torch.stack([raster(ellipsoids(seed * 100 + b, 30), 1, m, c["z"])[0, :c["y"], :c["x"]] for b in range(c["nb"])])
    fbp = (true + 1e-3 * torch.randn(shape, device="cuda", generator=g)).clamp_(min=0)
    p = F.avg_pool3d(true[:, None], 2)
    icd = F.interpolate(p, scale_factor=2, mode="nearest")[:, 0].contiguous()
    icd += 1e-4 * torch.randn(shape, device="cuda", generator=g)
    return fbp.contiguous(), icd, true.contiguous()


def conv_tensors(c, seed):
    """bf16 input [nb][y][x][z][cin], weights [27][cin][cout], bias, output gradient."""
    g = gen(seed, 4)
    v = (c["nb"], c["y"], c["x"], c["z"])
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g)  # noqa: E731
    x = F.relu(rnd(*v, c["cin"])).bfloat16()
    w = (rnd(27, c["cin"], c["cout"]) * math.sqrt(2 / (27 * c["cin"]))).bfloat16()
    return x, w, 0.1 * rnd(c["cout"]), rnd(*v, c["cout"]).bfloat16()


def k_major(w, transposed):
    """[27][cin][cout] -> rows of one output channel each, k = tap * inputs + input, padded to 64."""
    m = (w.permute(1, 0, 2) if transposed else w.permute(2, 0, 1)).reshape(w.shape[1 if transposed else 2], -1)
    return F.pad(m, (0, -m.shape[1] % 64)).contiguous()


class Net(xtg.WarmNet):
    """The network, its device buffers given back with it."""

    def __del__(self):
        self.close()


def prepare(c, seed):
    kind = c["kind"]
    if kind in ("icd", "step", "cost", "fbp", "multires"):
        s = scan_state(c, seed)
    elif kind == "nhicd":
        g = gen(seed, 5)
        n = (c["maps"], c["ny"], c["nx"])
        # update magnitudes: most columns near rest, a few moving
        m = 1e-3 * torch.exp(torch.randn(n, device="cuda", generator=g))
        m *= torch.rand(n, device="cuda", generator=g) > 0.2
        s = {"map": m, "kth": np.full(c["maps"], kth(c), np.int32), "thr": torch.zeros(c["maps"], device="cuda"),
             "sel": torch.zeros(n, dtype=torch.uint8, device="cuda"), "lib": xtg.gpu_lib()}
    elif kind in ("net", "train"):
        net = Net()
        net.load(WEIGHTS)
        f, q, t = images(c, seed)
        s = {"net": net, "fbp": f, "icd": q, "true": t, "out": torch.empty_like(f), "shape": tuple(f.shape)}
    else:
        x, w, b, dy = conv_tensors(c, seed)
        v = tuple(x.shape[:4])
        s = {"lib": xtg.gpu_lib(), "x": x, "b": b, "dy": dy, "w": k_major(w, False), "wt": k_major(w, True),
             "out": torch.empty(v + (c["cout"],), dtype=torch.bfloat16, device="cuda"),
             "dx": torch.empty(v + (c["cin"],), device="cuda"), "dw": torch.empty((27 * c["cin"], c["cout"]), device="cuda")}
    s["case"] = c
    torch.cuda.synchronize()
    return s


def kth(c):
    return c["ny"] * c["nx"] - c["ny"] * c["nx"] // 10


# -------------------------------------------------------------------- run --
def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def ok(rc):
    if rc:
        raise RuntimeError(xtg.gpu_lib().xtg_last_error().decode())


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "icd":
        st = s["ctx"].iteration(s["it"])
        s["it"] += 1
        s["ctx"].object_to_device(s["x"])
        return {"object": s["x"], "update_pct": st.avg_update_pct}
    if kind == "step":
        ctx = s["ctx"]
        ctx.upload_sino_start(s["y"], s["w"])
        ctx.iteration(s["it"])
        s["it"] += 1
        ctx.download_object_start(s["back"].data_ptr())
        ctx.download_wait()
        return s["back"]
    if kind == "cost":
        return s["ctx"].cost()
    if kind == "fbp":
        s["ctx"].init_fbp()
        s["ctx"].object_to_device(s["x"])
        return s["x"]
    if kind == "multires":
        s["ctx"].init_multires(c["iters"])
        s["ctx"].object_to_device(s["x"])
        return s["x"]
    if kind == "nhicd":
        ok(s["lib"].xtg_nhicd_threshold_noalloc(ptr(s["map"]), c["maps"], c["ny"], c["nx"],
                                                s["kth"].ctypes.data_as(ctypes.c_void_p), ptr(s["thr"]), ptr(s["sel"]),
                                                None))
        return s["thr"], s["sel"]
    if kind == "net":
        s["net"].forward(s["fbp"], s["icd"], s["out"], s["shape"])
        return s["out"]
    if kind == "train":
        loss = s["net"].backward(s["fbp"], s["icd"], s["true"], s["shape"])
        s["net"].adam_step(1e-4)
        return {"loss": loss, "gradients": s["net"].params(1)}
    dims = (c["nb"], c["y"], c["x"], c["z"])
    if c["op"] == "forward":
        ok(s["lib"].xtc_conv3d(ptr(s["x"]), ptr(s["w"]), ptr(s["b"]), ptr(s["out"]), *dims, c["cin"], c["cout"],
                               s["w"].shape[1], 0, 1))
        return s["out"]
    if c["op"] == "dgrad":
        ok(s["lib"].xtc_conv3d(ptr(s["dy"]), ptr(s["wt"]), None, ptr(s["dx"]), *dims, c["cout"], c["cin"],
                               s["wt"].shape[1], 2, -1))
        return s["dx"]
    s["dw"].zero_()
    ok(s["lib"].xtc_conv3d_wgrad(ptr(s["x"]), ptr(s["dy"]), ptr(s["dw"]), *dims, c["cin"], c["cout"]))
    return s["dw"]


# ------------------------------------------------------------------- work --
def work(c):
    kind = c["kind"]
    if kind == "nhicd":
        n = c["maps"] * c["ny"] * c["nx"]
        return {"bytes": 5.0 * n, "flops": 50.0 * n}
    if kind in ("net", "train"):
        vox = float(c["nb"] * c["y"] * c["x"] * c["z"])
        fl = sum(54.0 * ci * co * vox / 8 ** l for ci, co, l in LAYERS)
        return {"bytes": 12.0 * vox, "flops": fl * (3 if kind == "train" else 1)}
    if kind == "conv":
        vox = float(c["nb"] * c["y"] * c["x"] * c["z"])
        ci, co = c["cin"], c["cout"]
        by = {"forward": 2 * vox * (ci + co) + 54 * ci * co, "dgrad": 2 * vox * co + 4 * vox * ci + 54 * ci * co,
              "wgrad": 2 * vox * (ci + co) + 108 * ci * co}[c["op"]]
        return {"bytes": float(by), "flops": 54.0 * ci * co * vox}
    ns = float(c["views"]) * c["n"] * c["nz"]
    nvox = float(c["frames"]) * c["n"] ** 2 * c["nz"]
    hits = 2.2 * nvox * c["views"] / c["frames"]  # (voxel, sinogram entry) pairs
    if kind == "cost":
        return {"bytes": 8 * ns + 4 * nvox, "flops": 2 * hits}
    if kind == "fbp":  # the filter by FFT, two bins a (voxel, view), the error sinogram
        return {"bytes": 12 * ns + 8 * nvox, "flops": ns * 10 * math.log2(2 * c["n"]) + 4 * nvox * c["views"] / c["frames"] + 2 * hits}
    it = 2 * 8 * hits  # a random pass and as many selected columns; two sums and the update a pair
    if kind == "icd":
        return {"bytes": 12 * ns + 8 * nvox, "flops": it}
    if kind == "step":
        return {"bytes": 20 * ns + 12 * nvox, "flops": it + 2 * hits}
    return {"bytes": 12 * ns + 8 * nvox, "flops": c["iters"] * it / 4 + 2 * hits}


# ------------------------------------------------------------------ exact --
def exact_fbp(c, seed):
    """Ramp filter and interpolating backprojection of the sinogram."""
    y, _ = sinogram(c, ellipsoids(seed, 8 if c["frames"] > 1 else 30), seed)
    n, nz, f = c["n"], c["nz"], c["frames"]
    _, ang = views_of(c)
    th = torch.from_numpy(ang).cuda() * (math.pi / 180)
    m = (torch.arange(n, device="cuda")[:, None] - torch.arange(n, device="cuda")[None, :]).double()
    h = torch.where(m == 0, 0.25, torch.where(m.long() % 2 != 0, -1 / (m * math.pi).square().clamp(min=1), 0.0))
    g = torch.arange(n, device="cuda").double() + 0.5 - n / 2
    X, Y = g[None, :].expand(n, n).reshape(-1), g[:, None].expand(n, n).reshape(-1)
    out = torch.zeros((f, n * n, nz), dtype=torch.float64, device="cuda")
    per = c["views"] // f
    for p in range(c["views"]):
        q = F.pad(h @ y[p].double(), (0, 0, 1, 1))
        u = X * torch.cos(th[p]) - Y * torch.sin(th[p]) + n / 2 - 0.5
        i = torch.floor(u)
        w = (u - i)[:, None]
        i = i.long()
        at = lambda k: q[(k + 1).clamp(0, n + 1)]  # noqa: E731  (bins outside the detector read 0)
        out[min(p // per, f - 1)] += (1 - w) * at(i) + w * at(i + 1)
    cnt = torch.tensor([per] * (f - 1) + [c["views"] - per * (f - 1)], device="cuda").double()
    out *= (math.pi / cnt)[:, None, None]
    return out.clamp_(min=0).reshape(f, n, n, nz)


def exact_cost(c, seed):
    """(cost, data term, prior): generalized-Huber data term of y - A x and the qGGMRF prior."""
    ell = ellipsoids(seed, 8 if c["frames"] > 1 else 30)
    y, w = sinogram(c, ell, seed)
    x = start_image(c, ell, seed).double()
    n, f, p = c["n"], c["frames"], params_of(c)
    _, ang = views_of(c)
    g = torch.arange(n, device="cuda").double() + 0.5 - n / 2
    X, Y = g[None, :].expand(n, n).reshape(-1), g[:, None].expand(n, n).reshape(-1)
    off = (1 / math.sqrt(2) + 0.5) / 64  # the response is tabulated at 64 offsets
    q = torch.arange(512, device="cuda").double()
    beam = 0.54 - 0.46 * torch.cos(2 * math.pi / 512 * q)
    beam /= beam.sum()
    per, data = c["views"] // f, 0.0
    col = torch.arange(n * n, device="cuda")
    for v in range(c["views"]):
        th = math.radians(ang[v])
        # a voxel's line-integral profile (a trapezoid), 1536 samples over two voxel widths
        a = math.fmod(th, math.pi / 2)
        top = 1 / math.cos(a if a <= math.pi / 4 else math.pi / 2 - a)
        d1, d2 = math.cos(math.pi / 4) * math.cos(math.pi / 4 - a), math.cos(math.pi / 4) * abs(math.cos(math.pi / 4 + a))
        t = 2.0 * torch.arange(1536, device="cuda").double() / 1536
        prof = top * ((d1 - (t - 1).abs()) / max(d1 - d2, 1e-30)).clamp(0, 1)
        i = torch.floor(((-0.5 + q / 512)[None, :] - (torch.arange(64, device="cuda").double() * off - 1)[:, None]) * 768).long()
        hr = F.pad((torch.where((i >= 0) & (i < 1536), prof[i.clamp(0, 1535)], 0.0) * beam).sum(1), (0, 1))
        r = X * math.cos(th) - Y * math.sin(th) + n / 2
        b = torch.floor(r)[:, None].long() + torch.arange(-1, 2, device="cuda")
        d = (r[:, None] - (b + 0.5)).abs() / off
        k = torch.floor(d).long()
        A = torch.where(k < 64, hr[k.clamp(max=63)] * (1 - (d - k)) + hr[k.clamp(max=63) + 1] * (d - k), 0.0)
        keep = (b >= 0) & (b < n) & (A > 0)
        m = torch.sparse_coo_tensor(torch.stack([b[keep], col[:, None].expand(-1, 3)[keep]]), A[keep], (n, n * n))
        e = y[v].double() - torch.sparse.mm(m, x[min(v // per, f - 1)].reshape(n * n, -1))
        z = (e * w[v].double().sqrt()).abs()
        data += torch.where(z < p.zingerT, z * z, 2 * p.zingerDel * p.zingerT * z + p.zingerT ** 2 * (1 - 2 * p.zingerDel)).sum().item()
    slope = 1000.0 / (0.521225397034623 - 0.496372335005353 * 0.001205) / 0.0001
    chu = -slope * (0.496372335005353 * 0.001205 * 0.0001)
    inv = {(i, j, k): 1 / math.sqrt(i * i + j * j + k * k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1) if i or j or k}
    total = sum(inv.values()) + 2

    def rho(d, sig, cc):
        d = d.abs()
        return d * d / sig ** 2 / (cc + d ** (2 - p.p) / sig ** (2 - p.p))

    ss, prior = (p.sigma_s - chu) / slope, 0.0
    cut = lambda s: (slice(max(0, -s), None if s <= 0 else -s), slice(max(0, s), None if s >= 0 else s))  # noqa: E731
    for (i, j, k), v in inv.items():
        if (i, j, k) > (0, 0, 0):
            (z0, z1), (y0, y1), (x0, x1) = cut(i), cut(j), cut(k)
            prior += v * rho(x[:, y0, x0, z0] - x[:, y1, x1, z1], ss, p.c_s).sum().item()
    st = (p.sigma_t - chu) / slope * p.Rtime_delta
    prior += rho(x[1:] - x[:-1], st, p.c_t).sum().item() if f > 1 else 0.0
    prior *= p.Rtime_delta / total
    return data / 2 + prior, data / 2, prior


class Conv(torch.autograd.Function):
    """3x3x3 convolution, padding 1, [nb][y][x][z][cin] with [27][cin][cout], one tap at a time."""

    @staticmethod
    def shifted(x):
        nb, Y, X, Z, c = x.shape
        p = F.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        for t in range(27):
            dy, dx, dz = t // 9, t // 3 % 3, t % 3
            yield t, p[:, dy:dy + Y, dx:dx + X, dz:dz + Z]

    @staticmethod
    def forward(ctx, x, w):
        ctx.save_for_backward(x, w)
        out = x.new_zeros(x.shape[:4] + (w.shape[2],))
        for t, v in Conv.shifted(x):
            out += v @ w[t]
        return out

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        dx, dw = torch.zeros_like(x), torch.zeros_like(w)
        flat = dy.reshape(-1, dy.shape[-1])
        for t, v in Conv.shifted(x):
            dw[t] = v.reshape(-1, v.shape[-1]).T @ flat
        for t, v in Conv.shifted(dy):
            dx += v @ w[26 - t].T
        return dx, dw


def exact_net(flat, fbp, icd):
    """The network in 64 bits: flat parameters, images [nb][y][x][z]."""
    at, layers = 0, []
    for ci, co, _ in LAYERS:
        layers.append((flat[at:at + 27 * ci * co].view(27, ci, co), flat[at + 27 * ci * co:at + 27 * ci * co + co]))
        at += 27 * ci * co + co

    def conv(i, t):
        return torch.relu(Conv.apply(t, layers[i][0]) + layers[i][1])

    def pool(t):
        nb, Y, X, Z, ch = t.shape
        return t.view(nb, Y // 2, 2, X // 2, 2, Z // 2, 2, ch).mean((2, 4, 6))

    def up(t, skip):
        for d in (1, 2, 3):
            t = t.repeat_interleave(2, d)
        return torch.cat([t, skip], -1)

    s0 = conv(1, conv(0, torch.stack([fbp, icd], -1) * SCALE))
    s1 = conv(3, conv(2, pool(s0)))
    s2 = conv(5, conv(4, pool(s1)))
    t = conv(7, conv(6, pool(s2)))
    t = conv(9, conv(8, up(t, s2)))
    t = conv(11, conv(10, up(t, s1)))
    t = conv(13, conv(12, up(t, s0)))
    return icd + (t @ flat[at:at + 32] + flat[at + 32]) / SCALE


def exact(c, seed):
    kind = c["kind"]
    if kind == "fbp":
        return exact_fbp(c, seed)
    if kind == "cost":
        return exact_cost(c, seed)
    if kind == "nhicd":
        m = prepare(c, seed)["map"].double()
        h = torch.tensor([[0.0064, 0.0432, 0.08, 0.0432, 0.0064], [0.0432, 0.2916, 0.54, 0.2916, 0.0432],
                          [0.08, 0.54, 1.0, 0.54, 0.08], [0.0432, 0.2916, 0.54, 0.2916, 0.0432],
                          [0.0064, 0.0432, 0.08, 0.0432, 0.0064]], dtype=torch.float64, device="cuda")
        p = F.pad(m, (2, 2, 2, 2))
        f = sum(h[i, j] * p[:, i:i + c["ny"], j:j + c["nx"]] for i in range(5) for j in range(5))
        return f.reshape(c["maps"], -1).kthvalue(kth(c), 1).values, None
    if kind in ("net", "train"):
        flat = torch.from_numpy(np.fromfile(WEIGHTS, np.float32)[3:].astype(np.float64)).cuda()
        f, q, t = (v.double() for v in images(c, seed))
        if kind == "net":
            with torch.no_grad():
                return exact_net(flat, f, q)
        flat.requires_grad_(True)
        loss = torch.mean(((exact_net(flat, f, q) - t) * SCALE) ** 2)
        loss.backward()
        return {"loss": loss.item(), "gradients": flat.grad}
    if kind == "conv":
        x, w, b, dy = (v.double() for v in conv_tensors(c, seed))
        if c["op"] == "forward":
            return torch.relu(Conv.apply(x, w) + b)
        x.requires_grad_(True)
        w.requires_grad_(True)
        Conv.apply(x, w).backward(dy)
        return x.grad if c["op"] == "dgrad" else w.grad.reshape(27 * c["cin"], c["cout"])
    return None  # an iteration's result depends on which columns are in flight together
