"""The work a user of this framework has it do, as cases that can be timed one by one.

listed() names the cases, draw() gives more of the same ranges, prepare() makes what a program holds
before the call (frames, a context, parameters), run() is one pass through the public entry points of
the Python binding, work() the bytes and operations no implementation can do without, and exact() the
same result in plain FP64 torch.

A case's kind is the entry point:
  host    Context.scene_flow_two_frames: the drop-in call, one pair in host memory
  dimage  Context.scene_flow_multiscale: the reference's own entry point over FP64 planes
  seam    Context.scene_flow_single_scale: the per-level solver the reference calls
  device  Context.scene_flow_batch_device: n pairs in device memory, one solve (warm: from an estimate)
  noalloc scene_flow_noalloc: one pair in device memory, static workspace
  flow2d  Context.optical_flow_2d: the demo's flow type 1
"schedule" is "bench" (ratio 0.5, 5 levels, 10 outer, 30 SOR iterations, ISOTROPIC weights), "fine" (the
reference's pyramid ratio 0.75 with the bench's iteration counts) or "demo" (the reference's defaults:
ratio 0.75, 50 outer iterations, up to 10000 SOR iterations).
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "rgbd-flow_b200"))

import rgbdflow as rf  # noqa: E402
import synthetic as syn  # noqa: E402

# name of a mix -> (W, H, pairs)
MIXES = {"mix64": [(160, 120, 24), (320, 240, 24), (640, 480, 16)]}


def listed():
    return [
        # the smallest frame of the test configurations through the drop-in call: launches and latency
        dict(name="host_160x120", kind="host", W=160, H=120, schedule="bench", reg="iso"),
        # the drop-in call on the sensor's frame size, as a program that solves one pair at a time makes it
        dict(name="host_640x480", kind="host", W=640, H=480, schedule="bench", reg="iso"),
        # a cropped frame whose rows and levels are a multiple of nothing, on the reference's pyramid
        dict(name="host_501x377_ratio075", kind="host", W=501, H=377, schedule="fine", reg="iso"),
        # the command line's own call: halved sensor frames, every parameter at the reference's default
        dict(name="demo_320x240_hpb", kind="host", W=320, H=240, schedule="demo", reg="hpb"),
        # a program that links the reference's OpticalFlow class: FP64 planes in and out
        dict(name="dimage_320x240", kind="dimage", W=320, H=240, schedule="bench", reg="iso"),
        # a program that keeps the reference's pyramid and replaces its per-level solver
        dict(name="seam_160x120", kind="seam", W=160, H=120, schedule="bench", reg="iso"),
        # a control loop that may not allocate: one halved frame already on the device
        dict(name="noalloc_320x240", kind="noalloc", W=320, H=240, schedule="bench", reg="iso"),
        # the throughput workload of the benchmark
        dict(name="batch16_640x480", kind="device", W=640, H=480, n=16, schedule="bench", reg="iso", store="fp32", warm=0),
        # the benchmark's uneven batch: cameras of three resolutions solved together
        dict(name="mix64", kind="device", mix="mix64", schedule="bench", reg="iso", store="fp32", warm=0),
        # video: every stream starts from its previous flow (one full-resolution level)
        dict(name="warm8_640x480", kind="device", W=640, H=480, n=8, schedule="bench", reg="iso", store="fp32", warm=1),
        # FP16 pyramids, and the HPB weights the reference turns on by default, on a small batch
        dict(name="batch4_fp16_hpb_640x480", kind="device", W=640, H=480, n=4, schedule="bench", reg="hpb", store="fp16", warm=0),
        # the demo's other flow type on its halved frames
        dict(name="flow2d_320x240", kind="flow2d", W=320, H=240),
    ]


def draw(rng):
    """A case of the same ranges: widths 64..800 (half of them odd or otherwise ragged), batches up to 16
    pairs and at most the pixels of the listed batch."""
    kind = rng.choice(["host", "host", "device", "device", "device", "dimage", "seam", "noalloc", "flow2d"])
    top = {"host": 800, "device": 800, "dimage": 640, "seam": 320, "noalloc": 320, "flow2d": 240}[kind]
    W = int(round(math.exp(rng.uniform(math.log(64 if kind != "flow2d" else 80), math.log(top)))))
    H = max(48, int(W * rng.uniform(0.6, 0.8)))
    if rng.random() < 0.5:
        W, H = W & ~7, H & ~7
    if kind == "noalloc":
        H = min(H, 240)
    c = dict(kind=kind, W=W, H=H)
    if kind == "flow2d":
        return c
    c.update(schedule=rng.choice(["bench", "bench", "fine"]) if kind in ("host", "device") else "bench", reg="iso")
    if kind == "device":
        most = max(1, min(16, int(16 * 640 * 480 / (W * H))))
        c.update(n=rng.randint(1, most), store=rng.choice(["fp32", "fp32", "fp16", "bf16"]), warm=int(rng.random() < 0.25))
        if c["schedule"] == "bench" and not c["warm"] and rng.random() < 0.25:
            # the HPB weights' depth pyramid wants level sizes that halve evenly
            c.update(reg="hpb", W=max(64, W // 16 * 16), H=max(48, H // 16 * 16))
            c["n"] = min(c["n"], 4)
    return c


# ------------------------------------------------------------------------------------------
# schedules and inputs

def schedule(c, W):
    """The solve's parameters as plain numbers."""
    s = dict(alpha=0.02, gamma=1e-5, color_w=1.0, dvc=1.0, ratio=0.75, min_width=60, n_outer=50, n_sor=10000, period=25,
             omega=0.7, step=0.3, eps_d=1e-6, eps_z=1e-10, eps_s=1e-6, sor_tol=1e-5, outer_tol=4e-4, occ_margin=0.02,
             occ_penalty=0.01, max_grad=0.04, boundary=4)
    if c["schedule"] != "demo":
        s.update(n_outer=10, n_sor=30)
    if c["schedule"] == "bench":
        s.update(ratio=0.5, min_width=max(1, W // 16))
    return s


def params(c):
    p = rf.default_params()
    if c["schedule"] != "demo":
        p.n_outer, p.n_sor = 10, 30
    if c["schedule"] == "bench":
        p.pyramid_ratio, p.min_width = 0.5, -16
    p.regularization = {"iso": rf.REG_ISOTROPIC, "hpb": rf.REG_HPB}[c["reg"]]
    p.storage = {"fp32": rf.STORE_FP32, "fp16": rf.STORE_FP16, "bf16": rf.STORE_BF16}[c.get("store", "fp32")]
    return p


def focal(W):
    return 525.0 * W / 640


def camera(W, H):
    return rf.CameraParams.make(W, H, focal(W), (W - 1) / 2, (H - 1) / 2)


def scenes(W, H, n, seed, swap=True):
    """n frame pairs of one size: rendered scenes, each also mirrored in x, in y and in both, and (swap)
    with its frames exchanged, which are scenes of the same kind at none of the rendering cost."""
    out = []
    per = 8 if swap else 4
    for b in range((n + per - 1) // per):
        p = syn.make_pair(W=W, H=H, f=focal(W), cx=(W - 1) / 2, cy=(H - 1) / 2, n_patches=3 if W < 480 else 6,
                          hole_frac=0.05 if W < 480 else 0.08, seed=seed * 64 + b + W)
        for v in range(min(per, n - len(out))):
            fx, fy = v & 1, v >> 1 & 1
            q = {}
            for k in ("bgr1", "depth1", "bgr2", "depth2", "gt"):
                a = p[k]
                if k == "gt":
                    a = a * np.array([-1 if fx else 1, -1 if fy else 1, 1], np.float32)
                q[k] = np.ascontiguousarray(a[::-1 if fy else 1, ::-1 if fx else 1])
            if v & 4:
                q["bgr1"], q["bgr2"], q["depth1"], q["depth2"] = q["bgr2"], q["bgr1"], q["depth2"], q["depth1"]
            out.append(q)
    return out


def case_pairs(c, seed):
    """[(W, H, scene)] of a case."""
    sizes = MIXES[c["mix"]] if c.get("mix") else [(c["W"], c["H"], c.get("n", 1))]
    out = []
    for W, H, n in sizes:
        out += [(W, H, s) for s in scenes(W, H, n, seed, swap=not c.get("warm"))]
    if c.get("warm"):
        # the previous flow of a stream: the motion, damped, with what an estimate is off by
        g = np.random.default_rng(seed)
        for W, H, s in out:
            s["est"] = (0.8 * s["gt"] + g.normal(0, 1, s["gt"].shape) * np.array([0.1, 0.1, 0.002])).astype(np.float32)
    return out


def seam_inputs(c, seed):
    """One level's inputs as the reference's caller holds them: FP64 features, depths, weights, flow."""
    W, H = c["W"], c["H"]
    s = scenes(W, H, 1, seed)[0]
    dev = torch.device("cpu")
    col = [torch.from_numpy(s[k].astype(np.float64) / 255.0).permute(2, 0, 1).to(dev) for k in ("bgr1", "bgr2")]
    dep = [torch.from_numpy(s[k].astype(np.float64)).to(dev) for k in ("depth1", "depth2")]
    ddw = depth_weight(torch.from_numpy(s["depth1"]).to(dev), 4)
    dep = [fill_holes(d) for d in dep]
    f1, f2 = features(col[0]), features(col[1])
    g = np.random.default_rng(seed + 1)
    U = torch.from_numpy(0.7 * s["gt"].astype(np.float64) + g.normal(0, 1, s["gt"].shape) * np.array([0.05, 0.05, 0.001])).permute(2, 0, 1)
    wI, wD = warp(f1, dep[0], f2, dep[1], U)
    reg = torch.ones(H, W, 2, dtype=torch.float64)
    reg[:, -1, 0] = 0
    reg[-1, :, 1] = 0
    f = float(np.float32(focal(W)))
    return dict(Im1=f1, Im2=f2, dm1=dep[0], dm2=dep[1], wI=wI, wD=wD, U=U, ddw=ddw, dsw=torch.full((H, W), f * f, dtype=torch.float64),
                mag=(f / dep[0].clamp_min(1e-3)) ** 2, reg=reg, f=f)


def prepare(case, seed):
    c = case
    kind = c["kind"]
    if kind == "flow2d":
        s = scenes(c["W"], c["H"], 1, seed)[0]
        return dict(kind=kind, ctx=rf.Context(0), bgr1=s["bgr1"], bgr2=s["bgr2"])
    st = dict(kind=kind, prm=params(c))
    if kind != "noalloc":
        st["ctx"] = rf.Context(0)
    if kind == "seam":
        q = seam_inputs(c, seed)
        n = {k: np.ascontiguousarray(q[k].numpy()) for k in ("dm1", "dm2", "wD", "ddw", "dsw", "mag", "reg")}
        n.update({k: np.ascontiguousarray(q[k].permute(1, 2, 0).numpy()) for k in ("Im1", "Im2", "wI")})
        n.update({k: np.ascontiguousarray(q["U"][i].numpy()) for i, k in enumerate("uvw")})
        return dict(st, cam=camera(c["W"], c["H"]), n=n, k=schedule(c, c["W"]))
    pairs = case_pairs(c, seed)
    if kind in ("host", "dimage"):
        W, H, s = pairs[0]
        st.update(cam=camera(W, H), s=s)
        if kind == "dimage":
            sig = stereo_error1() / depth_weight(torch.from_numpy(s["depth1"]), 4)
            st.update(im1=s["bgr1"] / 255.0, im2=s["bgr2"] / 255.0, dm1=s["depth1"].astype(np.float64),
                      dm2=s["depth2"].astype(np.float64), sigma=sig.numpy().astype(np.float32))
        return st
    dev = []
    for W, H, s in pairs:
        d = {k: torch.from_numpy(s[k]).cuda() for k in ("bgr1", "depth1", "bgr2", "depth2")}
        if c.get("warm"):
            d["est"] = torch.from_numpy(s["est"]).cuda()
        dev.append(dict(d, W=W, H=H, cam=camera(W, H), out=torch.zeros(H, W, 3, device="cuda")))
    return dict(st, pairs=dev)


def run(state):
    kind, ctx = state["kind"], state.get("ctx")
    if kind == "host":
        s = state["s"]
        return ctx.scene_flow_two_frames(state["cam"], s["bgr1"], s["depth1"], s["bgr2"], s["depth2"], state["prm"], stats=False)
    if kind == "device":
        ctx.scene_flow_batch_device(state["pairs"], state["prm"])
        return [p["out"] for p in state["pairs"]]
    if kind == "noalloc":
        rf.scene_flow_noalloc(state["pairs"][0], state["prm"])
        return state["pairs"][0]["out"]
    if kind == "dimage":
        return list(ctx.scene_flow_multiscale(state["cam"], state["im1"], state["dm1"], state["im2"], state["dm2"], state["sigma"],
                                              state["prm"])[:3])
    if kind == "seam":
        n, k = state["n"], state["k"]
        return list(ctx.scene_flow_single_scale(state["cam"], n["Im1"], n["dm1"], n["Im2"], n["dm2"], n["wI"], n["wD"], n["u"], n["v"],
                                                n["w"], k["color_w"], n["ddw"], k["alpha"], n["dsw"], k["gamma"], n["mag"], n["reg"],
                                                k["n_outer"], 1, k["n_sor"], 1, state["prm"])[:5])
    return ctx.optical_flow_2d(state["bgr1"], state["bgr2"])


def work(case):
    """Inputs read once, outputs written once; operations of the shortest schedule the inputs can get (the
    convergence tests may end a level after one outer iteration of one check period; the coarsest level
    runs every outer iteration)."""
    c = case
    sizes = MIXES[c["mix"]] if c.get("mix") else [(c["W"], c["H"], c.get("n", 1))]
    if c["kind"] == "flow2d":
        n = c["W"] * c["H"]
        return {"bytes": n * (6 + 8), "flops": n * 40.0}
    nbytes = flops = 0.0
    for W, H, n in sizes:
        per = {"dimage": 24 + 24 + 8 + 8 + 4 + 24, "seam": 80 + 16 + 24 + 40 + 48 + 24 + 24}.get(c["kind"], 3 + 3 + 4 + 4 + 12)
        nbytes += n * W * H * (per + (12 if c.get("warm") else 0))
        s = schedule(c, W)
        sz = [(W, H)] if c.get("warm") or c["kind"] == "seam" else [x[:2] for x in pyramid_shape(W, H, s["ratio"], s["min_width"])]
        for k, (w, h) in enumerate(sz):
            last = k == len(sz) - 1 and c["kind"] != "seam"
            outer = s["n_outer"] if last else 1
            flops += n * w * h * outer * (min(s["n_sor"], s["period"]) * 84.0 + 400.0)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------------------------------
# the solve in FP64 torch

def stereo_error1():
    return 1.0 / (1.0 / .00285 + 1.0)


def shifted(x, di, dj, fill):
    """y[..., i, j] = x[..., i + di, j + dj], `fill` outside."""
    H, W = x.shape[-2:]
    y = torch.full_like(x, fill)
    i0, i1, j0, j1 = max(0, -di), min(H, H - di), max(0, -dj), min(W, W - dj)
    y[..., i0:i1, j0:j1] = x[..., i0 + di:i1 + di, j0 + dj:j1 + dj]
    return y


AROUND = [(a, b) for a in (-1, 0, 1) for b in (-1, 0, 1) if a or b]


def fill_holes(d):
    """Rounds: a hole pixel whose count of known neighbours none of its hole neighbours exceeds takes the
    (upper) median of its known neighbours; every decision reads the state before the round."""
    d = d.clone()
    known = d > 0
    for _ in range(253):
        if bool(known.all()):
            break
        nb = torch.stack([shifted(known, a, b, False) for a, b in AROUND])
        count = nb.sum(0)
        rival = torch.where(known, torch.full_like(count, -1), count)
        best = torch.stack([shifted(rival, a, b, -1) for a, b in AROUND]).amax(0)
        fill = ~known & (count > 0) & (best <= count)
        v = torch.stack([shifted(d, a, b, 0.0) for a, b in AROUND])
        v = torch.where(nb, v, torch.full_like(v, float("inf"))).sort(0).values
        med = v.gather(0, (count // 2).clamp(max=7).unsqueeze(0))[0]
        d = torch.where(fill, med, d)
        known = known | fill
    return d


def depth_weight(depth32, md):
    """The depth-data weight: stereo error at 1 m over the depth sigma, which grows tenfold towards a depth
    boundary over md pixels.  The boundary test takes the FP32 difference of two FP32 depths."""
    z = depth32.double()
    e1 = stereo_error1()
    ser = lambda q: (q * q / (1.0 / .00285 + q)) / e1  # noqa: E731
    s = torch.where(z > 0, (e1 * ser(z)).clamp_min(1e-4), torch.ones_like(z))

    def edge(di, dj):
        n = shifted(depth32, di, dj, 0.0)
        return (n > 0) & ((depth32 - n).abs().double() > .02 * ser(torch.minimum(z, n.double())))

    near = edge(1, 0) | edge(0, 1)
    best = torch.where(near, 0, md + 1)
    for t in range(1, md + 1):
        near = near | shifted(near, 1, 0, False) | shifted(near, -1, 0, False) | shifted(near, 0, 1, False) | shifted(near, 0, -1, False)
        best = torch.where(near & (best > t), t, best)
    a = best.double() / md
    s = torch.where(best <= md, torch.exp((1 - a) * torch.log(10 * s) + a * torch.log(s)), s)
    return e1 / s


def pyramid_shape(W, H, ratio, min_width):
    """[(w, h, source level, resize rate, filter sigma)] of the Gaussian pyramid, finest first."""
    n_levels, w = 1, W * ratio
    while w >= min_width:
        n_levels += 1
        w *= ratio
    base, n = 1 / ratio - 1, int(math.log(0.25) / math.log(ratio))
    out = [(W, H, 0, 1.0, 0.0)]
    for i in range(1, n_levels):
        if i <= n:
            r = ratio ** i
            out.append((int(W * r), int(H * r), 0, r, base * i))
        else:
            sl = i - n
            r = ratio ** i * W / out[sl][0]
            out.append((int(out[sl][0] * r), int(out[sl][1] * r), sl, r, base * n))
    return out


def along(x, dim, taps):
    """Correlation along a dimension, edges clamped."""
    fs, n = len(taps) // 2, x.shape[dim]
    at = torch.arange(n, device=x.device)
    return sum(t * x.index_select(dim, (at + l - fs).clamp(0, n - 1)) for l, t in enumerate(taps) if t != 0)


def resample(x, w, h, rx, ry):
    """Bilinear resize: (j, i) samples ((j + 1) / rx - 1, (i + 1) / ry - 1)."""
    H, W = x.shape[-2:]

    def axis(n, r, size):
        p = (torch.arange(n, device=x.device, dtype=torch.float64) + 1) / r - 1
        a = p.trunc()
        return a.long().clamp(0, size - 1), (a.long() + 1).clamp(0, size - 1), (p - a).clamp(0, 1)

    u0, u1, dx = axis(w, rx, W)
    v0, v1, dy = axis(h, ry, H)
    row = x[..., v0, :] * (1 - dy)[:, None] + x[..., v1, :] * dy[:, None]
    return row[..., u0] * (1 - dx) + row[..., u1] * dx


D5 = [1 / 12, -8 / 12, 0, 8 / 12, -1 / 12]


def features(col):
    g = .114 * col[0] + .587 * col[1] + .299 * col[2]
    return torch.stack([g, along(g, 1, D5), along(g, 0, D5), col[1] - col[0], col[1] - col[2]])


def warp(f1, d1, f2, d2, U):
    """Frame 2's features and depth at the flow, frame 1's where it leaves the image."""
    H, W = d1.shape
    jj = torch.arange(W, device=d1.device, dtype=torch.float64)
    ii = torch.arange(H, device=d1.device, dtype=torch.float64)[:, None]
    x, y = jj + U[0], ii + U[1]
    out = (x < 0) | (x > W - 1) | (y < 0) | (y > H - 1)
    xa, ya = x.floor().clamp(0, W - 1), y.floor().clamp(0, H - 1)
    ax, ay = x - xa, y - ya
    xa, ya = xa.long(), ya.long()
    xb, yb = (xa + 1).clamp(max=W - 1), (ya + 1).clamp(max=H - 1)
    s = torch.cat([f2, d2[None]])
    v = (1 - ax) * (1 - ay) * s[:, ya, xa] + (1 - ax) * ay * s[:, yb, xa] + ax * (1 - ay) * s[:, ya, xb] + ax * ay * s[:, yb, xb]
    v = torch.where(out, torch.cat([f1, d1[None]]), v)
    return v[:5], v[5] - U[2]


def system(U, f1, d1, f2, d2, ddw, dsw, mag, rh, rv, k):
    """One outer iteration's linear system: (1 / diagonal, off-diagonal couplings, right-hand sides, the four
    neighbour coefficients of the u and v rows, those of the w row)."""
    wI, wD = warp(f1, d1, f2, d2, U)
    mix = 0.4 * torch.cat([f1, d1[None]]) + 0.6 * torch.cat([wI, wD[None]])
    Ix, Iy = along(mix, 2, D5), along(mix, 1, D5)
    It = torch.cat([wI - f1, (wD - d1)[None]])
    m = k["max_grad"]
    Zx, Zy, Zt = Ix[5].clamp(-m, m), Iy[5].clamp(-m, m), It[5].clamp(-m, m)
    Ix, Iy, It = Ix[:5], Iy[:5], It[:5]
    q = torch.where(d1 + U[2] < d2 + k["occ_margin"] * d1 * d1, 1.0, k["occ_penalty"])
    psi = 0.5 / torch.sqrt((It * q) ** 2 + k["eps_d"]) * k["color_w"]
    pi = 0.5 / torch.sqrt(Zt * Zt + k["eps_z"]) * ddw
    right, down = shifted(U, 0, 1, 0.0) - U, shifted(U, 1, 0, 0.0) - U
    right[..., -1] = 0
    down[..., -1, :] = 0
    g = right ** 2 + down ** 2
    phi = 0.5 / torch.sqrt(g[0] + g[1] + dsw * g[2] + k["eps_s"])
    eR, eD = phi * rh, phi * rv
    eL, eU = shifted(eR, 0, -1, 0.0), shifted(eD, -1, 0, 0.0)
    lap = (U - shifted(U, 0, -1, 0.0)) * eL - right * eR + (U - shifted(U, -1, 0, 0.0)) * eU - down * eD
    inside = torch.ones_like(d1)
    nrm = rh + rv + shifted(rh, 0, -1, 0.0) + shifted(rv, -1, 0, 0.0)
    cnt = sum(shifted(inside, a, b, 0.0) for a, b in ((0, 1), (0, -1), (1, 0), (-1, 0)))
    lap = torch.where(nrm.abs() < 1e-5, torch.zeros_like(lap), lap / (nrm / cnt))
    sL, sU = shifted(dsw, 0, -1, 0.0), shifted(dsw, -1, 0, 0.0)
    al, ga = k["alpha"], k["gamma"]
    sxy, szz = eL + eU + eR + eD, eL * sL + eU * sU + (eR + eD) * dsw
    mean = lambda t: t.sum(0) / 5  # noqa: E731
    dinv = 1.0 / torch.stack([-(mean(psi * Ix * Ix) + pi * Zx * Zx + al * sxy) - ga, -(mean(psi * Iy * Iy) + pi * Zy * Zy + al * sxy) - ga,
                              -(pi + al * szz) - ga * mag])
    uv = -mean(psi * Ix * Iy) - pi * Zx * Zy
    uw, vw = pi * Zx, pi * Zy
    rhs = torch.stack([mean(psi * Ix * It) * q * q + pi * Zx * Zt + al * lap[0] + ga * U[0],
                       mean(psi * Iy * It) * q * q + pi * Zy * Zt + al * lap[1] + ga * U[1],
                       -(pi * Zt - al * dsw * lap[2]) + ga * mag * U[2]])
    a = torch.stack([al * e for e in (eL, eU, eR, eD)])
    aw = a * torch.stack([sL, sU, dsw, dsw])
    return dinv, (uv, uw, vw), rhs, a, aw


def solve_level(U, f1, d1, f2, d2, ddw, dsw, mag, rh, rv, f_level, early, k):
    H, W = d1.shape
    odd = (torch.arange(H, device=d1.device)[:, None] + torch.arange(W, device=d1.device)) % 2
    red = [odd == 0, odd == 1]
    for _ in range(k["n_outer"]):
        dinv, (uv, uw, vw), rhs, a, aw = system(U, f1, d1, f2, d2, ddw, dsw, mag, rh, rv, k)
        A = torch.stack([a, a, aw], 1)  # [neighbour][row]
        zero = torch.zeros_like(uv)
        C = torch.stack([torch.stack([zero, uv, uw]), torch.stack([uv, zero, vw]), torch.stack([uw, vw, zero])])
        xp = torch.zeros(3, H + 2, W + 2, dtype=torch.float64, device=d1.device)
        x = xp[:, 1:-1, 1:-1]
        for it in range(k["n_sor"]):
            check = it % k["period"] == k["period"] - 1
            old = x.clone() if check else None
            for c in range(2):
                nb = A[0] * xp[:, 1:-1, :-2]
                nb.addcmul_(A[1], xp[:, :-2, 1:-1]).addcmul_(A[2], xp[:, 1:-1, 2:]).addcmul_(A[3], xp[:, 2:, 1:-1])
                v = (rhs - nb - (C * x).sum(1)) * dinv
                v = k["omega"] * v + (1 - k["omega"]) * x
                x.copy_(torch.where(red[c], torch.minimum(torch.maximum(v, x - k["step"]), x + k["step"]), x))
            if check:
                md = float((x - old).abs().max())
                if md < k["sor_tol"] or md >= k["step"]:
                    break
        U = U + x
        stat = float((x[0] ** 2 + x[1] ** 2 + x[2] ** 2 * f_level / d1).sum()) / (3 * H * W)
        if early and stat < k["outer_tol"]:
            break
    return U


def solve(W, H, col1, dep1, col2, dep2, ddw, f, k, est=None):
    """The coarse-to-fine solve (isotropic weights) of filled depths; est: one full-resolution level from it."""
    shape = pyramid_shape(W, H, k["ratio"], k["min_width"])[: 1 if est is not None else None]
    base = torch.cat([col1, col2, dep1[None], dep2[None], ddw[None], torch.full_like(ddw, f * f)[None]])
    pyr = [base]
    for w, h, sl, rate, sigma in shape[1:]:
        fs = int(sigma * 3)
        g = [math.exp(-(l * l) / (sigma * sigma * 2)) for l in range(-fs, fs + 1)]
        g = [t / sum(g) for t in g]
        pyr.append(resample(along(along(pyr[sl], 2, g), 1, g), w, h, rate, rate))
    U = est
    for lv in range(len(shape) - 1, -1, -1):
        w, h = shape[lv][:2]
        P = pyr[lv]
        if est is None:
            if U is None:
                U = torch.zeros(3, h, w, dtype=torch.float64, device=P.device)
            else:
                U = resample(U, w, h, w / U.shape[2], h / U.shape[1])
                U = U * torch.tensor([1 / k["ratio"], 1 / k["ratio"], 1.0], dtype=torch.float64, device=P.device)[:, None, None]
        at = torch.arange(w * h, device=P.device)
        z = P[6].reshape(-1)[at // W * w + at % W].reshape(h, w)  # the reference indexes with the full width
        mag = torch.where(z > 0, f / z, torch.full_like(z, f / 2)) ** 2
        rh, rv = torch.ones_like(z), torch.ones_like(z)
        rh[:, -1] = 0
        rv[-1] = 0
        U = solve_level(U, features(P[0:3]), P[6], features(P[3:6]), P[7], P[8], P[9], mag, rh, rv,
                        float(np.float32(f * (w / W))), lv < len(shape) - 1, k)
    return U.permute(1, 2, 0).contiguous()


def exact(case, seed):
    """FP64 torch.  None for HPB weights and the 2-D flow (their order of operations is part of the result:
    8-bit colours and a lexicographic sweep that FP64 already runs), and for the 64-pair mix (over 20 s)."""
    c = case
    if c["kind"] == "flow2d" or c["reg"] != "iso" or c.get("mix"):
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    k = schedule(c, c["W"])
    if c["kind"] == "seam":
        q = {n: (v.to(dev) if torch.is_tensor(v) else v) for n, v in seam_inputs(c, seed).items()}
        U = solve_level(q["U"], q["Im1"], q["dm1"], q["Im2"], q["dm2"], q["ddw"], q["dsw"], q["mag"],
                        q["reg"][..., 0], q["reg"][..., 1], q["f"], True, k)
        wI, wD = warp(q["Im1"], q["dm1"], q["Im2"], q["dm2"], U)
        return [U[0].cpu(), U[1].cpu(), U[2].cpu(), wI.permute(1, 2, 0).cpu(), wD.cpu()]
    flows = []
    for i, (W, H, s) in enumerate(case_pairs(c, seed)):
        if i >= 4:  # the time of four pairs; the others of a batch are the same kind of scene
            flows.append(None)
            continue
        col = [torch.from_numpy(s[n]).to(dev).double().permute(2, 0, 1) / 255.0 for n in ("bgr1", "bgr2")]
        d32 = [torch.from_numpy(s[n]).to(dev) for n in ("depth1", "depth2")]
        ddw = depth_weight(d32[0], k["boundary"])
        if c["kind"] == "dimage":  # this entry point takes the FP32 sigma
            e1 = stereo_error1()
            ddw = e1 / (e1 / depth_weight(torch.from_numpy(s["depth1"]), k["boundary"])).float().double().to(dev)
        est = torch.from_numpy(s["est"]).to(dev).double().permute(2, 0, 1) if c.get("warm") else None
        flows.append(solve(W, H, col[0], fill_holes(d32[0].double()), col[1], fill_holes(d32[1].double()), ddw,
                           float(np.float32(focal(W))), k, est).cpu())
    if c["kind"] == "dimage":
        return [flows[0][..., j].contiguous() for j in range(3)]
    return flows if c["kind"] == "device" else flows[0]
