"""What a user of this package has it do, as measurable cases.

Families (the "kind" of a case), each through the package's public entry
points as a user's program calls them:

* step      -- advance a lattice by a batch of time steps and read rho, u, the
               wall shear stress, OSI and TAWSS into pinned host arrays (the
               end-to-end loop of every simulation);
* voxelize  -- a surface's triangles to the node-flag lattice (host data in
               and out, once per vessel);
* lattice   -- a mask and a surface to a ready lattice: classes, boundary
               lists, wall normals (once per vessel, before the first step);
* conv_fwd, conv_bwd -- one convolution layer of the warm-start network and
               its gradients through the C ABI;
* forward   -- the warm-start network's forward pass (a prediction);
* gradient  -- one training sample: forward, masked loss, backward;
* prior     -- the network-free part of a warm start: mask to network input,
               Poiseuille prior, smoothing and the per-node start fields.

Vessels are curved tubes with a stenosis, swept along z; each case states its
radius and length in lattice units.  A case's seed draws the flow state, the
inlet, the weights and the activations.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from pv_dec_original_gb300 import capi

# --------------------------------------------------------------------------- cases


def listed():
    return [
        # a single small vessel (the size of a 24 x 24 x 104 lattice): a step
        # is shorter than a launch, so latency and launches count
        dict(name="step_small_f32", kind="step", Q=19, precision="f32", mode="physics", collision="bgk", tau=0.8,
             radius=5.2, length=98, steps=100),
        # the ordinary run: about 0.95M nodes, FP32, regularized collision at
        # tau 0.55 as the pulsatile runs over several periods use it
        dict(name="step_f32", kind="step", Q=19, precision="f32", mode="physics", collision="regularized", tau=0.55,
             radius=24.6, length=509, steps=100),
        # a large lattice in FP16 storage (the precision option for capacity and throughput)
        dict(name="step_large_f16", kind="step", Q=19, precision="f16", mode="physics", collision="bgk", tau=0.8,
             radius=52.7, length=347, steps=100),
        # D3Q27 of a daughter vessel
        dict(name="step_q27_f32", kind="step", Q=27, precision="f32", mode="physics", collision="bgk", tau=0.8,
             radius=16.9, length=301, steps=100),
        # the drop-in semantics of the CPU code this engine replaces: FP64, its step order and wall rule
        dict(name="step_parity_f64", kind="step", Q=19, precision="f64", mode="parity", collision="bgk", tau=0.8,
             radius=11.8, length=163, steps=50),
        # STL triangles to the flag lattice: an artery-sized surface
        dict(name="voxelize", kind="voxelize", radius=24.6, length=509, h=1.5),
        # mask + surface to a ready lattice
        dict(name="lattice_setup", kind="lattice", Q=19, precision="f32", radius=17.3, length=253, h=2.0),
        # the network's first-level layer at the full prediction grid: forward
        dict(name="conv_fwd_16", kind="conv_fwd", D=256, H=128, W=128, ci=16, co=16, ksize=3, stride=1, relu=1),
        # a second-level layer's gradients (input, weights, bias) in training
        dict(name="conv_bwd_32", kind="conv_bwd", D=128, H=64, W=64, ci=32, co=32, ksize=3, stride=1),
        # a prediction at the scaled-down training grid
        dict(name="net_forward", kind="forward", D=128, H=64, W=64),
        # one training sample at the full grid
        dict(name="net_gradient", kind="gradient", D=256, H=128, W=128),
        # a warm start's geometry features and prior for a new vessel
        dict(name="prior_fields", kind="prior", D=128, H=64, W=64),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "voxelize", "lattice", "conv_fwd", "conv_bwd", "forward",
                       "gradient", "prior"])
    if kind == "step":
        mode = rng.choice(["physics", "physics", "physics", "parity"])
        precision = "f64" if mode == "parity" else rng.choice(["f32", "f32", "f16", "bf16", "f64"])
        q = 19 if mode == "parity" else rng.choice([19, 19, 27])
        nodes = _log(rng, 5e3, 1.5e5 if precision == "f64" else 1.5e6)
        radius = max(5.0, min(50.0, (nodes / (8.0 * math.pi)) ** (1.0 / 3.0) * rng.uniform(0.6, 1.3)))
        length = max(24, min(600, int(nodes / (math.pi * radius * radius))))
        reg = mode == "physics" and rng.random() < 0.5
        return dict(kind=kind, Q=q, precision=precision, mode=mode, collision="regularized" if reg else "bgk",
                    tau=0.55 if reg else 0.8, radius=round(radius, 2), length=length,
                    steps=50 if precision == "f64" else 100)
    if kind == "voxelize":
        radius = _log(rng, 6.0, 26.0)
        return dict(kind=kind, radius=round(radius, 2), length=int(_log(rng, 40, 500)), h=round(rng.uniform(1.5, 3.0), 2))
    if kind == "lattice":
        return dict(kind=kind, Q=rng.choice([19, 19, 27]), precision=rng.choice(["f32", "f16", "f64"]),
                    radius=round(_log(rng, 5.0, 18.0), 2), length=int(_log(rng, 24, 250)), h=2.0)
    if kind in ("conv_fwd", "conv_bwd"):
        level = rng.choice([0, 1, 1, 2])
        ci, co, stride = rng.choice([[(16, 16, 1), (32, 16, 1), (16, 32, 2)], [(32, 32, 1), (64, 32, 1), (32, 64, 2)],
                                     [(64, 64, 1), (64, 64, 2)]][level])
        # grids of the prediction's range at that level, ragged ones among them
        D, H, W = [max(8, (8 * rng.randint(lo, hi)) >> level) for lo, hi in ((6, 28), (4, 15), (4, 15))]
        if rng.random() < 0.5:
            H, W = max(16, H // 16 * 16), max(16, W // 16 * 16)
        c = dict(kind=kind, D=D, H=H, W=W, ci=ci, co=co, ksize=3, stride=stride)
        return dict(c, relu=1) if kind == "conv_fwd" else c
    # whole predictions: grids of the tiling the network is run at
    g = rng.choice([(1, 1), (1, 1), (2, 1), (1, 2)])
    if kind == "prior":
        return dict(kind=kind, D=8 * rng.randint(6, 30), H=8 * rng.randint(4, 15), W=8 * rng.randint(4, 15))
    return dict(kind=kind, D=32 * rng.randint(2, 6), H=64 * g[0], W=64 * g[1])


# --------------------------------------------------------------------------- vessels


def _centre(z, c, depth=0.25):
    """Centre line and radius of the vessel at height z (arrays); depth: of
    the stenosis, which lies where the vessel's bounding box does not depend
    on it."""
    R, L = c["radius"], float(c["length"])
    half = R + 2.0 + 0.12 * R
    t = np.clip(z / L, 0.0, 1.0)
    cx = half + 0.173 + 0.10 * R * np.sin(2.0 * math.pi * t)
    cy = half + 0.061 + 0.07 * R * np.sin(4.0 * math.pi * t)
    s = (t - 0.45) / 0.18
    r = R * (1.0 - depth * np.where(np.abs(s) < 1.0, 0.5 * (1.0 + np.cos(math.pi * s)), 0.0))
    return cx, cy, r


def vessel_mask(c):
    """uint8 [z][y][x]: 1 inside the vessel; one solid layer below and above."""
    nz = int(c["length"]) + 2
    n = int(math.ceil(2.0 * (1.12 * c["radius"] + 2.0))) + 1
    z = np.arange(nz, dtype=np.float64) - 1.0
    cx, cy, r = _centre(z, c)
    x = np.arange(n, dtype=np.float64)
    dx = (x[None, :] - cx[:, None]) ** 2
    dy = (x[None, :] - cy[:, None]) ** 2
    m = (dy[:, :, None] + dx[:, None, :]) < (r ** 2)[:, None, None]
    m[0] = m[-1] = False
    return np.ascontiguousarray(m.astype(np.uint8))


def vessel_surface(c, h, depth=0.25):
    """The vessel's closed surface as rows x1..z3, facet normal (float64 [n, 12])."""
    L = float(c["length"])
    na = max(12, int(round(2.0 * math.pi * c["radius"] / h)))
    nl = max(2, int(round(L / h)))
    z = np.linspace(0.5, L + 0.5, nl + 1)
    cx, cy, r = _centre(z - 1.0, c, depth)
    th = 2.0 * math.pi * np.arange(na) / na + 0.037
    ring = np.stack([cx[:, None] + r[:, None] * np.cos(th), cy[:, None] + r[:, None] * np.sin(th),
                     np.repeat(z[:, None], na, 1)], axis=-1)  # [nl + 1, na, 3]
    nx = np.roll(ring, -1, axis=1)
    a, b, d, e = ring[:-1], nx[:-1], ring[1:], nx[1:]
    wall = np.concatenate([np.stack([a, b, e], 2).reshape(-1, 3, 3), np.stack([a, e, d], 2).reshape(-1, 3, 3)])
    c0 = np.array([cx[0], cy[0], z[0]])
    c1 = np.array([cx[-1], cy[-1], z[-1]])
    low = np.stack([np.broadcast_to(c0, nx[0].shape), nx[0], ring[0]], 1)
    top = np.stack([np.broadcast_to(c1, nx[-1].shape), ring[-1], nx[-1]], 1)
    v = np.concatenate([wall, low, top])
    n = np.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    n /= np.maximum(np.linalg.norm(n, axis=1, keepdims=True), 1e-300)
    return np.ascontiguousarray(np.concatenate([v.reshape(-1, 9), n], axis=1))


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# --------------------------------------------------------------------------- inputs (shared by prepare and exact)

PERIOD = 4000


def step_inputs(c, seed):
    """Mask, surface, start fields (FP32 rho [n], u [n, 3]) and inlet table."""
    rng = np.random.default_rng(seed)
    mask = vessel_mask(c)
    tri = vessel_surface(c, max(1.5, c["radius"] / 8.0))
    k, j, i = np.nonzero(mask)
    cx, cy, r = _centre(k - 1.0, c)
    mean = float(rng.uniform(0.02, 0.04))
    prof = np.clip(1.0 - ((i - cx) ** 2 + (j - cy) ** 2) / r ** 2, 0.0, None)
    u = rng.normal(0.0, 0.03 * mean, (len(k), 3))
    u[:, 2] += mean * prof
    rho = 1.0 + rng.normal(0.0, 1e-4, len(k))
    s = np.arange(PERIOD, dtype=np.float64) * (2.0 * math.pi / PERIOD)
    amp = mean * (1.0 + 0.5 * np.sin(s) + 0.2 * np.sin(2.0 * s))
    return mask, tri, rho.astype(np.float32), u.astype(np.float32), amp


def inlet(c):
    cx, cy, r = _centre(np.array([0.0]), c)
    return float(cx[0]), float(cy[0]), float(r[0])


def conv_inputs(c, seed):
    """Activations (after a ReLU), weights [co][27][ci], bias and output gradient, BF16 on the GPU."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(seed)
    n = c["D"] * c["H"] * c["W"]
    taps = c["ksize"] ** 3
    x = torch.randn(n * c["ci"], generator=g, device=dev).relu_().to(torch.bfloat16)
    w = (torch.randn(c["co"] * taps * c["ci"], generator=g, device=dev)
         * math.sqrt(2.0 / (taps * c["ci"]))).to(torch.bfloat16)
    b = torch.randn(c["co"], generator=g, device=dev) * 0.1
    no = np.prod([(v - 1) // c["stride"] + 1 for v in (c["D"], c["H"], c["W"])])
    dy = None
    if c["kind"] == "conv_bwd":
        dy = torch.randn(int(no) * c["co"], generator=g, device=dev).to(torch.bfloat16)
    return x, w, b, dy, int(no)


# (name, source, input channels, output channels, kernel, stride, ReLU, tensor added to the result); "up:" = the
# source upsampled by two
NET = [("c0a", "x", 16, 16, 3, 1, 1, None), ("c0b", "c0a", 16, 16, 3, 1, 1, None), ("d1", "c0b", 16, 32, 3, 2, 1, None),
       ("c1", "d1", 32, 32, 3, 1, 1, None), ("d2", "c1", 32, 64, 3, 2, 1, None), ("c2", "d2", 64, 64, 3, 1, 1, None),
       ("d3", "c2", 64, 64, 3, 2, 1, None), ("c3", "d3", 64, 64, 3, 1, 1, None),
       ("u2", "up:c3", 64, 64, 3, 1, 1, "c2"), ("c2u", "u2", 64, 64, 3, 1, 1, None),
       ("u1", "up:c2u", 64, 32, 3, 1, 1, "c1"), ("c1u", "u1", 32, 32, 3, 1, 1, None),
       ("u0", "up:c1u", 32, 16, 3, 1, 1, "c0b"), ("c0u", "u0", 16, 16, 3, 1, 1, None),
       ("out", "c0u", 16, 16, 1, 1, 0, None)]


def net_vessel(c, seed):
    """A straight tube with a stenosis along z filling a D x H x W box; the
    seed draws which way round it lies and the inlet."""
    rng = np.random.default_rng(seed + 77)
    D, H, W = c["D"], c["H"], c["W"]
    R = 0.37 * min(H, W)
    t = (np.arange(D) / D - 0.4) / 0.2
    r = R * (1.0 - 0.3 * np.where(np.abs(t) < 1, 0.5 * (1 + np.cos(math.pi * t)), 0.0))
    if rng.random() < 0.5:
        r = r[::-1].copy()
    y = np.arange(H) - 0.5 * (H - 1) - 0.13 * rng.choice([-1.0, 1.0])
    x = np.arange(W) - 0.5 * (W - 1) + 0.07 * rng.choice([-1.0, 1.0])
    rad = np.sqrt(y[:, None] ** 2 + x[None, :] ** 2)
    mask = (rad[None] < r[:, None, None]).astype(np.uint8)
    mask[0] = mask[-1] = 0
    return np.ascontiguousarray(mask), r, rad, float(rng.uniform(0.01, 0.04)), float(rng.uniform(2000.0, 6000.0))


def net_inputs(c, seed):
    """Network input (BF16 [D*H*W*16]) and training target (FP32 [D*H*W*4]), mask, on the GPU."""
    dev = _device()
    D, H, W = c["D"], c["H"], c["W"]
    mask, r, rad, mean, period = net_vessel(c, seed)
    R = torch.from_numpy(r).to(dev, torch.float32)[:, None, None]
    q = torch.from_numpy(rad).to(dev, torch.float32)[None]
    m = torch.from_numpy(mask).to(dev)
    x = torch.zeros((D, H, W, 16), device=dev)
    x[..., 0] = ((R - q) * 0.2).clamp(-3.0, 3.0)
    x[..., 1] = m
    x[..., 2] = mean * 30.0
    x[..., 3] = period / 4000.0
    x[..., 4] = (torch.arange(D, device=dev) / D)[:, None, None]
    x[..., 5] = (1.0 - (q / R) ** 2).clamp(0.0) * m * (R[0] / R) ** 2
    x[..., 6] = (1.0 - torch.arange(D, device=dev) / D)[:, None, None] * 0.1 * m
    g = torch.Generator(device=dev).manual_seed(seed)
    # the correction a pulsatile solution leaves: smooth fields in the fluid
    ph = torch.rand(4, 3, generator=g, device=dev) * 6.28
    z = torch.arange(D, device=dev)[:, None, None] * (6.28 / D)
    yy = torch.arange(H, device=dev)[None, :, None] * (6.28 / H)
    xx = torch.arange(W, device=dev)[None, None, :] * (6.28 / W)
    t = torch.stack([0.3 * torch.sin(z + p[0]) * torch.cos(yy + p[1]) * torch.cos(xx + p[2]) + 0.2 for p in ph], dim=-1)
    t = t * m[..., None]
    return x.to(torch.bfloat16).reshape(-1), t.reshape(-1).contiguous(), m.reshape(-1), float(m.sum())


# --------------------------------------------------------------------------- prepare


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _pinned(n):
    return torch.zeros(n, dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "step":
        mask, tri, rho, u, amp = step_inputs(c, seed)
        s = capi.Solver(c["Q"], c["precision"], capi.LBM_PARITY if c["mode"] == "parity" else capi.LBM_PHYSICS, c["tau"],
                        1.0, (0.0, 0.0, 0.0), 1.0, 1.0,
                        collision=capi.LBM_COLLISION_REGULARIZED if c["collision"] == "regularized" else 0)
        cx, cy, r = inlet(c)
        s.set_geometry(mask, [capi.bc_spec(capi.LBM_BC_VELOCITY, "z-", -1, 1.0, 1, cx, cy, r),
                              capi.bc_spec(capi.LBM_BC_PRESSURE, "z+", -1, 1.0)])
        s.set_normals(tri)
        s.set_inlet_table(amp)
        s.init_from_macro(rho, u, regularized=False)
        s.set_graph_steps(c["steps"])
        n, nn = len(rho), s.counts()["next_to_wall"]
        return dict(c=c, s=s, rho=_pinned(n), u=_pinned(3 * n), wss=_pinned(nn), osi=_pinned(nn), tawss=_pinned(nn))
    if kind in ("voxelize", "lattice"):
        if kind == "voxelize":
            # the seed draws the stenosis
            return dict(c=c, tri=vessel_surface(c, c["h"], float(np.random.default_rng(seed).uniform(0.15, 0.4))))
        # the seed moves surface and lattice by a fraction of the spacing
        tri, shift = _moved(vessel_surface(c, c["h"]), seed)
        return dict(c=c, tri=tri, mask=vessel_mask(c), origin=shift)
    if kind in ("conv_fwd", "conv_bwd"):
        x, w, b, dy, no = conv_inputs(c, seed)
        st = dict(c=c, x=x, w=w, b=b, dims=(C.c_int * 3)(c["D"], c["H"], c["W"]), L=capi.load())
        if kind == "conv_fwd":
            st["y"] = torch.empty(no * c["co"], dtype=torch.bfloat16, device=x.device)
        else:
            st.update(dy=dy, dx=torch.empty_like(x), wt=torch.empty_like(w),
                      dw=torch.zeros(w.numel(), device=x.device), db=torch.zeros(c["co"], device=x.device))
        return st
    if kind == "prior":
        mask, _, _, mean, period = net_vessel(c, seed)
        return dict(c=c, mask=mask, mean=mean, period=period)
    from pv_dec_original_gb300 import warmstart
    net = warmstart.WarmStartNet((c["D"], c["H"], c["W"]), seed=seed)
    x, t, m, nfl = net_inputs(c, seed)
    return dict(c=c, net=net, x=x, t=t, m=m, inv=1.0 / (4.0 * nfl))


def _moved(tri, seed):
    """The surface and lattice origin shifted together by a seeded amount."""
    shift = np.random.default_rng(seed).uniform(-0.02, 0.02, 3)
    t = tri.copy()
    t[:, :9] += np.tile(2.0 * shift, 3)
    return np.ascontiguousarray(t), tuple(float(v) for v in shift)


# --------------------------------------------------------------------------- run


def run(state):
    c = state["c"]
    kind = c["kind"]
    if kind == "step":
        s = state["s"]
        s.step_async(c["steps"])
        s.outputs_async(state["rho"], state["u"], state["wss"], state["osi"], state["tawss"])
        s.wait_outputs()
        return {k: state[k] for k in ("rho", "u", "wss", "osi", "tawss")}
    if kind == "voxelize":
        mask, d = capi.voxelize(state["tri"], 1.0)
        return {"mask": mask, "fluid": int(d.fluid_count), "dims": np.array(d.dims[:], np.int64)}
    if kind == "lattice":
        cx, cy, r = inlet(c)
        s = capi.Solver(c["Q"], c["precision"], capi.LBM_PHYSICS, 0.8, 1.0, state["origin"], 1.0, 1.0)
        s.set_geometry(state["mask"], [capi.bc_spec(capi.LBM_BC_VELOCITY, "z-", -1, 1.0, 1, cx, cy, r),
                                       capi.bc_spec(capi.LBM_BC_PRESSURE, "z+", -1, 1.0)])
        s.set_normals(state["tri"])
        w = s.wss()
        k = s.counts()
        out = {"classes": s.classes(), "pt": w["pt"], "normal": w["normal"],
               "counts": np.array([k["active"], k["fluid"], k["wall"], k["next_to_wall"], k["segments"]], np.int64)}
        s.close()
        return out
    if kind == "conv_fwd":
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        capi._check(state["L"].lbm_nn_conv3d_fwd(_ptr(state["x"]), state["dims"], c["ci"], _ptr(state["w"]),
                                                 _ptr(state["b"]), c["co"], c["ksize"], c["stride"], c["relu"],
                                                 _ptr(state["y"]), None, st))
        return {"y": state["y"]}
    if kind == "conv_bwd":
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        state["dw"].zero_()
        state["db"].zero_()
        capi._check(state["L"].lbm_nn_conv3d_bwd(_ptr(state["x"]), state["dims"], c["ci"], _ptr(state["w"]),
                                                 _ptr(state["wt"]), c["co"], c["ksize"], c["stride"], _ptr(state["dy"]),
                                                 _ptr(state["dx"]), _ptr(state["dw"]), _ptr(state["db"]), st))
        return {"dx": state["dx"], "dw": state["dw"], "db": state["db"]}
    from pv_dec_original_gb300 import warmstart
    if kind == "prior":
        x, prior = warmstart.features(state["mask"], state["mean"], state["period"], tau=0.55)
        rho, u = warmstart.prediction_to_device(warmstart.zero_output(prior), prior)
        return {"x": x, "rho": rho, "u": u}
    net = state["net"]
    if kind == "forward":
        # the network computes in BF16: its BF16 result (the FP32 copy holds the same values)
        net.forward(state["x"])
        return {"y": net.act["out"]}
    net.zero_grad()
    net.loss.zero_()
    y = net.forward(state["x"])
    net.backward(net.loss_and_grad(y, state["t"], state["m"], state["inv"]))
    return {"loss": net.loss, "gw": net.gw, "gb": net.gb}


# --------------------------------------------------------------------------- work


def _conv_work(D, H, W, ci, co, ks, stride):
    no = 1
    for v in (D, H, W):
        no *= (v - 1) // stride + 1
    return no, 2.0 * no * co * ks ** 3 * ci


def work(case):
    c = case
    kind = c["kind"]
    if kind == "step":
        nodes = int(vessel_mask(c).sum())
        es = {"f64": 8, "f32": 4, "f16": 2, "bf16": 2}[c["precision"]]
        # every step reads and writes each population once; rho and u are written out at the end
        return {"bytes": c["steps"] * nodes * 2.0 * c["Q"] * es + 32.0 * nodes,
                "flops": c["steps"] * nodes * 13.0 * c["Q"]}
    if kind == "voxelize":
        n = (2.0 * 1.12 * c["radius"] + 4.0) ** 2 * c["length"]
        nt = 2.0 * (2.0 * math.pi * c["radius"] / c["h"]) * (c["length"] / c["h"])
        return {"bytes": 96.0 * nt + n, "flops": 100.0 * nt}
    if kind == "lattice":
        mask = vessel_mask(c)
        nodes = float(mask.sum())
        near = 2.0 * math.pi * c["radius"] * c["length"]
        nt = 2.0 * (2.0 * math.pi * c["radius"] / c["h"]) * (c["length"] / c["h"])
        es = {"f64": 8, "f32": 4, "f16": 2}[c["precision"]]
        # class bytes, node words, the start state of both buffers; the normals sum every (node, triangle) pair
        return {"bytes": 2.0 * mask.size + nodes * (12.0 + 2.0 * c["Q"] * es) + 96.0 * nt, "flops": near * nt * 15.0}
    if kind == "conv_fwd":
        no, fl = _conv_work(c["D"], c["H"], c["W"], c["ci"], c["co"], c["ksize"], c["stride"])
        return {"bytes": 2.0 * (c["D"] * c["H"] * c["W"] * c["ci"] + no * c["co"]), "flops": fl}
    if kind == "conv_bwd":
        no, fl = _conv_work(c["D"], c["H"], c["W"], c["ci"], c["co"], c["ksize"], c["stride"])
        return {"bytes": 2.0 * (2.0 * c["D"] * c["H"] * c["W"] * c["ci"] + no * c["co"]), "flops": 2.0 * fl}
    n = c["D"] * c["H"] * c["W"]
    if kind == "prior":
        # mask in; distance, prior and input channels, the start fields out
        return {"bytes": n * (1.0 + 32.0 + 16.0), "flops": 100.0 * n}
    fl = by = 0.0
    for _, src, ci, co, ks, stride, _, _ in NET:
        lvl = {"x": 0, "c0a": 0, "c0b": 0, "d1": 1, "c1": 1, "d2": 2, "c2": 2, "d3": 3, "up:c3": 2, "u2": 2,
               "up:c2u": 1, "u1": 1, "up:c1u": 0, "u0": 0, "c0u": 0}[src]
        no, f = _conv_work(c["D"] >> lvl, c["H"] >> lvl, c["W"] >> lvl, ci, co, ks, stride)
        fl += f
        by += 2.0 * no * co  # each layer's activation is kept for the backward pass
    if kind == "forward":
        return {"bytes": n * (32.0 + 32.0 + 64.0), "flops": fl}
    return {"bytes": n * (32.0 + 16.0 + 1.0) + 3.0 * by, "flops": 3.0 * fl}


# --------------------------------------------------------------------------- exact: the same results in 64 bits

C19 = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1),
       (-1, 1, 0), (-1, -1, 0), (-1, 0, 1), (-1, 0, -1), (0, 1, 1), (0, 1, -1), (0, -1, 1), (0, -1, -1), (0, 0, 0)]
C27 = [(x, y, z) for x in (0, 1, -1) for y in (0, 1, -1) for z in (0, 1, -1)]


class _Exact:
    """The lattice-Boltzmann step in FP64 torch operations over the fluid nodes."""

    def __init__(self, c, mask, origin=(0.0, 0.0, 0.0)):
        dev = _device()
        self.c, self.dev = c, dev
        self.cs = C19 if c["Q"] == 19 else C27
        self.Q = len(self.cs)
        wt = ({0: 12 / 36, 1: 2 / 36, 2: 1 / 36} if self.Q == 19 else {0: 8 / 27, 1: 2 / 27, 2: 1 / 54, 3: 1 / 216})
        self.w = [wt[sum(abs(v) for v in e)] for e in self.cs]
        self.opp = [self.cs.index(tuple(-v for v in e)) for e in self.cs]
        m = torch.from_numpy(np.pad(mask, 1)).to(dev)
        idx = torch.full(m.shape, -1, dtype=torch.int64, device=dev)
        p = m.nonzero()
        self.n = len(p)
        idx[p[:, 0], p[:, 1], p[:, 2]] = torch.arange(self.n, device=dev)
        self.xyz = torch.stack([p[:, 2], p[:, 1], p[:, 0]], 1).double() - 1.0
        # index of the node at x + c_q, -1 where solid or outside
        self.nb = [idx[p[:, 0] + e[2], p[:, 1] + e[1], p[:, 2] + e[0]] for e in self.cs]
        bnd = torch.zeros(self.n, dtype=torch.bool, device=dev)
        for b in self.nb:
            bnd |= b < 0
        z = self.xyz[:, 2]
        self.inl = (bnd & (z == z.min())).nonzero().flatten()
        outl = bnd & (z == z.max()) & (z != z.min())
        self.out = outl.nonzero().flatten()
        wall = bnd.clone()
        wall[self.inl] = False
        wall &= ~outl
        self.wall = wall.nonzero().flatten()
        near = torch.zeros_like(bnd)
        for b in self.nb:
            near |= (b >= 0) & wall[b.clamp(min=0)]
        self.nw = (near & ~bnd).nonzero().flatten()
        self.pts = self.xyz + torch.tensor(origin, dtype=torch.float64, device=dev)

    def normals(self, tri):
        t = torch.from_numpy(tri).to(self.dev)
        v = t[:, :9].reshape(-1, 3, 3)
        cr = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
        nrm = cr.norm(dim=1)
        unit = cr / nrm.clamp(min=1e-300)[:, None]
        area, cen = 0.5 * nrm, v.sum(1) / 3.0
        out = []
        x = self.pts[self.nw]
        for k in range(0, len(x), 1024):
            d2 = ((x[k:k + 1024, None, :] - cen[None]) ** 2).sum(2)
            s = (area[None] / d2) @ unit
            out.append(s / s.norm(dim=1, keepdim=True))
        return torch.cat(out) if out else x

    def feq(self, rho, u, at=None):
        usq = (u * u).sum(1)
        out = []
        for e, w in zip(self.cs, self.w):
            cu = u[:, 0] * e[0] + u[:, 1] * e[1] + u[:, 2] * e[2]
            out.append(w * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * usq))
        return out

    def moments(self, f):
        rho = sum(f)
        u = torch.stack([sum(f[q] * e[a] for q, e in enumerate(self.cs) if e[a]) for a in range(3)], 1)
        return rho, u / rho[:, None]

    def collide(self, f, rho, u):
        om = 1.0 / self.c["tau"]
        fe = self.feq(rho, u)
        if self.c["collision"] != "regularized":
            return [a + om * (b - a) for a, b in zip(f, fe)]
        P = {}
        for a in range(3):
            for b in range(a, 3):
                P[a, b] = sum((f[q] - fe[q]) * (e[a] * e[b]) for q, e in enumerate(self.cs) if e[a] * e[b])
        tr = (P[0, 0] + P[1, 1] + P[2, 2]) / 3.0
        out = []
        for q, e in enumerate(self.cs):
            cpc = sum(P[a, b] * (e[a] * e[b] * (1 if a == b else 2)) for a, b in P if e[a] * e[b])
            out.append(fe[q] + (1.0 - om) * self.w[q] * 4.5 * (cpc - tr))
        return out

    def zou_he(self, f, at, sg, pressure, value):
        """Zou-He on a z face: sg = +1 at the low end, -1 at the high end."""
        if not len(at):
            return
        g = [v[at] for v in f]
        S0 = sum(g[q] for q, e in enumerate(self.cs) if e[2] == 0)
        Sm = sum(g[q] for q, e in enumerate(self.cs) if e[2] == -sg)
        S = S0 + 2.0 * Sm
        if pressure:
            rho = torch.full_like(S, value)
            uz = sg * (1.0 - S / rho)
        else:
            uz = sg * value
            rho = S / (1.0 - sg * uz)
        M = 2.0 if self.Q == 19 else 6.0
        N = [sum(g[q] * e[t] for q, e in enumerate(self.cs) if e[2] == 0 and e[t]) / M for t in (0, 1)]
        for q, e in enumerate(self.cs):
            if e[2] == sg:
                corr = sum(N[t] * e[t] for t in (0, 1) if e[t])
                f[q][at] = g[self.opp[q]] + 6.0 * self.w[q] * rho * (e[2] * uz) - corr

    def run(self, rho, u, tri, amp):
        c, Q, dev = self.c, self.Q, self.dev
        parity = c["mode"] == "parity"
        f = self.feq(torch.from_numpy(rho).to(dev).double(), torch.from_numpy(u).to(dev).double())
        r, v = self.moments(f)
        post = self.collide(f, r, v)
        nrm = self.normals(tri)
        nw = self.nw
        cx, cy, R = inlet(c)
        xi = self.xyz[self.inl]
        prof = (1.0 - ((xi[:, 0] - cx) ** 2 + (xi[:, 1] - cy) ** 2) / (R * R)).clamp(min=0.0)
        miss = [b < 0 for b in self.nb]
        acc = torch.zeros((len(nw), 3), dtype=torch.float64, device=dev)
        accm = torch.zeros(len(nw), dtype=torch.float64, device=dev)
        for k in range(c["steps"]):
            g = []
            for q in range(Q):
                o = self.opp[q]
                pulled = post[q][self.nb[o].clamp(min=0)]
                g.append(torch.where(miss[o], f[q] if parity else post[o], pulled))
            self.zou_he(g, self.inl, 1, False, float(amp[k % len(amp)]) * prof)
            self.zou_he(g, self.out, -1, True, 1.0)
            if parity:
                for q in range(Q):
                    at = self.wall[miss[q][self.wall]]
                    g[self.opp[q]][at] = g[q][at]
            fe = self.feq(r[nw], v[nw])  # parity: the equilibrium of the previous collision
            f = g
            r, v = self.moments(f)
            if not parity:
                fe = self.feq(r[nw], v[nw])
            scale = 1.0 if parity else -(1.0 - 0.5 / c["tau"])
            tau = torch.zeros_like(acc)
            for q, e in enumerate(self.cs):
                cn = nrm[:, 0] * e[0] + nrm[:, 1] * e[1] + nrm[:, 2] * e[2]
                ev = torch.tensor(e, dtype=torch.float64, device=dev)
                tau += ((f[q][nw] - fe[q]) * cn)[:, None] * (ev[None] - cn[:, None] * nrm)
            tau *= scale
            wss = tau.norm(dim=1)
            acc += tau
            accm += wss
            post = self.collide(f, r, v)
        return {"rho": r, "u": v.reshape(-1), "wss": wss, "osi": 0.5 * (1.0 - acc.norm(dim=1) / accm), "tawss": accm}


def _conv64(x, w, stride, ks):
    """conv3d of [C][D][H][W] float64 as one matrix product per tap."""
    ci, D, H, W = x.shape
    co = w.shape[0]
    Do, Ho, Wo = ((v - 1) // stride + 1 for v in (D, H, W))
    p = ks // 2
    xp = torch.nn.functional.pad(x, (p, p, p, p, p, p))
    y = torch.zeros((co, Do * Ho * Wo), dtype=x.dtype, device=x.device)
    wt = w.reshape(co, ks ** 3, ci)
    for t in range(ks ** 3):
        a, b, d = t // (ks * ks), (t // ks) % ks, t % ks
        s = xp[:, a:a + stride * (Do - 1) + 1:stride, b:b + stride * (Ho - 1) + 1:stride,
               d:d + stride * (Wo - 1) + 1:stride]
        y = y + wt[:, t] @ s.reshape(ci, -1)
    return y.reshape(co, Do, Ho, Wo)


def _net64(x, w, b):
    """The network's layers over NET; w, b: lists of tensors per layer."""
    act = {"x": x}
    for (name, src, _, _, ks, stride, relu, skip), wl, bl in zip(NET, w, b):
        if src.startswith("up:"):
            a = act[src[3:]]
            for d in (1, 2, 3):
                a = a.repeat_interleave(2, dim=d)
        else:
            a = act[src]
        y = _conv64(a, wl, stride, ks) + bl[:, None, None, None]
        y = y.relu() if relu else y
        act[name] = y + act[skip] if skip else y
    return act["out"]


def _net_weights(dims, seed):
    """The network's start weights (the documented He initialisation), rounded to BF16, and zero biases."""
    rng = np.random.default_rng(seed)
    w, b = [], []
    for name, src, ci, co, ks, _, _, _ in NET:
        cr, orr = (7 if src == "x" else ci), (4 if name == "out" else co)
        std = math.sqrt(2.0 / (ks ** 3 * cr)) * (0.3 if name == "out" else 1.0)
        blk = np.zeros((co, ks ** 3, ci), np.float32)
        blk[:orr, :, :cr] = rng.normal(0.0, std, (orr, ks ** 3, cr))
        w.append(torch.from_numpy(blk).to(_device()).to(torch.bfloat16).double())
        b.append(torch.zeros(co, dtype=torch.float64, device=_device()))
    return w, b


def _edt(cells, seeds):
    """Euclidean distance of every cell [n, k] to the nearest seed [m, k]."""
    out = []
    s2 = (seeds * seeds).sum(1)
    for k in range(0, len(cells), 8192):
        a = cells[k:k + 8192]
        out.append(((a * a).sum(1)[:, None] + s2[None] - 2.0 * a @ seeds.T).min(1).values.clamp(min=0.0).sqrt())
    return torch.cat(out)


def _prior64(c, seed):
    mask, _, _, mean, period = net_vessel(c, seed)
    dev = _device()
    D, H, W = mask.shape
    m = torch.from_numpy(mask).to(dev).bool()
    pad = torch.nn.functional.pad(m, (1, 1, 1, 1, 1, 1))
    near = [pad[1 + a:1 + a + D, 1 + b:1 + b + H, 1 + e:1 + e + W] for a, b, e in
            ((0, 0, 1), (0, 0, -1), (0, 1, 0), (0, -1, 0), (1, 0, 0), (-1, 0, 0))]
    flat = m & ~(near[0] & near[1] & near[2] & near[3])
    full = m & ~(near[0] & near[1] & near[2] & near[3] & near[4] & near[5])
    seeds = full.nonzero().double()
    if len(seeds) * m.numel() > 6e10 or not len(seeds):
        return None
    grid = torch.ones_like(m).nonzero().double()
    sdf = (_edt(grid, seeds) + 0.5).reshape(D, H, W)
    sdf = torch.where(m, sdf, -sdf)
    dist = torch.zeros((D, H, W), dtype=torch.float64, device=dev)
    cell = torch.ones((H, W), device=dev).nonzero().double()
    for k in range(D):
        s = flat[k].nonzero().double()
        if len(s):
            dist[k] = torch.where(m[k], (_edt(cell, s) + 0.5).reshape(H, W), dist[k])
    R = dist.reshape(D, -1).max(1).values
    fluid = (R > 0).nonzero().flatten()
    Q = math.pi * float(R[fluid[0]]) ** 2 * mean / 2.0
    Rs = R.clamp(min=1.0)
    peak = 2.0 * Q / (math.pi * Rs ** 2)
    fall = torch.where(R > 0, 24.0 * ((0.55 - 0.5) / 3.0) * Q / (math.pi * Rs ** 4), torch.zeros_like(R))
    tail = fall.flip(0).cumsum(0).flip(0) - fall
    e = Rs[:, None, None] - dist
    uz = torch.where(m, peak[:, None, None] * (1.0 - e * e / Rs[:, None, None] ** 2).clamp(0.0, 1.0), 0.0)
    drho = torch.where(m, tail[:, None, None].expand(D, H, W), 0.0)
    x = torch.zeros((D, H, W, 16), dtype=torch.float64, device=dev)
    x[..., 0] = (sdf * 0.2).clamp(-3.0, 3.0)
    x[..., 1] = m
    x[..., 2] = mean * 30.0
    x[..., 3] = period / 4000.0
    x[..., 4] = (torch.arange(D, device=dev).double() / D)[:, None, None]
    x[..., 5] = uz / mean
    x[..., 6] = drho / mean * 0.5
    md = m.double()

    def smooth(f):
        for axis in (0, 1, 2):
            p = [0, 0, 0, 0, 0, 0]
            p[4 - 2 * axis] = p[5 - 2 * axis] = 1
            pf, pm = torch.nn.functional.pad(f * md, p), torch.nn.functional.pad(md, p)
            n = f.shape[axis]
            num = 2.0 * f * md + pf.narrow(axis, 0, n) + pf.narrow(axis, 2, n)
            den = 2.0 + pm.narrow(axis, 0, n) + pm.narrow(axis, 2, n)
            f = num / den * md
        return f

    rho = 1.0 + smooth(drho)[m]
    u = torch.zeros((int(m.sum()), 3), dtype=torch.float64, device=dev)
    u[:, 2] = smooth(uz)[m]
    return {"x": x.reshape(-1), "rho": rho, "u": u.reshape(-1)}


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "step":
        mask, tri, rho, u, amp = step_inputs(c, seed)
        out = _Exact(c, mask).run(rho, u, tri, amp)
        if c["precision"] in ("f16", "bf16"):
            out["osi"] = None  # 1/2 (1 - |sum tau| / sum |tau|) cancels to the storage's rounding here
        return out
    if kind == "voxelize":
        return None
    if kind == "lattice":
        tri, origin = _moved(vessel_surface(c, c["h"]), seed)
        e = _Exact(dict(c, tau=0.8, collision="bgk"), vessel_mask(c), origin)
        return {"classes": None, "pt": None, "normal": e.normals(tri), "counts": None}
    if kind in ("conv_fwd", "conv_bwd"):
        x, w, b, dy, _ = conv_inputs(c, seed)
        x = x.double().reshape(c["D"], c["H"], c["W"], c["ci"]).permute(3, 0, 1, 2).contiguous()
        w = w.double().reshape(c["co"], -1, c["ci"])
        if kind == "conv_fwd":
            y = _conv64(x, w, c["stride"], c["ksize"]) + b.double()[:, None, None, None]
            return {"y": (y.relu() if c["relu"] else y).permute(1, 2, 3, 0).reshape(-1)}
        x.requires_grad_(True)
        w = w.clone().requires_grad_(True)
        y = _conv64(x, w, c["stride"], c["ksize"])
        g = dy.double().reshape(*y.shape[1:], c["co"]).permute(3, 0, 1, 2)
        dx, dw = torch.autograd.grad(y, (x, w), g)
        return {"dx": dx.permute(1, 2, 3, 0).reshape(-1), "dw": dw.reshape(-1), "db": g.sum((1, 2, 3))}
    if kind == "prior":
        return _prior64(c, seed)
    if kind == "gradient" and c["D"] * c["H"] * c["W"] > 1 << 21:
        return None  # the FP64 backward pass at the full grid takes too long
    x, t, m, nfl = net_inputs(c, seed)
    D, H, W = c["D"], c["H"], c["W"]
    x = x.double().reshape(D, H, W, 16).permute(3, 0, 1, 2).contiguous()
    w, b = _net_weights((D, H, W), seed)
    if kind == "forward":
        return {"y": _net64(x, w, b).permute(1, 2, 3, 0).reshape(-1)}
    for v in w + b:
        v.requires_grad_(True)
    y = _net64(x, w, b)[:4].permute(1, 2, 3, 0)
    d = (y - t.double().reshape(D, H, W, 4)) * m.reshape(D, H, W, 1)
    loss = (d * d).sum() / (4.0 * nfl)
    g = torch.autograd.grad(loss, w + b)
    return {"loss": loss.detach().reshape(1), "gw": torch.cat([v.reshape(-1) for v in g[:len(w)]]),
            "gb": torch.cat([v.reshape(-1) for v in g[len(w):]])}
