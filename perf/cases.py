"""The work that users of this package have it do, as cases that can be timed.

Each case goes through the public entry points: the Schafer-Turek rig and the towing tank step by
step with their recorded histories, the periodic box of seeded disks, a batch of seeded tunnels, a
monitored run that renders frames, and the warm-start network (one convolution layer, inference, one
training step). `exact` restates every case in plain torch / numpy in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import vortexlab_b200 as V
from vortexlab_b200 import cylinder
from vortexlab_b200 import warmstart as WS
from vortexlab_b200._lib import check, lib
from vortexlab_b200.batch import Batch, seeded_tunnels
from vortexlab_b200.tunnel import Tunnel
from vortexlab_b200.workloads import build_disk_box, disk_field

BYTES = {"f64": 8, "f32": 4, "f16s": 2, "f16c": 2, "f16x": 2}
FLOPS_PER_UPDATE = 200          # one collision of D2Q9


# ====================================================================== the cases
def listed():
    return [
        # the validation rig at its published coarse resolution (442 x 84): tens of thousands of
        # very short steps, forces and pressure drop recorded at each
        {"name": "rig20_f64", "kind": "rig", "n": 20, "prec": "f64", "steps": 1000},
        # the same rig at the resolution the published benchmark is quoted on (1762 x 330)
        {"name": "rig80_f64", "kind": "rig", "n": 80, "prec": "f64", "steps": 600},
        # one towing tank of the tunnel population, odd sizes, run alone in FP64 (the plain form
        # that converged statistics are judged against)
        {"name": "tunnel37_f64", "kind": "tunnel", "body": "star", "d": 37, "up": 5.0, "down": 15.0, "height": 10.0,
         "prec": "f64", "steps": 600},
        # the square of the precision sweep (1802 x 902) in FP32
        {"name": "square60_f32", "kind": "tunnel", "body": "square", "d": 60, "up": 10.0, "down": 20.0,
         "height": 15.0, "prec": "f32", "steps": 300},
        # a monitored run: some steps, then a vorticity frame and the conservation checks, repeated
        {"name": "frames24_f32", "kind": "frames", "body": "ellipse", "d": 24, "up": 5.0, "down": 15.0,
         "height": 10.0, "prec": "f32", "steps": 50, "frames": 4},
        # the throughput box (seeded disks, BGK) in FP64, larger than the L2
        {"name": "box4096_f64", "kind": "box", "nx": 4096, "ny": 2048, "prec": "f64", "steps": 200},
        # the box in FP32 at a row length that no power of two divides far, with an odd row count
        {"name": "box4000_f32", "kind": "box", "nx": 4000, "ny": 2001, "prec": "f32", "steps": 400},
        # the box in 16-bit storage, rows that are even but not a multiple of four
        {"name": "box3002_f16x", "kind": "box", "nx": 3002, "ny": 1501, "prec": "f16x", "steps": 400},
        # tunnels of uneven size, shape and Reynolds number in one batch, a chunk of steps at a time
        # with every tunnel's force history read after it (the on-line stopping loop's chunk)
        {"name": "batch24_f32", "kind": "batch", "count": 24, "dmin": 15, "dmax": 40, "prec": "f32", "steps": 400},
        # one 3x3 convolution of the warm-start network, forward, backward and its Adam update
        {"name": "conv64", "kind": "conv", "cin": 64, "cout": 64, "h": 64, "w": 128, "batch": 16, "stride": 1},
        # the network's prediction for a batch of 16 tunnels (the start of a warm batch)
        {"name": "unet_predict", "kind": "predict", "batch": 16},
        # the gradients of one training step at the training batch size
        {"name": "unet_train", "kind": "train", "batch": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rig", "tunnel", "tunnel", "frames", "box", "box", "batch", "conv", "conv", "predict", "train"])
    prec = rng.choice(["f64", "f64", "f32", "f32", "f16x", "f16c", "f16s"])
    if kind == "rig":
        return {"kind": kind, "n": 10 * rng.randint(1, 8), "prec": rng.choice(["f64", "f64", "f32"]),
                "steps": rng.randint(100, 600)}
    if kind in ("tunnel", "frames"):
        up = rng.randint(4, 8)
        c = {"kind": kind, "body": rng.choice(["ellipse", "square", "star"]), "d": _log_int(rng, 15, 60), "up": float(up),
             "down": float(rng.randint(8, 16)), "height": float(rng.randint(8, 12)), "prec": prec,
             "steps": rng.randint(100, 400)}
        if kind == "frames":
            c["d"] = _log_int(rng, 15, 36)
            c["steps"] = rng.randint(10, 60)
            c["frames"] = rng.randint(1, 4)
        return c
    if kind == "box":
        nx = _log_int(rng, 256, 4096)
        return {"kind": kind, "nx": nx, "ny": max(200, _log_int(rng, nx // 4, nx // 2)), "prec": prec,
                "steps": rng.randint(50, 200)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 24), "dmin": 15, "dmax": rng.randint(20, 40),
                "prec": rng.choice(["f32", "f32", "f64", "f16x"]), "steps": rng.randint(50, 400)}
    if kind == "conv":
        stride = rng.choice([1, 1, 2])
        if rng.random() < 0.5:      # a layer of the network on its own grid or a batch of another size
            lev = rng.randint(0, 3)
            h, w = 128 >> lev, 256 >> lev
        else:
            h, w = 2 * rng.randint(4, 48), 2 * rng.randint(8, 72)
        return {"kind": kind, "cin": rng.choice([32, 64, 96, 128, 192, 256]), "cout": rng.choice([32, 64, 128]),
                "h": h, "w": w, "batch": rng.randint(1, 8), "stride": stride}
    return {"kind": kind, "batch": rng.randint(1, 24)}


# ====================================================================== inputs from the seed
def _flow_inputs(case, seed):
    """Flow parameters and the body of a rig or a tank, as plain numbers."""
    g = np.random.default_rng([int(seed), 17])
    kind = case["kind"]
    if kind == "rig":
        return {"u": float(g.uniform(0.045, 0.055)), "re": float(g.uniform(80.0, 120.0))}
    p = {"u": float(g.uniform(0.045, 0.055)), "re": float(g.uniform(60.0, 150.0)), "angle": float(g.uniform(0.05, 0.5))}
    d = case["d"]
    if case["body"] == "ellipse":
        p["a"], p["b"] = 0.5 * d * float(g.uniform(1.0, 3.0)), 0.5 * d
    elif case["body"] == "star":
        p["radii"] = [0.5 * d * float(v) for v in g.uniform(0.6, 1.0, int(g.integers(6, 13)))]
        p["phase"] = float(g.uniform(0.0, 2.0 * math.pi))
    return p


def _tank(case, p):
    return Tunnel(d=case["d"], re=p["re"], u=p["u"], upstream=case["up"], downstream=case["down"], height=case["height"],
                  precision=case["prec"])


def _body(case, p, cx, cy):
    if case["body"] == "ellipse":
        s = V.Ellipse(cx, cy, p["a"], p["b"])
    elif case["body"] == "square":
        return V.section(V.Corner.Sharp, cx, cy, float(case["d"]), p["angle"])
    else:
        s = V.Star(cx, cy, p["radii"], p["phase"])
    return V.Rotated(s, cx, cy, p["angle"])


def _box_inputs(case, seed):
    g = np.random.default_rng([int(seed), 23])
    return disk_field(case["nx"], case["ny"], seed=0x5EED0001 + 7919 * (int(seed) + 1)), float(g.uniform(0.04, 0.06))


def _batch_sizes(case):
    return [int(round(d)) for d in np.linspace(case["dmin"], case["dmax"], case["count"])]


def _batch_cases(case, seed):
    """Seeded bodies and Reynolds numbers over the sizes, with steps for any number of chunks."""
    return [seeded_tunnels(seed=0x5EED0004 + 7919 * (int(seed) + 1) + 104729 * k, count=1, dmin=d, dmax=d,
                           re=(50.0, 150.0), units=1000.0, precision=case["prec"])[0]
            for k, d in enumerate(_batch_sizes(case))]


def _net_inputs(b, seed):
    """Encoded tunnels (body mask, Reynolds feature, coordinates) and wake-like targets, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 2 + 1)
    r = torch.rand(b, 4, generator=g, device="cuda")
    x = torch.linspace(-1, 1, WS.W, device="cuda")[None, None, :]
    y = torch.linspace(-1, 1, WS.H, device="cuda")[None, :, None]
    w, h = (0.05 + 0.07 * r[:, 0])[:, None, None], (0.05 + 0.1 * r[:, 1])[:, None, None]
    mask = (((x + 0.5) / w) ** 2 + (y / h) ** 2 < 1.0).float()
    re = (2.0 * r[:, 2] - 1.0)[:, None, None]
    inp = torch.stack([mask, re.expand_as(mask), x.expand_as(mask), y.expand_as(mask)], -1)
    down = torch.sigmoid(12.0 * (x + 0.5))
    ph = 6.28318 * r[:, 3][:, None, None]
    wake = torch.exp(-((y / (2.0 * h)) ** 2)) * down
    tgt = torch.stack([-0.6 * wake, 0.3 * wake * torch.sin(9.0 * x + ph), -0.2 * wake * torch.cos(9.0 * x + ph)], -1)
    return inp.contiguous(), tgt.contiguous(), (1.0 - mask).contiguous()


# ====================================================================== prepare
def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()     # the array keeps the memory


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "rig":
        p = _flow_inputs(case, seed)
        r = cylinder.rig(cylinder.Setup(n=case["n"], u_mean=p["u"], precision=case["prec"]), p["re"], 1.0)
        s.update(rig=r, out=_pinned(9 * r.ch.sim.n))
    elif kind in ("tunnel", "frames"):
        p = _flow_inputs(case, seed)
        tn = _tank(case, p)
        ch = V.Channel(tn.spec_warm(_body(case, p, *tn.centre())), precision=case["prec"])
        ch.sim.autotune()
        s.update(ch=ch, u=p["u"])
        if kind == "tunnel":
            s["out"] = _pinned(9 * ch.sim.n)
    elif kind == "box":
        disks, u = _box_inputs(case, seed)
        sim = build_disk_box(V, case["nx"], case["ny"], disks, precision=case["prec"])
        sim.autotune()
        s.update(sim=sim, u=u, out=_pinned(9 * sim.n))
    elif kind == "batch":
        cs = _batch_cases(case, seed)
        b = Batch(case["prec"])
        for c in cs:
            b.add(c.tunnel.spec_warm(c.body), c.steps)
        b.build()
        b.autotune()
        s["batch"] = b
    elif kind == "conv":
        g = torch.Generator(device="cuda").manual_seed(int(seed) * 2 + 1)
        c = WS.Conv(case["cin"], case["cout"], stride=case["stride"], seed=int(seed) % (1 << 20))
        c.alloc(case["batch"], case["h"], case["w"])
        x = torch.relu(torch.randn(case["batch"], case["h"], case["w"], case["cin"], generator=g, device="cuda"))
        s.update(conv=c, x=x.to(torch.bfloat16), err=WS._Err(), step=0,
                 dy=torch.randn(c.rows, c.cout, generator=g, device="cuda"),
                 dx=torch.zeros(case["batch"] * case["h"] * case["w"], case["cin"], device="cuda"))
    else:
        b = case["batch"]
        inp, tgt, wt = _net_inputs(b, seed)
        net = WS.load_pretrained() if kind == "predict" else WS.UNet(seed=1 + int(seed) % 1000)
        net.alloc(b)
        s.update(net=net, x=inp.to(torch.bfloat16))
        if kind == "train":
            s.update(tgt=tgt, w=wt, inv=1.0 / (float(wt.sum().item()) * WS.NT),
                     dout=torch.zeros(b * WS.H * WS.W, net.cout, device="cuda"),
                     partial=torch.zeros(296, dtype=torch.float64, device="cuda"))
    return s


# ====================================================================== run
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "rig":
        sim = s["rig"].ch.sim
        sim.init((1.0, 0.0, 0.0))
        cd, cl, dp = cylinder.run_record(s["rig"], case["steps"])
        return {"cd": cd, "cl": cl, "dp": dp, "f": sim.populations(s["out"])}
    if kind in ("tunnel", "box"):
        sim = s["ch"].sim if kind == "tunnel" else s["sim"]
        sim.init((1.0, s["u"], 0.0))
        sim.record(case["steps"])
        (s["ch"] if kind == "tunnel" else sim).step(case["steps"])
        return {"history": sim.history(), "f": sim.populations(s["out"])}
    if kind == "frames":
        ch = s["ch"]
        ch.sim.init((1.0, s["u"], 0.0))
        out = []
        for _ in range(case["frames"]):
            ch.step(case["steps"])
            out.append((ch.sim.vorticity(), ch.sim.total_mass(), ch.sim.max_speed(), ch.sim.force))
        return out
    if kind == "batch":
        b = s["batch"]
        first = b.global_step()
        b.run(case["steps"])
        return {"history": b.history_copy([(k, first, case["steps"]) for k in range(b.count)]),
                "fields": b.macros_field(0)}
    if kind == "conv":
        c = s["conv"]
        s["step"] += 1
        y = c.forward(s["x"], s["err"])
        c.backward(s["dy"], s["dx"], False, s["err"])
        c.adam(s["step"], 1e-4)
        return {"y": y, "dx": s["dx"], "gw": c.gw, "gb": c.gb, "w": c.w, "b": c.b}
    net = s["net"]
    out = net.forward(s["x"])
    if kind == "predict":
        return out
    rows = out.shape[0]
    check(lib.vl_nn_mse(WS._p(out), WS._p(s["tgt"]), WS._p(s["w"]), rows, net.cout, WS.NT, s["inv"], WS._p(s["dout"]),
                        WS._p(s["partial"]), 296, None))
    net.backward(s["dout"])
    return {"out": out, "grads": [(c.gw, c.gb) for c in net.layers()]}


# ====================================================================== work
def _grid(case):
    if case["kind"] == "rig":
        return 22 * case["n"] + 2, 41 * case["n"] // 10 + 2
    if case["kind"] == "box":
        return case["nx"], case["ny"]
    d = case["d"]
    return int((case["up"] + case["down"]) * d) + 2, int(case["height"] * d) + 2


def _conv_work(rows_in, rows_out, cin, cout, k, need_dx, train):
    """(bytes, flops) of a convolution layer: BF16 activations and weights; gradients FP32."""
    mac = rows_out * cout * cin * k * k
    bytes_ = 2.0 * (rows_in * cin + rows_out * cout + k * k * cin * cout)
    flops = 2.0 * mac
    if train:       # dy, y, x and the weights again; dx and the weight gradient
        bytes_ += rows_out * cout * (4 + 2) + 2.0 * rows_in * cin + 4.0 * k * k * cin * cout
        flops += 2.0 * mac
        if need_dx:
            bytes_ += 4.0 * rows_in * cin + 2.0 * k * k * cin * cout
            flops += 2.0 * mac
    return bytes_, flops


def work(case):
    kind = case["kind"]
    if kind in ("rig", "tunnel", "frames", "box"):
        nx, ny = _grid(case)
        # each step reads and writes nine populations of every fluid cell
        upd = nx * ny * case["steps"] * (0.95 if kind == "box" else 1.0) * case.get("frames", 1)
        read = {"rig": 72, "tunnel": 72, "box": 72, "frames": 4 * case.get("frames", 1)}[kind]
        return {"bytes": upd * 18 * BYTES[case["prec"]] + nx * ny * read, "flops": upd * FLOPS_PER_UPDATE}
    if kind == "batch":
        upd = float(sum((20 * d + 2) * (10 * d + 2) for d in _batch_sizes(case))) * case["steps"]
        return {"bytes": upd * 18 * BYTES[case["prec"]], "flops": upd * FLOPS_PER_UPDATE}
    if kind == "conv":
        st = case["stride"]
        ri = case["batch"] * case["h"] * case["w"]
        ro = case["batch"] * ((case["h"] + st - 1) // st) * ((case["w"] + st - 1) // st)
        b, f = _conv_work(ri, ro, case["cin"], case["cout"], 3, True, True)
        return {"bytes": b + 9 * case["cin"] * case["cout"] * 30, "flops": f}
    ch, px = [32, 64, 128, 256], [case["batch"] * (WS.H >> l) * (WS.W >> l) for l in range(4)]
    layers = []
    for l in range(4):
        layers += [(px[l - 1] if l else px[0], px[l], ch[l - 1] if l else 4, ch[l], 3), (px[l], px[l], ch[l], ch[l], 3)]
    for l in (2, 1, 0):
        layers += [(px[l], px[l], ch[l + 1] + ch[l], ch[l], 3), (px[l], px[l], ch[l], ch[l], 3)]
    layers.append((px[0], px[0], 32, 8, 1))
    tot = [_conv_work(*a, i > 0, kind == "train") for i, a in enumerate(layers)]
    return {"bytes": sum(t[0] for t in tot), "flops": sum(t[1] for t in tot)}


# ====================================================================== 64-bit restatement: flows
CX = [0, 1, 0, -1, 0, 1, -1, -1, 1]
CY = [0, 0, 1, 0, -1, 1, 1, -1, -1]
OPP = [0, 3, 4, 1, 2, 7, 8, 5, 6]
WT = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
FLUID, INLET, OUTLET, SIDE_WALL, SIDE_OPEN, BODY = range(6)


def _in_polygon(pts):
    pts = np.asarray(pts, float)

    def inside(x, y):
        res = np.zeros(np.shape(x), bool)
        j = len(pts) - 1
        for i in range(len(pts)):
            (xi, yi), (xj, yj) = pts[i], pts[j]
            j = i
            if yi == yj:
                continue
            res ^= ((yi > y) != (yj > y)) & (x < (xj - xi) * (y - yi) / (yj - yi) + xi)
        return res
    return inside


def _rotated(f, cx, cy, angle):
    s, c = math.sin(angle), math.cos(angle)
    return lambda x, y: f(cx + c * (x - cx) + s * (y - cy), cy - s * (x - cx) + c * (y - cy))


def _ellipse(cx, cy, a, b):
    return lambda x, y: ((x - cx) / a) ** 2 + ((y - cy) / b) ** 2 < 1.0


def _star(cx, cy, radii, phase):
    t = phase + 2.0 * math.pi * np.arange(len(radii)) / len(radii)
    return _in_polygon(np.stack([cx + radii * np.cos(t), cy + radii * np.sin(t)], 1))


def _square(cx, cy, d):
    h = 0.5 * d
    return _in_polygon([(cx + h, cy + h), (cx - h, cy + h), (cx - h, cy - h), (cx + h, cy - h)])


def _disks(disks, nx, ny):
    """Inside test of a union of disks through the disks near each cell."""
    side = 32
    gx, gy = nx // side + 3, ny // side + 3
    near = [[] for _ in range(gx * gy)]
    for k, (cx, cy, r) in enumerate(disks):
        for j in range(int((cy - r) // side) + 1, int((cy + r) // side) + 2):
            for i in range(int((cx - r) // side) + 1, int((cx + r) // side) + 2):
                near[j * gx + i].append(k)
    table = np.full((gx * gy, max(len(v) for v in near)), -1)
    for k, v in enumerate(near):
        table[k, :len(v)] = v
    far = np.vstack([disks, [[-1e9, -1e9, 0.0]]])       # index -1: no disk

    def inside(x, y):
        b = (np.floor(y / side).astype(int) + 1) * gx + np.floor(x / side).astype(int) + 1
        res = np.zeros(x.shape, bool)
        for c in range(table.shape[1]):
            d = far[table[b, c]]
            res |= (x - d[..., 0]) ** 2 + (y - d[..., 1]) ** 2 < d[..., 2] ** 2
        return res
    return inside


def _cut(inside, x, y, cx, cy):
    lo, hi = np.zeros(x.shape), np.ones(x.shape)
    for _ in range(40):
        m = 0.5 * (lo + hi)
        hit = inside(x + m * cx, y + m * cy)
        hi = np.where(hit, m, hi)
        lo = np.where(hit, lo, m)
    return np.clip(0.5 * (lo + hi), 1e-9, 1.0)


class _Flow:
    """A domain and its time step in FP64: pull, boundary links, collide. `paint`: the kind of every
    cell (or None: only the body in a periodic box); `profile(y)`: the inlet velocity."""

    def __init__(self, nx, ny, inside, tau, bgk, paint=None, profile=None, u_ref=0.0, moving_sides=0.0):
        self.nx, self.ny, self.bgk, self.u_ref = nx, ny, bgk, u_ref
        self.op = 1.0 / tau
        self.om = self.op if bgk else 1.0 / (0.5 + (3.0 / 16.0) / (tau - 0.5))
        X, Y = np.meshgrid(np.arange(nx, dtype=float), np.arange(ny, dtype=float))
        kind = np.zeros((ny, nx), np.int64) if paint is None else paint.copy()
        if paint is None:
            for y0 in range(0, ny, 256):            # in strips: the disk test's temporaries
                kind[y0:y0 + 256][inside(X[y0:y0 + 256], Y[y0:y0 + 256])] = BODY
        else:
            kind[inside(X, Y)] = BODY
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=self.dev)  # noqa: E731
        fluid = kind == FLUID
        self.fluid = t(fluid)
        idx = np.arange(nx * ny).reshape(ny, nx)
        wall, opened = [], []
        isopen = (kind == OUTLET) | (kind == SIDE_OPEN)
        for j in range(1, 9):
            sh = lambda a, sx, sy: np.roll(a, (-sy, -sx), (0, 1))  # noqa: E731  value at (x + sx, y + sy)
            nk = sh(kind, CX[j], CY[j])
            m = fluid & (nk != FLUID)
            k, at = nk[m], idx[m]
            x, y = X[m], Y[m]
            behind = np.where(sh(fluid, -CX[j], -CY[j])[m], sh(idx, -CX[j], -CY[j])[m], -1)
            q = np.full(k.shape, 0.5)
            b = k == BODY
            q[b] = _cut(inside, x[b], y[b], float(CX[j]), float(CY[j]))
            ux = np.zeros(k.shape)
            if profile is not None:
                ux[k == INLET] = profile(y[k == INLET] + 0.5 * CY[j])
                ux[k == SIDE_WALL] = moving_sides
            beside = sh(isopen, CX[j], 0)[m]
            o = (k == OUTLET) | (k == SIDE_OPEN)
            wall.append([np.full((~o).sum(), j), at[~o], behind[~o], q[~o], ux[~o], b[~o], (k == INLET)[~o]])
            opened.append([np.full(o.sum(), j), at[o], np.where(beside[o], CX[j], 0), np.where(beside[o], 0, CY[j]),
                           (k == SIDE_OPEN)[o]])
        w = [np.concatenate(c) for c in zip(*wall)]
        self.wj, self.wat, self.wbehind = t(w[0]), t(w[1]), t(w[2])
        self.wq, self.wux, self.wbody = t(w[3]), t(w[4]), t(w[5])
        o = [np.concatenate(c) for c in zip(*opened)]
        self.oj, self.oat, self.onx, self.ony, self.orad = t(o[0]), t(o[1]), t(o[2].astype(float)), t(o[3].astype(float)), t(o[4])
        self.pn = t(np.unique(o[1][~o[4]])) if len(o[0]) else None       # outlet nodes (outward normal +x)
        f8 = dict(dtype=torch.float64, device=self.dev)
        self.cx, self.cy, self.w = torch.tensor(CX, **f8), torch.tensor(CY, **f8), torch.tensor(WT, **f8)
        self.opp = torch.tensor(OPP, device=self.dev)

    def start(self, ux):
        u = torch.where(self.fluid, torch.tensor(float(ux), dtype=torch.float64, device=self.dev), 0.0)
        self.f = self._eq(torch.ones_like(u), u, torch.zeros_like(u))

    def _eq(self, rho, ux, uy):
        usq = 1.5 * (ux * ux + uy * uy)
        out = torch.empty((9,) + tuple(rho.shape), dtype=torch.float64, device=self.dev)
        for i in range(9):
            cu = 3.0 * (CX[i] * ux + CY[i] * uy)
            out[i] = WT[i] * rho * (1.0 + cu + 0.5 * cu * cu - usq)
        return out

    def moments(self, f):
        rho = f.sum(0)
        return rho, (f[1] - f[3] + f[5] - f[6] - f[7] + f[8]) / rho, (f[2] - f[4] + f[5] + f[6] - f[7] - f[8]) / rho

    def step(self, scale):
        """One step with the inlet at `scale` of its profile. Returns (force, outlet offset)."""
        a = self.f
        flat = a.reshape(9, -1)
        new = torch.stack([torch.roll(a[i], (CY[i], CX[i]), (0, 1)) for i in range(9)])
        nf = new.view(9, -1)
        j, i = self.wj, self.opp[self.wj]
        out, own, q = flat[j, self.wat], flat[i, self.wat], self.wq
        corr = 6.0 * self.w[j] * self.cx[j] * self.wux * scale
        beh = flat[j, self.wbehind.clamp(min=0)]
        back = torch.where(q >= 0.5, 0.5 / q * (out - corr) + (1.0 - 0.5 / q) * own,
                           torch.where(self.wbehind >= 0, 2.0 * q * out + (1.0 - 2.0 * q) * beh - corr, out - corr))
        nf[i, self.wat] = back
        fx = torch.where(self.wbody, self.cx[j] * (out + back), 0.0).sum()
        fy = torch.where(self.wbody, self.cy[j] * (out + back), 0.0).sum()
        drho = torch.zeros((), dtype=torch.float64, device=self.dev)
        if self.pn is not None:
            cs = math.sqrt(1.0 / 3.0)
            drho = (self.moments(flat[:, self.pn])[1].mean() - self.u_ref * scale) / cs
            j, i = self.oj, self.opp[self.oj]
            _, ux, uy = self.moments(flat[:, self.oat])
            rho = torch.where(self.orad, 1.0 + (self.onx * ux + self.ony * uy) / cs, 1.0 + drho)
            cu = 3.0 * (self.cx[j] * ux + self.cy[j] * uy)
            nf[i, self.oat] = -flat[j, self.oat] + 2.0 * self.w[j] * rho * (1.0 + 0.5 * cu * cu - 1.5 * (ux * ux + uy * uy))
        rho, ux, uy = self.moments(new)
        eq = self._eq(rho, ux, uy)
        if self.bgk:
            new = new - self.op * (new - eq)
        else:
            opp, e = new[self.opp], eq[self.opp]
            new = new - 0.5 * self.op * (new + opp - eq - e) - 0.5 * self.om * (new - opp - eq + e)
        self.f = torch.where(self.fluid, new, a)
        return torch.stack([fx, fy]), drho


def _ramp(t, steps):
    return 1.0 if t >= steps else (t / steps) ** 2 * (3.0 - 2.0 * t / steps)


def _channel_paint(nx, ny, open_sides):
    p = np.zeros((ny, nx), np.int64)
    p[:, 0], p[:, -1] = INLET, OUTLET
    if open_sides:
        p[0, 1:-1] = p[-1, 1:-1] = SIDE_OPEN
    else:
        p[0], p[-1] = SIDE_WALL, SIDE_WALL
    return p


def _half_away(v):
    return math.floor(v + 0.5)


def _tank_flow(d, up, down, height, re, u, inside_of):
    nx, ny = int(_half_away((up + down) * d)) + 2, int(_half_away(height * d)) + 2
    cx, cy = 0.5 + _half_away(up * d), 0.5 + 0.5 * _half_away(height * d)
    fl = _Flow(nx, ny, inside_of(cx, cy), 3.0 * u * d / re + 0.5, False, _channel_paint(nx, ny, True),
               lambda y: np.full(np.shape(y), u), u)
    fl.start(u)
    return fl


def _exact_body(case, p):
    def make(cx, cy):
        if case["body"] == "ellipse":
            f = _ellipse(cx, cy, p["a"], p["b"])
        elif case["body"] == "square":
            f = _square(cx, cy, float(case["d"]))
        else:
            f = _star(cx, cy, np.array(p["radii"]), p["phase"])
        return _rotated(f, cx, cy, p["angle"])
    return make


def _exact_rig(case, seed):
    p = _flow_inputs(case, seed)
    n, u = float(case["n"]), p["u"]
    nx, ny = 22 * case["n"] + 2, 41 * case["n"] // 10 + 2
    c, r, h = 0.5 + 2.0 * n, 0.5 * n, float(ny - 2)
    s_of = lambda y: np.clip(y - 0.5, 0.0, h)  # noqa: E731
    fl = _Flow(nx, ny, _ellipse(c, c, r, r), 3.0 * u * n / p["re"] + 0.5, False, _channel_paint(nx, ny, False),
               lambda y: 6.0 * u * s_of(y) * (h - s_of(y)) / (h * h), u)
    fl.start(0.0)
    # pressure on the cylinder's front and back, extrapolated from three bilinear samples each
    at, wt = [], []
    for side in (-1.0, 1.0):
        for dist, k in ((1, 3.0), (2, -3.0), (3, 1.0)):
            px, py = c + side * (r + dist), c
            i, jj = math.floor(px), math.floor(py)
            cor = [(i + a, jj + b, (px - i if a else 1 - px + i) * (py - jj if b else 1 - py + jj))
                   for b in (0, 1) for a in (0, 1)]
            cor = [(a, b, v) for a, b, v in cor if v > 0 and bool(fl.fluid[b, a])]
            tot = sum(v for _, _, v in cor)
            at += [b * nx + a for a, b, _ in cor]
            wt += [-side * k * v / tot for _, _, v in cor]
    at, wt = torch.tensor(at, device=fl.dev), torch.tensor(wt, dtype=torch.float64, device=fl.dev)
    ramp = int(1.0 * n / u)
    force, dp = [], []
    for t in range(case["steps"]):
        force.append(fl.step(_ramp(t, ramp))[0])
        dp.append((fl.f.reshape(9, -1)[:, at].sum(0) * wt).sum() / 3.0 / (u * u))
    k = 2.0 / (u * u * n)
    force = torch.stack(force).cpu().numpy() * k
    return {"cd": np.ascontiguousarray(force[:, 0]), "cl": np.ascontiguousarray(force[:, 1]), "dp": torch.stack(dp).cpu().numpy(),
            "f": fl.f.cpu().numpy()}


def _record(fl, steps):
    h = torch.zeros(steps, 10, dtype=torch.float64, device=fl.dev)
    for t in range(steps):
        h[t, :2], h[t, 8] = fl.step(1.0)
    return h.cpu().numpy()


def _vorticity(fl):
    _, ux, uy = fl.moments(fl.f)
    ux, uy = torch.where(fl.fluid, ux, 0.0), torch.where(fl.fluid, uy, 0.0)

    def diff(v, dim):
        n = v.shape[dim]
        ok, val = [], []
        for s in (1, -1):       # the neighbours ahead and behind, inside the domain and fluid
            i = torch.arange(n, device=fl.dev) + s
            inb = (i >= 0) & (i < n)
            i = i.clamp(0, n - 1)
            shape = [-1, 1] if dim == 0 else [1, -1]
            ok.append(fl.fluid.index_select(dim, i) & inb.reshape(shape))
            val.append(v.index_select(dim, i))
        zero = torch.zeros_like(v)
        return torch.where(ok[0] & ok[1], 0.5 * (val[0] - val[1]),
                           torch.where(ok[0], val[0] - v, torch.where(ok[1], v - val[1], zero)))
    return torch.where(fl.fluid, diff(uy, 1) - diff(ux, 0), 0.0)


# ====================================================================== 64-bit restatement: network
def _bf(x):
    return x.to(torch.bfloat16).to(torch.float64)


class _Stored(torch.autograd.Function):
    """A tensor that is stored in BF16 on its way forward, and (or) its gradient on the way back."""

    @staticmethod
    def forward(ctx, x, fwd, bwd):
        ctx.bwd = bwd
        return _bf(x) if fwd else x.clone()

    @staticmethod
    def backward(ctx, g):
        return (_bf(g) if ctx.bwd else g), None, None


def _conv64(x, w, b, stride, relu):
    """x [B, C, H, W]; w [cout, cin, k, k] and b in FP64. Activations and gradients of a layer's sum are BF16."""
    z = _Stored.apply(torch.nn.functional.conv2d(x, w, b, stride=stride, padding=w.shape[2] // 2), False, True)
    return _Stored.apply(torch.relu(z), True, False) if relu else z


def _w64(master, cin, k):
    """Padded [cout, kp] weights in (ky, kx, c) order -> [cout, cin, k, k], rounded to BF16."""
    return _bf(master[:, :k * k * cin]).reshape(-1, k, k, cin).permute(0, 3, 1, 2).contiguous().requires_grad_(True)


def _flat_grad(g, kp):
    out = torch.zeros(g.shape[0], kp, dtype=torch.float64, device=g.device)
    out[:, :g[0].numel()] = g.permute(0, 2, 3, 1).reshape(g.shape[0], -1)
    return out


def _conv_init(cin, cout, k, relu, seed):
    """The layer's initial weights as its class documents them: He-scaled normals, (ky, kx, c) columns."""
    fan = k * k * cin
    kp = (9 * cin + 63) // 64 * 64 if k == 3 else cin
    w = torch.zeros(cout, kp)
    w[:, :fan] = torch.randn(cout, fan, generator=torch.Generator().manual_seed(seed)) * math.sqrt(2.0 / fan) * (1.0 if relu else 0.1)
    return w.cuda()


def _exact_conv(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 2 + 1)
    B, h, w, cin, cout, st = (case[k] for k in ("batch", "h", "w", "cin", "cout", "stride"))
    x = torch.relu(torch.randn(B, h, w, cin, generator=g, device="cuda")).to(torch.bfloat16).double()
    ho, wo = (h + st - 1) // st, (w + st - 1) // st
    dy = torch.randn(B * ho * wo, cout, generator=g, device="cuda").double()
    master = _conv_init(cin, cout, 3, True, int(seed) % (1 << 20))
    xt = x.permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    wt = _w64(master, cin, 3)
    b = torch.zeros(cout, dtype=torch.float64, device="cuda", requires_grad=True)
    y = _conv64(xt, wt, b, st, True)
    y.backward(dy.reshape(B, ho, wo, cout).permute(0, 3, 1, 2))
    gw = _flat_grad(wt.grad, master.shape[1])
    lr, eps = 1e-4, 1e-8
    adam = lambda v, gr: v - lr * gr / (gr.abs() + eps)  # noqa: E731  the first update from zero moments
    return {"y": y.detach().permute(0, 2, 3, 1).reshape(-1, cout), "dx": xt.grad.permute(0, 2, 3, 1).reshape(-1, cin),
            "gw": gw, "gb": b.grad, "w": adam(master.double(), gw), "b": adam(torch.zeros_like(b.grad), b.grad)}


def _net_layers():
    """(key, cin, cout, stride, k, seed offset) of the four-level network in layer order."""
    ch, out = [32, 64, 128, 256], []
    for l in range(4):
        out += [(ch[l - 1] if l else 4, ch[l], 2 if l else 1, 3, 2 * l), (ch[l], ch[l], 1, 3, 2 * l + 1)]
    for l in (2, 1, 0):
        out += [(ch[l + 1] + ch[l], ch[l], 1, 3, 100 + 2 * l), (ch[l], ch[l], 1, 3, 101 + 2 * l)]
    return out + [(32, 8, 1, 1, 999)]


def _exact_net(case, seed):
    b = case["batch"]
    inp, tgt, wt = _net_inputs(b, seed)
    L = _net_layers()
    if case["kind"] == "predict":
        z = np.load(WS.PRETRAINED)
        masters = [torch.from_numpy((z["w%d" % i].astype(np.uint32) << 16).view(np.float32)).cuda() for i in range(len(L))]
        biases = [torch.from_numpy(z["b%d" % i]).cuda().double() for i in range(len(L))]
    else:
        s0 = (1 + int(seed) % 1000) * 1000
        masters = [_conv_init(ci, co, k, k == 3, s0 + off) for ci, co, _, k, off in L]
        biases = [torch.zeros(co, dtype=torch.float64, device="cuda") for _, co, _, _, _ in L]
    ws = [_w64(m, ci, k) for m, (ci, _, _, k, _) in zip(masters, L)]
    bs = [v.requires_grad_(True) for v in biases]
    lay = lambda i, x: _conv64(x, ws[i], bs[i], L[i][2], L[i][3] == 3)  # noqa: E731
    with torch.set_grad_enabled(case["kind"] == "train"):
        x, enc = _bf(inp).permute(0, 3, 1, 2).contiguous(), []
        for l in range(4):
            x = lay(2 * l + 1, lay(2 * l, x))
            enc.append(x)
        for n, l in enumerate((2, 1, 0)):
            up = torch.nn.functional.interpolate(x, scale_factor=2, mode="nearest")
            x = lay(9 + 2 * n, lay(8 + 2 * n, torch.cat([up, enc[l]], 1)))
        out = lay(14, x).permute(0, 2, 3, 1).reshape(-1, 8)
        if case["kind"] == "predict":
            return out
        d = (out[:, :3] - tgt.reshape(-1, 3).double()) * wt.reshape(-1, 1)
        ((d * d).sum() / (wt.double().sum() * 3)).backward()
    return {"out": out.detach(), "grads": [(_flat_grad(w.grad, m.shape[1]), v.grad) for w, m, v in zip(ws, masters, bs)]}


# ====================================================================== exact
def exact(case, seed):
    kind = case["kind"]
    if kind == "rig":
        return _exact_rig(case, seed)
    if kind in ("tunnel", "frames"):
        p = _flow_inputs(case, seed)
        fl = _tank_flow(case["d"], case["up"], case["down"], case["height"], p["re"], p["u"], _exact_body(case, p))
        if kind == "tunnel":
            h = _record(fl, case["steps"])
            return {"history": h, "f": fl.f.cpu().numpy()}
        out = []
        for _ in range(case["frames"]):
            for _ in range(case["steps"]):
                force, _ = fl.step(1.0)
            rho, ux, uy = fl.moments(fl.f)
            speed = torch.where(fl.fluid, (ux * ux + uy * uy).sqrt(), 0.0).max()
            out.append((_vorticity(fl), float(torch.where(fl.fluid, rho, 0.0).sum()), float(speed), force.reshape(1, 2)))
        return out
    if kind == "box":
        disks, u = _box_inputs(case, seed)
        fl = _Flow(case["nx"], case["ny"], _disks(disks, case["nx"], case["ny"]), 0.55, True)
        fl.start(u)
        h = _record(fl, case["steps"])
        return {"history": h, "f": fl.f.cpu().numpy()}
    if kind == "batch":
        hist, fields = [], None
        for c in _batch_cases(case, seed):
            tn, b = c.tunnel, c.body
            inner = getattr(b, "inner", b)

            def shape(cx, cy, b=b, inner=inner):
                if hasattr(inner, "radii"):
                    f = _star(inner.cx, inner.cy, np.array(inner.radii), inner.phase)
                elif hasattr(inner, "pts"):
                    f = _in_polygon(inner.pts)
                else:
                    f = _ellipse(inner.cx, inner.cy, inner.a, inner.b)
                return _rotated(f, b.cx, b.cy, b.angle) if inner is not b else f
            fl = _tank_flow(tn.d, tn.upstream, tn.downstream, tn.height, tn.re, tn.u, shape)
            hist.append(np.ascontiguousarray(_record(fl, case["steps"])[:, :2]))
            if fields is None:
                fields = tuple(torch.where(fl.fluid, v, w).cpu().numpy() for v, w in zip(fl.moments(fl.f), (1.0, 0.0, 0.0)))
        return {"history": hist, "fields": fields}
    return _exact_conv(case, seed) if kind == "conv" else _exact_net(case, seed)
