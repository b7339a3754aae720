"""The work that is timed: shots of elastic forward modelling and of RTM as a program using this package runs them.

Every case is a run of whole calls of the public entry points: jv_forward_noalloc, Context.forward,
Context.forward_device, Context.rtm_shot_device, Context.rtm_batch with Context.images, and the request server.
Real surveys run 1000 to 3000 time steps a shot; the larger grids here run fewer, since every step is the same work.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the model, the survey, the observed traces and the context a program keeps
    run(state)          one pass
    exact(case, seed)   the same outputs in 64 bits, from plain torch
"""
import ctypes
import importlib
import math

import numpy as np
import torch

jv = importlib.import_module("domain-decomposition-release_b200")

PRECISIONS = {"fp32": jv.JV_FP32, "bf16": jv.JV_BF16, "fp16": jv.JV_FP16}
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def _case(name, kind, nx, ny, nz, pml, nt, rec_step, fm=20.0, d=5.0, dt=4e-4, rec_width=1, precision="fp32", shots=1):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, pml=pml, nt=nt, rec_step=rec_step, fm=fm, d=d, dt=dt,
             rec_width=rec_width, precision=precision, shots=shots)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: one shot of a small model in a caller that may not allocate device memory; launch-bound
        _case("forward_noalloc_32", "noalloc", 32, 28, 24, 8, 160, 2, fm=40.0),
        # small models in a parameter study: many short forward runs, traces left on the device
        _case("forward_48", "forward_device", 48, 48, 48, 10, 300, 4, fm=40.0),
        # the plain forward configuration of the benchmark, traces to the host
        _case("forward_100", "forward", 100, 100, 100, 10, 1000, 12),
        # a ragged crop of a larger model: odd extents and an odd absorbing layer
        _case("forward_odd_131", "forward_device", 131, 87, 75, 9, 240, 3, fm=40.0),
        # a mid-size survey's forward model, wider than one row tile
        _case("forward_320", "forward_device", 320, 320, 320, 20, 80, 8, fm=60.0),
        # migration of a batch of shots on one small model, images to the host (the batched benchmark's smallest grid)
        _case("rtm_batch_80", "batch", 80, 80, 80, 16, 500, 2, shots=2),
        # migration of a ragged crop with exact reconstruction (rec_width 4) and a 16-bit boundary store
        _case("rtm_odd_93_w4_fp16", "rtm", 93, 61, 47, 11, 260, 2, fm=40.0, rec_width=4, precision="fp16"),
        # the batched benchmark's one-model grid, one shot
        _case("rtm_160", "rtm", 160, 160, 160, 16, 240, 2, fm=40.0),
        # the benchmark's single-shot migration: full receiver plane, rec_width 1
        _case("rtm_200", "rtm", 200, 200, 200, 20, 300, 1, fm=30.0),
        # ... and at rec_width 4 with the store halved
        _case("rtm_200_w4_bf16", "rtm", 200, 200, 200, 20, 160, 1, fm=50.0, rec_width=4, precision="bf16"),
        # the large-model configuration, 16-bit boundary store
        _case("rtm_676_fp16", "rtm", 676, 676, 210, 20, 48, 4, fm=40.0, d=10.0, dt=8e-4, precision="fp16"),
        # a mixed queue of modelling and migration requests through the request server
        _case("server_mix", "server", 112, 112, 112, 10, 160, 4, fm=40.0, shots=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["noalloc", "forward", "forward_device", "rtm", "rtm", "batch"])
    pml = rng.randint(8, 20)
    if kind == "noalloc":  # the no-allocation path holds up to about 60 cells a side
        nx, ny, nz = (_log(rng, 16, 44) for _ in range(3))
        pml = rng.randint(5, 10)
    elif kind == "batch":
        nx, ny, nz = (rng.randint(40, 96) for _ in range(3))
    else:
        nx, ny, nz = (_log(rng, 32, 360) for _ in range(3))
    if rng.random() < 0.5:  # rows of the benchmark's kind: even extents
        nx, pml = nx + nx % 2, pml + pml % 2
    cells = (nx + 2 * pml) * (ny + 2 * pml) * (nz + 2 * pml)
    if kind == "batch":
        nt = rng.randint(300, 500)
    else:
        cost = 3 if kind == "rtm" else 1
        nt = int(min(_log(rng, 100, 1000), 6e9 / (cost * cells)))
    rtm = kind in ("rtm", "batch")
    fm = 20.0 if kind == "batch" else max(20.0, min(60.0, 1.3 / (0.3 * nt * 4e-4)))
    return _case(None, kind, nx, ny, nz, pml, nt, rng.randint(1, 8), fm=fm,
                 rec_width=rng.randint(1, 4) if rtm else 1,
                 precision=rng.choice(["fp32", "fp32", "bf16", "fp16"]) if rtm else "fp32",
                 shots=2 if kind == "batch" else 1)


# ------------------------------------------------------------------ inputs

# the requests of a server queue: (kind, cells a side, model number); sizes of the benchmark's mixed queue, two on
# one grid so that a pooled context is used again
SERVER_QUEUE = (("rtm", 48, 0), ("forward", 112, 1), ("rtm", 80, 2), ("forward", 64, 3), ("rtm", 96, 4), ("rtm", 80, 5))


def _problems(case):
    """The problems of a pass: the case itself, or a server queue's requests."""
    if case["kind"] != "server":
        return [case]
    return [dict(case, kind=k, nx=n, ny=n, nz=n, number=q, shots=1) for k, n, q in SERVER_QUEUE[:case["shots"]]]


def _model(case, seed):
    """vp, vs, rho (float32, (nz, ny, nx), on the device): layers with dipping interfaces and a smooth anomaly."""
    rng = np.random.default_rng([seed, case.get("number", 0)])
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ax = [torch.arange(n, dtype=torch.float32, device=DEVICE) for n in (nz, ny, nx)]
    z, y, x = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    speeds = rng.uniform(2000.0, 4000.0, size=5)
    vp = torch.full((nz, ny, nx), float(speeds[0]), dtype=torch.float32, device=DEVICE)
    for depth, speed in zip(np.sort(rng.uniform(0.1 * nz, 0.9 * nz, size=4)), speeds[1:]):
        sx, sy = rng.uniform(-0.15, 0.15, size=2)
        below = z >= float(depth) + float(sx) * (x - nx / 2) + float(sy) * (y - ny / 2)
        vp = torch.where(below, torch.full_like(vp, float(speed)), vp)
    r2 = (z - nz / 2) ** 2 + (y - ny / 2) ** 2 + (x - nx / 2) ** 2
    vp = vp * (1.0 + float(rng.uniform(-0.12, 0.12)) * torch.exp(-r2 / (2.0 * (0.1 * min(nx, ny, nz)) ** 2)))
    return vp, vp / 1.732, 310.0 * vp ** 0.25


def _survey(case, seed):
    """Shot and receiver cells: shots near the surface centre, receivers on a surface grid, both 5 cells deep."""
    rng = np.random.default_rng([seed, case.get("number", 0), 1])
    nx, ny, step = case["nx"], case["ny"], case["rec_step"]
    shots = [(int(rng.integers(nx // 3, 2 * nx // 3)), int(rng.integers(ny // 3, 2 * ny // 3)), 5)
             for _ in range(case["shots"])]
    j, i = np.meshgrid(np.arange(0, ny, step), np.arange(0, nx, step), indexing="ij")
    recs = np.stack([i.ravel(), j.ravel(), np.full(i.size, 5)], axis=1)
    return np.asarray(shots), recs


def _observed(case, seed, shot, recs, number):
    """Observed traces (3, n_recv, nt) float32: three events with hyperbolic moveout per component, and noise."""
    rng = np.random.default_rng([seed, case.get("number", 0), 2 + number])
    nt, dt, fm, d = case["nt"], case["dt"], case["fm"], case["d"]
    off = torch.tensor(np.hypot(recs[:, 0] - shot[0], recs[:, 1] - shot[1]) * d, dtype=torch.float64, device=DEVICE)
    t = torch.arange(nt, dtype=torch.float64, device=DEVICE) * dt
    out = torch.zeros((3, recs.shape[0], nt), dtype=torch.float32, device=DEVICE)
    for q in range(3):
        for _ in range(3):
            t0, v, a = rng.uniform(0.1, 0.7) * nt * dt, rng.uniform(2000.0, 4000.0), rng.normal() * 1e-3
            arg = (math.pi * fm * (t[None, :] - torch.sqrt(t0 * t0 + (off / v) ** 2)[:, None])) ** 2
            out[q] += (a * (1.0 - 2.0 * arg) * torch.exp(-arg)).float()
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(int(rng.integers(1 << 31)))
    out += 2e-5 * torch.randn(out.shape, generator=gen, device=DEVICE)
    return out


def _metres(cells, d):
    return np.ascontiguousarray(np.asarray(cells, dtype=np.float64).reshape(-1, 3) * d, dtype=np.float32)


def _pinned(t):
    return t.cpu().pin_memory().numpy()


class _Server:
    """A request server that is closed with its state."""

    def __init__(self):
        self.server = jv.Server(slots=4, budget=16 << 30)

    def __del__(self):
        self.server.close()


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "server":
        state["server"] = _Server()
        state["requests"] = []
        for p in _problems(case):
            vp, vs, rho = (a.cpu().numpy() for a in _model(p, seed))
            shots, recs = _survey(p, seed)
            n, rtm = p["nx"], p["kind"] == "rtm"
            outs = (tuple(np.zeros((n, n, n), np.float64) for _ in range(5)) if rtm else
                    tuple(np.zeros((recs.shape[0], p["nt"]), np.float32) for _ in range(3)))
            state["requests"].append((jv.JOB_RTM if rtm else jv.JOB_FORWARD, dict(
                nx=n, ny=n, nz=n, pml=p["pml"], dx=p["d"], dy=p["d"], dz=p["d"], vp=vp, vs=vs, rho=rho, dt=p["dt"],
                fm=p["fm"], nt=p["nt"], shot_xyz=_metres(shots, p["d"])[0], recv_xyz=_metres(recs, p["d"]),
                **({"image": outs} if rtm else {"out": outs})), outs))
        return state
    vp, vs, rho = _model(case, seed)
    shots, recs = _survey(case, seed)
    nx, ny, nz, nt, d, nrec = case["nx"], case["ny"], case["nz"], case["nt"], case["d"], recs.shape[0]
    if kind == "noalloc":
        state["grid"] = jv.Grid(nx, ny, nz, case["pml"], d, d, d)
        state["model"] = [a.contiguous() for a in (vp, vs, rho)]
        state["src"], state["rec"] = _metres(shots, d), _metres(recs, d)
        state["out"] = torch.empty((3, nrec, nt), dtype=torch.float32, device=DEVICE)
        torch.cuda.synchronize()
        return state
    ctx = jv.Context.create(nx, ny, nz, case["pml"], d, d, d, *(a.cpu().numpy() for a in (vp, vs, rho)), case["dt"],
                            case["fm"], nt, rec_width=case["rec_width"], precision=PRECISIONS[case["precision"]])
    ctx.set_geometry(_metres(shots, d), _metres(recs, d))
    state["ctx"] = ctx
    if kind == "forward_device":
        state["out"] = torch.empty((3, nrec, nt), dtype=torch.float32, device=DEVICE)
    elif kind == "rtm":
        state["obs"] = _observed(case, seed, shots[0], recs, 0)
        state["out"] = torch.empty((5, nz, ny, nx), dtype=torch.float64, device=DEVICE)
    elif kind == "batch":
        state["obs"] = [list(_pinned(_observed(case, seed, s, recs, k))) for k, s in enumerate(shots)]
    torch.cuda.synchronize()
    return state


# ------------------------------------------------------------------ the pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "noalloc":
        lib, vp, out = jv.lib(), ctypes.c_void_p, state["out"]
        fp = ctypes.POINTER(ctypes.c_float)
        kept = ctypes.c_int()
        rc = lib.jv_forward_noalloc(ctypes.byref(state["grid"]), *(vp(a.data_ptr()) for a in state["model"]),
                                    case["dt"], case["fm"], case["nt"], state["src"].ctypes.data_as(fp),
                                    state["rec"].shape[0], state["rec"].ctypes.data_as(fp),
                                    *(vp(out[q].data_ptr()) for q in range(3)), ctypes.byref(kept),
                                    vp(torch.cuda.current_stream().cuda_stream))
        if rc != jv.JV_OK:
            raise jv.JvError(rc, lib.jv_last_error().decode())
        return out
    if kind == "forward":
        return state["ctx"].forward(0)
    if kind == "forward_device":
        state["ctx"].forward_device(0, [state["out"][q].data_ptr() for q in range(3)])
        return state["out"]
    if kind == "rtm":
        ctx = state["ctx"]
        ctx.image_reset()
        ctx.rtm_shot_device(0, [state["obs"][q].data_ptr() for q in range(3)])
        for k in range(5):
            ctx.image_to_device(k, state["out"][k].data_ptr())
        return state["out"]
    if kind == "batch":
        ctx = state["ctx"]
        ctx.image_reset()
        ctx.rtm_batch(list(range(case["shots"])), state["obs"])
        return ctx.images()
    server = state["server"].server
    ids = [server.submit(kind_, **args) for kind_, args, _ in state["requests"]]
    for i in ids:
        rc = server.wait(i)
        if rc != jv.JV_OK:
            raise jv.JvError(rc, "request failed")
    return [outs for _, _, outs in state["requests"]]


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """Per time step of a propagation: the nine fields read and written once and the four model arrays read once; the
    memory variables of the absorbing axes read and written once; in a migration also the pressure-like field and the
    P-wave velocities, the images and the boundary records.  Velocity and stress of a step are counted as one pass
    over memory: a step's velocities need not leave the chip before its stresses use them."""
    total, flops = 0, 0
    for p in _problems(case):
        m, nt = p["pml"], p["nt"]
        ext = [p[k] + 2 * m for k in ("nx", "ny", "nz")]
        cells, phy = math.prod(ext), p["nx"] * p["ny"] * p["nz"]
        psi = sum(2 * (m - 2) * cells // n for n in ext) * 6  # three arrays a set, a velocity and a stress set
        fwd = 4 * (9 * 2 + 4) * cells + 8 * psi
        area = 2 * (p["nx"] * p["ny"] + p["ny"] * p["nz"] + p["nx"] * p["nz"])
        nrec = -(-p["nx"] // p["rec_step"]) * -(-p["ny"] // p["rec_step"])
        if p["kind"] in ("rtm", "batch"):
            r = p["rec_width"]
            record = area * (7 * r - 3) * (4 if p["precision"] == "fp32" else 2)
            step = (fwd + 8 * cells                       # forward with the pressure-like field
                    + fwd + 8 * cells + 24 * phy          # receivers, with their P-wave velocities
                    + (4 * (13 * 2 + 3) + 40) * phy       # reconstruction, with the five images
                    + 2 * record)
            n, total = p["shots"] * nt, total + p["shots"] * (nt * step + 12 * nrec * nt) + 60 * phy
            flops += n * (2 * 330 * cells + 420 * phy)
            if case["kind"] == "server":  # a request without traces models them first
                total, flops = total + nt * (fwd + 12 * nrec), flops + nt * 300 * cells
        else:
            total, flops = total + nt * (fwd + 12 * nrec), flops + nt * 300 * cells
    return {"bytes": int(total), "flops": int(flops)}


def tolerance(case):
    """Hundreds of 32-bit sums follow one another in a propagation, and the imaging condition multiplies two of them;
    a 16-bit boundary store seeds the reconstruction with values of 8 or 11 bits.  About four times the largest error
    against 64 bits seen over the cases and a dozen draws: traces 3e-5, images 1.1e-4 (FP32 store), 2.8e-4 (FP16) and
    1.9e-3 (BF16)."""
    if case["kind"] in ("noalloc", "forward", "forward_device"):
        return {"rel": 1.2e-4}
    return {"rel": {"fp32": 4.5e-4, "fp16": 1.2e-3, "bf16": 8e-3}[case["precision"]]}


# ------------------------------------------------------------------ the same in 64 bits

TAPS = {1: (1.0,), 2: (9 / 8, -1 / 24), 3: (75 / 64, -25 / 384, 3 / 640),
        4: (1225 / 1024, -245 / 3072, 49 / 5120, -5 / 7168)}
SHEAR = {"sxy": (0, 1), "sxz": (0, 2), "syz": (1, 2)}
V, S = ("vx", "vy", "vz"), ("sxx", "syy", "szz", "sxy", "sxz", "syz")


class _Exact:
    """One wavefield in 64 bits.  Arrays are (z, y, x) over the grid and its absorbing layers; axis 0 is x."""

    def __init__(self, case, seed):
        self.m, self.dt, self.h, self.nt = case["pml"], float(np.float32(case["dt"])), case["d"], case["nt"]
        self.n = [case[k] + 2 * self.m for k in ("nx", "ny", "nz")]
        self.p = [case[k] for k in ("nx", "ny", "nz")]
        at = [(torch.arange(n, device=DEVICE) - self.m).clamp(0, p - 1) for n, p in zip(self.n, self.p)]
        vp, vs, rho = (a.double()[at[2]][:, at[1]][:, :, at[0]] for a in _model(case, seed))
        self.vp, self.bdt = vp, self.dt / rho
        self.lam, self.mu = rho * (vp * vp - 2 * vs * vs), rho * vs * vs
        self.l2m = self.lam + 2 * self.mu
        self.outer = [(2, n - 2) for n in self.n]
        self.inner = [(self.m, self.m + p) for p in self.p]
        self.alpha = math.pi * case["fm"]
        self.coef = {}
        n0 = math.floor(float(np.float32(np.float32(1.3) / np.float32(case["fm"])) / np.float32(case["dt"])
                              + np.float32(0.5)))
        a2 = (math.pi * case["fm"] * (np.arange(self.nt) - n0) * self.dt) ** 2
        self.wavelet = 1e4 * (1 - 2 * a2) * np.exp(-a2)

    def field(self):
        return torch.zeros(self.n[::-1], dtype=torch.float64, device=DEVICE)

    def state(self, names):
        return {k: self.field() for k in names}

    @staticmethod
    def cut(a, box, axis=0, shift=0):
        s = [slice(lo + (shift if k == axis else 0), hi + (shift if k == axis else 0)) for k, (lo, hi) in
             enumerate(box)]
        return a[s[2], s[1], s[0]]

    def diff(self, a, axis, plus, box, order=4, rows=None):
        """The staggered difference of `a` over a box: plus, at the half cell above; else at the one below.  With
        rows, the order changes along the axis: rows[r] is the r-th tap there."""
        out = None
        for r in range(order):
            up, down = (r + 1, -r) if plus else (r, -r - 1)
            t = self.cut(a, box, axis, up) - self.cut(a, box, axis, down)
            t *= rows[r] if rows is not None else TAPS[order][r]
            out = t if out is None else out.add_(t)
        return out.mul_(1 / self.h)

    def damping(self, axis, side, half):
        """(box within the updated cells, a, b) of one absorbing side of one axis."""
        key = (axis, side, half)
        if key not in self.coef:
            n, m = self.n[axis], self.m
            lo, hi = (2, m) if side == 0 else (n - m, n - 2)
            c = torch.arange(lo, hi, dtype=torch.float64, device=DEVICE)
            depth = m - c - (0.5 if half else 0.0) if side == 0 else c - (n - m - 1) - (0.0 if half else 0.5)
            q = depth / (m - 2)
            shape = [1, 1, 1]
            shape[2 - axis] = hi - lo
            k = (21.0 / (2.0 * (m - 2) * self.h) * q * q).reshape(shape)
            alpha = (self.alpha * (1 - q)).clamp(min=0.0).reshape(shape)
            box = list(self.outer)
            box[axis] = (lo, hi)
            d = self.cut(self.vp, box) * k
            b = torch.exp(-(d + alpha) * self.dt)
            self.coef[key] = ([(x0 - 2, x1 - 2) for x0, x1 in box], d * (b - 1) / (d + alpha), b)
        return self.coef[key]

    def damped(self, psi, name, a, axis, plus):
        """The 4th-order difference over the updated cells, with its memory variables in the absorbing ranges."""
        d = self.diff(a, axis, plus, self.outer, order=2)
        for side in (0, 1):
            box, ca, cb = self.damping(axis, side, plus)
            part = self.cut(d, box)
            key = (name, axis, side)
            new = ca * part
            if key in psi:
                new += cb * psi[key]
            psi[key] = new
            part += new
        return d

    def inside(self):
        return [(self.m - 2, self.m - 2 + p) for p in self.p]

    def velocity(self, w, psi):
        """One velocity update of the grid and its absorbing layers; with P-wave velocities where w has them."""
        rows = (("vx", (("sxx", 0, True), ("sxy", 1, False), ("sxz", 2, False))),
                ("vy", (("sxy", 0, False), ("syy", 1, True), ("syz", 2, False))),
                ("vz", (("sxz", 0, False), ("syz", 1, False), ("szz", 2, True))))
        for v, terms in rows:
            edge = inner = None
            for f, axis, plus in terms:
                e = self.damped(psi, v + f, w[f], axis, plus)
                i = self.diff(w[f], axis, plus, self.inner)
                edge, inner = (e, i) if edge is None else (edge.add_(e), inner.add_(i))
            self.cut(edge, self.inside()).copy_(inner)
            self.cut(w[v], self.outer).add_(self.cut(self.bdt, self.outer) * edge)
        if "vxp" in w:
            for axis, v in enumerate(("vxp", "vyp", "vzp")):
                self.cut(w[v], self.inner).add_(self.cut(self.bdt, self.inner)
                                                * self.diff(w["sau"], axis, True, self.inner))

    def stress(self, w, psi, source=None, it=0):
        if source is not None:
            for f in S[:3]:
                w[f][source[2] + self.m, source[1] + self.m, source[0] + self.m] += float(self.wavelet[it])
        d = {}
        for axis, v in enumerate(V):
            for f, other, plus in ((("n", axis), axis, False),) + tuple(
                    ((k, v), b if a == axis else a, True) for k, (a, b) in SHEAR.items() if axis in (a, b)):
                e = self.damped(psi, str(f), w[v], other, plus)
                self.cut(e, self.inside()).copy_(self.diff(w[v], other, plus, self.inner))
                key = f if f[0] == "n" else f[0]
                d[key] = e if key not in d else d[key].add_(e)
        self.add_stress(w, d, self.outer, self.dt)

    def add_stress(self, w, d, box, dt):
        lam, mu, l2m = (self.cut(a, box) for a in (self.lam, self.mu, self.l2m))
        both = d["n", 0] + d["n", 1] + d["n", 2]
        if "sau" in w:
            self.cut(w["sau"], box).add_(l2m * both, alpha=dt)
        both *= lam
        for axis, f in enumerate(S[:3]):
            self.cut(w[f], box).add_(both + 2 * mu * d["n", axis], alpha=dt)
        for f in SHEAR:
            self.cut(w[f], box).add_(mu * d[f], alpha=dt)

    def rim(self, width):
        """Per axis the taps of every inner cell: fewer near the faces, never below the stored width."""
        out = []
        for axis, p in enumerate(self.p):
            e = np.minimum(np.arange(p), p - 1 - np.arange(p))
            order = np.where(e >= 4, 4, np.maximum(e + 1, width))
            t = np.array([[TAPS[o][r] if r < o else 0.0 for o in order] for r in range(4)])
            shape = [4, 1, 1, 1]
            shape[3 - axis] = p
            out.append(torch.tensor(t, device=DEVICE).reshape(shape))
        return out

    def back_stress(self, w, rim, source, it):
        for f in S[:3]:
            w[f][source[2] + self.m, source[1] + self.m, source[0] + self.m] -= float(self.wavelet[it])
        d = {}
        for axis, v in enumerate(V):
            d["n", axis] = self.diff(w[v], axis, False, self.inner, rows=rim[axis])
            for k, (a, b) in SHEAR.items():
                if axis in (a, b):
                    o = b if a == axis else a
                    t = self.diff(w[v], o, True, self.inner, rows=rim[o])
                    d[k] = t if k not in d else d[k].add_(t)
        self.add_stress(w, d, self.inner, -self.dt)

    def back_velocity(self, w, rim):
        b = self.cut(self.bdt, self.inner)
        for v, terms in (("vx", (("sxx", 0, True), ("sxy", 1, False), ("sxz", 2, False))),
                         ("vy", (("sxy", 0, False), ("syy", 1, True), ("syz", 2, False))),
                         ("vz", (("sxz", 0, False), ("syz", 1, False), ("szz", 2, True))),
                         ("vxp", (("sau", 0, True),)), ("vyp", (("sau", 1, True),)), ("vzp", (("sau", 2, True),))):
            for f, axis, plus in terms:
                self.cut(w[v], self.inner).sub_(b * self.diff(w[f], axis, plus, self.inner, rows=rim[axis]))

    def faces(self, width):
        """The stored boxes of each field: layers outside the inner grid that the reconstruction reads."""
        r = width
        wide = {"vx": (r - 1, r, r - 1, r, r, r - 1), "vy": (r - 1, r, r, r - 1, r - 1, r),
                "vz": (r, r - 1, r - 1, r, r - 1, r), "sxx": (0, 0, 0, 0, r - 1, r), "syy": (0, 0, r - 1, r, 0, 0),
                "szz": (r - 1, r, 0, 0, 0, 0), "sau": (r - 1, r, r - 1, r, r - 1, r),
                "sxy": (0, 0, r, r - 1, r, r - 1), "sxz": (r, r - 1, 0, 0, r, r - 1), "syz": (r, r - 1, r, r - 1, 0, 0)}
        out = []
        for f, ws in wide.items():
            for face, k in enumerate(ws):
                if k > 0:
                    axis = (2, 1, 0)[face // 2]
                    lo, hi = self.inner[axis]
                    box = list(self.inner)
                    box[axis] = (lo - k, lo) if face % 2 == 0 else (hi, hi + k)
                    out.append((f, box))
        return out


def _forward64(case, seed, shot, recs):
    e = _Exact(case, seed)
    w, psi = e.state(V + S), {}
    at = [torch.tensor(recs[:, k] + e.m, device=DEVICE) for k in range(3)]
    out = torch.empty((3, recs.shape[0], e.nt), dtype=torch.float64, device=DEVICE)
    for it in range(e.nt):
        e.velocity(w, psi)
        e.stress(w, psi, shot, it)
        for q, v in enumerate(V):
            out[q, :, it] = w[v][at[2], at[1], at[0]]
    return out


def _rtm64(case, seed, shot, recs, obs):
    """The five images of one shot."""
    e = _Exact(case, seed)
    w, psi = e.state(V + S + ("sau",)), {}
    faces, kept = e.faces(case["rec_width"]), []
    for it in range(e.nt):
        e.velocity(w, psi)
        e.stress(w, psi, shot, it)
        if it < e.nt - 1:
            kept.append([e.cut(w[f], box).clone() for f, box in faces])
    P = ("vxp", "vyp", "vzp")
    w.update(e.state(P))
    r, psi = e.state(V + S + ("sau",) + P), {}
    rim = e.rim(case["rec_width"])
    images = torch.zeros((5,) + tuple(e.p[::-1]), dtype=torch.float64, device=DEVICE)
    at = (torch.tensor(recs[:, 2] + e.m, device=DEVICE), torch.tensor(recs[:, 1] + e.m, device=DEVICE),
          torch.tensor(recs[:, 0] + e.m, device=DEVICE))
    for it in range(e.nt - 1, -1, -1):
        for q, v in enumerate(V):
            r[v].index_put_(at, obs[q, :, it].double(), accumulate=True)
        e.back_stress(w, rim, shot, it)
        e.velocity(r, psi)
        record = kept.pop() if it > 0 else []
        for (f, box), a in zip(faces, record):
            if f not in V:
                e.cut(w[f], box).copy_(a)
        e.back_velocity(w, rim)
        for v, p in zip(V, P):
            sp, rp = e.cut(w[p], e.inner), e.cut(r[p], e.inner)
            ss, rs = e.cut(w[v], e.inner) - sp, e.cut(r[v], e.inner) - rp
            for k, (a, b) in enumerate(((sp, sp), (sp, rp), (sp, rs), (ss, rp), (ss, rs))):
                images[k].addcmul_(a, b)
        e.stress(r, psi)
        for (f, box), a in zip(faces, record):
            if f in V:
                e.cut(w[f], box).copy_(a)
    return images


def exact(case, seed):
    steps = case["nt"] * case["shots"] * (1 if "forward" in case["kind"] or case["kind"] == "noalloc" else 4)
    cells = math.prod(case[k] + 2 * case["pml"] for k in ("nx", "ny", "nz"))
    if cells > 5e7 or steps * cells > 1.7e10:  # over about 20 seconds
        return None
    out = []
    for p in _problems(case):
        shots, recs = _survey(p, seed)
        if p["kind"] in ("noalloc", "forward", "forward_device"):
            out.append(_forward64(p, seed, shots[0], recs))
            continue
        if case["kind"] == "server":
            images = _rtm64(p, seed, shots[0], recs, _forward64(p, seed, shots[0], recs))
        else:
            images = sum(_rtm64(p, seed, s, recs, _observed(p, seed, s, recs, k)) for k, s in enumerate(shots))
        out.append(images)
    if case["kind"] == "server":
        return [tuple(o.cpu().numpy() for o in q) for q in out]
    if case["kind"] == "forward":
        return tuple(out[0].cpu().numpy())
    if case["kind"] == "batch":
        return dict(zip(("ip", "pp", "ps", "sp", "ss"), out[0].cpu().numpy()))
    return out[0]
