"""The tile kernels (variant 4) at the sizes where they can go wrong, through
the C ABI against the FP64 oracle: rows that end just before, on and after a
32-column tile, 16-row tiles with one row or one short of full, odd extents
and absorbing layers (pairs that straddle gridphy's edge and the rim), the
thinnest layer, the source in a tile's corner cells.

Tolerances are those of the other parity tests: traces 2e-5 and images 5e-5
relative L2 (FP32 sums over some hundred time steps)."""
import ctypes

import numpy as np
import pytest

from conftest import pkg, rel_l2

jv = pkg()
pytestmark = pytest.mark.gpu


def _problem(oracle, s, w):
    return oracle.Problem(s.nx, s.ny, s.nz, s.pml, s.dx, s.dy, s.dz, s.dt, s.fm, s.T, w, s.shots, s.recvs,
                          s.vp, s.vs, s.rho)


CASES = [
    dict(n=(24, 16, 9), pml=4, nt=90, seed=71, shot_idx=[(0, 0, 0)]),              # thinnest layer, corner source
    dict(n=(25, 17, 10), pml=5, nt=90, seed=72, shot_idx=[(24, 16, 9)]),           # odd everything
    dict(n=(31, 20, 12), pml=7, nt=90, seed=73, nrec=30, rec_width=3),
    dict(n=(32, 21, 11), pml=6, nt=90, seed=74, rec_width=2, shot_idx=[(31, 4, 5)]),
    dict(n=(33, 8, 8), pml=9, nt=80, seed=75, rec_width=4, anomaly=(0.1, 3.0)),
    dict(n=(65, 33, 8), pml=8, nt=70, seed=76, shot_idx=[(32, 16, 4)]),
    # the source near the receivers: from the far end (z = 38) nothing reaches them in 80 steps but images of
    # 1e-36, whose FP32 products are subnormal
    dict(n=(8, 8, 40), pml=11, nt=110, seed=77, shot_idx=[(3, 4, 7)]),
]


@pytest.mark.parametrize("kw", CASES)
def test_tile_kernels_vs_oracle(oracle, synth, kw):
    s = synth.small_case(**kw)
    p = _problem(oracle, s, s.rec_width)
    obs = oracle.forward(p)
    ref = oracle.rtm_shot(p, obs)
    with jv.Context.from_survey(s) as ctx:
        cfg = ctx.kernel_config()
        assert cfg["kernel_variant"] == 4 and cfg["run_chunks"] > 0
        tr = ctx.forward(0)
        ctx.rtm_shot(0, [o.astype(np.float32) for o in obs])
        raw = ctx.images()
    for a, b in zip(tr, obs):
        assert np.all(np.isfinite(a))
        assert rel_l2(a, b) <= 2e-5, rel_l2(a, b)
    for k in ("ip", "pp", "ps", "sp", "ss"):
        assert rel_l2(raw[k], ref[k]) <= 5e-5, (k, rel_l2(raw[k], ref[k]))


@pytest.mark.parametrize("dx,dy,dz", [(10.0, 12.5, 8.0)])
def test_tile_kernels_unequal_spacing(oracle, synth, dx, dy, dz):
    """Each axis' differences carry its own spacing."""
    s = synth.small_case(n=(21, 18, 16), pml=6, nt=100, seed=78, dx=dx)
    s.dy, s.dz = dy, dz
    scale = np.array([1.0, dy / dx, dz / dx], np.float32)
    s.shots, s.recvs = s.shots * scale, s.recvs * scale
    p = _problem(oracle, s, 1)
    obs = oracle.forward(p)
    with jv.Context.from_survey(s) as ctx:
        tr = ctx.forward(0)
    for a, b in zip(tr, obs):
        assert rel_l2(a, b) <= 2e-5, rel_l2(a, b)


# ------------------------------------------------ rounding, bit for bit

F32 = np.float32


def _fma(a, b, c):
    """a b + c in FP32 with one rounding: the exact product, its sum with c rounded to odd in FP64, then to FP32."""
    p = np.asarray(a, F32).astype(np.float64) * np.asarray(b, F32).astype(np.float64)
    p, c = np.broadcast_arrays(p, np.asarray(c, F32).astype(np.float64))
    s = p + c
    t = s - p
    err = (p - (s - t)) + (c - t)
    bits = s.view(np.int64)
    step = np.where((err != 0) & (bits & 1 == 0), np.where((err > 0) == (s > 0), 1, -1), 0)
    return (bits + step).view(np.float64).astype(F32)


class _Interior:
    """One FP32 wavefield of a grid so large that nothing reaches its faces; arrays (z, y, x), axis 0 is x."""
    TAPS = [F32(c) for c in (1225 / 1024, -245 / 3072, 49 / 5120, -5 / 7168)]
    SUMS = (("vx", (("sxx", 0, True), ("sxy", 1, False), ("sxz", 2, False))),
            ("vy", (("sxy", 0, False), ("syy", 1, True), ("syz", 2, False))),
            ("vz", (("sxz", 0, False), ("syz", 1, False), ("szz", 2, True))))

    def __init__(self, s):
        vp, vs, rho = (np.asarray(a, F32) for a in (s.vp, s.vs, s.rho))
        self.dt, self.rd, self.bdt = F32(s.dt), [F32(1) / F32(d) for d in (s.dx, s.dy, s.dz)], F32(s.dt) / rho
        vs2 = vs * vs
        self.lam, self.mu = rho * (vp * vp - F32(2) * vs2), rho * vs2
        self.f = {k: np.zeros_like(vp) for k in ("vx", "vy", "vz", "sxx", "syy", "szz", "sxy", "sxz", "syz", "sau",
                                                 "px", "py", "pz")}

    def diff(self, k, axis, plus):
        def at(n):
            return np.roll(self.f[k], -n, 2 - axis)
        d = [at(q + 1) - at(-q) if plus else at(q) - at(-q - 1) for q in range(4)]
        t = self.TAPS[0] * d[0]
        for q in (1, 2, 3):
            t = _fma(self.TAPS[q], d[q], t)
        return t

    def velocity(self, forward, sign=1):
        rx, ry, rz = self.rd
        for v, terms in self.SUMS:
            x, y, z = (self.diff(*t) for t in terms)
            d = _fma(y, ry, x * rx) if forward else _fma(x, rx, y * ry)
            self.f[v] = _fma(F32(sign) * self.bdt, _fma(z, rz, d), self.f[v])

    def p_velocity(self, sign):
        for axis, p in enumerate(("px", "py", "pz")):
            self.f[p] = _fma(F32(sign) * self.bdt, self.diff("sau", axis, True) * self.rd[axis], self.f[p])

    def stress(self, sign=1, source=None, value=0):
        f, dt, (rx, ry, rz) = self.f, F32(sign) * self.dt, self.rd
        if source is not None:
            for k in ("sxx", "syy", "szz"):
                f[k][source] = f[k][source] + F32(sign) * value
        nx, ny, nz = (self.diff(k, a, False) * self.rd[a] for a, k in enumerate(("vx", "vy", "vz")))
        lam, mu = self.lam, self.mu
        l2m = _fma(mu, F32(2), lam)
        new = {"sxx": _fma(dt, _fma(lam, nz, _fma(l2m, nx, lam * ny)), f["sxx"]),
               "syy": _fma(dt, _fma(lam, nz, _fma(lam, nx, l2m * ny)), f["syy"]),
               "szz": _fma(dt, _fma(l2m, nz, _fma(lam, nx, lam * ny)), f["szz"]),
               "sau": _fma(dt * l2m, (nx + ny) + nz, f["sau"])}
        for k, (a, i, r), (b, j, q) in (("sxy", ("vy", 0, rx), ("vx", 1, ry)), ("sxz", ("vz", 0, rx), ("vx", 2, rz)),
                                        ("syz", ("vz", 1, ry), ("vy", 2, rz))):
            new[k] = _fma(dt * mu, _fma(self.diff(a, i, True), r, self.diff(b, j, True) * q), f[k])
        f.update(new)


def _wavelet(s):
    n0 = int(np.floor(F32(1.3) / F32(s.fm) / F32(s.dt) + F32(0.5)))
    a2 = [(np.pi * float(F32(s.fm)) * float(F32(i - n0) * F32(s.dt))) ** 2 for i in range(s.nt)]
    return [F32(1e4 * (1 - 2 * x) * np.exp(-x)) for x in a2]


@pytest.mark.parametrize("n,dx,dy,dz", [((57, 58, 60), 10.0, 10.0, 10.0), ((64, 56, 58), 10.0, 12.5, 8.0)])
def test_sums_of_differences_round_once(synth, n, dx, dy, dz):
    """Three steps of modelling and of migration from the middle of a grid, where no layer is reached: every trace
    and image equals its FP32 sums with the stated fused multiply-adds, bit for bit (no tolerance)."""
    c = tuple(k // 2 for k in n)
    s = synth.small_case(n=n, pml=4, nt=3, seed=81, dx=dx, fm=300.0, dt=2e-4, shot_idx=[c])
    recs = np.array([(c[0] + i, c[1] + j, c[2] + k) for i in range(-9, 10, 3) for j in (-7, 0, 2) for k in (-5, 1)])
    s.dy, s.dz = dy, dz
    s.shots = (np.array([c]) * np.array([dx, dy, dz])).astype(F32)
    s.recvs = (recs * np.array([dx, dy, dz])).astype(F32)
    obs = [(1e-3 * np.random.default_rng(q).standard_normal((len(recs), s.nt))).astype(F32) for q in range(3)]
    with jv.Context.from_survey(s) as ctx:
        tr = ctx.forward(0)
        ctx.rtm_shot(0, obs)
        raw = ctx.images()
    w, src, at = _Interior(s), c[::-1], tuple(recs.T[::-1])
    wavelet, V, P = _wavelet(s), ("vx", "vy", "vz"), ("px", "py", "pz")
    for it in range(s.nt):
        w.velocity(True)
        w.stress(1, src, wavelet[it])
        for q, v in enumerate(V):
            assert np.array_equal(tr[q][:, it], w.f[v][at]), (it, v)
    r = _Interior(s)
    img = {k: np.zeros_like(w.lam) for k in ("ip", "pp", "ps", "sp", "ss")}
    for it in range(s.nt - 1, -1, -1):
        for q, v in enumerate(V):
            r.f[v][at] += obs[q][:, it]
        w.stress(-1, src, wavelet[it])
        w.velocity(False, -1)
        r.velocity(False)
        w.p_velocity(-1)
        r.p_velocity(1)
        sp, rp = [w.f[k] for k in P], [r.f[k] for k in P]
        ss, rs = ([u.f[v] - p for v, p in zip(V, pp)] for u, pp in ((w, sp), (r, rp)))
        for k, a, b in (("ip", sp, sp), ("pp", sp, rp), ("ps", sp, rs), ("sp", ss, rp), ("ss", ss, rs)):
            img[k] = img[k] + _fma(a[2], b[2], _fma(a[0], b[0], a[1] * b[1]))
        r.stress()
    for k in img:
        assert np.abs(img[k]).max() > 0 and np.array_equal(raw[k].astype(F32), img[k]), k


@pytest.mark.parametrize("precision", [jv.JV_FP32, jv.JV_FP16])
def test_captured_migration_repeats_itself(synth, precision):
    """A migration large enough to fill the chip, twelve times from captured graphs and three times from direct
    launches: the same images, bit for bit.  A plane refilled under a late reader showed in every captured run."""
    s = synth.scaled_cfg2(144, 160, pml=16)
    out = []
    for graphs in (1, 0):
        with jv.Context.from_survey(s, use_graphs=graphs, precision=precision) as ctx:
            tr = ctx.forward(0)
            for _ in range(12 if graphs else 3):
                ctx.image_reset()
                ctx.rtm_shot(0, tr)
                out.append((tr, ctx.images()))
    for tr, im in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(tr, out[0][0]))
        for k in im:
            assert np.array_equal(im[k], out[0][1][k]), k


def test_arrays_of_4_gb_and_more():
    """A shot near the end of arrays of 4.4 GB, whose byte offsets pass 32 bits, against variant 3's kernels."""
    import os
    import torch

    nx, ny, nz, pml, nt = 1000, 1000, 960, 20, 6
    if torch.cuda.mem_get_info(0)[0] < 135e9 or os.sysconf("SC_AVPHYS_PAGES") * os.sysconf("SC_PAGE_SIZE") < 40e9:
        pytest.skip("needs 125 GB of device memory and 30 GB of host memory")
    vp = np.empty((nz, ny, nx), np.float32)
    vp[:] = np.linspace(2000, 3000, nz, dtype=np.float32)[:, None, None]
    vs, rho = vp / np.float32(1.732), np.full_like(vp, 2000)
    shot = np.array([(nx // 2, ny // 2, nz - 6)])
    recs = shot + np.array([(3 * i, 2 * j, -k) for i in (-2, 0, 2) for j in (0, 3) for k in (0, 5, 8)])
    out = []
    for variant in (4, 3):
        with jv.Context.create(nx, ny, nz, pml, 5.0, 5.0, 5.0, vp, vs, rho, 4e-4, 100.0, nt, kernel_variant=variant,
                               autotune=0) as ctx:
            ctx.set_geometry((shot * 5.0).astype(np.float32), (recs * 5.0).astype(np.float32))
            out.append(ctx.forward(0))
            assert (ctx.kernel_config()["run_chunks"] > 0) == (variant == 4)
    for a, b in zip(*out):
        assert np.abs(b).max() > 0 and rel_l2(a, b) <= 1e-6  # sums of six steps in other orders


@pytest.mark.parametrize("n,pml", [((48, 20, 18), 10), ((32, 28, 24), 8), ((33, 9, 17), 5)])
def test_tile_layout_covers_every_cell(synth, n, pml):
    """jv_forward_noalloc runs the same kernels on rows as short as can be and the cost model's chunks: other row
    offsets, tiles and chunks than a context's, and the same traces bit for bit, of receivers at every cell of two
    planes (one along the layer's edge)."""
    import torch
    from test_zz_no_alloc import _run

    s = synth.small_case(n=n, pml=pml, nt=60, seed=82)
    s.recvs = (np.array([(i, j, k) for k in (0, n[2] // 2) for j in range(n[1]) for i in range(n[0])])
               * np.array([s.dx, s.dy, s.dz])).astype(np.float32)
    with jv.Context.from_survey(s, autotune=0, run_chunks=3) as ctx:
        ref = ctx.forward(0)
    out = torch.full((3, len(s.recvs), s.nt), float("nan"), dtype=torch.float32, device="cuda:0")
    kept = ctypes.c_int(-1)
    assert _run(s, out, kept) == jv.JV_OK and kept.value == len(s.recvs)
    for a, b in zip(out.cpu().numpy(), ref):
        assert np.abs(b).max() > 0 and np.array_equal(a, b)
