"""The tile kernels (variant 4) at the sizes where they can go wrong, through
the C ABI against the FP64 oracle: rows that end just before, on and after a
32-column tile, 16-row tiles with one row or one short of full, odd extents
and absorbing layers (pairs that straddle gridphy's edge and the rim), the
thinnest layer, the source in a tile's corner cells.

Tolerances are those of the other parity tests: traces 2e-5 and images 5e-5
relative L2 (FP32 sums over some hundred time steps)."""
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


def test_tile_layout_covers_every_cell():
    """The columns of every grid fall in exactly one tile, start pairs on
    8-byte boundaries, and the memory variables of a pair lie within their
    row, for the offset make_layout picks (restated)."""
    for m in range(4, 24):
        for px in list(range(8, 76)) + [100, 160, 200, 338, 676]:
            nx = px + 2 * m
            tiles = lambda xo: (4 * ((xo + nx - 2 - (xo + 2) // 32 * 32 + 31) // 32)
                                + 3 * ((xo + m + px - (xo + m) // 32 * 32 + 31) // 32))
            x0 = (32 - m % 32) % 32
            xoff = x0
            for xo in range(x0 % 4, 32, 4):
                if tiles(xo) < tiles(xoff):
                    xoff = xo
            assert (xoff + m) % 4 == 0
            xl = (xoff + 2) & ~1
            wl = ((xoff + m + 1) & ~1) - xl
            xh = (xoff + m + px) & ~1
            wh = ((xoff + nx - 1) & ~1) - xh
            wy = ((xoff + nx - 1) & ~1) - xl
            for lo, hi in ((2, nx - 2), (m, m + px)):
                e0 = (xoff + lo) // 32 * 32
                seen = set()
                for e in range(e0, e0 + (xoff + hi - e0 + 31) // 32 * 32, 2):
                    x = e - xoff
                    cells = [c for c in (x, x + 1) if lo <= c < hi]
                    assert not seen & set(cells)
                    seen |= set(cells)
                    if not cells or lo != 2:
                        continue
                    col = e - xl
                    assert col % 2 == 0 and 0 <= col and col + 1 < wy
                    if any(c < m or c >= m + px for c in cells):
                        xc = e - xl if x < m else wl + e - xh
                        assert xc % 2 == 0 and (0 <= xc < wl if x < m else wl <= xc < wl + wh)
                assert seen == set(range(lo, hi))
