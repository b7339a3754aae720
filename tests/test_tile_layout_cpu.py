"""The row layout and the tile kernels' geometry as the library computes them, on the host: the columns of every grid
fall in exactly one tile, pairs start on 8-byte boundaries, and the memory variables of a pair lie in its row."""
import os
import subprocess

import pytest

from conftest import PKG, ROOT

SOURCE = r"""
#include <cstdio>
#include "engine.hpp"
int main() {
    int v[6];
    while (std::scanf("%d %d %d %d %d", v, v + 1, v + 2, v + 3, v + 4) == 5) {
        jv_grid grid{};
        grid.nx = v[0]; grid.ny = v[1]; grid.nz = v[2]; grid.pml = v[3];
        grid.dx = grid.dy = grid.dz = 1.f;
        size_t fe = 0;
        const jv::GridDev g = jv::make_layout(grid, &fe, v[4] != 0);
        long long slabs = 0;
        jv::make_pml_slabs(g, 1, &slabs);
        std::printf("%lld %lld %lld %zu %lld %lld", (long long)g.xoff, (long long)g.sy, (long long)g.sz, fe,
                    jv::tile_psi_floats(g), slabs);
        for (int phy = 0; phy < 2; phy++) {
            const jv::TileGeo q = jv::tile_geometry(g, phy != 0);
            std::printf(" %d %d %d %d %d %d %d %d %d %d %d", q.lo[0], q.hi[0], q.e0, q.ntx, q.nty, q.PX, q.PY, q.W,
                        q.cxl, q.cxh, q.cy);
        }
        std::printf("\n");
    }
}
"""
TILE = ("lo", "hi", "e0", "ntx", "nty", "PX", "PY", "W", "cxl", "cxh", "cy")


@pytest.fixture(scope="module")
def layout(tmp_path_factory):
    d = tmp_path_factory.mktemp("layout")
    cuda, lib, csrc = os.environ.get("CUDA_HOME", "/usr/local/cuda"), os.path.join(ROOT, PKG), os.path.join(ROOT, PKG, "csrc")
    (d / "l.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I", csrc, "-I",
                    os.path.join(cuda, "include"), str(d / "l.cpp"), "-L", lib, "-ljv", "-L",
                    os.path.join(cuda, "lib64"), "-lcudart", f"-Wl,-rpath,{lib}", "-o", str(d / "l")], check=True)

    def run(grids):
        text = "".join("%d %d %d %d %d\n" % g for g in grids)
        out = subprocess.run([str(d / "l")], input=text, capture_output=True, text=True, check=True).stdout
        for line in out.splitlines():
            n = [int(x) for x in line.split()]
            yield n[:6], [dict(zip(TILE, n[6 + 11 * k:])) for k in (0, 1)]
    return run


def _tiles(px, m, xoff):
    """Tiles of a migration step's four updates over gridext and three over gridphy."""
    hi, lo = xoff + px + 2 * m - 2, xoff + 2
    return 4 * -(-(hi - lo // 32 * 32) // 32) + 3 * -(-(xoff + m + px - (xoff + m) // 32 * 32) // 32)


@pytest.mark.parametrize("tight", [0, 1])
@pytest.mark.parametrize("ny,nz", [(8, 8), (17, 300), (400, 400)])
def test_layout_covers_every_cell(layout, ny, nz, tight):
    grids = [(px, ny, nz, m, tight) for m in range(4, 24)
             for px in list(range(8, 76)) + [93, 100, 131, 160, 200, 230, 250, 338, 676]]
    for (px, _, _, m, _), ((xoff, sy, sz, fe, psi, slabs), geo) in zip(grids, layout(grids)):
        nx, NY, NZ = px + 2 * m, ny + 2 * m, nz + 2 * m
        assert (xoff + m) % 4 == 0 and sy % 32 == 0 and sy >= xoff + nx and sz == sy * NY and fe >= sz * NZ + 128
        # the fewest tiles of the offsets whose rows are no longer than with gridphy on a 128-byte line, or whose
        # fields stay below 64 MB
        first, row = -m % 32, lambda xo: -(-(xo + nx) // 32) * 32
        assert _tiles(px, m, xoff) == min(
            _tiles(px, m, xo) for xo in range(first % 4, 32, 4)
            if row(xo) <= row(first) or (not tight and row(xo) * NY * NZ < 1 << 24))
        for q in geo:
            assert q["e0"] % 32 == 0 and q["e0"] <= xoff + q["lo"] < q["e0"] + 32
            seen, cols = set(), {}
            for e in range(q["e0"], q["e0"] + 32 * q["ntx"], 2):
                cells = [c for c in (e - xoff, e - xoff + 1) if q["lo"] <= c < q["hi"]]
                assert not seen & set(cells)
                seen |= set(cells)
                if not cells or q["lo"] != 2:
                    continue
                x = e - xoff
                col = x + q["cy"]
                assert col % 2 == 0 and 0 <= col and col + 1 < q["PY"]
                if any(c < m or c >= m + px for c in cells):
                    xc = x + (q["cxl"] if x < m else q["cxh"])
                    assert xc % 2 == 0 and 0 <= xc and xc + 1 < q["PX"] and xc not in cols
                    cols[xc] = x
            assert seen == set(range(q["lo"], q["hi"]))
            assert q["nty"] * 16 >= (NY - 4 if q["lo"] == 2 else ny) and q["PX"] % 4 == 0 and q["PY"] % 4 == 0
        q = geo[0]
        assert psi == 6 * (q["PX"] * (NY - 4) * (NZ - 4) + q["PY"] * q["W"] * (NZ - 4) + q["PY"] * (NY - 4) * q["W"])
        assert psi <= slabs  # no more than the split kernels', so what fitted the no-allocation scratch still does
