// tile.hpp -- host side of the z-marching tile kernels (tile.cu).
#pragma once

#include "jv_internal.hpp"

namespace jv {

// One updated region and its tiles.
//  - Region: cells [lo, hi) of gridext per axis: the whole of gridext but its
//    two outer cells in the steps with absorbing layers, gridphy in the
//    source reconstruction.
//  - Tiles: 32 columns x 16 rows, the first at element column e0 (a
//    multiple of 32: rows start on 128-byte lines) and row lo[1]; ntx x nty
//    of them, each cut into Q chunks of L planes.  Block b: x tile fastest,
//    then y tile, then chunk, so that neighbours march together and share
//    their halo rows in L2.
//  - Memory variables (set 0 velocity, 1 stress) are axis-major: per axis
//    three arrays over the cells that absorb on that axis: x arrays
//    [t][z-2][y-2][xc] of pitch PX, y arrays [t][z-2][yc][col] and z arrays
//    [t][zc][y-2][col] of pitch PY; W = 2 (m - 2) absorbing indices on an
//    axis.  Columns follow the element index, so a pair is 8-byte aligned
//    for any pml_num: xc = x + cxl below and x + cxh above gridphy, col = x + cy.
struct TileGeo {
    int lo[3], hi[3];
    int e0, ntx, nty, Q, L;
    int PX, PY, W, cxl, cxh, cy;
    float *psx[2][3], *psy[2][3], *psz[2][3];
    const float4 *ax[3];  // per axis and index {K, K_half, alpha, alpha_half}, all 0 outside the layers
    float taps[5][4];  // difference weights by half-order, zero past it
};

// One wavefield's descriptors and launch facts for one region.
struct TileMaps {
    bool ok = false;
    TileGeo geo{};
    FieldMap s[3];          // vx vy vz with their x and y halo (stress)
    FieldMap v[6];          // sxz (x halo), syz (y halo), szz, sxy (both), syy (y), sxx (x)
    FieldMap p;             // sau with both halos
    int qcand[3] = {0, 0, 0};  // the cost model's three best chunk counts, best first
    int *err = nullptr;
};

// the region and tiles over gridext (phy false) or gridphy, and the places of
// the memory variables: everything of a TileGeo that neither a device nor a
// wavefield decides
TileGeo tile_geometry(const GridDev &g, bool phy);
// floats of one wavefield's memory variables (both sets)
long long tile_psi_floats(const GridDev &g);

// Descriptors of wavefield w over gridext (phy false) or gridphy (phy true);
// chunks: 0 for the cost model's choice.  m->ok stays false when the driver
// entry point is missing.  Returns a cudaError_t.
int k_make_tile_maps(const GridDev &g, const WaveDev &w, bool phy, float4 *const ax[3], float *psi, int *err_flag,
                     int chunks, TileMaps *m);

int k_stress_tile(int mode, const GridDev &g, const WaveDev &w, const float *lam, const float *mu, const float *vp,
                  float dt, int rec_w, const float *wavelet, const StepState *st, int it_off, const TileMaps &m,
                  void *stream);
// velocity update without the P-wave velocities (mode kBwd: gridphy, backwards)
int k_vel_tile(int mode, const GridDev &g, const WaveDev &w, const float *bdt, const float *vp, float dt, int rec_w,
               const TileMaps &m, void *stream);
// P-wave velocities over gridphy: of the receiver wavefield r (and nothing
// else, f and img NULL), or of the reconstructed source wavefield f
// backwards in time followed by the imaging condition against r, with r's
// own P-wave update first when r_too is set
int k_pvel_tile(const GridDev &g, const WaveDev *f, const TileMaps *fm, const WaveDev &r, const TileMaps &rm,
                bool r_too, const float *bdt, int rec_w, const ImageDev *img, void *stream);

}  // namespace jv
