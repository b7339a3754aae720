// tile.cu -- z-marching tile kernels of the time loops (kernel variant 4).
//
// Every stencil update of a time step runs in one of three kernels over x/y
// tiles: the stress update, the velocity update, and the P-wave velocities
// with the imaging condition.  The first two cover the whole of gridext in
// the steps that carry absorbing layers (8th order in gridphy, 4th order
// with C-PML memory variables elsewhere) and gridphy with the rtm_backward
// rim orders in the source reconstruction.  Reference (FD =
// src/jarvis_cpp/jarvis/.jarvis_2_app/.jarvis_3_seismology/
// elastic_1_fdtd3d_model_mpi, RTM = .../elastic_1_rtm3d_model_mpi):
//   interior velocity   FD/fdtd3d_2_phy_mpi_module/fdtd3d_phy_mpi_2_vel_kernel.hpp:7-2088
//   interior stress     FD/fdtd3d_2_phy_mpi_module/fdtd3d_phy_mpi_3_stress_kernel.hpp:7-1364
//   CPML                FD/fdtd3d_1_cpml_mpi_module/fdtd3d_cpml_mpi_2_kernel_device_{x,y,z}_meat.hpp
//   damping profile     FD/fdtd3d_1_cpml_mpi_module/fdtd3d_cpml_mpi_1_host_meat.hpp:147-620
//   imaging             RTM/rtm3d_0_image_module/rtm3d_iamge_kernel.hpp:6-51
//
// Shape.  Eight warps own a tile of 32 x 16 cells, one x pair per thread, and
// march it through a chunk of z planes.  x and y neighbours come from shared
// memory, where TMA brings each plane of the differenced fields with its
// 4-cell halo.  A field that is also differenced in z arrives four planes
// ahead, so that the planes above are read from the same buffers and only the
// three or four planes below are carried in registers.  What a cell reads
// alone (model, the updated fields) goes straight to registers, behind an L2
// prefetch a plane ahead.  A warp gives a plane back with one arrival once its
// differences are taken and runs on; nothing in the loop waits for the slowest
// warp of the block, and two blocks share an SM.
//
// Cells of the absorbing layers take the same 8-tap differences with their
// outer two weights zero, so a warp that holds both kinds does not run two
// paths; the memory variables and the rounding of the sums are branches.
//
// What bounds them, 200^3 + 20 (us, and GB/s of arrays read and written once;
// a copy moves 6460): with absorbing layers instruction issue, 0.5 a cycle and
// scheduler -- stress 272 (4280), velocity 237 (3590), against 259 and 227 for
// the persistent kernels of one CTA an SM that they replaced, with a separate
// launch for wide or odd grids; over gridphy DRAM latency -- imaging with
// P-wave velocities 192 (5160), backward stress 133 (4590), backward velocity
// 113 (3690), against 250 for imaging with the backward velocity update, 147
// for the backward stress and 147 + 124 for the receivers' velocity update and
// its layers.  The 200^3 migration gains 3 %, small, odd and wide grids 10 to
// 100 %.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <utility>

#include "damping.hpp"
#include "jv_internal.hpp"
#include "tile.hpp"
#include "tma.cuh"

namespace jv {

namespace {

constexpr int kTX = 32, kTY = 16;             // cells of a tile
constexpr int kThreads = kTX * kTY / 2;       // one pair of cells a thread
constexpr int kAhead = 1;  // planes the L2 prefetch of the pointwise rows runs ahead (2: 1394, 3: 1428 against 1377 us)
constexpr int kDepth = 2;  // planes in flight or in use ahead of the four that the z differences hold (3: less L1, 0-5 % slower)
constexpr int kHalo = 4;
constexpr int kPW = kTX + 2 * kHalo, kPH = kTY + 2 * kHalo;

// ------------------------------------------------ pairs of floats
//
// An x pair in one 64-bit register: the y and z differences and the updates
// are packed two-wide instructions (half the issue slots of scalar ones).
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void up(f2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return fma2(b, pk(-1.f, -1.f), a); }
__device__ __forceinline__ f2 dup(float a) { return pk(a, a); }

__device__ __forceinline__ f2 at2(const float *p) { return *reinterpret_cast<const f2 *>(p); }
__device__ __forceinline__ f2 lds2(uint32_t a) {
    f2 r;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(r) : "r"(a));
    return r;
}
// a pair at byte offset o of an array (32-bit offsets, for arrays below 4 GB,
// gave the same times within 0.1 % from 32^3 to 676 x 676 x 210)
__device__ __forceinline__ f2 get2(const float *p, uint64_t o) {
    return *reinterpret_cast<const f2 *>(reinterpret_cast<const char *>(p) + o);
}
__device__ __forceinline__ f2 &ref2(float *p, uint64_t o) {
    return *reinterpret_cast<f2 *>(reinterpret_cast<char *>(p) + o);
}
// store the cells of N pairs that the update covers (bit c of mask: cell c)
template <int N>
__device__ __forceinline__ void put2(float *const (&p)[N], const f2 (&v)[N], uint64_t o, int mask) {
    if (mask == 3) {
#pragma unroll
        for (int j = 0; j < N; j++) ref2(p[j], o) = v[j];
    } else if (mask) {
#pragma unroll
        for (int j = 0; j < N; j++) {
            float a, b;
            up(v[j], a, b);
            float *q = reinterpret_cast<float *>(&ref2(p[j], o));
            q[mask == 2] = mask == 2 ? b : a;
        }
    }
}
// from global to shared memory, by the thread (or warp) that will read it
__device__ __forceinline__ void copy8(uint32_t dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy16(uint32_t dst, const float4 *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the last committed group have landed
__device__ __forceinline__ void copy_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void prefetch_line(const float *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// ------------------------------------------------ differences
//
// Dp f = sum_q c_q (f[i+(q+1)s] - f[i-qs]);  Dm f = sum_q c_q (f[i+qs] - f[i-(q+1)s])
// in cells of the grid (callers multiply by 1 / spacing).  Single cells of an
// image are differences of nearly equal numbers, where one rounding more or
// another order shows at 1 %; so the rounding here and in the sums of
// differences is fixed, and a test pins it bit for bit.  gridphy sums its four
// terms from q = 0 on, an absorbing layer its two from q = 1 on: with AB
// (kernels that run in layers) the term q = 0 has a weight at either end of
// the chain, C[0] and C[4], one of them zero.

// along x, at the pair F[0..1] of a row in shared memory; C: the weights of
// the two cells; mid: the pair itself
template <bool PLUS, bool AB>
__device__ __forceinline__ f2 diff_x(const float *F, const f2 *C, f2 &mid) {
    float e[10];
    mid = at2(F);
#pragma unroll
    for (int j = 0; j < 5; j++) up(j == 2 ? mid : at2(F - 4 + 2 * j), e[2 * j], e[2 * j + 1]);
    constexpr int o = PLUS ? 5 : 4;
    const f2 d0 = pk(e[o] - e[o - 1], e[o + 1] - e[o]);
    f2 t = mul2(C[0], d0);
#pragma unroll
    for (int q = 1; q < 4; q++) t = fma2(C[q], pk(e[o + q] - e[o - 1 - q], e[o + 1 + q] - e[o - q]), t);
    return AB ? fma2(C[4], d0, t) : t;
}
// along y: rows PITCH floats apart
template <bool PLUS, bool AB, int PITCH>
__device__ __forceinline__ f2 diff_y(const float *F, const f2 *C) {
    constexpr int o = PLUS ? 1 : 0;
    const f2 d0 = sub2(at2(F + o * PITCH), at2(F - (1 - o) * PITCH));
    f2 t = mul2(C[0], d0);
#pragma unroll
    for (int q = 1; q < 4; q++) t = fma2(C[q], sub2(at2(F + (q + o) * PITCH), at2(F - (q + 1 - o) * PITCH)), t);
    return AB ? fma2(C[4], d0, t) : t;
}
// along z: mid is this plane's pair, F the field's place in a buffer and off
// the buffers of this plane and the four above; w the pairs of the planes
// below, oldest first (three of them with PLUS, else four), which move on
template <bool PLUS, bool AB>
__device__ __forceinline__ f2 diff_z(const float *F, const int off[5], f2 mid, f2 *w, const f2 *C) {
    f2 d0, t;
    if (PLUS) {
        d0 = sub2(at2(F + off[1]), mid);
        t = mul2(C[0], d0);
        t = fma2(C[1], sub2(at2(F + off[2]), w[2]), t);
        t = fma2(C[2], sub2(at2(F + off[3]), w[1]), t);
        t = fma2(C[3], sub2(at2(F + off[4]), w[0]), t);
        w[0] = w[1];
        w[1] = w[2];
        w[2] = mid;
    } else {
        d0 = sub2(mid, w[3]);
        t = mul2(C[0], d0);
        t = fma2(C[1], sub2(at2(F + off[1]), w[2]), t);
        t = fma2(C[2], sub2(at2(F + off[2]), w[1]), t);
        t = fma2(C[3], sub2(at2(F + off[3]), w[0]), t);
        w[0] = w[1];
        w[1] = w[2];
        w[2] = w[3];
        w[3] = mid;
    }
    return AB ? fma2(C[4], d0, t) : t;
}
// weights of the two cells of a pair; p0, p1: whether they lie in gridphy
__device__ __forceinline__ void set_weights(f2 C[5], bool p0, bool p1, const TileGeo &q) {
    C[0] = pk(p0 ? q.taps[4][0] : 0.f, p1 ? q.taps[4][0] : 0.f);
    C[4] = pk(p0 ? 0.f : q.taps[2][0], p1 ? 0.f : q.taps[2][0]);
#pragma unroll
    for (int j = 1; j < 4; j++) C[j] = pk(p0 ? q.taps[4][j] : q.taps[2][j], p1 ? q.taps[4][j] : q.taps[2][j]);
}
// Adding a difference t to another one: in gridphy one fused multiply-add, t r
// + sum with r = 1 / spacing; in a layer t r is rounded first, for its memory
// variable, and then added.  (t S) R + sum serves a pair with a cell of
// either kind: S = 1 and R = r, or S = r and R = 1.  Pairs of gridphy, most of
// them, take the fused form from a branch of their own: with S and R kept in
// registers for all pairs the stress update ran at 275 against 264 us
// (200^3 + 20), short of registers.
struct Join {
    f2 S, R;
    __device__ __forceinline__ Join(bool p0, bool p1, float r)
        : S(pk(p0 ? 1.f : r, p1 ? 1.f : r)), R(pk(p0 ? r : 1.f, p1 ? r : 1.f)) {}
};

// Order of one axis in the rtm_backward rim: within 4 cells of a gridphy
// face the order drops to e+1 (e = distance to the face) but never below
// rec_width (FD/fdtd3d_2_phy_mpi_module/fdtd3d_phy_mpi_2_vel_kernel.hpp:132-152,240-261).
__device__ __forceinline__ int rim_order(int p, int np, int w) {
    const int e = min(p, np - 1 - p);
    return e >= kPhyHalf ? kPhyHalf : max(e + 1, w);
}

// ------------------------------------------------ absorbing layers
//
// damping of a pair; a cell that does not absorb has K and alpha zero
__device__ __forceinline__ void damping(f2 vp, f2 K, f2 alpha, f2 dt, f2 &A, f2 &B) {
    float v0, v1, k0, k1, l0, l1, t0, t1, a0, a1, b0, b1;
    up(vp, v0, v1);
    up(K, k0, k1);
    up(alpha, l0, l1);
    up(dt, t0, t1);
    damping_ab(v0, k0, l0, t0, a0, b0);
    damping_ab(v1, k1, l1, t1, a1, b1);
    A = pk(a0, a1);
    B = pk(b0, b1);
}

// the thread's place in its tile
struct Place {
    int X0, Y0, z0, n;  // element column, row and plane of the tile's first cell; planes
    int r, c;           // row; the pair's column
    int x, y;           // gridext cell of the pair's first cell
    int mask, i0;       // cells of the pair that are updated; element index in plane z0
    int rows, nlive;    // rows of the tile; warps that have some
    __device__ __forceinline__ Place(const GridDev &g, const TileGeo &q) {
        const int b = blockIdx.x;
        const int xt = b % q.ntx, t = b / q.ntx, yt = t % q.nty, o = t / q.nty;
        // the two chunks with absorbing planes first: they are the longest
        const int ch = o == 1 && q.Q > 1 ? q.Q - 1 : o > 1 ? o - 1 : 0;
        X0 = q.e0 + xt * kTX;
        Y0 = q.lo[1] + yt * kTY;
        z0 = q.lo[2] + ch * q.L;
        n = min(q.L, q.hi[2] - z0);
        rows = min(kTY, q.hi[1] - Y0);
        nlive = (rows + 1) / 2;
        r = threadIdx.x / (kTX / 2);
        c = 2 * (threadIdx.x % (kTX / 2));
        x = X0 + c - (int)g.xoff;
        y = Y0 + r;
        mask = 0;
        if (r < rows) mask = (x >= q.lo[0] && x < q.hi[0] ? 1 : 0) | (x + 1 >= q.lo[0] && x + 1 < q.hi[0] ? 2 : 0);
        // a thread without cells reads along at the nearest pair that has some, and stores nothing
        const int ec = min(max(X0 + c, ((int)g.xoff + q.lo[0]) & ~1), ((int)g.xoff + q.hi[0] - 1) & ~1);
        i0 = ec + (int)g.sy * min(y, q.hi[1] - 1) + (int)g.sz * z0;
    }
    // the two rows of a warp start here in plane z0: two lanes an array prefetch them
    __device__ __forceinline__ int line(const GridDev &g, const TileGeo &q) const {
        const int row = Y0 + 2 * (threadIdx.x >> 5) + (threadIdx.x & 1);
        return X0 + (int)g.sy * min(row, q.hi[1] - 1) + (int)g.sz * z0;
    }
};

// The planes of a block's march.  Event e delivers plane e + 4 of the fields
// differenced in z (buffers A, four deeper than B) and plane e of the others
// (buffers B) under one barrier; events -4 .. -1 only the former.  Plane k
// is given back by one arrival of each live warp, its lanes' reads fenced
// against the copies that follow, and event e waits for plane e - D: D planes
// are in flight or in use ahead of the four.
template <int A_FLOATS, int B_FLOATS, int DEPTH>
struct Flow {
    static constexpr int D = DEPTH, SA = DEPTH + 4;
    static constexpr int a0 = 0, b0 = SA * A_FLOATS, floats = b0 + DEPTH * B_FLOATS;
    uint32_t bars;  // full[SA], empty[D]
    __device__ __forceinline__ uint32_t full(int p) const { return bars + 8u * (uint32_t)(p % SA); }
    __device__ __forceinline__ uint32_t empty(int k) const { return bars + 8u * (uint32_t)(SA + k % D); }
    __device__ __forceinline__ void init(int nlive) const {
        for (int s = 0; s < SA; s++) mbar_init(bars + 8u * s, 1);
        for (int s = 0; s < D; s++) mbar_init(bars + 8u * (SA + s), nlive);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // one lane: the copies of plane p of the A fields and plane p - 4 of the B
    // fields (la and lb start one plane's)
    template <class LA, class LB>
    __device__ __forceinline__ void issue(float *sm, int p, LA la, LB lb) const {
        mbar_expect(full(p), 4u * (uint32_t)(A_FLOATS + (p >= 4 ? B_FLOATS : 0)));
        la(p, sm + a0 + (p % SA) * A_FLOATS, full(p));
        if (B_FLOATS && p >= 4) lb(p - 4, sm + b0 + ((p + D - 4) % D) * B_FLOATS, full(p));
    }
    // the same lane, before it leaves: no copy is in flight when the block
    // ends, whatever became of its readers (p: the next plane it would issue)
    __device__ __forceinline__ void drain(int p) const {
        for (int j = max(0, p - SA); j < p; j++) mbar_wait_bounded(full(j), (uint32_t)((j / SA) & 1));
    }
};
// A reader's side of it: the buffers of plane k and the four above.
template <class F>
struct Reader {
    F flow;
    int off[5];    // of plane k .. k + 4 (floats from the first A buffer)
    int s, par;    // buffer and phase of plane k + 4
    int b;         // B buffer of plane k
    // waits for planes 0 .. 3; false when one did not arrive in time
    __device__ __forceinline__ bool start(const F &f, int afloats) {
        flow = f;
        bool ok = true;
        for (int p = 0; p < 4; p++) ok = ok && mbar_wait_bounded(f.full(p), 0);
#pragma unroll
        for (int j = 0; j < 5; j++) off[j] = j * afloats;
        s = 4;
        par = 0;
        b = 0;
        return __all_sync(0xffffffffu, ok);
    }
    __device__ __forceinline__ bool wait() const {
        return __all_sync(0xffffffffu, mbar_wait_bounded(flow.bars + 8u * s, (uint32_t)par));
    }
    __device__ __forceinline__ void release() const {
        reads_before_bulk_copies();
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(flow.bars + 8u * (F::SA + b));
    }
    __device__ __forceinline__ void next(int afloats) {
#pragma unroll
        for (int j = 0; j < 4; j++) off[j] = off[j + 1];
        if (++s == F::SA) {
            s = 0;
            par ^= 1;
        }
        off[4] = s * afloats;
        if (++b == F::D) b = 0;
    }
};

// What the absorbing layers add to the item of one thread, set SET of the
// memory-variable layout: its memory variables and vp are copied to the
// thread's own slots in shared memory, and the damping row of the plane to
// its warp's, while the item before it runs (nothing is synchronised but
// the warp); the damping rows of the tile's columns and rows are there from
// the start.
template <int SET>
struct Psi {
    int ox, oy, oz;  // the pair's place in an x, y and z array, plane 0 (z: absorbing plane 0)
    int px, py, pz;  // floats of one plane of them
    uint32_t slot;   // the thread's first slot: vp, then three of each axis; two sets
    float4 *tab;     // damping rows: columns and rows of the tile; planes, two sets by warp
    static constexpr uint32_t kStep = 8u * kThreads, kSet = 10u * kStep;
    static constexpr int kRows = kTX + kTY, kZ = kThreads / 32;
    static constexpr uint32_t kTab = 2u * kSet, kBytes = kTab + 16u * (kRows + 2 * kZ);
    __device__ __forceinline__ Psi(const GridDev &g, const TileGeo &q, const Place &t, float *sm) {
        const int x = t.x, y = t.y;
        px = (g.ny - 4) * q.PX;
        py = q.W * q.PY;
        pz = (g.ny - 4) * q.PY;
        ox = (y - 2) * q.PX + x + (x < g.m ? q.cxl : q.cxh);
        oy = (y < g.m ? y - 2 : y - g.py - 2) * q.PY + x + q.cy;
        oz = (y - 2) * q.PY + x + q.cy;
        slot = smem_u32(sm) + 8u * threadIdx.x;
        tab = reinterpret_cast<float4 *>(reinterpret_cast<char *>(sm) + kTab);
    }
    // before a barrier of the block; rows outside gridext are never used
    __device__ __forceinline__ void fill(const GridDev &g, const TileGeo &q, const Place &t) const {
        const int i = threadIdx.x;
        if (i < kTX) {
            const int x = t.X0 + i - (int)g.xoff;
            tab[i] = x >= 0 && x < g.nx ? q.ax[0][x] : make_float4(0.f, 0.f, 0.f, 0.f);
        } else if (i < kRows) {
            tab[i] = q.ax[1][min(t.Y0 + i - kTX, g.ny - 1)];
        }
    }
    __device__ __forceinline__ int ix(int z) const { return ox + (z - 2) * px; }
    __device__ __forceinline__ int iy(int z) const { return oy + (z - 2) * py; }
    __device__ __forceinline__ int iz(const GridDev &g, int z) const { return oz + (z < g.m ? z - 2 : z - g.pz - 2) * pz; }
    __device__ __forceinline__ float4 &zrow(int s) const { return tab[kRows + s * kZ + (threadIdx.x >> 5)]; }
    __device__ __forceinline__ void fetch3(uint32_t d, float *const p[3], int i) const {
#pragma unroll
        for (int a = 0; a < 3; a++)
            copy8(d + a * kStep, reinterpret_cast<const float *>(&ref2(p[a], 4ull * (uint32_t)i)));
    }
    // start the copies of plane z into set s; o: the pair's byte offset in that plane
    __device__ __forceinline__ void fetch(const GridDev &g, const TileGeo &q, const float *vpm, uint64_t o, int z, int s,
                                          bool live, bool xab, bool yab, bool zab) const {
        const uint32_t d = slot + (uint32_t)s * kSet;
        if (xab || yab || (zab && live)) copy8(d, reinterpret_cast<const float *>(reinterpret_cast<const char *>(vpm) + o));
        if (xab) fetch3(d + kStep, q.psx[SET], ix(z));
        if (yab) fetch3(d + 4 * kStep, q.psy[SET], iy(z));
        if (zab) {
            if (live) fetch3(d + 7 * kStep, q.psz[SET], iz(g, z));
            if ((threadIdx.x & 31) == 0) copy16(smem_u32(&zrow(s)), q.ax[2] + z);
        }
    }
    __device__ __forceinline__ f2 vp(int s) const { return lds2(slot + (uint32_t)s * kSet); }
    __device__ __forceinline__ uint32_t at(int s, int a) const { return slot + (uint32_t)s * kSet + (uint32_t)a * kStep; }
};

// One absorbing axis of a pair: the three memory variables (from d on in
// shared memory, element i of the arrays p) and the differences they are
// added to, the normal one (n) first.  The nodes are the integer one for the
// normal difference and the half one for the others in the stress update,
// the other way round in the velocity update (HALF_N).
template <bool HALF_N>
__device__ __forceinline__ void absorb3(uint32_t d, float *const p[3], int i, f2 vp, f2 dt, f2 K, f2 Kh, f2 al, f2 alh,
                                        f2 &n, f2 &a, f2 &b) {
    constexpr uint32_t st = 8u * kThreads;
    const uint64_t o = 4ull * (uint32_t)i;
    f2 A, B;
    damping(vp, HALF_N ? Kh : K, HALF_N ? alh : al, dt, A, B);
    f2 v = fma2(B, lds2(d), mul2(A, n));
    ref2(p[0], o) = v;
    n = add2(n, v);
    damping(vp, HALF_N ? K : Kh, HALF_N ? al : alh, dt, A, B);
    v = fma2(B, lds2(d + st), mul2(A, a));
    ref2(p[1], o) = v;
    a = add2(a, v);
    v = fma2(B, lds2(d + 2 * st), mul2(A, b));
    ref2(p[2], o) = v;
    b = add2(b, v);
}
// x: a damping row for each cell
template <bool HALF_N>
__device__ __forceinline__ void absorb_x(uint32_t d, float *const p[3], int i, const float4 &t, const float4 &u, f2 vp, f2 dt,
                                         f2 &n, f2 &a, f2 &b) {
    absorb3<HALF_N>(d, p, i, vp, dt, pk(t.x, u.x), pk(t.y, u.y), pk(t.z, u.z), pk(t.w, u.w), n, a, b);
}
// y and z: one for both
template <bool HALF_N>
__device__ __forceinline__ void absorb_yz(uint32_t d, float *const p[3], int i, const float4 &t, f2 vp, f2 dt, f2 &n, f2 &a,
                                          f2 &b) {
    absorb3<HALF_N>(d, p, i, vp, dt, dup(t.x), dup(t.y), dup(t.z), dup(t.w), n, a, b);
}

// ------------------------------------------------ stress

struct StressMaps {
    CUtensorMap v[3];
};
constexpr int kSField = kPW * kPH;  // one field's plane
using StressFlow = Flow<3 * kSField, 0, kDepth>;

// MODE kFwd, kRtmFwd, kRev: gridext with its absorbing layers; kBwd: gridphy
// with the rim orders, backwards in time (dt < 0, the source subtracted).
template <int MODE>
__global__ void __launch_bounds__(kThreads, 2)
    stress_tile(GridDev g, const __grid_constant__ StressMaps maps, const __grid_constant__ WaveDev w,
                const float *__restrict__ lam, const float *__restrict__ mu, const float *__restrict__ vpm, float dt,
                int rec_w, const float *__restrict__ wavelet, const StepState *__restrict__ st, int it_off,
                const __grid_constant__ TileGeo q, int *err) {
    using FL = StressFlow;
    constexpr bool kCp = MODE != kBwd, kSau = MODE != kFwd;
    constexpr int AF = 3 * kSField;
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(8) uint64_t bars[FL::SA + FL::D];
    __shared__ f2 rows[5][4];  // the difference weights of every order, as pairs
    const Place t(g, q);
    if (t.n <= 0) return;
    const int tid = threadIdx.x;
    const FL flow{smem_u32(bars)};
    const Psi<1> psi(g, q, t, sm + FL::floats);
    if (tid == 0) flow.init(t.nlive);
    if (!kCp && tid < 20) rows[tid / 4][tid % 4] = dup(q.taps[tid / 4][tid % 4]);
    if (kCp) psi.fill(g, q, t);
    __syncthreads();
    if ((tid >> 5) >= t.nlive) return;
    auto la = [&](int p, float *buf, uint32_t bar) {
        for (int f = 0; f < 3; f++)
            tma_load_3d(smem_u32(buf + f * kSField), &maps.v[f], t.X0 - kHalo, t.Y0 - kHalo, t.z0 + p, bar);
    };
    auto lb = [](int, float *, uint32_t) {};
    int next = 0;  // the next plane to issue (thread 0)
    if (tid == 0)
        for (; next < min(t.n, FL::D) + 4; next++) flow.issue(sm, next, la, lb);
    const int sz = (int)g.sz, m = g.m;
    const bool live = t.mask != 0;
    f2 wx[3], wy[3], wz[4];  // the planes below, of vx, vy, vz
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const bool in = t.z0 + j >= 4;
        const int i = t.i0 + (j - 4) * sz;
        if (j) wx[j - 1] = in ? at2(w.f[VX] + i) : 0ull;
        if (j) wy[j - 1] = in ? at2(w.f[VY] + i) : 0ull;
        wz[j] = in ? at2(w.f[VZ] + i) : 0ull;
    }
    const float *pf = nullptr;  // the row this lane prefetches
    {
        const int a = (tid & 31) >> 1;
        if (a < 2) pf = a == 0 ? lam : mu;
        else if (a < (kSau ? 9 : 8)) pf = w.f[SXX + a - 2];
        if (pf) pf += t.line(g, q) + kAhead * sz;
    }
    const f2 rdx = dup(1.0f / g.dx), rdy = dup(1.0f / g.dy), rdz = dup(1.0f / g.dz), dt2 = dup(dt);
    const bool ph0 = t.x >= m && t.x < m + g.px, ph1 = t.x + 1 >= m && t.x + 1 < m + g.px;
    const bool yph = t.y >= m && t.y < m + g.py;
    const bool xab = kCp && ((t.mask & 1 && !ph0) || (t.mask & 2 && !ph1)), yab = kCp && live && !yph;
    auto zabs = [&](int z) { return z < m || z >= m + g.pz; };
    if (kCp) {
        psi.fetch(g, q, vpm, 4ull * (uint32_t)t.i0, t.z0, 0, live, xab, yab, zabs(t.z0));
        copy_commit();
    }
    int zclass = -1;  // whether the weights are those of a plane of gridphy
    f2 cx[5];
    if (!kCp) {
        const int o0 = rim_order(min(max(t.x - m, 0), g.px - 1), g.px, rec_w);
        const int o1 = rim_order(min(max(t.x + 1 - m, 0), g.px - 1), g.px, rec_w);
#pragma unroll
        for (int j = 0; j < 4; j++) cx[j] = pk(q.taps[o0][j], q.taps[o1][j]);
    }
    // the item that holds the source, if it lies in this thread's pair
    int src_k = -1, src_c = 0;
    if (MODE != kRev && live) {
        const long long d = st->src - t.i0;
        const long long k = d >= 0 ? d / sz : -1;
        if (k >= 0 && k < t.n && d - k * sz < 2 && (t.mask >> (int)(d - k * sz)) & 1) {
            src_k = (int)k;
            src_c = (int)(d - k * sz);
        }
    }
    Reader<FL> rd;
    bool ok = rd.start(flow, AF);
    const float *S = sm + (t.r + kHalo) * kPW + t.c + kHalo;  // the pair in a buffer's first field
#pragma unroll 1
    for (int k = 0; k < t.n && ok; k++) {
        // opaque to the compiler, which would otherwise keep a running pointer per array
        uint64_t o = 4ull * (uint32_t)(t.i0 + k * sz);
        int z = t.z0 + k;
        asm volatile("" : "+l"(o), "+r"(z));
        const f2 pl = get2(lam, o), pm = get2(mu, o);
        f2 ps[7];
#pragma unroll
        for (int f = 0; f < (kSau ? 7 : 6); f++) ps[f] = get2(w.f[SXX + f], o);
        if (kCp) {
            __syncwarp();  // the set to be filled has been read
            if (k + 1 < t.n) psi.fetch(g, q, vpm, o + 4ull * (uint32_t)sz, z + 1, (k + 1) & 1, live, xab, yab, zabs(z + 1));
            copy_commit();
        }
        if (pf && k + kAhead < t.n) prefetch_line(pf + (long long)k * sz);
        ok = rd.wait();
        if (!ok) break;
        const bool zph = !zabs(z), p0 = ph0 && yph && zph, p1 = ph1 && yph && zph;
        const bool ab = kCp && !(p0 && p1);  // a cell of the pair lies in a layer
        f2 vp = 0;
        if (kCp) {
            if (zclass != (int)zph) {
                zclass = zph;
                set_weights(cx, p0, p1, q);
            }
            copy_wait1();
            __syncwarp();
            if (xab || yab || !zph) vp = psi.vp(k & 1);
        }
        const float *F = S + rd.off[0];
        // normal differences Nx = d vx/dx, ...; shear sums Sxy = d vy/dx + d vx/dy, ...
        f2 mx, my, mz;
        f2 Nx = mul2(diff_x<false, kCp>(F, cx, mx), rdx);
        f2 Sxy = diff_x<true, kCp>(F + kSField, cx, my);
        f2 Sxz = diff_x<true, kCp>(F + 2 * kSField, cx, mz);
        if (ab) {
            const Join jx(p0, p1, 1.0f / g.dx);
            Sxy = mul2(Sxy, jx.S);
            Sxz = mul2(Sxz, jx.S);
            if (xab)
                absorb_x<false>(psi.at(k & 1, 1), q.psx[1], psi.ix(z), psi.tab[t.c], psi.tab[t.c + 1], vp, dt2, Nx, Sxy, Sxz);
        }
        f2 Ny, Syz;
        {
            f2 cy[5];
#pragma unroll
            for (int j = 0; j < (kCp ? 5 : 4); j++) cy[j] = kCp ? cx[j] : rows[rim_order(t.y - m, g.py, rec_w)][j];
            Ny = mul2(diff_y<false, kCp, kPW>(F + kSField, cy), rdy);
            f2 a = mul2(diff_y<true, kCp, kPW>(F, cy), rdy);
            Syz = diff_y<true, kCp, kPW>(F + 2 * kSField, cy);
            if (ab) {
                Syz = mul2(Syz, Join(p0, p1, 1.0f / g.dy).S);
                if (yab)
                    absorb_yz<false>(psi.at(k & 1, 4), q.psy[1], psi.iy(z), psi.tab[kTX + t.r], vp, dt2, Ny, a, Syz);
                Sxy = fma2(Sxy, Join(p0, p1, 1.0f / g.dx).R, a);
            } else {
                Sxy = fma2(Sxy, rdx, a);
            }
        }
        f2 cz[5];
#pragma unroll
        for (int j = 0; j < (kCp ? 5 : 4); j++) cz[j] = kCp ? cx[j] : rows[rim_order(z - m, g.pz, rec_w)][j];
        f2 Nz = mul2(diff_z<false, kCp>(S + 2 * kSField, rd.off, mz, wz, cz), rdz);
        f2 a = mul2(diff_z<true, kCp>(S, rd.off, mx, wx, cz), rdz);
        f2 b = mul2(diff_z<true, kCp>(S + kSField, rd.off, my, wy, cz), rdz);
        rd.release();
        rd.next(AF);
        if (ab) {
            if (live && !zph)
                absorb_yz<false>(psi.at(k & 1, 7), q.psz[1], psi.iz(g, z), psi.zrow(k & 1), vp, dt2, Nz, a, b);
            Sxz = fma2(Sxz, Join(p0, p1, 1.0f / g.dx).R, a);
            Syz = fma2(Syz, Join(p0, p1, 1.0f / g.dy).R, b);
        } else {
            Sxz = fma2(Sxz, rdx, a);
            Syz = fma2(Syz, rdy, b);
        }
        if (MODE != kRev && k == src_k) {
            // explosive source, applied before the stress update of step it
            // (FD/fdtd3d_2_phy_mpi_module/fdtd3d_phy_mpi_3_stress_kernel.hpp:1308-1364)
            const float v = wavelet[st->it + it_off];
            const float sv = MODE == kBwd ? -v : v;
            const f2 s2 = src_c == 0 ? pk(sv, 0.f) : pk(0.f, sv);
#pragma unroll
            for (int f = 0; f < 3; f++) ps[f] = add2(ps[f], s2);
        }
        const f2 l2m = fma2(pm, dup(2.0f), pl), dm = mul2(dt2, pm);
        f2 v[kSau ? 7 : 6];
        v[0] = fma2(dt2, fma2(pl, Nz, fma2(l2m, Nx, mul2(pl, Ny))), ps[0]);
        v[1] = fma2(dt2, fma2(pl, Nz, fma2(pl, Nx, mul2(l2m, Ny))), ps[1]);
        v[2] = fma2(dt2, fma2(l2m, Nz, fma2(pl, Nx, mul2(pl, Ny))), ps[2]);
        v[3] = fma2(dm, Sxy, ps[3]);
        v[4] = fma2(dm, Sxz, ps[4]);
        v[5] = fma2(dm, Syz, ps[5]);
        if constexpr (kSau) {
            v[6] = fma2(mul2(dt2, l2m), add2(add2(Nx, Ny), Nz), ps[6]);
            float *const dst[7] = {w.f[SXX], w.f[SYY], w.f[SZZ], w.f[SXY], w.f[SXZ], w.f[SYZ], w.f[SAU]};
            put2(dst, v, o, t.mask);
        } else {
            float *const dst[6] = {w.f[SXX], w.f[SYY], w.f[SZZ], w.f[SXY], w.f[SXZ], w.f[SYZ]};
            put2(dst, v, o, t.mask);
        }
        // the first warp refills what every live warp has given back
        if (tid < 32 && k + FL::D < t.n) {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(flow.empty(k), (uint32_t)((k / FL::D) & 1)));
            if (tid == 0 && ok) flow.issue(sm, next++, la, lb);
        }
    }
    if (!ok) atomicExch(err, 1);
    if (tid == 0) flow.drain(next);
}

// ------------------------------------------------ velocity

struct VelMaps {
    CUtensorMap f[6];  // sxz (x halo), syz (y halo), szz | sxy (both), syy (y), sxx (x)
};
// A buffers: sxz, syz, szz; B buffers: sxy, syy, sxx
constexpr int kVsyz = kPW * kTY, kVszz = kVsyz + kTX * kPH, kVA = kVszz + kTX * kTY;
constexpr int kVsyy = kPW * kPH, kVsxx = kVsyy + kTX * kPH, kVB = kVsxx + kPW * kTY;
using VelFlow = Flow<kVA, kVB, kDepth>;

// MODE kFwd, kRev: gridext with its absorbing layers; kBwd: gridphy with the
// rim orders, backwards in time.  Of the three differences of a velocity, kFwd
// rounds the x term and joins y, then z; the others round y and join x, then z.
template <int MODE>
__global__ void __launch_bounds__(kThreads, 2)
    vel_tile(GridDev g, const __grid_constant__ VelMaps maps, const __grid_constant__ WaveDev w,
             const float *__restrict__ bdt, const float *__restrict__ vpm, float dt, int rec_w,
             const __grid_constant__ TileGeo q, int *err) {
    using FL = VelFlow;
    constexpr bool kCp = MODE != kBwd, kXFirst = MODE == kFwd;
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(8) uint64_t bars[FL::SA + FL::D];
    __shared__ f2 rows[5][4];
    const Place t(g, q);
    if (t.n <= 0) return;
    const int tid = threadIdx.x;
    const FL flow{smem_u32(bars)};
    const Psi<0> psi(g, q, t, sm + FL::floats);
    if (tid == 0) flow.init(t.nlive);
    if (!kCp && tid < 20) rows[tid / 4][tid % 4] = dup(q.taps[tid / 4][tid % 4]);
    if (kCp) psi.fill(g, q, t);
    __syncthreads();
    if ((tid >> 5) >= t.nlive) return;
    auto la = [&](int p, float *buf, uint32_t bar) {
        tma_load_3d(smem_u32(buf), &maps.f[0], t.X0 - kHalo, t.Y0, t.z0 + p, bar);
        tma_load_3d(smem_u32(buf + kVsyz), &maps.f[1], t.X0, t.Y0 - kHalo, t.z0 + p, bar);
        tma_load_3d(smem_u32(buf + kVszz), &maps.f[2], t.X0, t.Y0, t.z0 + p, bar);
    };
    auto lb = [&](int k, float *buf, uint32_t bar) {
        tma_load_3d(smem_u32(buf), &maps.f[3], t.X0 - kHalo, t.Y0 - kHalo, t.z0 + k, bar);
        tma_load_3d(smem_u32(buf + kVsyy), &maps.f[4], t.X0, t.Y0 - kHalo, t.z0 + k, bar);
        tma_load_3d(smem_u32(buf + kVsxx), &maps.f[5], t.X0 - kHalo, t.Y0, t.z0 + k, bar);
    };
    int next = 0;  // the next plane to issue (thread 0)
    if (tid == 0)
        for (; next < min(t.n, FL::D) + 4; next++) flow.issue(sm, next, la, lb);
    const int sz = (int)g.sz, m = g.m;
    const bool live = t.mask != 0;
    f2 wx[4], wy[4], wz[3];  // the planes below, of sxz, syz, szz
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const bool in = t.z0 + j >= 4;
        const int i = t.i0 + (j - 4) * sz;
        wx[j] = in ? at2(w.f[SXZ] + i) : 0ull;
        wy[j] = in ? at2(w.f[SYZ] + i) : 0ull;
        if (j) wz[j - 1] = in ? at2(w.f[SZZ] + i) : 0ull;
    }
    const float *pf = nullptr;  // the row this lane prefetches
    {
        const int a = (tid & 31) >> 1;
        if (a < 4) pf = (a == 0 ? bdt : w.f[VX + a - 1]) + t.line(g, q) + kAhead * sz;
    }
    const f2 rdx = dup(1.0f / g.dx), rdy = dup(1.0f / g.dy), dt2 = dup(dt);
    const bool ph0 = t.x >= m && t.x < m + g.px, ph1 = t.x + 1 >= m && t.x + 1 < m + g.px;
    const bool yph = t.y >= m && t.y < m + g.py;
    const bool xab = kCp && ((t.mask & 1 && !ph0) || (t.mask & 2 && !ph1)), yab = kCp && live && !yph;
    auto zabs = [&](int z) { return z < m || z >= m + g.pz; };
    if (kCp) {
        psi.fetch(g, q, vpm, 4ull * (uint32_t)t.i0, t.z0, 0, live, xab, yab, zabs(t.z0));
        copy_commit();
    }
    int zclass = -1;
    f2 cx[5];
    if (!kCp) {
        const int o0 = rim_order(min(max(t.x - m, 0), g.px - 1), g.px, rec_w);
        const int o1 = rim_order(min(max(t.x + 1 - m, 0), g.px - 1), g.px, rec_w);
#pragma unroll
        for (int j = 0; j < 4; j++) cx[j] = pk(q.taps[o0][j], q.taps[o1][j]);
    }
    Reader<FL> rd;
    bool ok = rd.start(flow, kVA);
    const float *A0 = sm + t.r * kPW + t.c + kHalo;                         // sxz in an A buffer
    const float *A1 = sm + kVsyz + (t.r + kHalo) * kTX + t.c;               // syz
    const float *A2 = sm + kVszz + t.r * kTX + t.c;                         // szz
    const float *B0 = sm + FL::b0 + (t.r + kHalo) * kPW + t.c + kHalo;      // sxy in a B buffer
    const float *B1 = sm + FL::b0 + kVsyy + (t.r + kHalo) * kTX + t.c;      // syy
    const float *B2 = sm + FL::b0 + kVsxx + t.r * kPW + t.c + kHalo;        // sxx
#pragma unroll 1
    for (int k = 0; k < t.n && ok; k++) {
        uint64_t o = 4ull * (uint32_t)(t.i0 + k * sz);
        int z = t.z0 + k;
        asm volatile("" : "+l"(o), "+r"(z));
        const f2 pb = get2(bdt, o), pv[3] = {get2(w.f[VX], o), get2(w.f[VY], o), get2(w.f[VZ], o)};
        if (kCp) {
            __syncwarp();  // the set to be filled has been read
            if (k + 1 < t.n) psi.fetch(g, q, vpm, o + 4ull * (uint32_t)sz, z + 1, (k + 1) & 1, live, xab, yab, zabs(z + 1));
            copy_commit();
        }
        if (pf && k + kAhead < t.n) prefetch_line(pf + (long long)k * sz);
        ok = rd.wait();
        if (!ok) break;
        const bool zph = !zabs(z), p0 = ph0 && yph && zph, p1 = ph1 && yph && zph;
        const bool ab = kCp && !(p0 && p1);  // a cell of the pair lies in a layer
        f2 vp = 0;
        if (kCp) {
            if (zclass != (int)zph) {
                zclass = zph;
                set_weights(cx, p0, p1, q);
            }
            copy_wait1();
            __syncwarp();
            if (xab || yab || !zph) vp = psi.vp(k & 1);
        }
        const int ob = rd.b * kVB;
        f2 mx, my, mz, no;
        f2 Dx = diff_x<true, kCp>(B2 + ob, cx, no);            // sxx
        f2 Dy = diff_x<false, kCp>(B0 + ob, cx, no);           // sxy
        f2 Dz = diff_x<false, kCp>(A0 + rd.off[0], cx, mx);    // sxz
        if (kXFirst) {
            Dx = mul2(Dx, rdx);
            Dy = mul2(Dy, rdx);
            Dz = mul2(Dz, rdx);
        }
        if (ab) {
            if (!kXFirst) {
                const Join j(p0, p1, 1.0f / g.dx);
                Dx = mul2(Dx, j.S);
                Dy = mul2(Dy, j.S);
                Dz = mul2(Dz, j.S);
            }
            if (xab)
                absorb_x<true>(psi.at(k & 1, 1), q.psx[0], psi.ix(z), psi.tab[t.c], psi.tab[t.c + 1], vp, dt2, Dx, Dy, Dz);
        }
        {
            f2 cy[5];
#pragma unroll
            for (int j = 0; j < (kCp ? 5 : 4); j++) cy[j] = kCp ? cx[j] : rows[rim_order(t.y - m, g.py, rec_w)][j];
            f2 a = diff_y<false, kCp, kPW>(B0 + ob, cy);          // sxy
            f2 b = diff_y<true, kCp, kTX>(B1 + ob, cy);           // syy
            f2 c = diff_y<false, kCp, kTX>(A1 + rd.off[0], cy);   // syz
            if (!kXFirst) {
                a = mul2(a, rdy);
                b = mul2(b, rdy);
                c = mul2(c, rdy);
            }
            f2 R = kXFirst ? rdy : rdx;
            if (ab) {
                const Join j(p0, p1, kXFirst ? 1.0f / g.dy : 1.0f / g.dx);
                if (kXFirst) {
                    a = mul2(a, j.S);
                    b = mul2(b, j.S);
                    c = mul2(c, j.S);
                }
                if (yab)
                    absorb_yz<true>(psi.at(k & 1, 4), q.psy[0], psi.iy(z), psi.tab[kTX + t.r], vp, dt2, b, a, c);
                R = j.R;
            }
            Dx = kXFirst ? fma2(a, R, Dx) : fma2(Dx, R, a);
            Dy = kXFirst ? fma2(b, R, Dy) : fma2(Dy, R, b);
            Dz = kXFirst ? fma2(c, R, Dz) : fma2(Dz, R, c);
        }
        f2 cz[5];
#pragma unroll
        for (int j = 0; j < (kCp ? 5 : 4); j++) cz[j] = kCp ? cx[j] : rows[rim_order(z - m, g.pz, rec_w)][j];
        my = at2(A1 + rd.off[0]);
        mz = at2(A2 + rd.off[0]);
        f2 a = diff_z<false, kCp>(A0, rd.off, mx, wx, cz);  // sxz
        f2 b = diff_z<false, kCp>(A1, rd.off, my, wy, cz);  // syz
        f2 c = diff_z<true, kCp>(A2, rd.off, mz, wz, cz);   // szz
        rd.release();
        rd.next(kVA);
        f2 R = dup(1.0f / g.dz);
        if (ab) {
            const Join j(p0, p1, 1.0f / g.dz);
            a = mul2(a, j.S);
            b = mul2(b, j.S);
            c = mul2(c, j.S);
            if (live && !zph)
                absorb_yz<true>(psi.at(k & 1, 7), q.psz[0], psi.iz(g, z), psi.zrow(k & 1), vp, dt2, c, a, b);
            R = j.R;
        }
        Dx = fma2(a, R, Dx);
        Dy = fma2(b, R, Dy);
        Dz = fma2(c, R, Dz);
        // the stored dt / rho is of the forward step
        const f2 b1 = MODE == kBwd ? mul2(pb, pk(-1.f, -1.f)) : pb;
        const f2 v[3] = {fma2(b1, Dx, pv[0]), fma2(b1, Dy, pv[1]), fma2(b1, Dz, pv[2])};
        float *const dst[3] = {w.f[VX], w.f[VY], w.f[VZ]};
        put2(dst, v, o, t.mask);
        // the first warp refills what every live warp has given back
        if (tid < 32 && k + FL::D < t.n) {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(flow.empty(k), (uint32_t)((k / FL::D) & 1)));
            if (tid == 0 && ok) flow.issue(sm, next++, la, lb);
        }
    }
    if (!ok) atomicExch(err, 1);
    if (tid == 0) flow.drain(next);
}

// ------------------------------------------------ P-wave velocities, imaging

struct PvelMaps {
    CUtensorMap f, r;  // sau of the source and of the receiver wavefield
};
template <bool FB, bool RP>
using PvelFlow = Flow<((FB ? 1 : 0) + (RP ? 1 : 0)) * kSField, 0, kDepth>;

__device__ __forceinline__ f2 dot3(const f2 *a, const f2 *b) { return fma2(a[2], b[2], fma2(a[0], b[0], mul2(a[1], b[1]))); }

// The P-wave velocities over gridphy, from the pressure-like field sau (Dp on
// every axis): with RP the receiver wavefield's, forwards in time; with FB
// the reconstructed source wavefield's, backwards and with the rim orders,
// and then the zero-lag imaging condition (RTM/rtm3d_0_image_module/
// rtm3d_iamge_kernel.hpp:6-51): P = p, S = v - p of the source (f) and of
// the receiver wavefield (r), added into the shot's FP32 images.  vx, vy, vz
// of both wavefields are those after this step's velocity updates.
template <bool FB, bool RP>
__global__ void __launch_bounds__(kThreads, 2)
    pvel_tile(GridDev g, const __grid_constant__ PvelMaps maps, const __grid_constant__ WaveDev f,
              const __grid_constant__ WaveDev r, const float *__restrict__ bdt, int rec_w,
              const __grid_constant__ ImageDev img, const __grid_constant__ TileGeo q, int *err) {
    using FL = PvelFlow<FB, RP>;
    constexpr int AF = ((FB ? 1 : 0) + (RP ? 1 : 0)) * kSField;
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(8) uint64_t bars[FL::SA + FL::D];
    __shared__ f2 rows[5][4];
    const Place t(g, q);
    if (t.n <= 0) return;
    const int tid = threadIdx.x;
    const FL flow{smem_u32(bars)};
    if (tid == 0) flow.init(t.nlive);
    if (tid < 20) rows[tid / 4][tid % 4] = dup(q.taps[tid / 4][tid % 4]);
    __syncthreads();
    if ((tid >> 5) >= t.nlive) return;
    auto la = [&](int p, float *buf, uint32_t bar) {
        if (FB) tma_load_3d(smem_u32(buf), &maps.f, t.X0 - kHalo, t.Y0 - kHalo, t.z0 + p, bar);
        if (RP) tma_load_3d(smem_u32(buf + (FB ? kSField : 0)), &maps.r, t.X0 - kHalo, t.Y0 - kHalo, t.z0 + p, bar);
    };
    auto lb = [](int, float *, uint32_t) {};
    int next = 0;  // the next plane to issue (thread 0)
    if (tid == 0)
        for (; next < min(t.n, FL::D) + 4; next++) flow.issue(sm, next, la, lb);
    const int sz = (int)g.sz, m = g.m;
    f2 wf[3], wr[3];  // the planes below, of sau (inside gridext: pml_num >= 4)
#pragma unroll
    for (int j = 0; j < 3; j++) {
        if (FB) wf[j] = at2(f.f[SAU] + t.i0 + (j - 3) * sz);
        if (RP) wr[j] = at2(r.f[SAU] + t.i0 + (j - 3) * sz);
    }
    const float *pf = nullptr;  // the row this lane prefetches
    {
        const int a = (tid & 31) >> 1;
        if (a == 0) pf = bdt;
        else if (a < 4) pf = r.f[VXP + a - 1];
        else if (FB && a < 7) pf = r.f[VX + a - 4];
        else if (FB && a < 10) pf = f.f[VX + a - 7];
        else if (FB && a < 13) pf = f.f[VXP + a - 10];
        if (pf) pf += t.line(g, q) + kAhead * sz;
    }
    const f2 rdx = dup(1.0f / g.dx), rdy = dup(1.0f / g.dy), rdz = dup(1.0f / g.dz);
    f2 cx[4];
    if (FB) {
        const int o0 = rim_order(min(max(t.x - m, 0), g.px - 1), g.px, rec_w);
        const int o1 = rim_order(min(max(t.x + 1 - m, 0), g.px - 1), g.px, rec_w);
#pragma unroll
        for (int j = 0; j < 4; j++) cx[j] = pk(q.taps[o0][j], q.taps[o1][j]);
    }
    // images are dense over gridphy: a pair of them is one 8-byte access where its row starts on one
    const bool odd_row = (g.px & 1) != 0;
    float *im[5] = {img.ip, img.pp, img.ps, img.sp, img.ss};
    Reader<FL> rd;
    bool ok = rd.start(flow, AF);
    const float *S = sm + (t.r + kHalo) * kPW + t.c + kHalo;
#pragma unroll 1
    for (int k = 0; k < t.n && ok; k++) {
        uint64_t o = 4ull * (uint32_t)(t.i0 + k * sz);
        int z = t.z0 + k;
        asm volatile("" : "+l"(o), "+r"(z));
        const long long io = (t.x - m) + (long long)g.px * ((t.y - m) + (long long)g.py * (z - m));
        const bool wide = t.mask == 3 && !(odd_row && (io & 1));
        f2 pb = get2(bdt, o), pi[5], p[3], pr[3], vf[3], vr[3];
#pragma unroll
        for (int a = 0; a < 5; a++) pi[a] = FB && wide ? at2(im[a] + io) : 0ull;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            pr[a] = get2(r.f[VXP + a], o);
            if (FB) {
                p[a] = get2(f.f[VXP + a], o);
                vf[a] = get2(f.f[VX + a], o);
                vr[a] = get2(r.f[VX + a], o);
            }
        }
        if (pf && k + kAhead < t.n) prefetch_line(pf + (long long)k * sz);
        ok = rd.wait();
        if (!ok) break;
        const float *F = S + rd.off[0];
        f2 mid, d[3], e[3], c[4];
        if (FB) {
            d[0] = mul2(diff_x<true, false>(F, cx, mid), rdx);
#pragma unroll
            for (int j = 0; j < 4; j++) c[j] = rows[rim_order(t.y - m, g.py, rec_w)][j];
            d[1] = mul2(diff_y<true, false, kPW>(F, c), rdy);
#pragma unroll
            for (int j = 0; j < 4; j++) c[j] = rows[rim_order(z - m, g.pz, rec_w)][j];
            d[2] = mul2(diff_z<true, false>(S, rd.off, mid, wf, c), rdz);
        }
        if (RP) {
            constexpr int R = FB ? kSField : 0;
#pragma unroll
            for (int j = 0; j < 4; j++) c[j] = rows[kPhyHalf][j];
            e[0] = mul2(diff_x<true, false>(F + R, c, mid), rdx);
            e[1] = mul2(diff_y<true, false, kPW>(F + R, c), rdy);
            e[2] = mul2(diff_z<true, false>(S + R, rd.off, mid, wr, c), rdz);
        }
        rd.release();
        rd.next(AF);
        if (RP) {
#pragma unroll
            for (int a = 0; a < 3; a++) pr[a] = fma2(pb, e[a], pr[a]);
            float *const dst[3] = {r.f[VXP], r.f[VYP], r.f[VZP]};
            put2(dst, pr, o, t.mask);
        }
        if (FB) {
            pb = mul2(pb, pk(-1.f, -1.f));
            f2 s[3], rs[3];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                p[a] = fma2(pb, d[a], p[a]);
                s[a] = sub2(vf[a], p[a]);
                rs[a] = sub2(vr[a], pr[a]);
            }
            float *const dst[3] = {f.f[VXP], f.f[VYP], f.f[VZP]};
            put2(dst, p, o, t.mask);
            const f2 add[5] = {dot3(p, p), dot3(p, pr), dot3(p, rs), dot3(s, pr), dot3(s, rs)};
#pragma unroll
            for (int a = 0; a < 5; a++) {
                if (wide) {
                    *reinterpret_cast<f2 *>(im[a] + io) = add2(pi[a], add[a]);
                } else {
                    float u, v;
                    up(add[a], u, v);
                    if (t.mask & 1) im[a][io] += u;
                    if (t.mask & 2) im[a][io + 1] += v;
                }
            }
        }
        // the first warp refills what every live warp has given back
        if (tid < 32 && k + FL::D < t.n) {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(flow.empty(k), (uint32_t)((k / FL::D) & 1)));
            if (tid == 0 && ok) flow.issue(sm, next++, la, lb);
        }
    }
    if (!ok) atomicExch(err, 1);
    if (tid == 0) flow.drain(next);
}

}  // namespace

// --------------------------------------------------------------- hosts

namespace {

int round4(int n) { return (n + 3) / 4 * 4; }

// the element columns of the x memory variables: [xl, xl + wl) below and [xh, xh + wh) above gridphy
struct PsiCols {
    int xl, wl, xh, wh, yl, wy;
};
PsiCols psi_cols(const GridDev &g) {
    const int o = (int)g.xoff;
    PsiCols c;
    c.xl = (o + 2) & ~1;
    c.wl = ((o + g.m + 1) & ~1) - c.xl;
    c.xh = (o + g.m + g.px) & ~1;
    c.wh = ((o + g.nx - 2 + 1) & ~1) - c.xh;
    c.yl = c.xl;
    c.wy = ((o + g.nx - 2 + 1) & ~1) - c.yl;
    return c;
}

template <int MODE>
constexpr size_t stress_smem() {
    return StressFlow::floats * sizeof(float) + (MODE == kBwd ? 0 : Psi<1>::kBytes);
}
template <int MODE>
constexpr size_t vel_smem() {
    return VelFlow::floats * sizeof(float) + (MODE == kBwd ? 0 : Psi<0>::kBytes);
}
template <bool FB, bool RP>
constexpr size_t pvel_smem() {
    return PvelFlow<FB, RP>::floats * sizeof(float);
}
// two blocks an SM: 228 KB, of which 1 KB a block is the system's and the barriers and weights are static
static_assert(stress_smem<kFwd>() <= 115200 && vel_smem<kFwd>() <= 115200 && stress_smem<kBwd>() <= 115200, "shared memory");

}  // namespace

long long tile_psi_floats(const GridDev &g) {
    const PsiCols c = psi_cols(g);
    const long long PX = round4(c.wl + c.wh), PY = round4(c.wy), W = 2 * (g.m - 2), ny = g.ny - 4, nz = g.nz - 4;
    return 2 * 3 * (PX * ny * nz + PY * W * nz + PY * ny * W);
}

TileGeo tile_geometry(const GridDev &g, bool phy) {
    TileGeo q{};
    const int n[3] = {g.nx, g.ny, g.nz}, p[3] = {g.px, g.py, g.pz};
    for (int a = 0; a < 3; a++) {
        q.lo[a] = phy ? g.m : 2;
        q.hi[a] = phy ? g.m + p[a] : n[a] - 2;
    }
    // tiles start on 128-byte lines: rows that straddle them measured 240
    // against 303 us (stress update, 200^3 + 20), more than the tile that a
    // shifted start can save
    q.e0 = ((int)g.xoff + q.lo[0]) / kTX * kTX;
    q.ntx = ((int)g.xoff + q.hi[0] - q.e0 + kTX - 1) / kTX;
    q.nty = (q.hi[1] - q.lo[1] + kTY - 1) / kTY;
    const PsiCols c = psi_cols(g);
    q.PX = round4(c.wl + c.wh);
    q.PY = round4(c.wy);
    q.W = 2 * (g.m - 2);
    q.cxl = (int)g.xoff - c.xl;
    q.cxh = c.wl + (int)g.xoff - c.xh;
    q.cy = (int)g.xoff - c.yl;
    return q;
}

int k_make_tile_maps(const GridDev &g, const WaveDev &w, bool phy, float4 *const ax[3], float *psi, int *err_flag,
                     int chunks, TileMaps *m) {
    m->ok = false;
    TileGeo q = tile_geometry(g, phy);
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaError_t e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return (int)e;
    // Planes per chunk.  Over gridphy: waves of two blocks an SM, a chunk's
    // start (barriers, the planes below and the first four above) costing
    // about ten of its planes.  Over gridext a plane costs more, the start
    // about five, and blocks differ: one in a corner of the absorbing layers
    // takes twice as long as one of gridphy, so that the others wait for most
    // of the last block (0.8 of one) and a single wave of long chunks is the
    // worst split (160^3 + 16, 4 chunks against 10, 986 against 830 us a
    // migration step).
    const int nz = q.hi[2] - q.lo[2];
    const long long slots = 2 * nsm;
    long long qc[3] = {-1, -1, -1};
    int qn[3] = {0, 0, 0};
    for (int Q = 1; Q <= nz; Q++) {
        const int L = (nz + Q - 1) / Q;
        if ((nz + L - 1) / L != Q) continue;  // an empty last chunk
        const long long R = (long long)q.ntx * q.nty * Q;
        const long long cost = phy ? (R + slots - 1) / slots * (L + 10) : (std::max(R, slots) * 10 / slots + 8) * (L + 5);
        for (int k = 0; k < 3; k++) {
            if (qc[k] < 0 || cost < qc[k]) {
                for (int j = 2; j > k; j--) {
                    qc[j] = qc[j - 1];
                    qn[j] = qn[j - 1];
                }
                qc[k] = cost;
                qn[k] = Q;
                break;
            }
        }
    }
    for (int k = 0; k < 3; k++) m->qcand[k] = qn[k];
    q.Q = chunks >= 1 && chunks <= nz ? chunks : qn[0];
    q.L = (nz + q.Q - 1) / q.Q;
    const long long nx3 = 3LL * q.PX * (g.ny - 4) * (g.nz - 4), ny3 = 3LL * q.PY * q.W * (g.nz - 4),
                    nz3 = 3LL * q.PY * (g.ny - 4) * q.W;
    for (int s = 0; s < 2; s++) {
        for (int a = 0; a < 3 && psi; a++) {
            q.psx[s][a] = psi + s * (nx3 + ny3 + nz3) + a * (nx3 / 3);
            q.psy[s][a] = psi + s * (nx3 + ny3 + nz3) + nx3 + a * (ny3 / 3);
            q.psz[s][a] = psi + s * (nx3 + ny3 + nz3) + nx3 + ny3 + a * (nz3 / 3);
        }
    }
    for (int a = 0; a < 3; a++) q.ax[a] = ax[a];
    staggered_taps(q.taps);
    static PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &r) != cudaSuccess ||
            r != cudaDriverEntryPointSuccess)
            return (PFN_cuTensorMapEncodeTiled_v12000) nullptr;
        return (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }();
    if (!encode) return 0;
    // the pitched gridext array as a 3-D tensor; boxes of one plane
    auto make = [&](const float *base, int bw, int bh, FieldMap *out) {
        CUtensorMap tm;
        const cuuint64_t dims[3] = {(cuuint64_t)g.sy, (cuuint64_t)g.ny, (cuuint64_t)g.nz};
        const cuuint64_t strides[2] = {(cuuint64_t)g.sy * sizeof(float), (cuuint64_t)g.sz * sizeof(float)};
        const cuuint32_t box[3] = {(cuuint32_t)bw, (cuuint32_t)bh, 1}, estr[3] = {1, 1, 1};
        if (encode(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void *)base, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
        static_assert(sizeof(tm) == sizeof(FieldMap), "descriptor size");
        std::memcpy(out->bytes, &tm, sizeof(tm));
        return true;
    };
    for (int f = 0; f < 3; f++)
        if (!make(w.f[VX + f], kPW, kPH, &m->s[f])) return 0;
    if (!make(w.f[SXZ], kPW, kTY, &m->v[0]) || !make(w.f[SYZ], kTX, kPH, &m->v[1]) ||
        !make(w.f[SZZ], kTX, kTY, &m->v[2]) || !make(w.f[SXY], kPW, kPH, &m->v[3]) ||
        !make(w.f[SYY], kTX, kPH, &m->v[4]) || !make(w.f[SXX], kPW, kTY, &m->v[5]))
        return 0;
    if (w.f[SAU] && !make(w.f[SAU], kPW, kPH, &m->p)) return 0;
    // the attribute belongs to the kernel: every caller sets the same value
    const std::pair<const void *, size_t> fns[] = {{(const void *)stress_tile<kFwd>, stress_smem<kFwd>()},
                                                   {(const void *)stress_tile<kRtmFwd>, stress_smem<kRtmFwd>()},
                                                   {(const void *)stress_tile<kRev>, stress_smem<kRev>()},
                                                   {(const void *)stress_tile<kBwd>, stress_smem<kBwd>()},
                                                   {(const void *)vel_tile<kFwd>, vel_smem<kFwd>()},
                                                   {(const void *)vel_tile<kRev>, vel_smem<kRev>()},
                                                   {(const void *)vel_tile<kBwd>, vel_smem<kBwd>()},
                                                   {(const void *)pvel_tile<true, true>, pvel_smem<true, true>()},
                                                   {(const void *)pvel_tile<true, false>, pvel_smem<true, false>()},
                                                   {(const void *)pvel_tile<false, true>, pvel_smem<false, true>()}};
    for (const auto &f : fns) {
        e = cudaFuncSetAttribute(f.first, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f.second);
        if (e != cudaSuccess) return (int)e;
    }
    m->geo = q;
    m->err = err_flag;
    m->ok = true;
    return 0;
}

int k_stress_tile(int mode, const GridDev &g, const WaveDev &w, const float *lam, const float *mu, const float *vp,
                  float dt, int rec_w, const float *wavelet, const StepState *st, int it_off, const TileMaps &m,
                  void *stream) {
    if (!m.ok) return (int)cudaErrorInvalidValue;
    StressMaps sm;
    static_assert(sizeof(sm) == sizeof(m.s), "descriptor layout");
    std::memcpy(&sm, m.s, sizeof(sm));
    const int grid = m.geo.ntx * m.geo.nty * m.geo.Q;
    cudaStream_t s = (cudaStream_t)stream;
#define JV_ST(M)                                                                                                 \
    stress_tile<M><<<grid, kThreads, stress_smem<M>(), s>>>(g, sm, w, lam, mu, vp, dt, rec_w, wavelet, st, it_off, \
                                                            m.geo, m.err)
    switch (mode) {
    case kFwd: JV_ST(kFwd); break;
    case kRtmFwd: JV_ST(kRtmFwd); break;
    case kRev: JV_ST(kRev); break;
    case kBwd: JV_ST(kBwd); break;
    default: return (int)cudaErrorInvalidValue;
    }
#undef JV_ST
    return (int)cudaGetLastError();
}

int k_vel_tile(int mode, const GridDev &g, const WaveDev &w, const float *bdt, const float *vp, float dt, int rec_w,
               const TileMaps &m, void *stream) {
    if (!m.ok) return (int)cudaErrorInvalidValue;
    VelMaps vm;
    static_assert(sizeof(vm) == sizeof(m.v), "descriptor layout");
    std::memcpy(&vm, m.v, sizeof(vm));
    const int grid = m.geo.ntx * m.geo.nty * m.geo.Q;
    cudaStream_t s = (cudaStream_t)stream;
#define JV_VT(M) vel_tile<M><<<grid, kThreads, vel_smem<M>(), s>>>(g, vm, w, bdt, vp, dt, rec_w, m.geo, m.err)
    switch (mode) {
    case kFwd:
    case kRtmFwd: JV_VT(kFwd); break;
    case kRev: JV_VT(kRev); break;
    case kBwd: JV_VT(kBwd); break;
    default: return (int)cudaErrorInvalidValue;
    }
#undef JV_VT
    return (int)cudaGetLastError();
}

int k_pvel_tile(const GridDev &g, const WaveDev *f, const TileMaps *fm, const WaveDev &r, const TileMaps &rm,
                bool r_too, const float *bdt, int rec_w, const ImageDev *img, void *stream) {
    if (!rm.ok || (f && (!fm || !fm->ok || !img)) || (!f && !r_too)) return (int)cudaErrorInvalidValue;
    PvelMaps pm{};
    if (f) std::memcpy(&pm.f, fm->p.bytes, sizeof(pm.f));
    std::memcpy(&pm.r, rm.p.bytes, sizeof(pm.r));
    const TileGeo &q = rm.geo;
    const int grid = q.ntx * q.nty * q.Q;
    cudaStream_t s = (cudaStream_t)stream;
    const WaveDev fw = f ? *f : WaveDev{};
    const ImageDev im = img ? *img : ImageDev{};
#define JV_PV(FB, RP) \
    pvel_tile<FB, RP><<<grid, kThreads, pvel_smem<FB, RP>(), s>>>(g, pm, fw, r, bdt, rec_w, im, q, rm.err)
    if (f && r_too) {
        JV_PV(true, true);
    } else if (f) {
        JV_PV(true, false);
    } else {
        JV_PV(false, true);
    }
#undef JV_PV
    return (int)cudaGetLastError();
}

}  // namespace jv
