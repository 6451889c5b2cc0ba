// Isotropic elastic (P-SV) standard-staggered-grid time step, 10th order: the two modes of
// forward/yang_version_2016_2_2 for a flat surface -- 'abc' (YPRI:234-386, cosine sponge on all
// four sides) and 'fsbc' (YPRI:57-230, free surface at row zs, no top sponge).  Every field is kept in the reference's split form (x and z parts), ten per cell:
//   vxx vxz vzx vzz | strxxx strxxz | strzzx strzzz | strxzx strxzz
// with the five sums vx, vz, strxx, strzz, strxz (YPUB:1410-1426) beside them, written by the
// kernel that completes them, and one step is two kernels
// (YPUB = Iso_multishot_fd_subroutine_fsbc_zy_m2_pub.f90):
//   velocity: strxx, strxz, strzz staged on the tile plus halo;
//             vxx += (dt/dx) busg2e Dx0 strxx, vxz += (dt/dz) busg2e Dz0 strxz,
//             vzx += (dt/dx) busg1e Dx1 strxz, vzz += (dt/dz) busg1e Dz1 strzz
//             (caluxabs / caluzabs, YPUB:1095-1157, 1347-1407), each part times its sponge
//   stress:   vx, vz staged on the tile plus halo;
//             strxxx += (dt/dx) lambmusg Dx1 vx, strxxz += (dt/dz) lambsg Dz0 vz,
//             strzzx += (dt/dx) lambsg Dx1 vx,   strzzz += (dt/dz) lambmusg Dz0 vz,
//             strxzx += (dt/dx) musge Dx0 vz,    strxzz += (dt/dz) musge Dz1 vx,
//             each part times its sponge, the Gaussian source added to strxxx and strzzx after
//             their sponge (YPRI:331-359, YPUB:1429-1466); records vx, vz at the receivers
// Dx0 u(i) = sum_m a_m (u(i+m) - u(i-1-m)), Dx1 u(i) = sum_m a_m (u(i+1+m) - u(i-m)), m = 0..4.
// Every multiply and add is rounded separately in the reference's order, so the kernels agree
// bit for bit with the FP32 restatement in oracle/iso_oracle.cpp.
//
// The surface row is per column: itopo(x) (1-based, the reference's itopoe), from a topography or
// flat.  abc mode updates the rows from t0 = itopo - npz - 1 (0-based) down, with the top sponge
// on rows t0 .. t0 + npz taking spgzn(z - t0 + 1) (YPUB:851-897); a flat surface has t0 = -1.
// Free surface (fsbc, zs = itopo - 1): rows above zs keep their values; the z derivatives of the five rows from
// zs down drop to 8th, 6th, 4th and 2nd order (YPUB:1160-1343); left and right sponges act from
// zs down, the bottom sponge everywhere, no top sponge (YPUB:901-934); strzz parts are zero on
// rows <= zs after their sponge and before the source (YPUB:978-1007), which enters strxx only for
// sources below the surface (YPRI:163-168).  After the stress kernel the surface kernel writes
// the image strxz(zs - 1) = -strxz(zs) (YPUB:1009-1024) and vz(zs - 1) from vz(zs) and dx vx(zs)
// (YPUB:938-976).  The reference writes that vz after summing the split parts, so its stress
// update reads it one step later; running the surface kernel after the stress kernel gives the
// same order.
//
// Bound: memory latency (DRAM at 4.2 TB/s with 18 warps an SM, issue 45%).  A step must read and write ten split fields and read five model arrays (100 B a
// cell); the two kernels move 140 B (the sums are written once and read once, the halos hit L2).
// The sums are slabs of their own so that one TMA box per field stages a tile with its halo (no
// registers, no address arithmetic in the threads) while the threads' own split parts are loaded,
// and so that the halos re-read one array per field instead of two.  Tiles are 64 rows of z by 8
// columns, one vector of four cells per thread, five CTAs of 128 threads per SM: the 2.25-fold halo
// hits L2, and many small CTAs cover one another's loads and the slow vectors at the surface.
// Free-surface step of 8 shots of 1280 x 483 (4.95 M cells): 277 us before, 122 us now (40.6 Gpts/s,
// DRAM at 4.2 TB/s).  Tiles of 16 and 32 columns 133 and 160 us; 64 columns and four vectors per
// thread, which loads and waits four times in turn, 250 us.
//
// Model preparation (host, per shot window): substagger (YPUB:323-547); then, in abc mode, on the
// device the PML smoothing of modipapml (YPUB:549-634), which overwrites each top-sponge cell with the
// Gaussian-weighted sum of its window while later cells read the already smoothed ones: a
// sequential chain, run as one thread per array and window in the reference's serial order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "sfd_internal.h"
#include "tile_stage.cuh"

namespace sfd {
namespace {

constexpr int TX = kTileX, TZ = kTileZ;
constexpr int H = 5;                  // staggered reach: Dx0 reads i-5..i+4, Dx1 i-4..i+5
constexpr int HZ = 8;                 // z halo rounded for float4 staging
constexpr int SW = TZ + 2 * HZ;       // 80
constexpr int TC = kIsoCols;          // columns of a CTA's tile
constexpr int kSmem = (TC + 2 * H) * SW;  // floats per staged field
constexpr int kThreads = TC * TZ / 4;     // one float4 of cells per thread

__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }

// Two cells per instruction with the same roundings as the scalar operations: a difference as
// fma(b, -1, a) and a sum as fma(a, one, b) are rounded once.  `one` is 1.0 from the kernel's
// arguments: the compiler, which contracts a paired multiply and a paired add into one paired FMA,
// cannot see that the factor does nothing.
__device__ __forceinline__ float2 bc(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 add2(float2 a, float2 b, float one) { return __ffma2_rn(a, bc(one), b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, bc(-1.0f), a); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float4 cat4(float2 a, float2 b) { return make_float4(a.x, a.y, b.x, b.y); }
__device__ __forceinline__ float4 add4(const float4& p, const float4& q, float one) {
    return cat4(add2(lo2(p), lo2(q), one), add2(hi2(p), hi2(q), one));
}
// u + (c k) d, each operation rounded
__device__ __forceinline__ float4 upd4(const float4& u, float c, const float4& k, const float4& d, float one) {
    return cat4(add2(mul2(mul2(bc(c), lo2(k)), lo2(d)), lo2(u), one),
                add2(mul2(mul2(bc(c), hi2(k)), hi2(d)), hi2(u), one));
}

struct TileRef {
    int shot, tile, x0, z0;
    ShotDev sd;
};

// CTA b covers TC columns; t.tile is the 64 x 64 tile (of the receiver lists) that holds them
__device__ __forceinline__ bool tile_of(const IArgs& a, TileRef& t) {
    t.shot = a.slot_to_shot[blockIdx.z];
    t.sd = a.shots[t.shot];
    t.x0 = (a.col0 + (int)blockIdx.y) * TC;
    t.z0 = blockIdx.x * TZ;
    t.tile = t.x0 / TX * a.L.ntz + blockIdx.x;
    return t.x0 < t.sd.nx;
}

__device__ __forceinline__ long long cell(const IArgs& a, int shot, int x, int z) {
    return (long long)shot * a.L.shot_stride + (long long)(x + a.L.gx) * a.L.pitch + a.L.gz + z;
}

// One thread requests the tile plus halo of NF sum fields, one TMA box each (z coordinate a multiple
// of 64, x coordinate at least 3: see Layout2D's margins), all completing on one mbarrier.
template <int NF>
__device__ __forceinline__ void stage(float* s, uint64_t* bar, const IArgs& a, const TileRef& t, const int* field) {
    tile::expect(bar, 4u * NF * kSmem);
#pragma unroll
    for (int f = 0; f < NF; f++)
        tile::box(s + f * kSmem, &a.tm[field[f] - I_VX], a.L.gz + t.z0 - HZ, a.L.gx + t.x0 - H, t.shot, bar);
}

// The same without the slabs of the sums, from the split parts f0, f0 + 1 (the caller's __syncthreads follows)
__device__ __forceinline__ void stage_parts(float* s, const IArgs& a, const TileRef& t, int f0) {
    for (int i = threadIdx.x; i < kSmem / 4; i += kThreads) {
        const int r = i / (SW / 4), c = 4 * (i % (SW / 4));
        const long long off = cell(a, t.shot, t.x0 - H + r, t.z0 - HZ + c);
        const float4 p = *reinterpret_cast<const float4*>(a.f[f0] + off), q = *reinterpret_cast<const float4*>(a.f[f0 + 1] + off);
        *reinterpret_cast<float4*>(s + r * SW + c) = add4(p, q, a.one);
    }
}

// one split-sponge factor in YPUB:851-897's order (near-side table, then far-side table)
__device__ __forceinline__ float xs(float u, int x, int n, int np, const float* tn, const float* tp) {
    if (x <= np) u = fm(u, tn[x]);
    if (x >= n - np - 1) u = fm(u, tp[n - 1 - x]);
    return u;
}

// Thread t takes the z-vector t % 16 (cells z0 + 4 (t % 16) .. + 3) of row t / 16 of the tile; a warp
// covers two whole tile rows, so every field access is one coalesced 16-byte load or store per lane.
// The stencils read float4 windows from shared memory: an x derivative of four cells is ten 16-byte
// loads, a z derivative five.

__device__ __forceinline__ float4 lds4(const float* s, int r, int c) { return *reinterpret_cast<const float4*>(s + r * SW + c); }
__device__ __forceinline__ float cmp(const float4& v, int q) { return q == 0 ? v.x : (q == 1 ? v.y : (q == 2 ? v.z : v.w)); }
__device__ __forceinline__ float& cmpr(float4& v, int q) { return q == 0 ? v.x : (q == 1 ? v.y : (q == 2 ? v.z : v.w)); }

// x derivative (YPUB:1095-1157) of the four cells (row r, columns c..c+3) of a staged field
template <int FLAG>
__device__ __forceinline__ float4 dx4(const float* s, int r, int c, const float* a, float one) {
    float2 l, h;
#pragma unroll
    for (int m = 0; m < 5; m++) {
        const float4 p = lds4(s, FLAG == 0 ? r + m : r + 1 + m, c);
        const float4 q = lds4(s, FLAG == 0 ? r - 1 - m : r - m, c);
        const float2 am = bc(a[m]);
        const float2 tl = mul2(am, sub2(lo2(p), lo2(q))), th = mul2(am, sub2(hi2(p), hi2(q)));
        l = m == 0 ? tl : add2(tl, l, one);
        h = m == 0 ? th : add2(th, h, one);
    }
    return cat4(l, h);
}

// z derivative (YPUB:1347-1407) of the same four cells: the window z-8 .. z+11 (c = column of z).
// d0: distance of the first cell below the free surface (large without one).  Cells d = 0..4
// rows below it take the lower orders of caluz (YPUB:1160-1343); the ones above it are not used.
template <int FLAG, bool FS>
__device__ __forceinline__ float4 dz4(const float* s, int r, int c, const IArgs& a, int d0) {
    float w[20];
#pragma unroll
    for (int j = 0; j < 5; j++) {
        const float4 v = lds4(s, r, c - 8 + 4 * j);
        w[4 * j] = v.x; w[4 * j + 1] = v.y; w[4 * j + 2] = v.z; w[4 * j + 3] = v.w;
    }
    float4 acc;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int d = d0 + q;
        const int M = !FS ? 5 : FLAG == 0 ? (d >= 5 ? 5 : (d < 1 ? 1 : d)) : (d >= 4 ? 5 : (d < 0 ? 1 : d + 1));
        float sum = 0.0f;
#pragma unroll
        for (int m = 0; m < 5; m++) {  // selects, not branches: neighbouring threads differ in M
            float cm = a.a[m];
            if (FS && m < 4) {
                cm = M == 4 ? a.cr[3][m] : cm;
                cm = m < 3 && M == 3 ? a.cr[2][m] : cm;
                cm = m < 2 && M == 2 ? a.cr[1][m] : cm;
                cm = m < 1 && M == 1 ? a.cr[0][m] : cm;
            }
            const int z = 8 + q;  // index of cell q in w
            const float t = FLAG == 0 ? fs(w[z + m], w[z - 1 - m]) : fs(w[z + 1 + m], w[z - m]);
            const float next = (m == 0) ? fm(cm, t) : fa(sum, fm(cm, t));
            sum = !FS || m < M ? next : sum;
        }
        cmpr(acc, q) = sum;
    }
    return acc;
}

// z-part sponge: abc, the top table on rows t0 .. t0 + npz then the bottom table (YPUB:851-897);
// fsbc, the bottom table only (YPUB:901-934)
template <bool FS>
__device__ __forceinline__ float zsp(float u, int z, int t0, const IArgs& a, const float* tn, const float* tp) {
    if (!FS && z >= t0 && z <= t0 + a.npz) u = fm(u, tn[z - t0]);
    if (z >= a.nz - a.npz - 1) u = fm(u, tp[a.nz - 1 - z]);
    return u;
}

// Four cells of a field.  The rows past nz of the last vector exist in the slab and hold zero, which
// the stencils rely on: Vec::keep clears them before a store.
__device__ __forceinline__ float4 ld4(const float* f, long long c) { return *reinterpret_cast<const float4*>(f + c); }
__device__ __forceinline__ void st4(float* f, long long c, const float4& v) { *reinterpret_cast<float4*>(f + c) = v; }

__device__ __forceinline__ void mul4(float4& v, float f) {
    v = cat4(mul2(lo2(v), bc(f)), mul2(hi2(v), bc(f)));
}

// One z-vector of a row: where it lies and which sponges, surface rows and orders it meets.  A plain
// vector (all but those at the surface and across the bottom edge) updates its four cells alike: the
// x sponge is one factor per row, the z sponge is applied only by the threads inside it.  Deciding
// this per cell took 237 (velocity) and 382 (stress) instructions a cell, which bound the kernels.
template <bool FS>
struct Vec {
    int gx, gz, top;
    long long c, mi;
    bool plain, pad, air;
    __device__ __forceinline__ Vec(const IArgs& a, const TileRef& t, int r, int z) {
        gx = t.x0 + r;
        gz = t.z0 + z;
        c = cell(a, t.shot, gx, gz);
        const int mc = min(t.sd.x0 + gx, a.nx_model - 1);
        mi = (long long)mc * a.mpitch + gz;
        // first updated row: zs = itopo - 1 (fsbc) or t0 = itopo - npz - 1 (abc)
        top = __ldg(a.itopo + mc) - (FS ? 1 : a.npz + 1);
        const bool zpad = (!FS && gz <= top + a.npz) || gz + 3 >= a.nz - a.npz - 1;
        plain = gz + 3 < a.nz && gz - top >= (FS ? 5 : 0);
        pad = zpad || gx <= a.npx || gx >= t.sd.nx - a.npx - 1;
        // above the row over the surface (which the surface kernel rewrites) nothing changes
        air = gz + 3 < top - 1 && !zpad;
    }
    // both sponge tables of the x part, near side then far side (YPUB:851-897)
    __device__ __forceinline__ void xsp(float4& v, const IArgs& a, int nx, const float* tn) const {
        if (gx <= a.npx) mul4(v, tn[gx]);
        if (gx >= nx - a.npx - 1) mul4(v, tn[a.spg_stride + nx - 1 - gx]);
    }
    __device__ __forceinline__ void zsp4(float4& v, const IArgs& a, const float* tn) const {
#pragma unroll
        for (int q = 0; q < 4; q++) cmpr(v, q) = zsp<FS>(cmp(v, q), gz + q, top, a, tn, tn + a.spg_stride);
    }
    __device__ __forceinline__ void keep(float4& v, int nz) const {
#pragma unroll
        for (int q = 1; q < 4; q++)
            if (gz + q >= nz) cmpr(v, q) = 0.0f;
    }
};

// SUMS = false: no memory for the slabs of the sums, a third of the state.  The tile and its halo are summed by
// the threads: 58 ms against 35 for 275 steps of 8 shots of 1280 x 483.
template <bool FS, bool SUMS>
__global__ void __launch_bounds__(kThreads, 5) iso_velocity_kernel(const __grid_constant__ IArgs a) {
    extern __shared__ __align__(128) float smem[];
    const float* sSxx = smem;
    const float* sSxz = smem + kSmem;
    const float* sSzz = smem + 2 * kSmem;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 3 * kSmem);
    TileRef t;
    const bool on = tile_of(a, t);
    tile::bar_init(bar);
    tile::release();
    tile::acquire();
    if (!on) return;
    if (!SUMS) {
        stage_parts(smem, a, t, I_SXXX);
        stage_parts(smem + kSmem, a, t, I_SXZX);
        stage_parts(smem + 2 * kSmem, a, t, I_SZZX);
        __syncthreads();
    } else if (threadIdx.x == 0) {
        const int f[3] = {I_SXX, I_SXZ, I_SZZ};
        stage<3>(smem, bar, a, t, f);
    }
    const int nx = t.sd.nx, nz = a.nz;
    const float* tb = a.spg;
    const int st = a.spg_stride;
    const int z = 4 * (threadIdx.x & 15);
    const int r = threadIdx.x >> 4;
    const Vec<FS> e(a, t, r, z);
    if (t.x0 + r >= nx || e.gz >= nz || e.air) {
        if (SUMS) tile::staged(bar, a.err_flag);  // leave with the CTA's copies landed
        return;
    }
    float4 vxx = ld4(a.f[I_VXX], e.c), vxz = ld4(a.f[I_VXZ], e.c);
    float4 vzx = ld4(a.f[I_VZX], e.c), vzz = ld4(a.f[I_VZZ], e.c);
    const float4 b2 = __ldg(reinterpret_cast<const float4*>(a.b2e + e.mi));
    const float4 b1 = __ldg(reinterpret_cast<const float4*>(a.b1e + e.mi));
    if (SUMS && !tile::staged(bar, a.err_flag)) return;
    const float4 d_xx = dx4<0>(sSxx, r + H, z + HZ, a.a, a.one);  // Dx0 strxx
    const float4 d_zx = dx4<1>(sSxz, r + H, z + HZ, a.a, a.one);  // Dx1 strxz
    // YPRI:310-326: vx parts with sponges spgxn/spgxp and spgzn/spgzp, vz parts with
    // spg1xn/spg2xp and spg1zn/spg2zp
    if (e.plain) {
        vxx = upd4(vxx, a.dtdx, b2, d_xx, a.one);
        vxz = upd4(vxz, a.dtdz, b2, dz4<0, false>(sSxz, r + H, z + HZ, a, 0), a.one);
        vzx = upd4(vzx, a.dtdx, b1, d_zx, a.one);
        vzz = upd4(vzz, a.dtdz, b1, dz4<1, false>(sSzz, r + H, z + HZ, a, 0), a.one);
        if (e.pad) {
            e.xsp(vxx, a, nx, tb);
            e.xsp(vzx, a, nx, tb + 4 * st);
            e.zsp4(vxz, a, tb + 2 * st);
            e.zsp4(vzz, a, tb + 6 * st);
        }
    } else {
        const int d0 = FS ? e.gz - e.top : (1 << 20);
        const float4 d_xz = dz4<0, FS>(sSxz, r + H, z + HZ, a, d0);  // Dz0 strxz
        const float4 d_zz = dz4<1, FS>(sSzz, r + H, z + HZ, a, d0);  // Dz1 strzz
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int zq = min(e.gz + q, nz - 1);      // cells past nz are computed, not stored
            const bool below = e.gz + q >= e.top;  // rows above the first updated row keep their values
            if (below) {
                const float n_xx = fa(cmp(vxx, q), fm(fm(a.dtdx, cmp(b2, q)), cmp(d_xx, q)));
                cmpr(vxx, q) = xs(n_xx, e.gx, nx, a.npx, tb + 0 * st, tb + 1 * st);
                cmpr(vxz, q) = fa(cmp(vxz, q), fm(fm(a.dtdz, cmp(b2, q)), cmp(d_xz, q)));
            }
            cmpr(vxz, q) = zsp<FS>(cmp(vxz, q), zq, e.top, a, tb + 2 * st, tb + 3 * st);
            if (below) {
                const float n_zx = fa(cmp(vzx, q), fm(fm(a.dtdx, cmp(b1, q)), cmp(d_zx, q)));
                cmpr(vzx, q) = xs(n_zx, e.gx, nx, a.npx, tb + 4 * st, tb + 5 * st);
                cmpr(vzz, q) = fa(cmp(vzz, q), fm(fm(a.dtdz, cmp(b1, q)), cmp(d_zz, q)));
            }
            cmpr(vzz, q) = zsp<FS>(cmp(vzz, q), zq, e.top, a, tb + 6 * st, tb + 7 * st);
        }
        e.keep(vxx, nz); e.keep(vxz, nz); e.keep(vzx, nz); e.keep(vzz, nz);
    }
    st4(a.f[I_VXX], e.c, vxx); st4(a.f[I_VXZ], e.c, vxz);
    st4(a.f[I_VZX], e.c, vzx); st4(a.f[I_VZZ], e.c, vzz);
    if (SUMS) {
        st4(a.f[I_VX], e.c, add4(vxx, vxz, a.one));  // YPRI:316
        st4(a.f[I_VZ], e.c, add4(vzx, vzz, a.one));  // YPRI:326
    }
}

template <bool FS, bool SUMS>
__global__ void __launch_bounds__(kThreads, 5) iso_stress_kernel(const __grid_constant__ IArgs a) {
    extern __shared__ __align__(128) float smem[];
    const float* sVx = smem;
    const float* sVz = smem + kSmem;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 2 * kSmem);
    TileRef t;
    const bool on = tile_of(a, t);
    tile::bar_init(bar);
    tile::release();
    tile::acquire();
    if (!on) return;
    if (!SUMS) {
        stage_parts(smem, a, t, I_VXX);
        stage_parts(smem + kSmem, a, t, I_VZX);
        __syncthreads();
    } else if (threadIdx.x == 0) {
        const int f[2] = {I_VX, I_VZ};
        stage<2>(smem, bar, a, t, f);
    }
    const int nx = t.sd.nx, nz = a.nz;
    const float* tb = a.spg;
    const int st = a.spg_stride;
    const ShotDev& sd = t.sd;
    const float wav = __ldg(a.wavelets + sd.wav_off + a.step);
    const int z = 4 * (threadIdx.x & 15);
    // YPRI:163-168: in fsbc mode strxx takes the source only below the surface at the source column
    const bool src_xx = !FS || sd.sz + 1 > __ldg(a.itopo + min(sd.x0 + sd.sx, a.nx_model - 1));
    // YPUB:1458 wavelet*gc2d*dt/(dz**2)
    auto source = [&](int bx, int bz) {
        return __fdiv_rn(fm(fm(wav, __ldg(a.stamps + sd.stamp_off + bx * sd.stamp_h + bz)), a.dt), a.dz2);
    };
    const int r = threadIdx.x >> 4;
    const Vec<FS> e(a, t, r, z);
    const int bx = e.gx - sd.stamp_x0, bz0 = e.gz - sd.stamp_z0;
    const bool stamp = bx >= 0 && bx < sd.stamp_w && bz0 + 3 >= 0 && bz0 < sd.stamp_h;
    const bool work = t.x0 + r < nx && e.gz < nz && (!e.air || stamp);
    float4 v[6], lm2, lam, mue;  // v: strxxx strxxz strzzx strzzz strxzx strxzz
    if (work) {
#pragma unroll
        for (int k = 0; k < 6; k++) v[k] = ld4(a.f[I_SXXX + k], e.c);
        lm2 = __ldg(reinterpret_cast<const float4*>(a.lm2 + e.mi));
        lam = __ldg(reinterpret_cast<const float4*>(a.lam + e.mi));
        mue = __ldg(reinterpret_cast<const float4*>(a.mue + e.mi));
    }
    if (SUMS && !tile::staged(bar, a.err_flag)) return;
    if (work) {
        const float4 d1 = dx4<1>(sVx, r + H, z + HZ, a.a, a.one);  // Dx1 vx
        const float4 d3 = dx4<0>(sVz, r + H, z + HZ, a.a, a.one);  // Dx0 vz
        if (e.plain) {
            const float4 d2 = dz4<0, false>(sVz, r + H, z + HZ, a, 0), d4 = dz4<1, false>(sVx, r + H, z + HZ, a, 0);
            v[0] = upd4(v[0], a.dtdx, lm2, d1, a.one);
            v[1] = upd4(v[1], a.dtdz, lam, d2, a.one);
            v[2] = upd4(v[2], a.dtdx, lam, d1, a.one);
            v[3] = upd4(v[3], a.dtdz, lm2, d2, a.one);
            v[4] = upd4(v[4], a.dtdx, mue, d3, a.one);
            v[5] = upd4(v[5], a.dtdz, mue, d4, a.one);
            if (e.pad) {
                e.xsp(v[0], a, nx, tb + 4 * st);
                e.zsp4(v[1], a, tb + 2 * st);
                e.xsp(v[2], a, nx, tb + 4 * st);
                e.zsp4(v[3], a, tb + 2 * st);
                e.xsp(v[4], a, nx, tb);
                e.zsp4(v[5], a, tb + 6 * st);
            }
            if (stamp) {
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (bz0 + q >= 0 && bz0 + q < sd.stamp_h) {
                        const float src = source(bx, bz0 + q);
                        if (src_xx) cmpr(v[0], q) = fa(src, cmp(v[0], q));
                        cmpr(v[2], q) = fa(src, cmp(v[2], q));
                    }
            }
        } else {
            const int d0 = FS ? e.gz - e.top : (1 << 20);
            const float4 d2 = dz4<0, FS>(sVz, r + H, z + HZ, a, d0);  // Dz0 vz
            const float4 d4 = dz4<1, FS>(sVx, r + H, z + HZ, a, d0);  // Dz1 vx
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int zq = min(e.gz + q, nz - 1);  // cells past nz are computed, not stored
                const int bz = zq - sd.stamp_z0;
                const bool in_stamp = stamp && bz >= 0 && bz < sd.stamp_h;
                const float src = in_stamp ? source(bx, bz) : 0.0f;
                // rows above the first updated row keep their values (the loops start at itopo or
                // itopo - npzn)
                const bool below = e.gz + q >= e.top;
                const bool zero_zz = FS && e.gz + q <= e.top;  // YPUB:978-1007, rows <= itopo
                // YPRI:331-338: strxx parts, sponge spg1xn/spg2xp, spgzn/spgzp, then the source
                float s0 = cmp(v[0], q), s1 = cmp(v[1], q), s2 = cmp(v[2], q), s3 = cmp(v[3], q);
                float s4 = cmp(v[4], q), s5 = cmp(v[5], q);
                if (below) {
                    s0 = xs(fa(s0, fm(fm(a.dtdx, cmp(lm2, q)), cmp(d1, q))), e.gx, nx, a.npx, tb + 4 * st, tb + 5 * st);
                    s1 = fa(s1, fm(fm(a.dtdz, cmp(lam, q)), cmp(d2, q)));
                }
                s1 = zsp<FS>(s1, zq, e.top, a, tb + 2 * st, tb + 3 * st);
                if (in_stamp && src_xx) s0 = fa(src, s0);
                // YPRI:342-349: strzz parts; fsbc: zero on rows <= the surface before the source
                if (below) {
                    s2 = xs(fa(s2, fm(fm(a.dtdx, cmp(lam, q)), cmp(d1, q))), e.gx, nx, a.npx, tb + 4 * st, tb + 5 * st);
                    s3 = fa(s3, fm(fm(a.dtdz, cmp(lm2, q)), cmp(d2, q)));
                }
                s3 = zsp<FS>(s3, zq, e.top, a, tb + 2 * st, tb + 3 * st);
                if (zero_zz) s2 = s3 = 0.0f;
                if (in_stamp) s2 = fa(src, s2);
                // YPRI:353-359: strxz parts, sponge spgxn/spgxp, spg1zn/spg2zp
                if (below) {
                    s4 = xs(fa(s4, fm(fm(a.dtdx, cmp(mue, q)), cmp(d3, q))), e.gx, nx, a.npx, tb + 0 * st, tb + 1 * st);
                    s5 = fa(s5, fm(fm(a.dtdz, cmp(mue, q)), cmp(d4, q)));
                }
                s5 = zsp<FS>(s5, zq, e.top, a, tb + 6 * st, tb + 7 * st);
                cmpr(v[0], q) = s0; cmpr(v[1], q) = s1; cmpr(v[2], q) = s2;
                cmpr(v[3], q) = s3; cmpr(v[4], q) = s4; cmpr(v[5], q) = s5;
            }
#pragma unroll
            for (int k = 0; k < 6; k++) e.keep(v[k], nz);
        }
#pragma unroll
        for (int k = 0; k < 6; k++) st4(a.f[I_SXXX + k], e.c, v[k]);
        if (SUMS) {
            st4(a.f[I_SXX], e.c, add4(v[0], v[1], a.one));
            st4(a.f[I_SZZ], e.c, add4(v[2], v[3], a.one));
            st4(a.f[I_SXZ], e.c, add4(v[4], v[5], a.one));
        }
    }
    // receivers: record1 = vx, record2 = vz after the step (YPRI:361-367, YPUB:2-16); the
    // velocities are final after the velocity kernel and staged here
    const int* trp = a.tile_rec_ptr + sd.tile_rec_base + t.tile;
    const int rb = trp[0], re = trp[1];
    for (int j = rb + threadIdx.x; j < re; j += kThreads) {
        const int ridx = a.tile_rec_idx[j];
        const int rr = a.rec_x[sd.rec_list + ridx] - t.x0 + H, rz = a.rec_z[sd.rec_list + ridx] - t.z0 + HZ;
        if (rr < H || rr >= H + TC) continue;  // another CTA of the 64 x 64 tile holds it
        const long long o = sd.rec_base + (long long)a.step * sd.nrec + ridx;
        a.records[o] = sVx[rr * SW + rz];
        a.records2[o] = sVz[rr * SW + rz];
    }
}

// Free surface, after the stress kernel (one thread per column, zs = itopo(x) - 1): the image strxz(zs - 1) =
// -strxz(zs) of both split parts (YPUB:1009-1024), and vz(zs - 1) = vz(zs) + lambsg/lambmusg
// (vx(zs, x + 1) - vx(zs, x)) for both pairs of split parts (YPUB:938-976, columns but the last).
// The velocity kernel that follows forms the sums of vx and vz again; the sum of strxz is written here.
__global__ void iso_surface_kernel(const __grid_constant__ IArgs a) {
    const int shot = a.slot_to_shot[blockIdx.y];
    const ShotDev sd = a.shots[shot];
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    tile::release();
    tile::acquire();
    if (x >= sd.nx) return;
    const int mc = min(sd.x0 + x, a.nx_model - 1);
    const int zs = __ldg(a.itopo + mc) - 1;
    if (zs < 1) return;  // the row above the surface is the split fields' unused row 0
    const long long c = cell(a, shot, x, zs), cu = c - 1;
    const float ux = -a.f[I_SXZX][c], uz = -a.f[I_SXZZ][c];
    a.f[I_SXZX][cu] = ux;
    a.f[I_SXZZ][cu] = uz;
    if (a.f[I_SXZ]) a.f[I_SXZ][cu] = fa(ux, uz);
    if (x + 1 < sd.nx) {
        const long long cn = cell(a, shot, x + 1, zs);
        const long long mi = (long long)mc * a.mpitch + zs;
        const float ratio = __fdiv_rn(__ldg(a.lam + mi), __ldg(a.lm2 + mi));
        a.f[I_VZX][cu] = fa(a.f[I_VZX][c], fm(ratio, fs(a.f[I_VXX][cn], a.f[I_VXX][c])));
        a.f[I_VZZ][cu] = fa(a.f[I_VZZ][c], fm(ratio, fs(a.f[I_VXZ][cn], a.f[I_VXZ][c])));
    }
}

// YPUB:592-634, one sequential chain per (window, array), one warp each: cells (z < itopo) in
// the serial loop order, each replaced by the weighted sum of its window as it stands at that
// moment.  The warp's lanes form the cell's products u(m, n) gc(idx1, idx2) in parallel (each
// is one rounded multiply, whoever computes it) into shared memory in the loop's (n, m) order;
// lane 0 then adds them in that order, so the sum is rounded exactly as the serial loop rounds
// it.  Terms with an exact zero weight (table columns outside [lo, hi], rows outside the
// column's non-zero range) are left out: adding them would leave the sum unchanged (it starts
// at +0 and never becomes -0).  __syncwarp orders lane 0's store of a cell before the loads of
// the next cells.
struct SmoothArgs {
    float* arr[5];
    const int* win;   // nwin (start column, width) pairs
    const int* rng;   // per table column idx2: first and last row idx1 with a non-zero weight
    const int* itopo; // per prepared column: rows z < itopo are smoothed
    int nwin, mpitch, ghost, nz, rgau, lo, hi;
    const float* gc;
};

__global__ void __launch_bounds__(32) iso_smooth_kernel(const __grid_constant__ SmoothArgs s) {
    extern __shared__ __align__(16) float prod[];
    const int t = blockIdx.x, lane = threadIdx.x;
    const int b = t / 5;
    float* u = s.arr[t - 5 * b] + (long long)s.win[2 * b] * s.mpitch;
    const int* itopo = s.itopo + s.win[2 * b];
    const int nxw = s.win[2 * b + 1];
    const int w = 2 * s.rgau - 1, r1 = s.rgau - 1;
    for (int i = 0; i < nxw; i++)
        for (int k = 0, kn = min(itopo[i], s.nz); k < kn; k++) {
            const int nlo = max(i - r1 + s.lo, 0), nhi = min(i - r1 + s.hi, nxw - 1);
            // lane L forms the products of columns nlo + L and nlo + L + 32; their offsets in the
            // loop order come from a warp prefix sum of the column lengths
            int mlo[2], cnt[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int n = nlo + lane + 32 * h;
                mlo[h] = 0;
                cnt[h] = 0;
                if (n <= nhi) {
                    const int j2 = n - i + r1;  // idx2 - 1
                    mlo[h] = max(k - r1 + s.rng[2 * j2], 0);
                    cnt[h] = max(min(k - r1 + s.rng[2 * j2 + 1], s.nz - 1) - mlo[h] + 1, 0);
                }
            }
            int off[2], total = 0;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                int x = cnt[h];
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, x, d);
                    if (lane >= d) x += y;
                }
                off[h] = total + x - cnt[h];
                total += __shfl_sync(0xffffffffu, x, 31);
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (cnt[h] == 0) continue;
                const int n = nlo + lane + 32 * h;
                const float* col = u + (long long)n * s.mpitch + mlo[h];
                const float* g = s.gc + (n - i + r1) * w + r1 - k + mlo[h];  // gc(m - k + r1 + 1, idx2)
                float* p = prod + off[h];
#pragma unroll 4
                for (int q = 0; q < cnt[h]; q++) p[q] = fm(col[q], g[q]);
            }
            __syncwarp();
            if (lane == 0) {
                float acc = 0.0f;
                int q = 0;
#pragma unroll 4
                for (; q + 4 <= total; q += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(prod + q);
                    acc = fa(fa(fa(fa(acc, v.x), v.y), v.z), v.w);
                }
                for (; q < total; q++) acc = fa(acc, prod[q]);
                u[(long long)i * s.mpitch + k] = acc;
            }
            __syncwarp();
        }
    for (int c = lane; c < nxw; c += 32)  // the replicated rows above z = 0 follow the smoothed row
        for (int g = 1; g <= s.ghost; g++) u[(long long)c * s.mpitch - g] = u[(long long)c * s.mpitch];
}

}  // namespace

namespace {

template <bool FS, bool SUMS>
cudaError_t launch_pair(const IArgs& a, int active, cudaStream_t st, int* launches) {
    const int ntz = a.L.ntz, ncol = a.L.ntx * (TX / TC);
    const int sv = (int)sizeof(float) * (3 * kSmem + 4), ss = (int)sizeof(float) * (2 * kSmem + 4);
    const void* kv = (const void*)iso_velocity_kernel<FS, SUMS>;
    const void* ks = (const void*)iso_stress_kernel<FS, SUMS>;
    static bool attr0[kMaxDevices] = {}, attr1[kMaxDevices] = {};
    if (cudaError_t e = smem_attr_once(kv, sv, attr0)) return e;
    if (cudaError_t e = smem_attr_once(ks, ss, attr1)) return e;
    if (cudaError_t e = tile::launch_columns(kv, ntz, ncol, active, kThreads, sv, st, a, launches)) return e;
    return tile::launch_columns(ks, ntz, ncol, active, kThreads, ss, st, a, launches);
}

}  // namespace

void elastic2d_box(int box[2]) {
    box[0] = SW;
    box[1] = TC + 2 * H;
}

cudaError_t elastic2d_launch_step(const IArgs& a, int active, int nx_max, cudaStream_t st, int* launches) {
    const bool sums = a.f[I_VX] != nullptr;
    const cudaError_t e = a.fs ? (sums ? launch_pair<true, true>(a, active, st, launches)
                                       : launch_pair<true, false>(a, active, st, launches))
                               : (sums ? launch_pair<false, true>(a, active, st, launches)
                                       : launch_pair<false, false>(a, active, st, launches));
    if (e != cudaSuccess || !a.fs) return e;
    ++*launches;
    return tile::launch((const void*)iso_surface_kernel, dim3((nx_max + 127) / 128, active), 128, 0, st, a);
}

cudaError_t elastic2d_smooth(float* const arrays[5], int mpitch, int ghost, int nz, const int* itopo_dev,
                             const int* win_host, int nwin, const std::vector<float>& gc, int rgau, int lo, int hi,
                             cudaStream_t st) {
    if (nwin <= 0) return cudaSuccess;
    SmoothArgs s{};
    for (int i = 0; i < 5; i++) s.arr[i] = arrays[i];
    const int w = 2 * rgau - 1;
    std::vector<int> rng(2 * (size_t)w), buf(2 * (size_t)nwin);  // per table column: non-zero rows
    for (int j = 0; j < w; j++) {
        int a = w, b = -1;
        for (int i = 0; i < w; i++)
            if (gc[(size_t)j * w + i] != 0.0f) {
                a = std::min(a, i);
                b = std::max(b, i);
            }
        rng[2 * j] = a;
        rng[2 * j + 1] = b;
    }
    for (int i = 0; i < 2 * nwin; i++) buf[i] = win_host[i];
    buf.insert(buf.end(), rng.begin(), rng.end());
    int* d_win = nullptr;
    float* d_gc = nullptr;
    cudaError_t e = cudaMalloc(&d_win, sizeof(int) * buf.size());
    if (e == cudaSuccess) e = cudaMalloc(&d_gc, sizeof(float) * gc.size());
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_win, buf.data(), sizeof(int) * buf.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_gc, gc.data(), sizeof(float) * gc.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        s.win = d_win;
        s.rng = d_win + 2 * nwin;
        s.gc = d_gc;
        s.nwin = nwin;
        s.mpitch = mpitch;
        s.ghost = ghost;
        s.nz = nz;
        s.itopo = itopo_dev;
        s.rgau = rgau;
        s.lo = lo;
        s.hi = hi;
        // shared memory: the products of one cell, at most (hi - lo + 1)^2; the kernel gives each
        // lane two table columns (the sigma = 2 table has at most 57 non-zero ones)
        const size_t smem = sizeof(float) * ((size_t)(hi - lo + 1) * (hi - lo + 1) + 4);
        if (smem > 200 * 1024 || hi - lo + 1 > 64) {
            e = cudaErrorInvalidValue;
        } else {
            if (smem > 48 * 1024)
                e = cudaFuncSetAttribute(iso_smooth_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e == cudaSuccess) {
                iso_smooth_kernel<<<5 * nwin, 32, smem, st>>>(s);
                e = cudaGetLastError();
            }
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d_win);
    cudaFree(d_gc);
    return e;
}

bool elastic2d_prepare(int nx, int nz, const float* vp, const float* vs, const float* rho, const int* itopo,
                       float* b2e, float* b1e, float* lm2, float* lam, float* mue) {
    const size_t n = (size_t)nx * nz;
    auto at = [nz](int k, int i) { return (size_t)i * nz + k; };  // Fortran (k, i), 0-based
    std::vector<float> mu(n), lamb(n), busg1(n, 0.0f), busg2(n), musg(n);
    for (int i = 0; i < nx; i++)
        for (int k = 0; k < nz; k++) {
            const size_t c = at(k, i);
            mu[c] = rho[c] * vs[c] * vs[c];
            lamb[c] = rho[c] * vp[c] * vp[c] - 2.0f * mu[c];
        }
    for (int i = 0; i < nx - 1; i++)
        for (int k = 0; k < nz - 1; k++)
            busg1[at(k, i)] = 0.25f * (rho[at(k, i)] + rho[at(k + 1, i)] + rho[at(k + 1, i + 1)] + rho[at(k, i + 1)]);
    for (int i = 0; i < nx; i++) busg1[at(nz - 1, i)] = busg1[at(nz - 2, i)];
    for (int k = 0; k < nz; k++) busg1[at(k, nx - 1)] = busg1[at(k, nx - 2)];
    for (size_t c = 0; c < n; c++) {
        if (busg1[c] == 0.0f || rho[c] == 0.0f) return false;  // YPUB:370, 400
        busg1[c] = 1.0f / busg1[c];
        busg2[c] = 1.0f / rho[c];
    }
    for (int i = 0; i < nx; i++) {
        for (int k = 1; k < nz; k++) b1e[at(k, i)] = 0.5f * (busg1[at(k, i)] + busg1[at(k - 1, i)]);
        b1e[at(0, i)] = busg1[at(0, i)];
    }
    for (int k = 0; k < nz; k++) {
        for (int i = 0; i < nx - 1; i++) b2e[at(k, i)] = 0.5f * (busg2[at(k, i)] + busg2[at(k, i + 1)]);
        b2e[at(k, nx - 1)] = busg2[at(k, nx - 1)];
    }
    for (int i = 0; i < nx; i++) {
        for (int k = 0; k < nz - 1; k++) musg[at(k, i)] = 0.5f * (mu[at(k + 1, i)] + mu[at(k, i)]);
        musg[at(nz - 1, i)] = mu[at(nz - 1, i)];
    }
    for (int i = 0; i < nx - 1; i++)
        for (int k = 1; k < nz; k++) {
            const float q0 = musg[at(k, i)], q1 = musg[at(k, i + 1)], q2 = musg[at(k - 1, i + 1)], q3 = musg[at(k - 1, i)];
            mue[at(k, i)] = (q0 != 0.0f && q1 != 0.0f && q2 != 0.0f && q3 != 0.0f)
                                ? 4.0f / (1.0f / q0 + 1.0f / q1 + 1.0f / q2 + 1.0f / q3)
                                : 0.0f;
        }
    for (int i = 0; i < nx; i++) mue[at(0, i)] = musg[at(0, i)];
    for (int k = 0; k < nz; k++) mue[at(k, nx - 1)] = musg[at(k, nx - 1)];
    for (int k = 0; k < nz; k++) {
        for (int i = 0; i < nx - 1; i++) {
            lam[at(k, i)] = 0.5f * (lamb[at(k, i + 1)] + lamb[at(k, i)]);
            lm2[at(k, i)] = 0.5f * (lamb[at(k, i)] + 2.0f * mu[at(k, i)] + lamb[at(k, i + 1)] + 2.0f * mu[at(k, i + 1)]);
        }
        lam[at(k, nx - 1)] = lamb[at(k, nx - 1)];
        lm2[at(k, nx - 1)] = lamb[at(k, nx - 1)] + 2.0f * mu[at(k, nx - 1)];
    }
    // YPUB:484-501: rows above itopo (1-based) take row itopo's values
    for (float* f : {b2e, b1e, lm2, lam, mue})
        for (int i = 0; i < nx; i++)
            for (int k = std::min(itopo[i], nz) - 1; k >= 1; k--) f[at(k - 1, i)] = f[at(k, i)];
    return true;
}

void elastic2d_gauss_table(int rgau, std::vector<float>* out, int* lo, int* hi) {
    const int w = 2 * rgau - 1, cen = (w + 1) / 2;
    const float pi = 3.1415926f, sigma2 = 2.0f * 2.0f;
    out->assign((size_t)w * w, 0.0f);
    for (int j = 1; j <= w; j++)
        for (int i = 1; i <= w; i++) {
            const float dis = (float)((j - cen) * (j - cen) + (i - cen) * (i - cen));
            (*out)[(size_t)(j - 1) * w + (i - 1)] = 1.0f / (2.0f * pi * sigma2) * std::exp(-(dis / (2.0f * sigma2)));
        }
    float sum = 0.0f;
    for (int j = 0; j < w; j++)
        for (int i = 0; i < w; i++) sum = sum + (*out)[(size_t)j * w + i];
    int l = w, h = -1;
    for (int j = 0; j < w; j++)
        for (int i = 0; i < w; i++) {
            float& v = (*out)[(size_t)j * w + i];
            v = v / sum;
            if (v != 0.0f) {
                l = std::min(l, std::min(i, j));
                h = std::max(h, std::max(i, j));
            }
        }
    *lo = l;
    *hi = h;
}

void elastic2d_stamp(int nx, int nz, int sx, int sz, int rgau, const std::vector<float>& gc, int* box,
                     std::vector<float>* out) {
    const int w = 2 * rgau - 1, r1 = rgau - 1;
    int xlo = 1 << 30, xhi = -1, zlo = 1 << 30, zhi = -1;
    for (int x = std::max(sx - r1, 0); x <= std::min(sx + r1, nx - 1); x++)
        for (int z = std::max(sz - r1, 0); z <= std::min(sz + r1, nz - 1); z++)
            if (gc[(size_t)(x - sx + r1) * w + (z - sz + r1)] != 0.0f) {
                xlo = std::min(xlo, x); xhi = std::max(xhi, x);
                zlo = std::min(zlo, z); zhi = std::max(zhi, z);
            }
    if (xhi < 0) {
        box[0] = box[1] = box[2] = box[3] = 0;
        return;
    }
    box[0] = xlo; box[1] = zlo; box[2] = xhi - xlo + 1; box[3] = zhi - zlo + 1;
    for (int x = xlo; x <= xhi; x++)
        for (int z = zlo; z <= zhi; z++) out->push_back(gc[(size_t)(x - sx + r1) * w + (z - sz + r1)]);
}

}  // namespace sfd
