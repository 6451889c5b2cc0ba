// Visco-elastic (P-SV, one standard-linear-solid memory variable per stress) rotated-staggered-
// grid time step: the full scheme of forward/Q_forward/Q_multishot_fd_subroutine_fsbc_zy_rotated.f90
// (QS:695-1337) with vs > 0, flat surface.  Every field is kept in the reference's split form
// (x, z and memory parts), 22 per cell:
//   vxx vxz vzx vzz | sxxx sxxz sxxr | szzx szzz szzr | sxzx sxzz sxzr | rxxx rxxz rxxr |
//   rzzx rzzz rzzr | rxzx rxzz rxzr
// with the five sums vx, vz, sxx, szz, sxz (QS:1273-1337) beside them, written by the kernel that
// completes them, and one step is two kernels:
//   velocity: sxx, sxz, szz staged on the tile plus halo;
//             vxx += dt b Dx0 sxx, vxz += dt b Dz0 sxz, vzx += dt b Dx0 sxz, vzz += dt b Dz0 szz,
//             x parts times the x sponge, z parts times the z sponge        (QS:713-748, 969-990)
//   stress:   vx, vz staged on the tile plus halo; d1 = Dx1 vx, d2 = Dx1 vz,
//             d3 = Dz1 vx, d4 = Dz1 vz; with r.. the memory sums of the previous step,
//             sxxx += dt (q1 d1), sxxz += dt (q2 d4), sxxr += dt rxx          (calpstrxx)
//             szzx += dt (q2 d1), szzz += dt (q1 d4), szzr += dt rzz          (calpstrzz)
//             sxzx += dt (q3 d2), sxzz += dt (q3 d3), sxzr += dt rxz          (calpstrxz)
//             rxxx += f (m1 d1), rxxz += f (m2 d4), rxxr += f rxx            (calprxx)
//             rzzz += f (m1 d4), rzzx += f (m2 d1), rzzr += f rzz            (calprzz)
//             rxzx += f (m3 d2), rxzz += f (m3 d3), rxzr += f rxz            (calprxz)
//             x parts times the x' sponge, z parts times the z' sponge, the source added to
//             sxxx and szzx after their sponge (QS:801, 1340-1390)
//   with q1 = lambda tau_p, q2 = lambda tau_p - 2 mu tau_s, q3 = mu tau_s, m1 = lambda (tau_p - 1),
//   m2 = lambda (tau_p - 1) - 2 mu (tau_s - 1), m3 = mu (tau_s - 1), f = dt (-1 / tau_sigma)
//   (QS:473-551), rounded in the reference's order.  Records: strzz (record1) and strxx (record2)
//   at the receivers after the step (QM:452-459).
// Every multiply and add is rounded separately in the reference's order, so the kernels agree
// bit for bit with the FP32 restatement in oracle/q_oracle.cpp.
//
// Bound: memory in the stress kernel (DRAM at 4.9 TB/s), issue and shared-memory loads in the velocity kernel
// (72% and 66%, DRAM at 3.0 TB/s).  The split fields (22 read and written) and seven model arrays are 204 B a cell; the
// two kernels move 244 B (sums written once and read once, halos from L2).  One TMA box per sum field
// stages a tile with its halo while every thread loads the split parts of its one cell, so that all
// loads of a CTA are in flight together; small CTAs cover one another's waits.
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "sfd_internal.h"
#include "tile_stage.cuh"

namespace sfd {
namespace {

constexpr int TX = kTileX, TZ = kTileZ;
// Tiles of 64 rows by 4 columns, one thread per cell, eight (velocity) and five (stress) CTAs per SM.
// Step of 8 shots of 780 x 580 (3.6 M cells): 64 x 64 tiles with 16 cells per thread in turn 225 us
// (before); 8 columns 195 us; 4 columns 168 us; 2 columns 165 us on this grid, with a
// sixfold halo.
constexpr int TC = 4, kThreads = TC * TZ;
constexpr int kMinV = 8, kMinS = 5;
constexpr int H = 5;                  // rotated-staggered reach
constexpr int HZ = 8;                 // z halo rounded for float4 staging
constexpr int SROWS = TC + 2 * H;
constexpr int SW = TZ + 2 * HZ;       // 80
constexpr int SMEM = SROWS * SW;      // floats per staged field

__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }

// QS:843-966, the same rounding order as viscoac2d.cu
template <bool XDIR, int FLAG>
__device__ __forceinline__ float rsg(const float* s, int r, int c, const float* a, float h) {
    auto u = [&](int dk, int di) { return s[(r + di) * SW + c + dk]; };
    float acc = 0.0f;
#pragma unroll
    for (int m = 0; m < 5; m++) {
        float t;
        if (FLAG == 0) {
            t = XDIR ? fs(fa(fs(u(m, m), u(-1 - m, -1 - m)), u(-1 - m, m)), u(m, -1 - m))
                     : fa(fs(fs(u(m, m), u(-1 - m, -1 - m)), u(-1 - m, m)), u(m, -1 - m));
        } else {
            t = XDIR ? fs(fa(fs(u(1 + m, 1 + m), u(-m, -m)), u(-m, 1 + m)), u(1 + m, -m))
                     : fa(fs(fs(u(1 + m, 1 + m), u(-m, -m)), u(-m, 1 + m)), u(1 + m, -m));
        }
        acc = (m == 0) ? fm(a[0], t) : fa(acc, fm(a[m], t));
    }
    return fm(h, acc);
}

// both derivatives of one field: their four-point differences share the first subtraction
template <int FLAG>
__device__ __forceinline__ void rsg_both(const float* s, int r, int c, const float* a, float hx, float hz, float* dx,
                                         float* dz) {
    float ax = 0.0f, az = 0.0f;
#pragma unroll
    for (int m = 0; m < 5; m++) {
        const int hi = FLAG == 0 ? m : 1 + m, lo = FLAG == 0 ? -1 - m : -m;
        const float t = fs(s[(r + hi) * SW + c + hi], s[(r + lo) * SW + c + lo]);
        const float p = s[(r + hi) * SW + c + lo], q = s[(r + lo) * SW + c + hi];
        const float tx = fm(a[m], fs(fa(t, p), q)), tz = fm(a[m], fa(fs(t, p), q));
        ax = m == 0 ? tx : fa(ax, tx);
        az = m == 0 ? tz : fa(az, tz);
    }
    *dx = fm(hx, ax);
    *dz = fm(hz, az);
}

struct TileRef {
    int shot, tile, x0, z0;
    ShotDev sd;
};

__device__ __forceinline__ bool tile_of(const EArgs& a, TileRef& t) {
    t.shot = a.slot_to_shot[blockIdx.z];
    t.sd = a.shots[t.shot];
    t.x0 = (a.col0 + (int)blockIdx.y) * TC;
    t.z0 = blockIdx.x * TZ;
    t.tile = t.x0 / TX * a.L.ntz + blockIdx.x;  // the 64 x 64 tile of the receiver lists
    return t.x0 < t.sd.nx;
}

__device__ __forceinline__ long long cell(const EArgs& a, int shot, int x, int z) {
    return (long long)shot * a.L.shot_stride + (long long)(x + a.L.gx) * a.L.pitch + a.L.gz + z;
}

// One thread requests the tile plus halo of NF sum fields (x coordinate at least 3, z a multiple of 64)
template <int NF>
__device__ __forceinline__ void stage(float* s, uint64_t* bar, const EArgs& a, const TileRef& t, const int* field) {
    tile::expect(bar, 4u * NF * SMEM);
#pragma unroll
    for (int f = 0; f < NF; f++)
        tile::box(s + f * SMEM, &a.tm[field[f] - E_VX], a.L.gz + t.z0 - HZ, a.L.gx + t.x0 - H, t.shot, bar);
}

// The same without the slabs of the sums, from the NP split parts from f0 on (the caller's __syncthreads follows)
template <int NP>
__device__ __forceinline__ void stage_parts(float* s, const EArgs& a, const TileRef& t, int f0) {
    for (int i = threadIdx.x; i < SMEM / 4; i += kThreads) {
        const int r = i / (SW / 4), c = 4 * (i % (SW / 4));
        const long long off = cell(a, t.shot, t.x0 - H + r, t.z0 - HZ + c);
        float4 v = *reinterpret_cast<const float4*>(a.f[f0] + off);
#pragma unroll
        for (int k = 1; k < NP; k++) {
            const float4 p = *reinterpret_cast<const float4*>(a.f[f0 + k] + off);
            v = make_float4(fa(v.x, p.x), fa(v.y, p.y), fa(v.z, p.z), fa(v.w, p.w));
        }
        *reinterpret_cast<float4*>(s + r * SW + c) = v;
    }
}

// one split-sponge factor applied in QS order (left table, then right table)
__device__ __forceinline__ float xs(float u, int x, int n, int np, const float* tn, const float* tp) {
    if (x <= np) u = fm(u, tn[x]);
    if (x >= n - np - 1) u = fm(u, tp[n - 1 - x]);
    return u;
}

// SUMS = false: no memory for the slabs of the sums.  The tile and its halo are summed by the threads: 52 ms
// against 41 for 230 steps of 8 shots of 780 x 580.
template <bool SUMS>
__global__ void __launch_bounds__(kThreads, kMinV) e_velocity_kernel(const __grid_constant__ EArgs a) {
    extern __shared__ __align__(128) float smem[];
    const float* sSxx = smem;
    const float* sSxz = smem + SMEM;
    const float* sSzz = smem + 2 * SMEM;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 3 * SMEM);
    TileRef t;
    const bool on = tile_of(a, t);
    tile::bar_init(bar);
    tile::release();
    tile::acquire();
    if (!on) return;
    if (!SUMS) {
        stage_parts<3>(smem, a, t, E_SXXX);
        stage_parts<3>(smem + SMEM, a, t, E_SXZX);
        stage_parts<3>(smem + 2 * SMEM, a, t, E_SZZX);
        __syncthreads();
    } else if (threadIdx.x == 0) {
        const int f[3] = {E_SXX, E_SXZ, E_SZZ};
        stage<3>(smem, bar, a, t, f);
    }
    const int nx = t.sd.nx, nz = a.nz;
    const int r = threadIdx.x / TZ, z = threadIdx.x % TZ, gx = t.x0 + r, gz = t.z0 + z;
    if (gx >= nx || gz >= nz) {
        if (SUMS) tile::staged(bar, a.err_flag);  // leave with the CTA's copies landed
        return;
    }
    const long long c = cell(a, t.shot, gx, gz);
    float n_xx = a.f[E_VXX][c], n_xz = a.f[E_VXZ][c], n_zx = a.f[E_VZX][c], n_zz = a.f[E_VZZ][c];
    const float dtb = fm(a.dt, __ldg(a.busg + (long long)min(t.sd.x0 + gx, a.nx_model - 1) * a.mpitch + gz));
    if (SUMS && !tile::staged(bar, a.err_flag)) return;
    n_xx = fa(n_xx, fm(dtb, rsg<true, 0>(sSxx, r + H, z + HZ, a.a, a.hx)));  // QS:713-720
    n_zz = fa(n_zz, fm(dtb, rsg<false, 0>(sSzz, r + H, z + HZ, a.a, a.hz)));  // QS:741-748
    float d_zx, d_xz;
    rsg_both<0>(sSxz, r + H, z + HZ, a.a, a.hx, a.hz, &d_zx, &d_xz);
    n_xz = fa(n_xz, fm(dtb, d_xz));  // QS:722-729
    n_zx = fa(n_zx, fm(dtb, d_zx));  // QS:733-740
    const float* tb = a.spg;
    const int st = a.spg_stride;
    if (gx <= a.npx || gx >= nx - a.npx - 1) {
        n_xx = xs(n_xx, gx, nx, a.npx, tb + 0 * st, tb + 1 * st);
        n_zx = xs(n_zx, gx, nx, a.npx, tb + 0 * st, tb + 1 * st);
    }
    if (gz <= a.npz || gz >= nz - a.npz - 1) {
        n_xz = xs(n_xz, gz, nz, a.npz, tb + 2 * st, tb + 3 * st);
        n_zz = xs(n_zz, gz, nz, a.npz, tb + 2 * st, tb + 3 * st);
    }
    a.f[E_VXX][c] = n_xx; a.f[E_VXZ][c] = n_xz; a.f[E_VZX][c] = n_zx; a.f[E_VZZ][c] = n_zz;
    if (SUMS) {
        a.f[E_VX][c] = fa(n_xx, n_xz);  // QS:1273-1291
        a.f[E_VZ][c] = fa(n_zx, n_zz);
    }
}

template <bool SUMS>
__global__ void __launch_bounds__(kThreads, kMinS) e_stress_kernel(const __grid_constant__ EArgs a) {
    extern __shared__ __align__(128) float smem[];
    const float* sVx = smem;
    const float* sVz = smem + SMEM;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 2 * SMEM);
    TileRef t;
    const bool on = tile_of(a, t);
    tile::bar_init(bar);
    tile::release();
    tile::acquire();
    if (!on) return;
    if (!SUMS) {
        stage_parts<2>(smem, a, t, E_VXX);
        stage_parts<2>(smem + SMEM, a, t, E_VZX);
        __syncthreads();
    } else if (threadIdx.x == 0) {
        const int f[2] = {E_VX, E_VZ};
        stage<2>(smem, bar, a, t, f);
    }
    const int nx = t.sd.nx, nz = a.nz;
    const ShotDev& sd = t.sd;
    const int r = threadIdx.x / TZ, z = threadIdx.x % TZ, gx = t.x0 + r, gz = t.z0 + z;
    const bool in = gx < nx && gz < nz;
    const long long c = cell(a, t.shot, gx, gz);
    float w[18];  // sxxx sxxz sxxr szzx szzz szzr sxzx sxzz sxzr rxxx rxxz rxxr rzzx rzzz rzzr rxzx rxzz rxzr
    float q1, q2, q3, m1, m2, m3;
    if (in) {
#pragma unroll
        for (int k = 0; k < 18; k++) w[k] = a.f[E_SXXX + k][c];
        const long long mi = (long long)min(sd.x0 + gx, a.nx_model - 1) * a.mpitch + gz;
        q1 = __ldg(a.q1 + mi); q2 = __ldg(a.q2 + mi); q3 = __ldg(a.q3 + mi);
        m1 = __ldg(a.m1 + mi); m2 = __ldg(a.m2 + mi); m3 = __ldg(a.m3 + mi);
    }
    const float wav = __ldg(a.wavelets + sd.wav_off + a.step);
    if (SUMS && !tile::staged(bar, a.err_flag)) return;
    if (in) {
        const float dt = a.dt, f = a.f_mem;
        float d1, d2, d3, d4;
        rsg_both<1>(sVx, r + H, z + HZ, a.a, a.hx, a.hz, &d1, &d3);  // Dx1 vx, Dz1 vx
        rsg_both<1>(sVz, r + H, z + HZ, a.a, a.hx, a.hz, &d2, &d4);  // Dx1 vz, Dz1 vz
        const float rxx = fa(fa(w[9], w[10]), w[11]);   // memory sums of the previous step
        const float rzz = fa(fa(w[12], w[13]), w[14]);
        const float rxz = fa(fa(w[15], w[16]), w[17]);
        // calpstrxx, calpstrzz, calpstrxz (QS:993-1132)
        w[0] = fa(w[0], fm(dt, fm(q1, d1)));
        w[1] = fa(w[1], fm(dt, fm(q2, d4)));
        w[2] = fa(w[2], fm(dt, rxx));
        w[3] = fa(w[3], fm(dt, fm(q2, d1)));
        w[4] = fa(w[4], fm(dt, fm(q1, d4)));
        w[5] = fa(w[5], fm(dt, rzz));
        w[6] = fa(w[6], fm(dt, fm(q3, d2)));
        w[7] = fa(w[7], fm(dt, fm(q3, d3)));
        w[8] = fa(w[8], fm(dt, rxz));
        // calprxx, calprzz, calprxz (QS:1135-1269)
        w[9] = fa(w[9], fm(f, fm(m1, d1)));
        w[10] = fa(w[10], fm(f, fm(m2, d4)));
        w[11] = fa(w[11], fm(f, rxx));
        w[12] = fa(w[12], fm(f, fm(m2, d1)));
        w[13] = fa(w[13], fm(f, fm(m1, d4)));
        w[14] = fa(w[14], fm(f, rzz));
        w[15] = fa(w[15], fm(f, fm(m3, d2)));
        w[16] = fa(w[16], fm(f, fm(m3, d3)));
        w[17] = fa(w[17], fm(f, rxz));
        // x parts (0, 3, ...) take the x sponge, z parts (1, 4, ...) the z sponge
        const float* tb = a.spg;
        const int st = a.spg_stride;
        if (gx <= a.npx || gx >= nx - a.npx - 1)
#pragma unroll
            for (int k = 0; k < 18; k += 3) w[k] = xs(w[k], gx, nx, a.npx, tb + 4 * st, tb + 5 * st);
        if (gz <= a.npz || gz >= nz - a.npz - 1)
#pragma unroll
            for (int k = 1; k < 18; k += 3) w[k] = xs(w[k], gz, nz, a.npz, tb + 6 * st, tb + 7 * st);
        const int bx = gx - sd.stamp_x0, bz = gz - sd.stamp_z0;
        if (bx >= 0 && bx < sd.stamp_w && bz >= 0 && bz < sd.stamp_h) {  // QS:801, 1384
            const float src = __fdiv_rn(fm(fm(wav, __ldg(a.stamps + sd.stamp_off + bx * sd.stamp_h + bz)), dt), a.dz2);
            w[0] = fa(src, w[0]);
            w[3] = fa(src, w[3]);
        }
#pragma unroll
        for (int k = 0; k < 18; k++) a.f[E_SXXX + k][c] = w[k];
        if (SUMS) {
            a.f[E_SXX][c] = fa(fa(w[0], w[1]), w[2]);  // QS:1294-1337
            a.f[E_SZZ][c] = fa(fa(w[3], w[4]), w[5]);
            a.f[E_SXZ][c] = fa(fa(w[6], w[7]), w[8]);
        }
    }
    // receivers: record1 = strzz, record2 = strxx after the step (QM:452-459)
    const int* trp = a.tile_rec_ptr + sd.tile_rec_base + t.tile;
    const int rb = trp[0], re = trp[1];
    if (re > rb) {
        __syncthreads();
        for (int j = rb + threadIdx.x; j < re; j += kThreads) {
            const int ridx = a.tile_rec_idx[j];
            const int x = a.rec_x[sd.rec_list + ridx];
            if (x < t.x0 || x >= t.x0 + TC) continue;  // another CTA of the 64 x 64 tile holds it
            const long long c = cell(a, t.shot, x, a.rec_z[sd.rec_list + ridx]);
            const long long o = sd.rec_base + (long long)a.step * sd.nrec + ridx;
            auto sum = [&](int s, int f0) { return SUMS ? a.f[s][c] : fa(fa(a.f[f0][c], a.f[f0 + 1][c]), a.f[f0 + 2][c]); };
            a.records[o] = sum(E_SZZ, E_SZZX);
            a.records2[o] = sum(E_SXX, E_SXXX);
        }
    }
}

}  // namespace

void viscoel2d_box(int box[2]) {
    box[0] = SW;
    box[1] = SROWS;
}

template <bool SUMS>
static cudaError_t launch_pair(const EArgs& a, int active, cudaStream_t st, int* launches) {
    const int ntz = a.L.ntz, ncol = a.L.ntx * (TX / TC);
    const int sv = (int)sizeof(float) * (3 * SMEM + 4), ss = (int)sizeof(float) * (2 * SMEM + 4);
    const void* kv = (const void*)e_velocity_kernel<SUMS>;
    const void* ks = (const void*)e_stress_kernel<SUMS>;
    static bool attr0[kMaxDevices] = {}, attr1[kMaxDevices] = {};
    if (cudaError_t e = smem_attr_once(kv, sv, attr0)) return e;
    if (cudaError_t e = smem_attr_once(ks, ss, attr1)) return e;
    if (cudaError_t e = tile::launch_columns(kv, ntz, ncol, active, kThreads, sv, st, a, launches)) return e;
    return tile::launch_columns(ks, ntz, ncol, active, kThreads, ss, st, a, launches);
}
cudaError_t viscoel2d_launch_step(const EArgs& a, int active, cudaStream_t st, int* launches) {
    return a.f[E_VX] ? launch_pair<true>(a, active, st, launches) : launch_pair<false>(a, active, st, launches);
}

// QS:434-469 (density averaged in place, then buoyancy) and QS:473-551 (Blanch's tau for P and S),
// single precision in the reference's operation order, and the six stress-update coefficients.
// qp / qs == nullptr: Q = 1e5 (QM:418-419).
void viscoel2d_prepare(int nx, int nz, const float* vp, const float* vs, const float* rho, const float* qp,
                       const float* qs, float f0, float* busg, float* q1, float* q2, float* q3, float* m1, float* m2,
                       float* m3, float* rtau_out) {
    std::vector<float> r(rho, rho + (size_t)nx * nz);
    auto R = [&](int k, int i) -> float& { return r[(size_t)i * nz + k]; };
    for (int i = 0; i < nx - 1; i++)
        for (int k = 0; k < nz - 1; k++) R(k, i) = 0.25f * (R(k, i) + R(k + 1, i) + R(k + 1, i + 1) + R(k, i + 1));
    for (int i = 0; i < nx; i++) R(nz - 1, i) = R(nz - 2, i);
    for (int k = 0; k < nz; k++) R(k, nx - 1) = R(k, nx - 2);
    const float pi = 3.1415926f;
    const float flow = 2.0f * 2.0f * pi;
    const float fup = 2.5f * f0 * 2.0f * pi;
    const float tss = 1.0f / ((fup - flow) / 2.0f);
    const float nlow = std::log((tss * tss) * (flow * flow) + 1.0f);
    const float nup = std::log((tss * tss) * (fup * fup) + 1.0f);
    const float dlow = std::atan(flow * tss) - (flow * tss) / (1.0f + (tss * tss) * (flow * flow));
    const float dup = std::atan(fup * tss) - (fup * tss) / (1.0f + (tss * tss) * (fup * fup));
    for (size_t c = 0; c < (size_t)nx * nz; c++) {
        const float rr = r[c];
        busg[c] = 1.0f / rr;
        const float mu = rr * (vs[c] * vs[c]);
        const float lambmu = rr * (vp[c] * vp[c]);
        const float qpv = (qp ? qp[c] : 100000.0f) * (18.0f / 20.0f);
        const float qsv = (qs ? qs[c] : 100000.0f) * (18.0f / 20.0f);
        float tp = 0.0f, ts = 0.0f;
        if (dup - dlow != 0.0f) {
            tp = 1.0f / qpv * (nup - nlow) / (dup - dlow);
            ts = 1.0f / qsv * (nup - nlow) / (dup - dlow);
        }
        const float taup = (tp * tss + tss) / tss;
        const float taus = (ts * tss + tss) / tss;
        q1[c] = lambmu * taup;
        q2[c] = lambmu * taup - 2.0f * mu * taus;
        q3[c] = mu * taus;
        m1[c] = lambmu * (taup - 1.0f);
        m2[c] = lambmu * (taup - 1.0f) - 2.0f * mu * (taus - 1.0f);
        m3[c] = mu * (taus - 1.0f);
    }
    *rtau_out = 1.0f / tss;
}

}  // namespace sfd
