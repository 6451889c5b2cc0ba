// Default (fast) viscoacoustic step of SFD_VISCOAC_2D: the rotated-staggered-grid scheme of
// forward/Q_forward/Q_multishot_fd_subroutine_fsbc_zy_rotated.f90 (QS:751-835 and its leaves
// QS:843-1337) with vs = 0, FMA contraction, two kernels per time step.
//
// State, all of it in place.  Everywhere: vx, vz, the merged stress sigma = (sx + sz) + sr (QS strxx) and
// the merged memory variable r = (rx + rz) + rr.  Away from the sponge bands the split parts only ever
// appear summed, so the step updates the sums:
//   sigma += dt (p1 (d1 + d4) + r_old) + source,   r += f (p2 (d1 + d4) + r_old),
// with f = -dt / tau_sigma, p1 = M tau_eps / tau_sigma, p2 = M (tau_eps / tau_sigma - 1),
// d1 = 0.5/dx Dx1 vx, d4 = 0.5/dz Dz1 vz.  In the bands (x <= npx, x >= nx - npx - 1, z <= npz,
// z >= nz - npz - 1) the split sponge of QS:609-654 multiplies the x and z parts separately, so
// there the split parts sx, sz, sr, rx, rz, rr are kept and updated in the reference's form; sigma and r
// are their sums.  Cells outside a shot's grid hold zeros.
//
// A CTA owns a tile of 64 rows by TC columns; the fields that a kernel differentiates arrive by TMA, a box
// with halo per field, while the threads load their own values.  The rotated stencils (QS:843-966,
// (0.5/d) sum_m a_m t_m over four-point differences t_m) are sums of products, one input column at a time:
// a thread owns four rows of four (velocity) or two (stress) columns, holds one input column's window of 16
// values in registers and adds each tap with one FMA into the outputs that use it.
//
// Bound: memory (40 B a cell and step of state, 88 B in the bands; the model stays in L2).  16 shots of
// 1124 x 1124 (20.2 M cells): 76 us velocity at 4.9 TB/s, 165 us stress at 4.2.  A kernel that marched down x
// with both phases in one CTA (32 B a cell, but 280 B of shared loads a cell, the velocities of the z halo
// computed twice, and a second kernel for the bands) took 258 + 63 us: few warps in flight behind its
// barriers, and the shared-memory pipe at 86%.  Stress with four columns per thread: 2% slower (10 warps an
// SM); with one: 17% slower (shared loads); tiles of 8 or 32 columns: 1-3% slower; the split parts requested
// a column ahead: 3% slower.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "sfd_internal.h"
#include "tile_stage.cuh"

namespace sfd {
namespace {

constexpr int TX = kTileX, TZ = kTileZ;
constexpr int TC = 16;                   // columns of a tile
constexpr int UV = 4, US = 2;            // columns per thread of the velocity and the stress kernel, four rows each
constexpr int threads_of(int u) { return TC / u * (TZ / 4); }
constexpr int H = 5;                     // RSG reach (offsets -5 .. +4 of sigma, -4 .. +5 of the velocities)
constexpr int HZ = 8;                    // z halo, a multiple of four
constexpr int SW = TZ + 2 * HZ;          // 80
constexpr int SROWS = TC + 2 * H - 1;
constexpr int SMEM = SROWS * SW;         // floats per staged field
constexpr int SMEM_A = (SMEM + 31) / 32 * 32;  // the second box starts on 128 bytes

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ void st4(float* p, const float* v) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void unpack(float* o, const float4& v) { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }

// Split-sponge factors of coordinate c (QS:609-654): table n applies at c <= np, table p at
// c >= n - np - 1 (both in the product for a grid narrower than two bands)
__device__ __forceinline__ float sponge_factor(int c, int n, int np, const float* tn, const float* tp) {
    float f = 1.0f;
    if (c >= 0 && c <= np) f *= __ldg(tn + c);
    if (c >= n - np - 1 && c < n) f *= __ldg(tp + n - 1 - c);
    return f;
}
__device__ __forceinline__ bool in_band(int c, int n, int np) { return c <= np || c >= n - np - 1; }

// a thread's place: columns x .. x + 3, rows z .. z + 3; the tile's first cell, whether it has band cells
struct Place {
    int shot, x0, z0, x, z, row, zq;
    bool edge;
    long long c;  // slab offset of (x, z)
};

template <int U>
__device__ __forceinline__ Place place(const QFastArgs& A, const ShotDev& sd, int shot) {
    const QArgs& a = A.q;
    Place t;
    t.shot = shot;
    t.x0 = (A.col0 + (int)blockIdx.y) * TC;
    t.z0 = blockIdx.x * TZ;
    t.row = U * (int)(threadIdx.x / (TZ / 4));
    t.zq = threadIdx.x % (TZ / 4);
    t.x = t.x0 + t.row;
    t.z = t.z0 + 4 * t.zq;
    t.edge = !(t.x0 > a.npx && t.x0 + TC <= sd.nx - a.npx - 1 && t.z0 > a.npz && t.z0 + TZ <= a.nz - a.npz - 1);
    t.c = (long long)shot * a.L.shot_stride + (long long)(t.x + a.L.gx) * a.L.pitch + a.L.gz + t.z;
    return t;
}

__device__ __forceinline__ const float* model_at(const QArgs& a, const ShotDev& sd, const float* m, int x, int z) {
    return m + (long long)min(sd.x0 + x, a.nx_model - 1) * a.mpitch + z;
}

__device__ __forceinline__ void window(float w[16], const float* row) {
#pragma unroll
    for (int i = 0; i < 4; i++) unpack(w + 4 * i, ld4(row + 4 * i));
}

__global__ void __launch_bounds__(threads_of(UV), 8) viscoac2d_fast_velocity_kernel(const __grid_constant__ QFastArgs A) {
    constexpr int U = UV;
    __shared__ __align__(128) float sS[SMEM_A];
    __shared__ uint64_t bar;
    const QArgs& a = A.q;
    const int shot = a.slot_to_shot[blockIdx.z];
    const ShotDev sd = a.shots[shot];
    const Place t = place<U>(A, sd, shot);
    tile::bar_init(&bar);
    tile::release();
    tile::acquire();
    const int nx = sd.nx, nz = a.nz;
    if (t.x0 >= nx) return;
    if (threadIdx.x == 0) {
        tile::expect(&bar, 4u * SMEM);
        tile::box(sS, &A.tm_s, a.L.gz + t.z0 - HZ, a.L.gx + t.x0 - H, shot, &bar);
    }
    float4 vxo[U], vzo[U], bu[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        vxo[u] = vzo[u] = bu[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t.x + u < nx && t.z < nz) {
            vxo[u] = ld4(A.vx + t.c + u * a.L.pitch);
            vzo[u] = ld4(A.vz + t.c + u * a.L.pitch);
            bu[u] = ldg4(model_at(a, sd, a.busg, t.x + u, t.z));
        }
    }
    if (!tile::staged(&bar, A.err_flag)) return;
    // d/dx = h (DE + DF), d/dz = h (DE - DF) with the main- and anti-diagonal sums
    //   DE = sum_m a_m [s(x+m, z+m) - s(x-1-m, z-1-m)],  DF = sum_m a_m [s(x+m, z-1-m) - s(x-1-m, z+m)];
    // staged column k is x - 5 + k; w[i] = s(., z - 8 + i)
    float de[U][4], df[U][4];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int j = 0; j < 4; j++) de[u][j] = df[u][j] = 0.0f;
#pragma unroll
    for (int k = 0; k < 9 + U; k++) {
        float w[16];
        window(w, sS + (t.row + k) * SW + 4 * t.zq);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int kk = k - u;
            if (kk < 0 || kk > 9) continue;
            const int m = kk >= 5 ? kk - 5 : 4 - kk;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (kk >= 5) {  // column x + m
                    de[u][j] = fmaf(a.a[m], w[8 + j + m], de[u][j]);
                    df[u][j] = fmaf(a.a[m], w[7 + j - m], df[u][j]);
                } else {        // column x - 1 - m
                    de[u][j] = fmaf(-a.a[m], w[7 + j - m], de[u][j]);
                    df[u][j] = fmaf(-a.a[m], w[8 + j + m], df[u][j]);
                }
            }
        }
    }
    if (t.z >= nz) return;
    const float cx = a.dt * a.hx, cz = a.dt * a.hz;
    float fz[4];
    if (t.edge) {
#pragma unroll
        for (int j = 0; j < 4; j++)  // spgzn, spgzp; zero outside the grid
            fz[j] = t.z + j < nz ? sponge_factor(t.z + j, nz, a.npz, a.spg + 2 * a.spg_stride, a.spg + 3 * a.spg_stride)
                                 : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        if (t.x + u >= nx) break;
        float vx[4], vz[4], b[4];
        unpack(vx, vxo[u]);
        unpack(vz, vzo[u]);
        unpack(b, bu[u]);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            vx[j] = fmaf(b[j] * cx, de[u][j] + df[u][j], vx[j]);
            vz[j] = fmaf(b[j] * cz, de[u][j] - df[u][j], vz[j]);
        }
        if (t.edge) {  // QS:609-654: vx in x, vz in z
            const float fx = sponge_factor(t.x + u, nx, a.npx, a.spg, a.spg + a.spg_stride);  // spgxn, spgxp
#pragma unroll
            for (int j = 0; j < 4; j++) {
                vx[j] = t.z + j < nz ? vx[j] * fx : 0.0f;
                vz[j] = t.z + j < nz ? vz[j] * fz[j] : 0.0f;
            }
        }
        st4(A.vx + t.c + u * a.L.pitch, vx);
        st4(A.vz + t.c + u * a.L.pitch, vz);
    }
}

__global__ void __launch_bounds__(threads_of(US), 5) viscoac2d_fast_stress_kernel(const __grid_constant__ QFastArgs A) {
    constexpr int U = US;
    __shared__ __align__(128) float sV[2 * SMEM_A];
    __shared__ uint64_t bar;
    const QArgs& a = A.q;
    const int shot = a.slot_to_shot[blockIdx.z];
    const ShotDev sd = a.shots[shot];
    const Place t = place<U>(A, sd, shot);
    tile::bar_init(&bar);
    tile::release();
    tile::acquire();
    const int nx = sd.nx, nz = a.nz;
    if (t.x0 >= nx) return;
    if (threadIdx.x == 0) {
        tile::expect(&bar, 8u * SMEM);
        tile::box(sV, &A.tm_vx, a.L.gz + t.z0 - HZ, a.L.gx + t.x0 - H + 1, shot, &bar);
        tile::box(sV + SMEM_A, &A.tm_vz, a.L.gz + t.z0 - HZ, a.L.gx + t.x0 - H + 1, shot, &bar);
    }
    float4 p1v[U], p2v[U], so[U], ro[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        p1v[u] = p2v[u] = so[u] = ro[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t.x + u < nx && t.z < nz) {
            so[u] = ld4(A.s + t.c + u * a.L.pitch);
            ro[u] = ld4(A.r + t.c + u * a.L.pitch);
            p1v[u] = ldg4(model_at(a, sd, a.p1, t.x + u, t.z));
            p2v[u] = ldg4(model_at(a, sd, a.p2, t.x + u, t.z));
        }
    }
    const float wav = __ldg(a.wavelets + sd.wav_off + a.step);
    if (!tile::staged(&bar, A.err_flag)) return;
    // d/dx of vx: sum_m a_m [(P(z+1+m) + P(z-m)) - (N(z-m) + N(z+1+m))], d/dz of vz:
    // sum_m a_m [(P(z+1+m) - P(z-m)) + (N(z+1+m) - N(z-m))], P = column x+1+m, N = column x-m;
    // staged column k is x - 4 + k; w[i] = v(., z - 4 + i)
    float d1[U][4], d4[U][4];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int j = 0; j < 4; j++) d1[u][j] = d4[u][j] = 0.0f;
#pragma unroll
    for (int f = 0; f < 2; f++) {
#pragma unroll
        for (int k = 0; k < 9 + U; k++) {
            float w[16];
            window(w, sV + f * SMEM_A + (t.row + k) * SW + 4 * t.zq + HZ - 4);
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int kk = k - u;
                if (kk < 0 || kk > 9) continue;
                const int m = kk >= 5 ? kk - 5 : 4 - kk;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float hi = w[5 + j + m], lo = w[4 + j - m];
                    if (f == 0) {  // P: +(hi + lo), N: -(lo + hi)
                        const float sg = kk >= 5 ? a.a[m] : -a.a[m];
                        d1[u][j] = fmaf(sg, hi, fmaf(sg, lo, d1[u][j]));
                    } else {       // P and N: +hi - lo
                        d4[u][j] = fmaf(a.a[m], hi, fmaf(-a.a[m], lo, d4[u][j]));
                    }
                }
            }
        }
    }
    if (t.z < nz) {
        float fz[4];
        if (t.edge) {
#pragma unroll
            for (int j = 0; j < 4; j++)  // spgzn1, spgzp2
                fz[j] = sponge_factor(t.z + j, nz, a.npz, a.spg + 6 * a.spg_stride, a.spg + 7 * a.spg_stride);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (t.x + u >= nx) break;
            const long long c = t.c + u * a.L.pitch;
            float s[4], r[4], p1[4], p2[4], e1[4], e4[4];
            unpack(s, so[u]);
            unpack(r, ro[u]);
            unpack(p1, p1v[u]);
            unpack(p2, p2v[u]);
            // source: the Gaussian stamp into strxx (QS:1340-1390), after the sponge
            float add[4] = {0.f, 0.f, 0.f, 0.f};
            const int bx = t.x + u - sd.stamp_x0;
            if (bx >= 0 && bx < sd.stamp_w && t.z + 4 > sd.stamp_z0 && t.z < sd.stamp_z0 + sd.stamp_h) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int bz = t.z + j - sd.stamp_z0;
                    if (bz >= 0 && bz < sd.stamp_h)
                        add[j] = (wav * __ldg(a.stamps + sd.stamp_off + bx * sd.stamp_h + bz) * a.dt) / a.dz2;
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                e1[j] = a.hx * d1[u][j];
                e4[j] = a.hz * d4[u][j];
                const float dv = e1[j] + e4[j];
                s[j] = fmaf(a.dt, fmaf(p1[j], dv, r[j]), s[j]) + add[j];
                r[j] = fmaf(a.f_mem, fmaf(p2[j], dv, r[j]), r[j]);
            }
            if (t.edge) {
                const bool xb = in_band(t.x + u, nx, a.npx);
                if (xb || in_band(t.z, nz, a.npz) || in_band(t.z + 3, nz, a.npz)) {
                    // the reference's split update (QS:993-1020, 1135-1170) and sponges (QS:800-834)
                    const float fx = sponge_factor(t.x + u, nx, a.npx, a.spg + 4 * a.spg_stride,
                                                   a.spg + 5 * a.spg_stride);  // spgxn1, spgxp2
                    float sx[4], sz[4], sr[4], rx[4], rz[4], rr[4];
                    unpack(sx, ld4(a.sx + c));
                    unpack(sz, ld4(a.sz + c));
                    unpack(sr, ld4(a.sr + c));
                    unpack(rx, ld4(a.rx + c));
                    unpack(rz, ld4(a.rz + c));
                    unpack(rr, ld4(a.rr + c));
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        if (!(xb || in_band(t.z + j, nz, a.npz)) || t.z + j >= nz) continue;
                        const float rold = (rx[j] + rz[j]) + rr[j];
                        sx[j] = fmaf(a.dt, p1[j] * e1[j], sx[j]) * fx;
                        sz[j] = fmaf(a.dt, p1[j] * e4[j], sz[j]) * fz[j];
                        sr[j] = fmaf(a.dt, rold, sr[j]);
                        rx[j] = fmaf(a.f_mem, p2[j] * e1[j], rx[j]) * fx;
                        rz[j] = fmaf(a.f_mem, p2[j] * e4[j], rz[j]) * fz[j];
                        rr[j] = fmaf(a.f_mem, rold, rr[j]);
                        s[j] = ((sx[j] + sz[j]) + sr[j]) + add[j];
                        sx[j] += add[j];
                        r[j] = (rx[j] + rz[j]) + rr[j];
                    }
                    st4(a.sx + c, sx);
                    st4(a.sz + c, sz);
                    st4(a.sr + c, sr);
                    st4(a.rx + c, rx);
                    st4(a.rz + c, rz);
                    st4(a.rr + c, rr);
                }
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (t.z + j >= nz) s[j] = r[j] = 0.0f;
            }
            st4(A.s + c, s);
            st4(A.r + c, r);
        }
    }
    // receivers: strzz = sigma (QM:452-459), from the lists of the 64 x 64 tiles
    const int* trp = a.tile_rec_ptr + sd.tile_rec_base + t.x0 / TX * a.L.ntz + blockIdx.x;
    const int rb = __ldg(trp), re = __ldg(trp + 1);
    if (re > rb) {
        __syncthreads();
        for (int j = rb + threadIdx.x; j < re; j += threads_of(US)) {
            const int ridx = a.tile_rec_idx[j];
            const int x = a.rec_x[sd.rec_list + ridx];
            if (x < t.x0 || x >= t.x0 + TC) continue;  // another CTA of the 64 x 64 tile holds it
            a.records[sd.rec_base + (long long)a.step * sd.nrec + ridx] =
                A.s[(long long)shot * a.L.shot_stride + (long long)(x + a.L.gx) * a.L.pitch + a.L.gz +
                    a.rec_z[sd.rec_list + ridx]];
        }
    }
}

}  // namespace

cudaError_t viscoac2d_fast_launch(const QFastArgs& A, int active, cudaStream_t st, int* launches) {
    const int ntz = A.q.L.ntz, ncol = A.q.L.ntx * (TX / TC);
    if (cudaError_t e = tile::launch_columns((const void*)viscoac2d_fast_velocity_kernel, ntz, ncol, active, threads_of(UV), 0,
                                             st, A, launches))
        return e;
    return tile::launch_columns((const void*)viscoac2d_fast_stress_kernel, ntz, ncol, active, threads_of(US), 0, st, A,
                                launches);
}

void viscoac2d_fast_box(int box[2]) {
    box[0] = SW;
    box[1] = SROWS;
}

}  // namespace sfd
