// Adjoint of one time step of the viscoacoustic scheme (the vs = 0 reduction of
// forward/Q_forward/Q_multishot_fd_subroutine_fsbc_zy_rotated.f90, QS:695-1337, as the
// kernels of viscoac2d.cu implement it) and the zero-lag imaging conditions for the two
// model parameters of the stress update, p1 = lambda tau_eps/tau_sigma and
// p2 = lambda (tau_eps/tau_sigma - 1).  The reference has no adjoint.
//
// Forward step k (fields in place, eight per cell):
//   S  = sx + sz + sr
//   vx = Ax (vx + dt b Dx0 S),  vz = Az (vz + dt b Dz0 S)                 (velocity kernel)
//   d1 = Dx1 vx, d4 = Dz1 vz, R = rx + rz + rr (old)
//   sx = A'x (sx + dt p1 d1) + stamp w_k,  sz = A'z (sz + dt p1 d4),  sr += dt R
//   rx = A'x (rx + f p2 d1),  rz = A'z (rz + f p2 d4),  rr += f R            (stress kernel)
//   record = S at the receivers
// Adjoint step k (hatted fields hold d misfit / d state after step k, with the residual of
// step k already added at the receivers to sx^, sz^, sr^):
//   T1 = A'x (dt p1 sx^ + f p2 rx^), T4 = A'z (dt p1 sz^ + f p2 rz^), kept as slabs by kernel B
//   kernel A: vx^ = Ax (vx^ + Dx1^T T1),  vz^ = Az (vz^ + Dz1^T T4)
//             Qx = dt b vx^, Qz = dt b vz^;   dw_k = sum stamp sx^
//   kernel B: u1 = A'x sx^, u4 = A'z sz^, w1 = A'x rx^, w4 = A'z rz^, aR = f rr^ + dt sr^
//             aS = Dx0^T Qx + Dz0^T Qz
//             sx^ = u1 + aS, sz^ = u4 + aS, sr^ += aS, rx^ = w1 + aR, rz^ = w4 + aR, rr^ += aR
//             g1 += d1 u1 + d4 u4,  g2 += d1 w1 + d4 w4;   then sx^, sz^, sr^ += res_{k-1}
// so that d misfit / d p1 = dt sum g1 and d misfit / d p2 = f sum g2.  The transposed
// rotated-staggered derivatives gather from the mirrored taps of QS:843-966.  Kernel A reads the halo of
// T1, T4 and writes only velocity adjoints and Qx, Qz; kernel B reads the halo of Qx, Qz and writes only
// its own cells (with its receivers' residuals in sx^, sz^, sr^ before T1 and T4 are formed), so neither
// launch races with itself.
//
// Bound: issue and shared-memory loads in the velocity kernel (72% and 67%, DRAM 1.8 TB/s), memory and issue in
// the stress kernel (4.1 TB/s, 61%); 132 B a cell.  Each kernel's two differentiated fields arrive by TMA on tiles of 64 rows
// by 8 columns with two cells per thread, as in viscoac2d.cu (measurements there); before, kernel A staged
// six arrays with their halo to form T1 and T4 again.
#include <cuda_runtime.h>

#include <algorithm>

#include "sfd_internal.h"
#include "tile_stage.cuh"

namespace sfd {
namespace {

constexpr int TX = kTileX, TZ = kTileZ;
constexpr int TC = kQCols, kThreads = TC * TZ / 2;  // columns of a tile, two cells per thread (TC / 2 columns apart)
constexpr int H = 5;               // rotated-staggered reach (offsets -5 .. +5)
constexpr int HZ = 8;              // z halo rounded to 16 bytes
constexpr int SW = TZ + 2 * HZ;    // staged columns z0-8 .. z0+TZ+7
constexpr int SMEM = (TC + 2 * H) * SW;

struct Tile {
    int shot, tile, x0, z0;
    ShotDev sd;
};

__device__ __forceinline__ bool tile_of(const QAdjArgs& a, Tile& t) {
    t.shot = a.slot_to_shot[blockIdx.z];
    t.sd = a.shots[t.shot];
    t.x0 = (a.col0 + (int)blockIdx.y) * TC;
    t.z0 = blockIdx.x * TZ;
    t.tile = t.x0 / TX * a.L.ntz + blockIdx.x;  // the 64 x 64 tile of the receiver lists
    return t.x0 < t.sd.nx;
}

__device__ __forceinline__ long long cell(const QAdjArgs& a, int shot, int x, int z) {
    return (long long)shot * a.L.shot_stride + (long long)(x + a.L.gx) * a.L.pitch + a.L.gz + z;
}

// product of the two split-sponge factors of a coordinate (left / right tables)
__device__ __forceinline__ float sp(int x, int n, int np, const float* tn, const float* tp) {
    float f = 1.0f;
    if (x <= np) f *= tn[x];
    if (x >= n - np - 1) f *= tp[n - 1 - x];
    return f;
}

// values of a thread's two cells, TC / 2 staged columns apart
__device__ __forceinline__ float2 pair(const float* s, int dx, int dz) {
    return make_float2(s[dx * SW + dz], s[(TC / 2 + dx) * SW + dz]);
}
__device__ __forceinline__ float2 bc(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, bc(-1.0f), a); }

__global__ void __launch_bounds__(kThreads, 8) q_adj_velocity_kernel(const __grid_constant__ QAdjArgs a) {
    __shared__ __align__(128) float sT[2 * SMEM];
    __shared__ uint64_t bar;
    __shared__ float s_dw;
    Tile t;
    const bool on = tile_of(a, t);
    if (threadIdx.x == 0) s_dw = 0.0f;
    tile::bar_init(&bar);
    tile::release();
    tile::acquire();
    if (!on) return;
    if (threadIdx.x == 0) {  // zero outside the grid: the forward never updates there
        tile::expect(&bar, 8u * SMEM);
        tile::box(sT, &a.tm_t1, a.L.gz + t.z0 - HZ, a.L.gx + t.x0 - H, t.shot, &bar);
        tile::box(sT + SMEM, &a.tm_t4, a.L.gz + t.z0 - HZ, a.L.gx + t.x0 - H, t.shot, &bar);
    }
    const int nx = t.sd.nx, nz = a.nz;
    const float* tb = a.spg;
    const int st = a.spg_stride;
    const int r0 = threadIdx.x / TZ, z = threadIdx.x % TZ, gz = t.z0 + z;
    const long long c0 = cell(a, t.shot, t.x0 + r0, gz);
    bool in[2];
    float vxo[2], vzo[2], bu[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int gx = t.x0 + r0 + u * (TC / 2);
        const long long c = c0 + (long long)u * (TC / 2) * a.L.pitch;
        in[u] = gx < nx && gz < nz;
        if (in[u]) {
            vxo[u] = a.avx[c];
            vzo[u] = a.avz[c];
            bu[u] = __ldg(a.busg + (long long)min(t.sd.x0 + gx, a.nx_model - 1) * a.mpitch + gz);
        }
    }
    if (!tile::staged(&bar, a.err_flag)) return;
    const float* p1s = sT + (r0 + H) * SW + z + HZ;
    const float* p4s = p1s + SMEM;
    float2 s1p = bc(0.0f), s4p = bc(0.0f);
#pragma unroll
    for (int m = 0; m < 5; m++) {
        // Dx1^T: t(x-1-m, z-1-m) - t(x+m, z+m) + t(x-1-m, z+m) - t(x+m, z-1-m); Dz1^T flips the cross terms
        const float2 a1 = sub2(pair(p1s, -1 - m, -1 - m), pair(p1s, m, m));
        const float2 b1 = sub2(pair(p1s, -1 - m, m), pair(p1s, m, -1 - m));
        const float2 a4 = sub2(pair(p4s, -1 - m, -1 - m), pair(p4s, m, m));
        const float2 b4 = sub2(pair(p4s, -1 - m, m), pair(p4s, m, -1 - m));
        s1p = __ffma2_rn(bc(a.a[m]), __fadd2_rn(a1, b1), s1p);
        s4p = __ffma2_rn(bc(a.a[m]), sub2(a4, b4), s4p);
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
        if (!in[u]) continue;
        const int gx = t.x0 + r0 + u * (TC / 2);
        const long long c = c0 + (long long)u * (TC / 2) * a.L.pitch;
        const float s1 = u ? s1p.y : s1p.x, s4 = u ? s4p.y : s4p.x;
        const float ax = sp(gx, nx, a.npx, tb + 0 * st, tb + 1 * st);
        const float az = sp(gz, nz, a.npz, tb + 2 * st, tb + 3 * st);
        const float vx = ax * fmaf(a.hx, s1, vxo[u]);
        const float vz = az * fmaf(a.hz, s4, vzo[u]);
        const float db = a.dt * bu[u];
        a.avx[c] = vx;
        a.avz[c] = vz;
        a.qx[c] = db * vx;
        a.qz[c] = db * vz;
    }
    // wavelet gradient: dw_k = dt / dz^2 sum over the source stamp of sx^ (QS:1384 transposed)
    const ShotDev& sd = t.sd;
    const int bx0 = max(sd.stamp_x0, t.x0), bx1 = min(sd.stamp_x0 + sd.stamp_w, min(t.x0 + TC, nx));
    const int bz0 = max(sd.stamp_z0, t.z0), bz1 = min(sd.stamp_z0 + sd.stamp_h, min(t.z0 + TZ, nz));
    if (a.lam_src && bx1 > bx0 && bz1 > bz0) {
        const int w = bz1 - bz0;
        float part = 0.0f;
        for (int i = threadIdx.x; i < (bx1 - bx0) * w; i += kThreads) {
            const int x = bx0 + i / w, zz = bz0 + i % w;
            const float g = __ldg(a.stamps + sd.stamp_off + (x - sd.stamp_x0) * sd.stamp_h + (zz - sd.stamp_z0));
            part = fmaf(g, a.asx[cell(a, t.shot, x, zz)], part);
        }
        for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
        if ((threadIdx.x & 31) == 0) atomicAdd(&s_dw, part);
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(a.lam_src + (long long)t.shot * a.nt_max + a.step, s_dw * (a.dt / a.dz2));
    }
}

__global__ void __launch_bounds__(kThreads, 5) q_adj_stress_kernel(const __grid_constant__ QAdjArgs a) {
    __shared__ __align__(128) float sQ[2 * SMEM];
    __shared__ float sR[TC * TZ];
    __shared__ uint64_t bar;
    Tile t;
    const bool on = tile_of(a, t);
    // receivers of the 64 x 64 tile (their lists, before the wait for the kernel before) ...
    const int* trp = a.tile_rec_ptr + t.sd.tile_rec_base + t.tile;
    const int rb = on ? __ldg(trp) : 0, re = on ? __ldg(trp + 1) : 0, j0 = rb + threadIdx.x;
    const bool res = a.step >= 1 && re > rb;
    int ridx = 0, rx = 0, rz = 0;
    auto receiver = [&](int j) {
        ridx = a.tile_rec_idx[j];
        rx = a.rec_x[t.sd.rec_list + ridx] - t.x0;
        rz = a.rec_z[t.sd.rec_list + ridx] - t.z0;
    };
    if (res) {
        if (j0 < re) receiver(j0);
        for (int i = threadIdx.x; i < TC * TZ; i += kThreads) sR[i] = 0.0f;
    }
    tile::bar_init(&bar);
    tile::release();
    tile::acquire();
    if (!on) return;
    if (threadIdx.x == 0) {
        tile::expect(&bar, 8u * SMEM);
        tile::box(sQ, &a.tm_qx, a.L.gz + t.z0 - HZ, a.L.gx + t.x0 - H, t.shot, &bar);
        tile::box(sQ + SMEM, &a.tm_qz, a.L.gz + t.z0 - HZ, a.L.gx + t.x0 - H, t.shot, &bar);
    }
    const int nx = t.sd.nx, nz = a.nz;
    const ShotDev& sd = t.sd;
    const int r0 = threadIdx.x / TZ, z = threadIdx.x % TZ, gz = t.z0 + z;
    const long long c0 = cell(a, t.shot, t.x0 + r0, gz);
    bool in[2];
    float hs[2][6], d1[2], d4[2], g1[2], g2[2], p1[2], p2[2];  // hs: sx^ sz^ sr^ rx^ rz^ rr^
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int gx = t.x0 + r0 + u * (TC / 2);
        const long long c = c0 + (long long)u * (TC / 2) * a.L.pitch;
        in[u] = gx < nx && gz < nz;
        if (in[u]) {
            hs[u][0] = a.asx[c]; hs[u][1] = a.asz[c]; hs[u][2] = a.asr[c];
            hs[u][3] = a.arx[c]; hs[u][4] = a.arz[c]; hs[u][5] = a.arr[c];
            d1[u] = a.d1[c]; d4[u] = a.d4[c];
            g1[u] = a.g1[c]; g2[u] = a.g2[c];
            const long long mi = (long long)min(sd.x0 + gx, a.nx_model - 1) * a.mpitch + gz;
            p1[u] = __ldg(a.p1 + mi); p2[u] = __ldg(a.p2 + mi);
        }
    }
    // ... and the residual of step k-1 there (QM:452-459 transposed), S^ -> sx^, sz^, sr^, summed per cell while
    // the boxes are on their way
    if (res) {
        for (int j = j0; j < re; j += kThreads) {
            if (j > j0) receiver(j);
            if (rx >= 0 && rx < TC)  // else another CTA of the 64 x 64 tile holds it
                atomicAdd(&sR[rx * TZ + rz], a.res[sd.rec_base + (long long)(a.step - 1) * sd.nrec + ridx]);
        }
        __syncthreads();
    }
    if (!tile::staged(&bar, a.err_flag)) return;
    const float* tb = a.spg;
    const int st = a.spg_stride;
    const float dt = a.dt, f = a.f_mem;
    const float* px = sQ + (r0 + H) * SW + z + HZ;
    const float* pz = px + SMEM;
    float2 sxp = bc(0.0f), szp = bc(0.0f);
#pragma unroll
    for (int m = 0; m < 5; m++) {
        // Dx0^T: t(x-m, z-m) - t(x+1+m, z+1+m) + t(x-m, z+1+m) - t(x+1+m, z-m); Dz0^T flips the cross terms
        const float2 ax_ = sub2(pair(px, -m, -m), pair(px, 1 + m, 1 + m));
        const float2 bx_ = sub2(pair(px, -m, 1 + m), pair(px, 1 + m, -m));
        const float2 az_ = sub2(pair(pz, -m, -m), pair(pz, 1 + m, 1 + m));
        const float2 bz_ = sub2(pair(pz, -m, 1 + m), pair(pz, 1 + m, -m));
        sxp = __ffma2_rn(bc(a.a[m]), __fadd2_rn(ax_, bx_), sxp);
        szp = __ffma2_rn(bc(a.a[m]), sub2(az_, bz_), szp);
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
        if (!in[u]) continue;
        const int gx = t.x0 + r0 + u * (TC / 2);
        const long long c = c0 + (long long)u * (TC / 2) * a.L.pitch;
        const float sx = u ? sxp.y : sxp.x, sz = u ? szp.y : szp.x;
        const float aS = fmaf(a.hx, sx, a.hz * sz);
        const float axs = sp(gx, nx, a.npx, tb + 4 * st, tb + 5 * st);
        const float azs = sp(gz, nz, a.npz, tb + 6 * st, tb + 7 * st);
        const float u1 = axs * hs[u][0], u4 = azs * hs[u][1];
        const float w1 = axs * hs[u][3], w4 = azs * hs[u][4];
        const float aR = fmaf(f, hs[u][5], dt * hs[u][2]);
        a.g1[c] = g1[u] + fmaf(d1[u], u1, d4[u] * u4);
        a.g2[c] = g2[u] + fmaf(d1[u], w1, d4[u] * w4);
        float nsx = u1 + aS, nsz = u4 + aS, nsr = hs[u][2] + aS;
        const float nrx = w1 + aR, nrz = w4 + aR;
        const float v = res ? sR[(r0 + u * (TC / 2)) * TZ + z] : 0.0f;
        if (v != 0.0f) {
            nsx += v;
            nsz += v;
            nsr += v;
        }
        a.asx[c] = nsx;
        a.asz[c] = nsz;
        a.asr[c] = nsr;
        a.arx[c] = nrx;
        a.arz[c] = nrz;
        a.arr[c] = hs[u][5] + aR;
        const float e1 = dt * p1[u], e2 = f * p2[u];
        a.t1[c] = axs * fmaf(e1, nsx, e2 * nrx);
        a.t4[c] = azs * fmaf(e1, nsz, e2 * nrz);
    }
}

// sx^, sz^, sr^ of every shot in [first, first + n) += res of the shot's last step (several receivers may share
// a cell, so the adds are atomic); then T1, T4 there, from the sums
__global__ void q_adjoint_init_kernel(QAdjArgs a, int first_shot) {
    const int s = first_shot + blockIdx.y;
    const ShotDev sd = a.shots[s];
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < sd.nrec; r += gridDim.x * blockDim.x) {
        const long long c = cell(a, s, a.rec_x[sd.rec_list + r], a.rec_z[sd.rec_list + r]);
        const float v = a.res[sd.rec_base + (long long)(sd.nt - 1) * sd.nrec + r];
        atomicAdd(a.asx + c, v);
        atomicAdd(a.asz + c, v);
        atomicAdd(a.asr + c, v);
    }
}
__global__ void q_adjoint_init_t_kernel(QAdjArgs a, int first_shot) {
    const int s = first_shot + blockIdx.y;
    const ShotDev sd = a.shots[s];
    const float* tb = a.spg;
    const int st = a.spg_stride;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < sd.nrec; r += gridDim.x * blockDim.x) {
        const int x = a.rec_x[sd.rec_list + r], z = a.rec_z[sd.rec_list + r];
        const long long c = cell(a, s, x, z), mi = (long long)min(sd.x0 + x, a.nx_model - 1) * a.mpitch + z;
        const float e1 = a.dt * __ldg(a.p1 + mi), e2 = a.f_mem * __ldg(a.p2 + mi);
        a.t1[c] = sp(x, sd.nx, a.npx, tb + 4 * st, tb + 5 * st) * fmaf(e1, a.asx[c], e2 * a.arx[c]);
        a.t4[c] = sp(z, a.nz, a.npz, tb + 6 * st, tb + 7 * st) * fmaf(e1, a.asz[c], e2 * a.arz[c]);
    }
}

// Model-grid gradients.  Shot s's column x reads prepared-model column sd.x0 + x, which is
// model column ap_x0[s] + x.  dJ/dp1 = dt g1, dJ/dp2 = f g2 (sums over the shots covering the
// cell); p1 = lambda tpss, p2 = lambda (tpss - 1) with lambda = rho_avg vp^2 and
// tpss = 1 + kappa / Q (QS:473-551), so dp/dvp = 2 p / vp and dp1/d(1/Q) = dp2/d(1/Q) = lambda kappa.
__global__ void q_gradient_reduce_kernel(const double* __restrict__ acc1, const double* __restrict__ acc2, Layout2D L,
                                         const ShotDev* __restrict__ shots, const int* __restrict__ ap_x0, int nshot,
                                         const float* __restrict__ vp, const float* __restrict__ p1,
                                         const float* __restrict__ p2, int mpitch, int nx_model, int nz, double dt,
                                         double f, double kappa, double* grad_vp, double* grad_invq) {
    const long long n = (long long)nx_model * nz;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int X = (int)(i / nz), z = (int)(i - (long long)X * nz);
        double gv = 0.0, gq = 0.0;
        for (int s = 0; s < nshot; s++) {
            const int x = X - ap_x0[s];
            if (x < 0 || x >= shots[s].nx) continue;
            const long long c = (long long)s * L.shot_stride + (long long)(x + L.gx) * L.pitch + L.gz + z;
            const double G1 = dt * acc1[c], G2 = f * acc2[c];
            const long long b = (long long)(shots[s].x0 + x) * mpitch + z;
            const double q1 = p1[b], q2 = p2[b];
            gv += 2.0 * (q1 * G1 + q2 * G2) / (double)vp[(long long)X * mpitch + z];
            gq += (q1 - q2) * kappa * (G1 + G2);
        }
        grad_vp[i] = gv;
        if (grad_invq) grad_invq[i] = gq;
    }
}

int grid_for(long long n) { return (int)std::min<long long>((n + 255) / 256, 148 * 16); }

}  // namespace

cudaError_t q_adjoint_launch_step(const QAdjArgs& a, int active, cudaStream_t st, int* launches) {
    const int ntz = a.L.ntz, ncol = a.L.ntx * (TX / TC);
    if (cudaError_t e = tile::launch_columns((const void*)q_adj_velocity_kernel, ntz, ncol, active, kThreads, 0, st, a, launches))
        return e;
    return tile::launch_columns((const void*)q_adj_stress_kernel, ntz, ncol, active, kThreads, 0, st, a, launches);
}

cudaError_t q_adjoint_launch_init(const QAdjArgs& a, int first_shot, int nshot, int nrec_max, cudaStream_t st) {
    if (nrec_max <= 0 || nshot <= 0) return cudaSuccess;
    dim3 grid((nrec_max + 255) / 256, nshot);
    q_adjoint_init_kernel<<<grid, 256, 0, st>>>(a, first_shot);
    if (cudaError_t e = cudaGetLastError()) return e;
    q_adjoint_init_t_kernel<<<grid, 256, 0, st>>>(a, first_shot);
    return cudaGetLastError();
}

cudaError_t q_launch_gradient_reduce(const double* acc1, const double* acc2, const Layout2D& L, const ShotDev* shots,
                                     const int* ap_x0, int nshot, const float* vp, const float* p1, const float* p2,
                                     int mpitch, int nx_model, int nz, double dt, double f, double kappa,
                                     double* grad_vp, double* grad_invq, cudaStream_t st) {
    const long long n = (long long)nx_model * nz;
    q_gradient_reduce_kernel<<<grid_for(n), 256, 0, st>>>(acc1, acc2, L, shots, ap_x0, nshot, vp, p1, p2, mpitch,
                                                           nx_model, nz, dt, f, kappa, grad_vp, grad_invq);
    return cudaGetLastError();
}

}  // namespace sfd
