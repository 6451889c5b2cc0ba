// Viscoacoustic (one standard-linear-solid memory variable) rotated-staggered-grid time step,
// the vs = 0 reduction of forward/Q_forward/Q_multishot_fd_subroutine_fsbc_zy_rotated.f90 (QS).
//
// With mu = 0, strxz and rxz stay exactly zero, so vxz = vzx = 0 and strxx = strzz (their
// split parts receive identical updates, sponges and sources).  The state per cell is
//   vx, vz                (QS vxx, vzz; vx is sponged in x only, vz in z only)
//   sx, sz, sr            (QS strxxx, strxxz, strxxr; sigma = (sx + sz) + sr)
//   rx, rz, rr            (QS rxxx, rxxz, rxxr;       r     = (rx + rz) + rr)
// with sigma kept as a slab of its own, written by the stress kernel, and one step is two kernels:
//   velocity: d1 = Dx0(sigma), d2 = Dz0(sigma) (QS:843-966, xflag/zflag 0),
//             vx = (vx + dt b d1) * x-sponge, vz = (vz + dt b d2) * z-sponge   (QS:969-990, 609-654)
//   stress:   d1 = Dx1(vx), d4 = Dz1(vz) (flag 1),
//             sx = (sx + dt (p1 d1)) * x-sponge' + source, sz = (sz + dt (p1 d4)) * z-sponge',
//             sr = sr + dt r_old, rx = (rx + f (p2 d1)) * x-sponge', rz = (rz + f (p2 d4)) * z-sponge',
//             rr = rr + f r_old, f = dt (-1/tau_sigma)                       (QS:993-1337, 1340-1390)
// Every multiply and add is rounded separately in the reference's order, so the kernels agree
// bit for bit with the FP32 restatement in oracle/q_oracle.cpp.
//
// Bound: issue (79% in the velocity, 71% in the stress kernel; DRAM 1.8 and 3.1 TB/s): the prescribed order's
// arithmetic on 76 B a cell (eight fields read and written, three model arrays; the kernels move 100).
// The fields that a kernel differentiates arrive by TMA, a box with halo per field, on tiles of 64 rows by
// 8 columns with two cells per thread, while the threads load their own values.  8 shots of 700 x 420
// (2.4 M cells), forward and adjoint step together: 160 us with 64 x 64 tiles staged through registers and
// 16 cells per thread; 4 columns with one cell per thread 137 us (bound by issue: the fixed work of a thread
// is half of it); two cells per thread 122 us, with their stencils paired 119 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "sfd_internal.h"
#include "tile_stage.cuh"

namespace sfd {
namespace {

constexpr int TX = kTileX, TZ = kTileZ;
constexpr int TC = kQCols, kThreads = TC * TZ / 2;  // columns of a tile, two cells per thread (TC / 2 columns apart)
constexpr int H = 5;                    // RSG halo (offsets -5..+5)
constexpr int HZ = 8;                   // z halo rounded to 16 bytes
constexpr int SW = TZ + 2 * HZ;         // 80
constexpr int SMEM = (TC + 2 * H) * SW; // floats per staged field

__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }

// The derivatives of a thread's two cells at once, on paired FP32 instructions (half the arithmetic
// instructions).  A difference is fma(b, -1, a) and a sum fma(a, one, b), rounded once each: the compiler
// contracts a paired multiply and a paired add, but not through `one` (1.0 from the kernel's arguments).
__device__ __forceinline__ float2 bc(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 fs2(float2 a, float2 b) { return __ffma2_rn(b, bc(-1.0f), a); }
__device__ __forceinline__ float2 fa2(float2 a, float2 b, float one) { return __ffma2_rn(a, bc(one), b); }
__device__ __forceinline__ float2 pair(const float* s, int r, int c) {
    return make_float2(s[r * SW + c], s[(r + TC / 2) * SW + c]);
}

// QS:843-966: 0.5/d * sum_m a_m t_m with t_m the rotated four-point difference; (r, c) the staged position
// (row = x, column = z) of the first cell
template <bool XDIR, int FLAG>
__device__ __forceinline__ float2 rsg(const float* s, int r, int c, const float* a, float h, float one) {
    float2 acc;
#pragma unroll
    for (int m = 0; m < 5; m++) {
        const int hi = FLAG == 0 ? m : 1 + m, lo = FLAG == 0 ? -1 - m : -m;
        const float2 d = fs2(pair(s, r + hi, c + hi), pair(s, r + lo, c + lo));
        const float2 p = pair(s, r + hi, c + lo), q = pair(s, r + lo, c + hi);
        const float2 t = __fmul2_rn(bc(a[m]), XDIR ? fs2(fa2(d, p, one), q) : fa2(fs2(d, p), q, one));
        acc = m == 0 ? t : fa2(acc, t, one);
    }
    return __fmul2_rn(bc(h), acc);
}

// both derivatives of one field: their four-point differences share the first subtraction
template <int FLAG>
__device__ __forceinline__ void rsg_both(const float* s, int r, int c, const float* a, float hx, float hz, float one,
                                         float2* dx, float2* dz) {
    float2 ax, az;
#pragma unroll
    for (int m = 0; m < 5; m++) {
        const int hi = FLAG == 0 ? m : 1 + m, lo = FLAG == 0 ? -1 - m : -m;
        const float2 d = fs2(pair(s, r + hi, c + hi), pair(s, r + lo, c + lo));
        const float2 p = pair(s, r + hi, c + lo), q = pair(s, r + lo, c + hi);
        const float2 tx = __fmul2_rn(bc(a[m]), fs2(fa2(d, p, one), q));
        const float2 tz = __fmul2_rn(bc(a[m]), fa2(fs2(d, p), q, one));
        ax = m == 0 ? tx : fa2(ax, tx, one);
        az = m == 0 ? tz : fa2(az, tz, one);
    }
    *dx = __fmul2_rn(bc(hx), ax);
    *dz = __fmul2_rn(bc(hz), az);
}

struct TileRef {
    int shot, tile, x0, z0;
    ShotDev sd;
};

__device__ __forceinline__ bool tile_of(const QArgs& a, TileRef& t) {
    t.shot = a.slot_to_shot[blockIdx.z];
    t.sd = a.shots[t.shot];
    t.x0 = (a.col0 + (int)blockIdx.y) * TC;
    t.z0 = blockIdx.x * TZ;
    t.tile = t.x0 / TX * a.L.ntz + blockIdx.x;  // the 64 x 64 tile of the receiver lists
    return t.x0 < t.sd.nx;
}

__device__ __forceinline__ long long cell(const QArgs& a, int shot, int x, int z) {
    return (long long)shot * a.L.shot_stride + (long long)(x + a.L.gx) * a.L.pitch + a.L.gz + z;
}

// x / z factors of a split sponge: left/right (resp. top/bottom) tables, applied in QS order
__device__ __forceinline__ float xs(float u, int x, int nx, int np, const float* tn, const float* tp) {
    if (x <= np) u = fm(u, tn[x]);
    if (x >= nx - np - 1) u = fm(u, tp[nx - 1 - x]);
    return u;
}

// SUMS = false: no memory for the slab of sigma.  The tile and its halo are summed by the threads: 81 ms
// against 75 for 200 steps of 16 shots of 1124 x 1124.
template <bool SUMS>
__global__ void __launch_bounds__(kThreads, 8) q_velocity_kernel(const __grid_constant__ QArgs a) {
    __shared__ __align__(128) float sS[SMEM];
    __shared__ uint64_t bar;
    TileRef t;
    const bool on = tile_of(a, t);
    tile::bar_init(&bar);
    tile::release();
    tile::acquire();
    if (!on) return;
    if (!SUMS) {
        for (int i = threadIdx.x; i < SMEM / 4; i += kThreads) {
            const int r = i / (SW / 4), c = 4 * (i % (SW / 4));
            const long long o = cell(a, t.shot, t.x0 - H + r, t.z0 - HZ + c);
            const float4 x = *reinterpret_cast<const float4*>(a.sx + o), y = *reinterpret_cast<const float4*>(a.sz + o),
                         w = *reinterpret_cast<const float4*>(a.sr + o);
            *reinterpret_cast<float4*>(sS + r * SW + c) =
                make_float4(fa(fa(x.x, y.x), w.x), fa(fa(x.y, y.y), w.y), fa(fa(x.z, y.z), w.z), fa(fa(x.w, y.w), w.w));
        }
        __syncthreads();
    } else if (threadIdx.x == 0) {  // sigma = (sx + sz) + sr  (QS:1294-1314)
        tile::expect(&bar, 4u * SMEM);
        tile::box(sS, &a.tm_s, a.L.gz + t.z0 - HZ, a.L.gx + t.x0 - H, t.shot, &bar);
    }
    const int nx = t.sd.nx, nz = a.nz;
    const int r0 = threadIdx.x / TZ, z = threadIdx.x % TZ, gz = t.z0 + z;
    const long long c0 = cell(a, t.shot, t.x0 + r0, gz);
    bool in[2];
    float vx[2], vz[2], bu[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int gx = t.x0 + r0 + u * (TC / 2);
        const long long c = c0 + (long long)u * (TC / 2) * a.L.pitch;
        in[u] = gx < nx && gz < nz;
        if (in[u]) {
            vx[u] = a.vx[c];
            vz[u] = a.vz[c];
            bu[u] = __ldg(a.busg + (long long)min(t.sd.x0 + gx, a.nx_model - 1) * a.mpitch + gz);
        }
    }
    if (SUMS && !tile::staged(&bar, a.err_flag)) return;
    const float* tb = a.spg;
    const int st = a.spg_stride;
    float2 d1p, d2p;
    rsg_both<0>(sS, r0 + H, z + HZ, a.a, a.hx, a.hz, a.one, &d1p, &d2p);
#pragma unroll
    for (int u = 0; u < 2; u++) {
        if (!in[u]) continue;
        const int gx = t.x0 + r0 + u * (TC / 2);
        const long long c = c0 + (long long)u * (TC / 2) * a.L.pitch;
        const float d1 = u ? d1p.y : d1p.x, d2 = u ? d2p.y : d2p.x;
        const float dtb = fm(a.dt, bu[u]);
        float x = fa(vx[u], fm(dtb, d1)), y = fa(vz[u], fm(dtb, d2));
        x = xs(x, gx, nx, a.npx, tb + 0 * st, tb + 1 * st);   // spgxn, spgxp
        y = xs(y, gz, nz, a.npz, tb + 2 * st, tb + 3 * st);   // spgzn, spgzp
        a.vx[c] = fa(x, 0.0f);  // vx = vxx + vxz with vxz = 0
        a.vz[c] = fa(0.0f, y);  // vz = vzx + vzz with vzx = 0
    }
}

template <bool SUMS>
__global__ void __launch_bounds__(kThreads, 6) q_stress_kernel(const __grid_constant__ QArgs a) {
    __shared__ __align__(128) float sV[2 * SMEM];
    __shared__ uint64_t bar;
    const float* sVx = sV;
    const float* sVz = sV + SMEM;
    TileRef t;
    const bool on = tile_of(a, t);
    tile::bar_init(&bar);
    tile::release();
    tile::acquire();
    if (!on) return;
    if (threadIdx.x == 0) {
        tile::expect(&bar, 8u * SMEM);
        tile::box(sV, &a.tm_vx, a.L.gz + t.z0 - HZ, a.L.gx + t.x0 - H, t.shot, &bar);
        tile::box(sV + SMEM, &a.tm_vz, a.L.gz + t.z0 - HZ, a.L.gx + t.x0 - H, t.shot, &bar);
    }
    const int nx = t.sd.nx, nz = a.nz;
    const ShotDev& sd = t.sd;
    const int r0 = threadIdx.x / TZ, z = threadIdx.x % TZ, gz = t.z0 + z;
    const long long c0 = cell(a, t.shot, t.x0 + r0, gz);
    bool in[2];
    float p1[2], p2[2], o[2][6];  // o: sx sz sr rx rz rr
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int gx = t.x0 + r0 + u * (TC / 2);
        const long long c = c0 + (long long)u * (TC / 2) * a.L.pitch;
        in[u] = gx < nx && gz < nz;
        if (in[u]) {
            const long long mi = (long long)min(sd.x0 + gx, a.nx_model - 1) * a.mpitch + gz;
            p1[u] = __ldg(a.p1 + mi);
            p2[u] = __ldg(a.p2 + mi);
            o[u][0] = a.sx[c]; o[u][1] = a.sz[c]; o[u][2] = a.sr[c];
            o[u][3] = a.rx[c]; o[u][4] = a.rz[c]; o[u][5] = a.rr[c];
        }
    }
    const float wav = __ldg(a.wavelets + sd.wav_off + a.step);
    if (!tile::staged(&bar, a.err_flag)) return;
    const float* tb = a.spg;
    const int st = a.spg_stride;
    const float2 d1p = rsg<true, 1>(sVx, r0 + H, z + HZ, a.a, a.hx, a.one);
    const float2 d4p = rsg<false, 1>(sVz, r0 + H, z + HZ, a.a, a.hz, a.one);
#pragma unroll
    for (int u = 0; u < 2; u++) {
        if (!in[u]) continue;
        const int gx = t.x0 + r0 + u * (TC / 2);
        const long long c = c0 + (long long)u * (TC / 2) * a.L.pitch;
        const float d1 = u ? d1p.y : d1p.x, d4 = u ? d4p.y : d4p.x;
        const float rold = fa(fa(o[u][3], o[u][4]), o[u][5]);  // QS rxx of the previous step
        // calpstrxx (QS:993-1020) with mu = 0, split sponge (QS:800), source (QS:801)
        float sx = fa(o[u][0], fm(a.dt, fm(p1[u], d1)));
        float sz = fa(o[u][1], fm(a.dt, fm(p1[u], d4)));
        const float sr = fa(o[u][2], fm(a.dt, rold));
        sx = xs(sx, gx, nx, a.npx, tb + 4 * st, tb + 5 * st);   // spg1xn, spg2xp
        sz = xs(sz, gz, nz, a.npz, tb + 6 * st, tb + 7 * st);   // spg1zn, spg2zp
        const int bx = gx - sd.stamp_x0, bz = gz - sd.stamp_z0;
        if (bx >= 0 && bx < sd.stamp_w && bz >= 0 && bz < sd.stamp_h) {
            const float g = __ldg(a.stamps + sd.stamp_off + bx * sd.stamp_h + bz);
            sx = fa(__fdiv_rn(fm(fm(wav, g), a.dt), a.dz2), sx);   // QS:1384
        }
        // calprxx (QS:1135-1170)
        float rx = fa(o[u][3], fm(a.f_mem, fm(p2[u], d1)));
        float rz = fa(o[u][4], fm(a.f_mem, fm(p2[u], d4)));
        const float rr = fa(o[u][5], fm(a.f_mem, rold));
        rx = xs(rx, gx, nx, a.npx, tb + 4 * st, tb + 5 * st);
        rz = xs(rz, gz, nz, a.npz, tb + 6 * st, tb + 7 * st);
        a.sx[c] = sx; a.sz[c] = sz; a.sr[c] = sr;
        a.rx[c] = rx; a.rz[c] = rz; a.rr[c] = rr;
        if (SUMS) a.sg[c] = fa(fa(sx, sz), sr);
        if (a.d1_out) {  // gradient recomputation keeps the derivatives for the imaging condition
            a.d1_out[c] = d1;
            a.d4_out[c] = d4;
        }
    }
    // receivers: strzz (= strxx) = (sx + sz) + sr (QM:452-459)
    const int* trp = a.tile_rec_ptr + sd.tile_rec_base + t.tile;
    const int rb = trp[0], re = trp[1];
    if (re > rb) {
        __syncthreads();
        for (int j = rb + threadIdx.x; j < re; j += kThreads) {
            const int ridx = a.tile_rec_idx[j];
            const int x = a.rec_x[sd.rec_list + ridx];
            if (x < t.x0 || x >= t.x0 + TC) continue;  // another CTA of the 64 x 64 tile holds it
            const long long c = cell(a, t.shot, x, a.rec_z[sd.rec_list + ridx]);
            a.records[sd.rec_base + (long long)a.step * sd.nrec + ridx] = SUMS ? a.sg[c] : fa(fa(a.sx[c], a.sz[c]), a.sr[c]);
        }
    }
}

}  // namespace

void q_box(int box[2]) {
    box[0] = SW;
    box[1] = TC + 2 * H;
}

cudaError_t viscoac2d_launch_step(const QArgs& a, int active, cudaStream_t st, int* launches) {
    const int ntz = a.L.ntz, ncol = a.L.ntx * (TX / TC);
    const void* kv = a.sg ? (const void*)q_velocity_kernel<true> : (const void*)q_velocity_kernel<false>;
    const void* ks = a.sg ? (const void*)q_stress_kernel<true> : (const void*)q_stress_kernel<false>;
    if (cudaError_t e = tile::launch_columns(kv, ntz, ncol, active, kThreads, 0, st, a, launches)) return e;
    return tile::launch_columns(ks, ntz, ncol, active, kThreads, 0, st, a, launches);
}

// sigma = (sx + sz) + sr of n cells from each pointer on (n a multiple of four), as the stress kernel forms it
__global__ void q_sigma_kernel(const float4* sx, const float4* sz, const float4* sr, float4* sg, long long n4) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
        const float4 a = sx[i], b = sz[i], c = sr[i];
        sg[i] = make_float4(fa(fa(a.x, b.x), c.x), fa(fa(a.y, b.y), c.y), fa(fa(a.z, b.z), c.z), fa(fa(a.w, b.w), c.w));
    }
}
cudaError_t viscoac2d_launch_sigma(const QArgs& a, long long first, long long n, cudaStream_t st) {
    auto at = [&](float* f) { return reinterpret_cast<float4*>(f + first); };
    q_sigma_kernel<<<(unsigned)std::min<long long>((n / 4 + 255) / 256, 148 * 16), 256, 0, st>>>(at(a.sx), at(a.sz), at(a.sr),
                                                                                            at(a.sg), n / 4);
    return cudaGetLastError();
}

// QS:434-469 (density averaged in place, then buoyancy) and QS:473-551 (Blanch's tau method),
// single precision in the reference's operation order.  q == nullptr: Q = 1e5 (QM:418-419).
void viscoac2d_prepare(int nx, int nz, const float* vp, const float* rho, const float* q, float f0, float* busg,
                       float* p1, float* p2, float* rtau_out) {
    std::vector<float> r(rho, rho + (size_t)nx * nz);
    auto R = [&](int k, int i) -> float& { return r[(size_t)i * nz + k]; };  // 0-based (z, x)
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
        const float lambmu = rr * (vp[c] * vp[c]);
        const float qp = (q ? q[c] : 100000.0f) * (18.0f / 20.0f);
        float taup = 0.0f;
        if (dup - dlow != 0.0f) taup = 1.0f / qp * (nup - nlow) / (dup - dlow);
        const float tpe = taup * tss + tss;
        const float tpss = tpe / tss;
        p1[c] = lambmu * tpss;
        p2[c] = lambmu * (tpss - 1.0f);
    }
    *rtau_out = 1.0f / tss;
}

// QS:555-605 with R = 1e-3; tables xn, xp, zn, zp, 1xn, 2xp, 1zn, 2zp of `stride` entries
void viscoac2d_sponge_tables(int npx, int npz, float dx, float dz, int stride, float* out) {
    const float Rr = 1.0e-3f;
    const float fx = std::acos(Rr) / ((float)npx * dx), fz = std::acos(Rr) / ((float)npz * dz);
    for (int j = 0; j < 8 * stride; j++) out[j] = 1.0f;
    for (int i = 1; i <= npx + 1; i++) {
        out[0 * stride + i - 1] = std::cos(fx * (float)(npx - i + 1) * dx);
        out[1 * stride + i - 1] = std::cos(fx * (float)(npx - i + 1) * dx);
        out[4 * stride + i - 1] = (i == npx + 1) ? 1.0f : std::cos(fx * ((float)(npx - i + 1) * dx - dx / 2));
        out[5 * stride + i - 1] = std::cos(fx * ((float)(npx - i + 1) * dx + dx / 2));
    }
    for (int i = 1; i <= npz + 1; i++) {
        out[2 * stride + i - 1] = std::cos(fz * (float)(npz - i + 1) * dz);
        out[3 * stride + i - 1] = std::cos(fz * (float)(npz - i + 1) * dz);
        out[6 * stride + i - 1] = (i == npz + 1) ? 1.0f : std::cos(fz * ((float)(npz - i + 1) * dz - dz / 2));
        out[7 * stride + i - 1] = std::cos(fz * ((float)(npz - i + 1) * dz + dz / 2));
    }
}

// QS:1340-1444: the whole-grid Gaussian (sigma 1.5 cells) normalised by its single-precision
// sum, placed as the loop of QS:1378-1390 places it (centre offset by one cell for even sizes);
// the box of non-zero weights around the source.
void viscoac2d_stamp(int nx, int nz, int sx, int sz, int* box, std::vector<float>* out) {
    const int n1 = nz, n2 = nx;
    const int hw1 = (int)std::lround((n1 + 1) / 2.0), hw2 = (int)std::lround((n2 + 1) / 2.0);
    const int ixcen = (n1 + 1) / 2, izcen = (n2 + 1) / 2;
    const float pi = 3.1415926f, sigma2 = 1.5f * 1.5f;
    // g2c(i, j) before normalisation, 1-based; the squares in 64 bits (a grid of more than 92680 columns
    // would overflow 32)
    auto raw = [&](long long i, long long j) {
        const float dis = (float)((j - izcen) * (j - izcen) + (i - ixcen) * (i - ixcen));
        return 1.0f / (2.0f * pi * sigma2) * std::exp(-dis / (2.0f * sigma2));
    };
    float sum = 0.0f;
    for (int j = 1; j <= n2; j++)
        for (int i = 1; i <= n1; i++) sum = sum + raw(i, j);
    // 1-based source (isxe, isze) = (sx + 1, sz + 1); loop indices idx1 = m - (isze - hw1), idx2 likewise
    const int isxe = sx + 1, isze = sz + 1;
    int xlo = 1 << 30, xhi = -1, zlo = 1 << 30, zhi = -1;
    for (int n = isxe - (hw2 - 1); n <= isxe + (hw2 - 1); n++) {
        const int idx2 = n - (isxe - (hw2 - 1)) + 1;
        if (n < 1 || n > nx || idx2 > n2) continue;
        for (int m = isze - (hw1 - 1); m <= isze + (hw1 - 1); m++) {
            const int idx1 = m - (isze - (hw1 - 1)) + 1;
            if (m < 1 || m > nz || idx1 > n1) continue;
            if (raw(idx1, idx2) / sum != 0.0f) {
                xlo = std::min(xlo, n - 1); xhi = std::max(xhi, n - 1);
                zlo = std::min(zlo, m - 1); zhi = std::max(zhi, m - 1);
            }
        }
    }
    if (xhi < 0) {
        box[0] = box[1] = 0;
        box[2] = box[3] = 0;
        return;
    }
    box[0] = xlo; box[1] = zlo; box[2] = xhi - xlo + 1; box[3] = zhi - zlo + 1;
    for (int x = xlo; x <= xhi; x++)
        for (int z = zlo; z <= zhi; z++) {
            const int idx2 = (x + 1) - (isxe - (hw2 - 1)) + 1, idx1 = (z + 1) - (isze - (hw1 - 1)) + 1;
            out->push_back(raw(idx1, idx2) / sum);
        }
}

}  // namespace sfd
