// Small-tile step kernel of the 2-D acoustic velocity-pressure scheme (AFD:237-380) for launches that
// give the 64 x 64 tile kernel (acoustic2d_fma.cu) too few CTAs: same update, same values bit for bit
// (forward and adjoint mode), on tiles of 16 columns by 32 rows.
//
// Bound: latency.  One shot of 351 x 351 is 36 tiles of 64 x 64 on 148 SMs, each a serial chain of
// loads and three phases over 16 points per thread; here it is 242 tiles of one vector of four points
// per thread.  The price is the halo (P is read 2.5 times, Vx twice, Vz 1.5 times, from L2) and the
// velocities recomputed on it, which costs less than the idle SMs up to one wave of these CTAs and at
// low orders somewhat beyond (acoustic2d_use_small).
//
// A CTA of 128 threads: P on a cross (the tile with 2R columns on each side, and with 2 round4(R) rows
// above and below), Vx with R columns and Vz with round4(R) rows on each side, copied to shared memory
// asynchronously; phase A (Vx, two columns of one vector per thread from a register window), phase B
// (Vz), a barrier, phase C (P, one vector per thread).  Every stencil sum is the tile kernel's: first
// product, then fused multiply-adds in the order of m.
//
// The same tiles run SFD_EXACT at every size (kExact): each multiply and add rounded by itself in the
// reference's order, the scale factors and the divergence in double.  8 shots of 851 x 451 with variable
// density, order 16: 122 us a step on 64 x 64 tiles with one stencil point per shared-memory load, 60 us
// now (51 Gpts/s; latency: 18 warps an SM at 96 registers, issue 55%, L1 data pipe 58%, FP64 pipe 9%).
#include <cuda.h>
#include <cuda_runtime.h>

#include "sfd_internal.h"
#include "tile_stage.cuh"

namespace sfd {
namespace {

constexpr int TZ = 32;
enum Mode { kForward, kAdjoint, kExact };

__host__ __device__ constexpr int r4(int v) { return (v + 3) & ~3; }

template <int R, int TX>
struct SP {
    static constexpr int kThreads = TX * TZ / 4;
    static constexpr int RQ = r4(R), HX = 2 * R, HZ = 2 * RQ;
    static constexpr int PW = TZ + 2 * HZ, PR = TX + 2 * HX;    // staged P (its corners stay unused)
    static constexpr int VXR = TX + 2 * R, VZW = TZ + 2 * RQ;   // Vx rows, Vz width
    static constexpr int OFF_VX = PR * PW, OFF_VZ = OFF_VX + VXR * TZ;
    static constexpr int OFF_AX = OFF_VZ + TX * VZW, OFF_MX = OFF_AX + VXR;
    static constexpr int OFF_AZ = OFF_MX + VXR, OFF_MZ = OFF_AZ + VZW;
    static constexpr int FLOATS = OFF_MZ + VZW;
    static constexpr int NB = (RQ + 4 + R + 3) / 4;  // 16-byte loads of phase B's window
    static constexpr int NC = (RQ + R + 3 + 3) / 4;  // ... of phase C's
    static_assert(TZ + 2 * RQ - 4 + 4 * NB <= PW && TZ - 4 + 4 * NC <= VZW, "windows end inside the staged rows");
    static_assert(VXR % 2 == 0 && FLOATS * 4 <= 48 * 1024, "row pairs; static shared memory");
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float2 lo(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi(const float4& v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float4 cat(float2 a, float2 b) { return make_float4(a.x, a.y, b.x, b.y); }
__device__ __forceinline__ float2 bc(float c) { return make_float2(c, c); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, bc(-1.0f), a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float comp(const float4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }

__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tile::sptr(dst)), "l"(src) : "memory");
}
// four cells of column x from gz on: a vector inside the grid, else the cells below nz
__device__ __forceinline__ void put(float* f, long long c, const float4& v, int gz, int nz) {
    if (gz + 3 < nz) st4(f + c, v);
    else
        for (int q = 0; q < 4 && gz + q < nz; q++) f[c + q] = comp(v, q);
}

// kExact: one stencil sum in the reference's order, every operation rounded (AFD:255-302)
template <int R, class F>
__device__ __forceinline__ float sum_rn(const float* C, F diff) {
    float s = __fmul_rn(C[0], diff(0));
#pragma unroll
    for (int m = 1; m < R; m++) s = __fadd_rn(s, __fmul_rn(C[m], diff(m)));
    return s;
}
// ... of four cells, two per instruction: the sum as fma(t, one, s) with one = 1.0 from the arguments, which
// the compiler cannot contract with the product (see add2 in elastic2d.cu)
template <int R, class H, class L>
__device__ __forceinline__ float4 sum4_rn(const float* C, float one, H up, L down) {
    float2 sl, sh;
#pragma unroll
    for (int m = 0; m < R; m++) {
        const float4 p = up(m), q = down(m);
        const float2 tl = mul2(bc(C[m]), sub2(lo(p), lo(q))), th = mul2(bc(C[m]), sub2(hi(p), hi(q)));
        sl = m == 0 ? tl : fma2(tl, bc(one), sl);
        sh = m == 0 ? th : fma2(th, bc(one), sh);
    }
    return cat(sl, sh);
}
// kExact: a velocity, v a - (1 / den) (dt / d) s with the scale in double (AFD:259, 276)
__device__ __forceinline__ float vel_rn(float v, float a, double b, float s) {
    return __double2float_rn(__dsub_rn((double)__fmul_rn(v, a), __dmul_rn(b, (double)s)));
}

template <int R, int TX, bool VARDEN, Mode MODE>
__global__ void __launch_bounds__(TX * TZ / 4, 5) acoustic2d_small_kernel(const __grid_constant__ Acou2DArgs a) {
    using T = SP<R, TX>;
    constexpr bool ADJ = MODE == kAdjoint;
    constexpr int kThreads = T::kThreads;
    __shared__ __align__(16) float smem[T::FLOATS];
    float* sP = smem;
    float* sVx = smem + T::OFF_VX;
    float* sVz = smem + T::OFF_VZ;
    float *sAx = smem + T::OFF_AX, *sMx = smem + T::OFF_MX, *sAz = smem + T::OFF_AZ, *sMz = smem + T::OFF_MZ;
    const int tid = threadIdx.x, shot = a.slot_to_shot[blockIdx.y];
    const ShotDev sd = a.shots[shot];
    const int nzt = a.L.ntz * (kTileZ / TZ), txi = blockIdx.x / nzt;
    const int x0 = txi * TX, z0 = (blockIdx.x - txi * nzt) * TZ;
    const int nx = sd.nx, nz = a.nz, pitch = a.L.pitch;
    const long long soff = (long long)shot * a.L.shot_stride;
    auto cell = [&](int x, int z) -> long long { return soff + (long long)(x + a.L.gx) * pitch + a.L.gz + z; };
    tile::release();
    if (x0 >= nx || z0 >= nz) {
        tile::acquire();
        return;
    }
    // what no earlier kernel writes, before the wait for the previous step: the thread's own model vector,
    // and the sponge factors and update masks of the Vx columns and the Vz rows (x wins: ax < 0 outside
    // the x pads)
    const int row = tid >> 3, zo = 4 * (tid & 7), gx = x0 + row, gz = z0 + zo;
    const bool own = gx < nx && gz < nz;
    const long long c = cell(gx, gz);
    // Model values of four cells of a column.  kExact may be given the caller's own array
    // (sfd_forward_noalloc: any alignment, no rows around it), which is read cell by cell and only where
    // the scheme updates; elsewhere `out` stands in, for results that are not kept
    auto model4 = [&](const float* f, int x, int z, float out) -> float4 {
        const long long m = (long long)min(max(sd.x0 + x, 0), a.nx_model - 1) * a.mpitch + z;
        if (MODE != kExact || !a.model_raw) return __ldg(reinterpret_cast<const float4*>(f + m));
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
            v[q] = x >= R && x < nx - R && z + q >= R && z + q < nz - R ? __ldg(f + m + q) : out;
        return make_float4(v[0], v[1], v[2], v[3]);
    };
    const float4 vp = model4(a.vp, gx, gz, 0.0f);
    const float4 dn = VARDEN ? model4(a.den, gx, gz, 1.0f) : make_float4(a.den_c, a.den_c, a.den_c, a.den_c);
    for (int i = tid; i < T::VXR + T::VZW; i += kThreads) {
        const bool isx = i < T::VXR;
        const int p = isx ? x0 - R + i : z0 - T::RQ + i - T::VXR, n = isx ? nx : nz, pml = a.pml;
        float f = isx ? -1.0f : 1.0f;
        if (p >= 0 && p < n) {
            if (p < pml) f = a.sponge[pml - 1 - p];
            else if (p >= n - pml) f = a.sponge[p - (n - pml)];
        }
        (isx ? sAx : sAz - T::VXR)[i] = f;
        (isx ? sMx : sMz - T::VXR)[i] = (p >= R && p < n - R) ? 1.0f : 0.0f;
    }
    tile::acquire();

    // stage P's cross, Vx and Vz; the slabs' ghost margins (2R columns, 2 round4(R) rows) hold the halo
    for (int i = tid; i < T::PR * (TZ / 4); i += kThreads) {
        const int r = i / (TZ / 4), c = i % (TZ / 4);
        copy16(sP + r * T::PW + T::HZ + 4 * c, a.p_in + cell(x0 - T::HX + r, z0 + 4 * c));
    }
    for (int i = tid; i < TX * (2 * T::HZ / 4); i += kThreads) {
        const int r = i / (2 * T::HZ / 4), c = i % (2 * T::HZ / 4), z = 4 * c < T::HZ ? 4 * c : TZ + 4 * c;
        copy16(sP + (r + T::HX) * T::PW + z, a.p_in + cell(x0 + r, z0 - T::HZ + z));
    }
    for (int i = tid; i < T::VXR * (TZ / 4); i += kThreads) {
        const int r = i / (TZ / 4), c = i % (TZ / 4);
        copy16(sVx + r * TZ + 4 * c, a.vx_in + cell(x0 - R + r, z0 + 4 * c));
    }
    for (int i = tid; i < TX * (T::VZW / 4); i += kThreads) {
        const int r = i / (T::VZW / 4), c = i % (T::VZW / 4);
        copy16(sVz + r * T::VZW + 4 * c, a.vz_in + cell(x0 + r, z0 - T::RQ + 4 * c));
    }
    float4 dk = make_float4(0.f, 0.f, 0.f, 0.f), gk = dk;
    if (ADJ && own) {  // cells past nz lie in the slab and are not stored
        dk = ld4(a.adj_div + c);
        gk = ld4(a.adj_g + c);
    }
    float C[R];
#pragma unroll
    for (int m = 0; m < R; m++) C[m] = a.coef[m];
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // ---- phase A: Vx(t) on columns x0-R .. x0+TX+R (AFD:255-269), two columns of one vector each ----
    for (int i = tid; i < T::VXR / 2 * (TZ / 4); i += kThreads) {
        const int r0 = 2 * (i / (TZ / 4)), z = 4 * (i % (TZ / 4));
        float4 w[2 * R + 1];
#pragma unroll
        for (int j = 0; j < 2 * R + 1; j++) w[j] = ld4(sP + (r0 + 1 + j) * T::PW + T::HZ + z);
        const float4 az = ld4(sAz + T::RQ + z), mz = ld4(sMz + T::RQ + z);
#pragma unroll
        for (int o = 0; o < 2; o++) {
            if (MODE == kExact) {
                const float ax = sAx[r0 + o], mx = sMx[r0 + o];
                float* v = sVx + (r0 + o) * TZ + z;
                const float4 vo = ld4(v), sm = sum4_rn<R>(C, a.one, [&](int m) { return w[o + R + m]; },
                                                         [&](int m) { return w[o + R - 1 - m]; });
                float4 d = make_float4(1.f, 1.f, 1.f, 1.f);
                if (VARDEN) d = model4(a.den, x0 - R + r0 + o, z0 + z, 1.0f);
                float out[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const double b = VARDEN ? __dmul_rn(__drcp_rn((double)comp(d, q)), (double)a.dtdx) : a.bx_d;
                    const float n = vel_rn(comp(vo, q), ax >= 0.0f ? ax : comp(az, q), b, comp(sm, q));
                    out[q] = mx * comp(mz, q) != 0.0f ? n : 0.0f;
                }
                st4(v, make_float4(out[0], out[1], out[2], out[3]));
                continue;
            }
            float2 sl = mul2(bc(C[0]), sub2(lo(w[o + R]), lo(w[o + R - 1])));
            float2 sh = mul2(bc(C[0]), sub2(hi(w[o + R]), hi(w[o + R - 1])));
#pragma unroll
            for (int m = 1; m < R; m++) {
                sl = fma2(bc(C[m]), sub2(lo(w[o + R + m]), lo(w[o + R - 1 - m])), sl);
                sh = fma2(bc(C[m]), sub2(hi(w[o + R + m]), hi(w[o + R - 1 - m])), sh);
            }
            float* v = sVx + (r0 + o) * TZ + z;
            const float4 vo = ld4(v);
            float2 bl = bc(-a.bx_f), bh = bl;
            if (VARDEN) {
                const int g = min(max(sd.x0 + x0 - R + r0 + o, 0), a.nx_model - 1);
                const float4 d = __ldg(reinterpret_cast<const float4*>(a.bxm + (long long)g * a.mpitch + z0 + z));
                bl = make_float2(-d.x, -d.y);
                bh = make_float2(-d.z, -d.w);
            }
            const float ax = sAx[r0 + o], mx = sMx[r0 + o];
            float2 vl = lo(vo), vh = hi(vo);
            if (ADJ) {  // staged X'' = B M (X + rdx S+x nu), B = dt/(dx den) (1 here for constant density)
                vl = mul2(fma2(bc(a.rdx_f), sl, vl), mul2(bc(mx), lo(mz)));
                vh = mul2(fma2(bc(a.rdx_f), sh, vh), mul2(bc(mx), hi(mz)));
                if (VARDEN) {
                    vl = mul2(vl, make_float2(-bl.x, -bl.y));
                    vh = mul2(vh, make_float2(-bh.x, -bh.y));
                }
            } else {
                const float4 sa = ax >= 0.0f ? make_float4(ax, ax, ax, ax) : az;
                vl = mul2(vl, lo(sa));
                vh = mul2(vh, hi(sa));
                vl = mul2(fma2(bl, sl, vl), mul2(bc(mx), lo(mz)));
                vh = mul2(fma2(bh, sh, vh), mul2(bc(mx), hi(mz)));
            }
            st4(v, cat(vl, vh));
        }
    }
    // ---- phase B: Vz(t) on rows z0-RQ .. z0+TZ+RQ (AFD:272-286) ----
    for (int i = tid; i < TX * (T::VZW / 4); i += kThreads) {
        const int r = i / (T::VZW / 4), z = 4 * (i % (T::VZW / 4));
        float w[4 * T::NB];  // P(z0 - 2 RQ + z ..): cell q of the vector at RQ + q
#pragma unroll
        for (int j = 0; j < T::NB; j++) {
            const float4 v = ld4(sP + (r + T::HX) * T::PW + z + 4 * j);
            w[4 * j] = v.x; w[4 * j + 1] = v.y; w[4 * j + 2] = v.z; w[4 * j + 3] = v.w;
        }
        float* v = sVz + r * T::VZW + z;
        const float4 vo = ld4(v), az = ld4(sAz + z), mz = ld4(sMz + z);
        const float ax = sAx[r + R], mx = sMx[r + R];
        float out[4];
        float4 d = make_float4(1.f, 1.f, 1.f, 1.f);
        if (VARDEN) d = model4(MODE == kExact ? a.den : a.bzm, x0 + r, z0 - T::RQ + z, 1.0f);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (MODE == kExact) {
                const float s = sum_rn<R>(C, [&](int m) { return __fsub_rn(w[T::RQ + q + 1 + m], w[T::RQ + q - m]); });
                const double b = VARDEN ? __dmul_rn(__drcp_rn((double)comp(d, q)), (double)a.dtdz) : a.bz_d;
                const float n = vel_rn(comp(vo, q), ax >= 0.0f ? ax : comp(az, q), b, s);
                out[q] = mx * comp(mz, q) != 0.0f ? n : 0.0f;
                continue;
            }
            float s = __fmul_rn(C[0], __fsub_rn(w[T::RQ + q + 1], w[T::RQ + q]));
#pragma unroll
            for (int m = 1; m < R; m++) s = __fmaf_rn(C[m], __fsub_rn(w[T::RQ + q + 1 + m], w[T::RQ + q - m]), s);
            float b = a.bz_f;
            if (VARDEN)
                b = comp(d, q);
            const float mk = mx * comp(mz, q);
            if (ADJ) {  // staged Z'' = B M (Z + rdz S+z nu)
                out[q] = __fmul_rn(__fmaf_rn(a.rdz_f, s, comp(vo, q)), mk);
                if (VARDEN) out[q] = __fmul_rn(out[q], b);
            } else {
                out[q] = __fmul_rn(__fmaf_rn(-b, s, __fmul_rn(comp(vo, q), ax >= 0.0f ? ax : comp(az, q))), mk);
            }
        }
        st4(v, make_float4(out[0], out[1], out[2], out[3]));
    }
    __syncthreads();

    // ---- phase C: P(t) on the tile, one vector per thread (AFD:289-314, 337-338) ----
    const int step = a.step;
    float4 pn = make_float4(0.f, 0.f, 0.f, 0.f);
    if (MODE == kExact) {  // AFD:289-302: the divergence and the update in double
        const float* vx = sVx + (row + R) * TZ + zo;
        const float* vz = sVz + row * T::VZW + T::RQ + zo;
        float* pc = sP + (row + T::HX) * T::PW + T::HZ + zo;
        const float ax = sAx[row + R], mx = sMx[row + R];
        const float4 sx = sum4_rn<R>(C, a.one, [&](int m) { return ld4(vx + m * TZ); },
                                     [&](int m) { return ld4(vx - (m + 1) * TZ); });
        float w[4 * T::NC], out[4], pw[4];
#pragma unroll
        for (int j = 0; j < T::NC; j++) {
            const float4 v = ld4(vz - T::RQ + 4 * j);
            w[4 * j] = v.x; w[4 * j + 1] = v.y; w[4 * j + 2] = v.z; w[4 * j + 3] = v.w;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float sz = sum_rn<R>(C, [&](int m) { return __fsub_rn(w[T::RQ + q + m], w[T::RQ + q - 1 - m]); });
            const float kk = __fmul_rn(__fmul_rn(__fmul_rn(comp(dn, q), comp(vp, q)), comp(vp, q)), a.dt);
            const double div = __dadd_rn(__dmul_rn(a.rdx_d, (double)comp(sx, q)), __dmul_rn(a.rdz_d, (double)sz));
            const float p1 = __double2float_rn(__dsub_rn((double)pc[q], __dmul_rn((double)kk, div)));
            out[q] = mx * sMz[T::RQ + zo + q] != 0.0f ? __fmul_rn(p1, ax >= 0.0f ? ax : sAz[T::RQ + zo + q]) : 0.0f;
            pw[q] = out[q];
            if (gx == sd.sx && gz + q == sd.sz && step + 1 < sd.nt) {  // AFD:247-251 of the next step
                if (a.src_pre) a.src_pre[shot] = out[q];
                pw[q] = __fsub_rn(out[q], __fmul_rn(sd.inj_scale, __ldg(a.wavelets + sd.wav_off + step + 1)));
            }
        }
        st4(pc, make_float4(out[0], out[1], out[2], out[3]));  // receivers read the recorded value here
        if (own) {
            put(a.p_out, c, make_float4(pw[0], pw[1], pw[2], pw[3]), gz, nz);
            put(a.vx_out, c, ld4(vx), gz, nz);
            put(a.vz_out, c, ld4(vz), gz, nz);
        }
    } else {
        const float* vx = sVx + (row + R) * TZ + zo;
        float2 sl = mul2(bc(C[0]), sub2(lo(ld4(vx)), lo(ld4(vx - TZ))));
        float2 sh = mul2(bc(C[0]), sub2(hi(ld4(vx)), hi(ld4(vx - TZ))));
#pragma unroll
        for (int m = 1; m < R; m++) {
            const float4 p = ld4(vx + m * TZ), q = ld4(vx - (m + 1) * TZ);
            sl = fma2(bc(C[m]), sub2(lo(p), lo(q)), sl);
            sh = fma2(bc(C[m]), sub2(hi(p), hi(q)), sh);
        }
        sl = mul2(sl, bc(ADJ ? a.adj_cx : a.rdx_f));
        sh = mul2(sh, bc(ADJ ? a.adj_cx : a.rdx_f));
        const float sx[4] = {sl.x, sl.y, sh.x, sh.y};
        float w[4 * T::NC];  // Vz(gz - RQ ..): cell q of the vector at RQ + q
#pragma unroll
        for (int j = 0; j < T::NC; j++) {
            const float4 v = ld4(sVz + row * T::VZW + zo + 4 * j);
            w[4 * j] = v.x; w[4 * j + 1] = v.y; w[4 * j + 2] = v.z; w[4 * j + 3] = v.w;
        }
        float dv[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            float s = __fmul_rn(C[0], __fsub_rn(w[T::RQ + q], w[T::RQ + q - 1]));
#pragma unroll
            for (int m = 1; m < R; m++) s = __fmaf_rn(C[m], __fsub_rn(w[T::RQ + q + m], w[T::RQ + q - 1 - m]), s);
            dv[q] = __fadd_rn(sx[q], __fmul_rn(s, ADJ ? a.adj_cz : a.rdz_f));
        }
        float* pc = sP + (row + T::HX) * T::PW + T::HZ + zo;
        const float4 po = ld4(pc), vxo = ld4(vx);
        const float4 vzo = make_float4(w[T::RQ], w[T::RQ + 1], w[T::RQ + 2], w[T::RQ + 3]);
        const float4 az = ld4(sAz + T::RQ + zo), mz = ld4(sMz + T::RQ + zo);
        const float ax = sAx[row + R], mx = sMx[row + R];
        const float4 sa = ax >= 0.0f ? make_float4(ax, ax, ax, ax) : az;
        const float4 mk = make_float4(mx * mz.x, mx * mz.y, mx * mz.z, mx * mz.w);
        const float2 kl = mul2(mul2(mul2(lo(dn), lo(vp)), lo(vp)), bc(ADJ ? a.dt : -a.dt));
        const float2 kh = mul2(mul2(mul2(hi(dn), hi(vp)), hi(vp)), bc(ADJ ? a.dt : -a.dt));
        if (ADJ) {
            // bracket = nu_old / K + S-x(B M X') + S-z(B M Z') (= M a Q_old + ...), nu_new = M a K bracket
            const float2 bl = make_float2(__fadd_rn(dv[0], __fdividef(po.x, kl.x)), __fadd_rn(dv[1], __fdividef(po.y, kl.y)));
            const float2 bh = make_float2(__fadd_rn(dv[2], __fdividef(po.z, kh.x)), __fadd_rn(dv[3], __fdividef(po.w, kh.y)));
            pn = cat(mul2(mul2(bl, kl), mul2(lo(sa), lo(mk))), mul2(mul2(bh, kh), mul2(hi(sa), hi(mk))));
            if (own) {
                // X = a M X' and Z = a M Z' from the staged B M X', B M Z'
                float4 xf = sa, zf = sa;
                if (VARDEN) {
                    xf = make_float4(sa.x * dn.x * a.adj_xs, sa.y * dn.y * a.adj_xs, sa.z * dn.z * a.adj_xs,
                                     sa.w * dn.w * a.adj_xs);
                    zf = make_float4(sa.x * dn.x * a.adj_zs, sa.y * dn.y * a.adj_zs, sa.z * dn.z * a.adj_zs,
                                     sa.w * dn.w * a.adj_zs);
                }
                const float bq[4] = {bl.x, bl.y, bh.x, bh.y};
                if (gx == sd.sx && sd.sz >= gz && sd.sz < gz + 4)
                    for (int q = 0; q < 4; q++)
                        if (sd.sz == gz + q) a.adj_lam[(long long)shot * a.nt_max + step] = bq[q];
                put(a.adj_g, c, make_float4(fmaf(po.x, dk.x, gk.x), fmaf(po.y, dk.y, gk.y), fmaf(po.z, dk.z, gk.z),
                                            fmaf(po.w, dk.w, gk.w)), gz, nz);
                put(a.p_out, c, pn, gz, nz);
                put(a.vx_out, c, make_float4(vxo.x * xf.x, vxo.y * xf.y, vxo.z * xf.z, vxo.w * xf.w), gz, nz);
                put(a.vz_out, c, make_float4(vzo.x * zf.x, vzo.y * zf.y, vzo.z * zf.z, vzo.w * zf.w), gz, nz);
            }
        } else {
            const float2 pl = fma2(kl, make_float2(dv[0], dv[1]), lo(po)), ph = fma2(kh, make_float2(dv[2], dv[3]), hi(po));
            pn = cat(mul2(mul2(pl, lo(sa)), lo(mk)), mul2(mul2(ph, hi(sa)), hi(mk)));
            st4(pc, pn);  // receivers read the recorded value here
            if (own) {
                if (a.div_out != nullptr) put(a.div_out, c, make_float4(dv[0], dv[1], dv[2], dv[3]), gz, nz);
                float pw[4] = {pn.x, pn.y, pn.z, pn.w};
                if (gx == sd.sx && sd.sz >= gz && sd.sz < gz + 4 && step + 1 < sd.nt) {
                    const float inj = sd.inj_scale * __ldg(a.wavelets + sd.wav_off + step + 1);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (sd.sz == gz + q) {
                            if (a.src_pre) a.src_pre[shot] = pw[q];
                            pw[q] -= inj;
                        }
                }
                put(a.p_out, c, make_float4(pw[0], pw[1], pw[2], pw[3]), gz, nz);
                put(a.vx_out, c, vxo, gz, nz);
                put(a.vz_out, c, vzo, gz, nz);
            }
        }
    }
    // receivers of the 64 x 64 tile that lie in this one: the record (AFD:376-377), or its transpose for
    // step k-1, nu += M a K res (several receivers may share a cell, so the adds are atomic)
    const int* trp = a.tile_rec_ptr + sd.tile_rec_base + x0 / kTileX * a.L.ntz + z0 / kTileZ;
    const int rb = __ldg(trp), re = __ldg(trp + 1);
    if (re <= rb || (ADJ && step < 1)) return;
    __syncthreads();
    for (int j = rb + tid; j < re; j += kThreads) {
        const int ridx = a.tile_rec_idx[j];
        const int rx = a.rec_x[sd.rec_list + ridx], rz = a.rec_z[sd.rec_list + ridx];
        if (rx < x0 || rx >= x0 + TX || rz < z0 || rz >= z0 + TZ) continue;
        if (!ADJ) {
            a.records[sd.rec_base + (long long)step * sd.nrec + ridx] = sP[(rx - x0 + T::HX) * T::PW + (rz - z0) + T::HZ];
            continue;
        }
        if (rx < R || rx >= nx - R || rz < R || rz >= nz - R) continue;  // M = 0
        const long long m = (long long)min(sd.x0 + rx, a.nx_model - 1) * a.mpitch + rz;
        const float vpv = __ldg(a.vp + m), dnv = VARDEN ? __ldg(a.den + m) : a.den_c;
        float sa = 1.0f;
        if (rx < a.pml) sa = a.sponge[a.pml - 1 - rx];
        else if (rx >= nx - a.pml) sa = a.sponge[rx - (nx - a.pml)];
        else if (rz < a.pml) sa = a.sponge[a.pml - 1 - rz];
        else if (rz >= nz - a.pml) sa = a.sponge[rz - (nz - a.pml)];
        const float v = a.adj_res[sd.rec_base + (long long)(step - 1) * sd.nrec + ridx];
        atomicAdd(a.p_out + cell(rx, rz), dnv * vpv * vpv * a.dt * sa * v);
    }
}

template <int R, int TX, Mode MODE>
cudaError_t launch_r(const Acou2DArgs& a, int active, bool varden, cudaStream_t st) {
    const dim3 grid(a.L.ntx * (kTileX / TX) * a.L.ntz * (kTileZ / TZ), active);
    const void* k = varden ? (const void*)acoustic2d_small_kernel<R, TX, true, MODE>
                           : (const void*)acoustic2d_small_kernel<R, TX, false, MODE>;
    return tile::launch(k, grid, SP<R, TX>::kThreads, 0, st, a);
}

template <int TX, Mode MODE>
cudaError_t launch_mode(int radius, const Acou2DArgs& a, int active, bool varden, cudaStream_t st) {
    switch (radius) {
    case 1: return launch_r<1, TX, MODE>(a, active, varden, st);
    case 2: return launch_r<2, TX, MODE>(a, active, varden, st);
    case 4: return launch_r<4, TX, MODE>(a, active, varden, st);
    case 5: return launch_r<5, TX, MODE>(a, active, varden, st);
    case 8: return launch_r<8, TX, MODE>(a, active, varden, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t acoustic2d_small_launch(int radius, const Acou2DArgs& a, int active, bool varden, cudaStream_t st, bool adj) {
    if (varden && (!a.bxm || !a.bzm)) return cudaErrorInvalidValue;
    return adj ? launch_mode<16, kAdjoint>(radius, a, active, varden, st)
               : launch_mode<16, kForward>(radius, a, active, varden, st);
}

cudaError_t acoustic2d_exact_launch(int radius, const Acou2DArgs& a, int active, bool varden, cudaStream_t st) {
    return launch_mode<16, kExact>(radius, a, active, varden, st);
}

// One wave of small tiles (five CTAs per SM, 92 tiles of 64 x 64) takes the same time however few they are, and so
// do up to one of the tile kernel's persistent CTAs per SM.  Measured (us a step; small tiles / persistent CTAs
// / one tile per CTA): order 16, 64 to 90 tiles 5.4 / 7.2 / 9.5, 99 tiles 7.5 / 7.0 / 9.9, 147 tiles 9.2 / 7.4 / 8.9;
// order 16 with variable density 5.7 / 8.0 / 11, 8.0 / 7.8 / 11.8, 9.8 / 8.2 / 10.6; order 8 4.4 / 6.6 / 8.5, 6.2 / 6.4 /
// 9.0, 7.6 / 6.7 / 8.0; order 4 4.4 / 6.2 / 8, 4.4 / 6.1 / 8.2, 6.8 / 6.3 / 7.3; gradients alike.  So one wave runs the
// small tiles, and beyond it the tuner times both.  Steps with fewer tiles than SMs, but more than a wave, under
// a plan that does not run persistent CTAs (the last shots of an uneven batch) take the small tiles too.
bool acoustic2d_one_small_wave(const Layout2D& L, int active) {
    return (long long)active * L.ntx * L.ntz * (kTileX / 16) * (kTileZ / TZ) <= 5LL * num_sms();
}
bool acoustic2d_use_small(const Acou2DPlan& plan, const Layout2D& L, int active) {
    if (plan.pinned || plan.hooked) return false;
    return plan.small || acoustic2d_one_small_wave(L, active) ||
           (plan.stages == 1 && (long long)active * L.ntx * L.ntz < num_sms());
}

}  // namespace sfd
