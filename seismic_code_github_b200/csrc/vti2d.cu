// 2-D VTI pseudo-acoustic modelling for sm_100a: the coupled u / q second-order system of
// de-multiple/convolution_srm/vti_qa_2d_c3_demo1 (VS = VTI_multishot_qacoustic_fd_subroutine_c3.f90,
// VM = VTI_multishot_qacoustic_fd_main_c3.f90), every shot of a call in one launch per time step.
//
// Per time step the reference calls extrapolation_one_step_1 (new u from the current u and q,
// VS:432-960) and then extrapolation_one_step_2 (new q from the current u and q, VS:965-1258).
// Neither reads what the other writes -- step 2 takes the current u, not the new one -- so one
// kernel does both, updating the split PML fields of its cells in place and writing the new u and q
// into the slots of the old ones.  With SFD_EXACT the operation order is the reference's as written,
// every multiply, add and divide rounded separately (__fmul_rn, __fadd_rn, __fdiv_rn, __fsqrt_rn),
// so the records equal the FP32 restatement in oracle/vti_oracle.cpp bit for bit.  The default mode
// multiplies by dt^2 / h^2, takes the common factors h^2 and h out of the PML recurrences, leaving one
// division per PML cell, and forms every new value as the current one plus a small difference.  Its
// relative L2 distance from a 64-bit run is 2.2 to 4.1e-6 for grids of 220 to 490 columns and 350 to 630 steps,
// with or without a top PML; the reference order's is 2.3 to 3.2e-6 without and 4.9 to 9.6e-6 with one.
//
// Bound: issue (77%; DRAM at 3.5 TB/s): the stencil's arithmetic on 36 B a cell inside and 44 to 76 B more in
// the PML strips.  A CTA owns
// 64 x 2 cells, one per thread; u with a halo of 5 rows and 8 columns and q with a halo of 8 columns
// (q is only differentiated along x) arrive by two TMA boxes while each thread loads its cell's model
// and old u, q.  Addresses are 32-bit offsets from the shot's slab, formed on the host: with pointer
// arithmetic in the threads integer instructions were more than half of all.  16 shots of 698 x 348,
// 740 steps: 64 ms (default) and 83 ms (exact) with 32 x 8 tiles staged through registers; now 37 and
// 63 ms.  Tiles of 4 and 8 rows 39 and 49 ms; one vector of four cells per thread on 64 x 8 tiles, whose
// PML branch needs 160 registers, 44 ms.
//
// A one-thread-per-shot kernel adds the source to the current u before each step (VM:420-424,
// 468-472); the receiver row is written by the step kernel's threads on that row.  The per-shot model
// windows are built on the device from one copy of the model.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "sfd_internal.h"
#include "tile_stage.cuh"

namespace {

constexpr int kTX = 64, kTZ = 2, kH = 5;      // cells of a CTA's tile (x, z), stencil halo
constexpr int kThreads = kTX * kTZ;           // one cell per thread
constexpr int kGX = 8;                        // ghost columns: x halo rounded to 16 bytes
constexpr int kSX = kTX + 2 * kGX;            // staged columns
constexpr int kMinBlocks = 10;
constexpr int kGridY = 65535;                 // blocks that grid.y holds

// E = true: every operation rounded separately in the reference's order (bit-exact with the
// restatement); E = false: multiplies and adds may contract into FMAs (records within relative L2
// 1e-5 of the restatement)
template <bool E> __device__ __forceinline__ float fm(float a, float b) { return E ? __fmul_rn(a, b) : a * b; }
template <bool E> __device__ __forceinline__ float fa(float a, float b) { return E ? __fadd_rn(a, b) : a + b; }
template <bool E> __device__ __forceinline__ float fs(float a, float b) { return E ? __fsub_rn(a, b) : a - b; }
__device__ __forceinline__ float fd(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float fsq(float a) { return __fsqrt_rn(a); }

struct VtiDev {
    CUtensorMap tm_u[2], tm_q[2];  // u and q slots (column, row, shot), boxes kSX x (kTZ + 10) and kSX x kTZ
    int* err_flag;                 // set to 1 by a CTA whose bounded wait ran out
    // per shot: fields u[2], q[2] and the model vz, eps, delta on rows of `pitch` floats, cell (i, j)
    // (0-based) at (j + 5) * pitch + i + 8, all zero outside the grid; then the x-strip PML fields
    // (nz rows of nxl + nxr floats; u: four pairs, q: three) and the z-strip ones (nzu + nzd rows of
    // nx; u: four pairs)
    float* base;
    long long field, shot_stride;  // floats per field slab, per shot
    long long xs, zs;              // floats per x strip, per z strip
    int pitch, nx, nz, nxl, nxr, nzu, nzd, range, nt;
    float dx, dz, dt, L;
    float cx[2], cz[2];            // default mode: dt^2 / dx^2 and dt^2 / dz^2 as sums of two
    float cd[4], cdd[4];           // ... damping d = speed cd idx^2 and its derivative speed cdd idx (l, r, u, d)
    float cE[5], c1[5];    // coefficient_2nd(10) (fd_coe and fd_coe_pml_2nd alike), coefficient_1st
    float cx1;             // default mode: dt^2 / dx (after the coefficients, which it would shift off 8 bytes: 1%)
    const int* src;        // per shot: source cell i, j (1-based)
    const int* rrow;       // per shot: receiver row (1-based) and whether it is the row-6 fallback
    float* records;        // [shot][range][nt]
};

// Offsets (floats) of one step's arrays in a shot's slab: c = the current slots, o = the old ones that
// take the new values.  Formed on the host, so that a thread's address is one add: of 32 bits (I =
// unsigned) while a shot's slab has fewer than 2^32 floats, of 64 bits beyond.
template <class I>
struct VtiOff {
    int row0;  // first tile row of the launch (grid.y holds 65535)
    I uc, uo, qc, qo, vz, ep, de;
    I uxc[4], uxo[4], qxc[3], qxo[3], uzc[4], uzo[4];  // a1 a2 t2 a3
};

template <class I>
__device__ __forceinline__ I cell(const VtiDev& a, int i, int j) { return (I)(j + kH) * a.pitch + i + kGX; }

// second-derivative sum of VS:511-525: (c1 (f+1 + f-1 - 2 f0) + ... + c5 (...)) / h**2
// (default mode: the sum alone)
template <bool E>
__device__ __forceinline__ float d2(const float* f, int st, const float* cf, float h) {
    const float two_f0 = fm<E>(2.0f, f[0]);
    float s = fm<E>(cf[0], fs<E>(fa<E>(f[st], f[-st]), two_f0));
#pragma unroll
    for (int m = 2; m <= 5; m++) s = fa<E>(s, fm<E>(cf[m - 1], fs<E>(fa<E>(f[m * st], f[-m * st]), two_f0)));
    return E ? fd(s, fm<E>(h, h)) : s;
}
// default mode: s dt^2 / h^2 with the factor as the sum of two.  A grid constant that is rounded once has the
// same error at every cell and step, which shifts the wave's speed; this one is exact to 48 bits.
template <bool E> __device__ __forceinline__ float scaled(float s, const float* c) { return E ? s : fmaf(s, c[0], s * c[1]); }
// first-derivative sum of VS:567-578: (p1 (f+1 - f-1) + ... + p5 (...)) / h (default mode: times rh)
template <bool E>
__device__ __forceinline__ float d1(const float* f, int st, const float* cf, float h, float rh) {
    float s = fm<E>(cf[0], fs<E>(f[st], f[-st]));
#pragma unroll
    for (int m = 2; m <= 5; m++) s = fa<E>(s, fm<E>(cf[m - 1], fs<E>(f[m * st], f[-m * st])));
    return E ? fd(s, h) : s * rh;
}

// the split PML recurrences of one boundary cell (VS:651-663, 840-858): a1 (second-derivative
// part), t2 (first-derivative part with the damping derivative), a2; a1, t2 hold the old values and
// a1o, t2o, a2o the current ones; k2 = speed^2 dt^2, s2 and s1 the second and first derivative (default mode:
// dt^2 in s2 and s1 instead)
template <bool E>
__device__ __forceinline__ void pml_cell(float d, float dd, float dt, float h, float& a1, float a1o, float& t2,
                                         float t2o, float& a2, float a2o, float k2, float s2, float s1) {
    if (E) {
        const float k2s2 = fm<E>(k2, fm<E>(s2, fm<E>(h, h))), k2dd = fm<E>(fm<E>(k2, dd), fm<E>(s1, h));
        const float h2 = fm<E>(h, h);
        const float d2dt = fm<E>(fm<E>(2.0f, d), dt);
        const float P = fs<E>(fa<E>(fm<E>(2.0f, h2), fm<E>(d2dt, h2)), fm<E>(fm<E>(fm<E>(d, d), h2), fm<E>(dt, dt)));
        const float Den = fa<E>(h2, fm<E>(d2dt, h2));
        a1 = fd(fa<E>(fs<E>(fm<E>(a1o, P), fm<E>(h2, a1)), k2s2), Den);
        const float P2 = fs<E>(fa<E>(fm<E>(2.0f, h), fm<E>(d2dt, h)), fm<E>(fm<E>(fm<E>(dt, dt), h), fm<E>(d, d)));
        const float Den2 = fa<E>(h, fm<E>(d2dt, h));
        t2 = fd(fs<E>(fs<E>(fm<E>(t2o, P2), fm<E>(h, t2)), k2dd), Den2);
        a2 = fa<E>(fm<E>(a2o, fs<E>(1.0f, fm<E>(d, dt))), fm<E>(t2, dt));
    } else {
        // The same with h^2 and h taken out, as increments: 2 + 2 t - t^2 = (1 + 2 t) + (1 - t^2), so the rounded
        // reciprocal and t^2 scale only the small difference of two steps, not the value itself.
        const float t = d * dt, q = __frcp_rn(fmaf(2.0f, t, 1.0f)), tt = t * t;
        a1 = fmaf(q, fmaf(k2, s2, fmaf(-tt, a1o, a1o - a1)), a1o);
        t2 = fmaf(q, fmaf(-(k2 * dd), s1, fmaf(-tt, t2o, t2o - t2)), t2o);
        a2 = fmaf(t2, dt, fmaf(-t, a2o, a2o));
    }
}

// 2 c - o + f.  Default mode: as an increment, whose small difference loses nothing, so that a step rounds at the
// size of the field once instead of twice
template <bool E>
__device__ __forceinline__ float leap(float c, float o, float f) {
    return E ? fa<E>(fs<E>(fm<E>(2.0f, c), o), f) : c + ((c - o) + f);
}

__global__ void vti_inject_kernel(const __grid_constant__ VtiDev a, long long uc, float w) {
    sfd::tile::release();
    sfd::tile::acquire();
    const int s = blockIdx.x;
    if (threadIdx.x != 0) return;
    float* u = a.base + (long long)s * a.shot_stride + uc + cell<long long>(a, a.src[2 * s] - 1, a.src[2 * s + 1] - 1);
    *u = __fadd_rn(*u, w);
}

// The window of every shot (get_currshot_parameters, VS:268-338, and VM:405-408) from the model: vz with
// replicated edges, epsilon and delta only inside the window and below the rows nsz0 + nzu + 6.  mdl: the three
// arrays, marr floats apart, of shot s from mdl + s * mshot on (0: one copy for all), columns of nz_v values.
// win: per shot xmin, nsz0 and the model column that its copy starts with.
__global__ void vti_window_kernel(const __grid_constant__ VtiDev a, const float* mdl, long long mshot, long long marr,
                                  const int* win, int nx_v, int nz_v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, s = blockIdx.z;
    if (i >= a.nx) return;
    float* P = a.base + (long long)s * a.shot_stride + 4 * a.field;  // vz, eps, delta
    const float* vz = mdl + s * mshot;
    const float *ep = vz + marr, *de = ep + marr;
    win += 3 * s;
    const int il = min(max(i - a.nxl, 0), a.range - 1);
    for (int j = blockIdx.y; j < a.nz; j += gridDim.y) {
        const int jl = min(max(j - a.nzu, 0), nz_v - 1);
        const long long m = (long long)(min(max(il + win[0], 0), nx_v - 1) - win[2]) * nz_v + jl;
        const bool in = il == i - a.nxl && jl == j - a.nzu && j >= win[1] + a.nzu + 6;
        const long long c = cell<long long>(a, i, j);
        P[c] = vz[m];
        P[a.field + c] = in ? ep[m] : 0.0f;
        P[2 * a.field + c] = in ? de[m] : 0.0f;
    }
}

template <bool E, class I>
__global__ void __launch_bounds__(kThreads, kMinBlocks) vti_step_kernel(const __grid_constant__ VtiDev a,
                                                                        const __grid_constant__ VtiOff<I> o, int cu,
                                                                        int iit) {
    __shared__ __align__(128) float sU[(kTZ + 2 * kH) * kSX];
    __shared__ __align__(128) float sQ[kTZ * kSX];
    __shared__ uint64_t bar;
    const int s = blockIdx.z, tid = threadIdx.x, tx = tid % kTX, ty = tid / kTX;
    const int i0 = blockIdx.x * kTX, j0 = (o.row0 + (int)blockIdx.y) * kTZ;
    float* P = a.base + (long long)s * a.shot_stride;
    const int gi = i0 + tx, gj = j0 + ty;  // 0-based
    const bool in = gi < a.nx && gj < a.nz;
    const I g = cell<I>(a, gi, gj);
    sfd::tile::bar_init(&bar);
    sfd::tile::release();
    float v = 0.0f, de = 0.0f, ep = 0.0f, uo = 0.0f, qo = 0.0f;
    if (in) {
        v = P[o.vz + g];
        de = P[o.de + g];
        ep = P[o.ep + g];
    }
    sfd::tile::acquire();
    // u: rows j0 - 5 .. j0 + kTZ + 4, q: the tile's rows, columns i0 - 8 .. i0 + 71 (allocation columns
    // from i0, a multiple of 64, and rows from j0; rows past the allocation read as zero)
    if (tid == 0) {
        sfd::tile::expect(&bar, 4u * (2 * kTZ + 2 * kH) * kSX);
        sfd::tile::box(sU, &a.tm_u[cu], i0, j0, s, &bar);
        sfd::tile::box(sQ, &a.tm_q[cu], i0, j0 + kH, s, &bar);
    }
    if (in) {
        uo = P[o.uo + g];
        qo = P[o.qo + g];
    }
    if (!sfd::tile::staged(&bar, a.err_flag) || !in) return;
    const float dt = a.dt, dx = a.dx, dz = a.dz, L = a.L;
    const int nx = a.nx, nz = a.nz, nxl = a.nxl, nxr = a.nxr, nzu = a.nzu, nzd = a.nzd;
    const float* U = sU + (ty + kH) * kSX + kGX + tx;  // the cell in the staged u and q
    const float* Q = sQ + ty * kSX + kGX + tx;
    // The sums of the current u and q that both subroutines form: coefficient_2nd(10) is both
    // fd_coe and fd_coe_pml_2nd, the x sums of u and q appear in step 1 and step 2 (added in the
    // other order there, which IEEE addition does not distinguish), the z sum of u in every
    // region of step 1.  Each is formed once (in the default mode times dt^2).
    const float s2 = scaled<E>(fa<E>(d2<E>(U, 1, a.cE, dx), d2<E>(Q, 1, a.cE, dx)), a.cx);
    const float szu = scaled<E>(d2<E>(U, kSX, a.cE, dz), a.cz);
    const bool xin = gi >= nxl && gi < nx - nxr;
    float un, qn;
    if (xin) {  // extrapolation_one_step_1 (VS:432-960) and _2 (VS:965-1072) inside
        const float dv = E ? fm<E>(fm<E>(dt, dt), fm<E>(v, v)) : v * v;
        un = leap<E>(U[0], uo, fm<E>(dv, fa<E>(fm<E>(fa<E>(1.0f, fm<E>(2.0f, de)), s2), szu)));
        qn = leap<E>(Q[0], qo, fm<E>(dv, fm<E>(fm<E>(2.0f, fs<E>(ep, de)), s2)));
        if (gj < nzu || gj >= nz - nzd) {  // the top and bottom PML
            const bool top = gj < nzu;
            const int js = top ? gj : gj - (nz - nzd) + nzu, idx = top ? gj + 1 - (nzu + 1) : gj + 1 - (nz - nzd);
            const I z = (I)js * nx + gi;
            const float a1o = P[o.uzc[0] + z], a2o = P[o.uzc[1] + z], t2o = P[o.uzc[2] + z], a3o = P[o.uzc[3] + z];
            float a1 = P[o.uzo[0] + z], t2 = P[o.uzo[2] + z], a3 = P[o.uzo[3] + z], a2;
            const float sz1 = d1<E>(U, kSX, a.c1, dx, a.cx1);  // divided by dx as written (VS:796, 880)
            float d, dd, k2, n3;
            if (E) {
                const float vn = fm<E>(v, fsq(fa<E>(1.0f, fm<E>(2.0f, de))));
                const float axis = fm<E>((float)idx, dz), thick = fm<E>((float)(top ? nzu : nzd), dz);
                const float A = fd(fm<E>(3.0f, v), fm<E>(2.0f, thick));
                d = fm<E>(fm<E>(A, fm<E>(fd(axis, thick), fd(axis, thick))), L);
                dd = fm<E>(fm<E>(A, fd(fm<E>(2.0f, axis), fm<E>(thick, thick))), L);
                k2 = fm<E>(fm<E>(v, v), fm<E>(dt, dt));
                n3 = fm<E>(fm<E>(fm<E>(vn, vn), fm<E>(dt, dt)), s2);
            } else {
                const float fi = (float)idx;
                d = v * (a.cd[top ? 2 : 3] * (fi * fi));
                dd = v * (a.cdd[top ? 2 : 3] * fi);
                k2 = dv;
                n3 = k2 * (1.0f + 2.0f * de) * s2;
            }
            pml_cell<E>(d, dd, dt, dz, a1, a1o, t2, t2o, a2, a2o, k2, szu, sz1);
            a3 = leap<E>(a3o, a3, n3);
            un = fa<E>(fa<E>(a1, a2), a3);
            P[o.uzo[0] + z] = a1; P[o.uzo[1] + z] = a2; P[o.uzo[2] + z] = t2; P[o.uzo[3] + z] = a3;
        }
    } else {  // the left and right PML (all rows): u, then q (VS:1073-1150) with the same s1, s2, d, dd
        const bool left = gi < nxl;
        const int is = left ? gi : gi - (nx - nxr) + nxl, idx = left ? gi + 1 - (nxl + 1) : gi + 1 - (nx - nxr);
        const I x = (I)gj * (nxl + nxr) + is;
        const float a1o = P[o.uxc[0] + x], a2o = P[o.uxc[1] + x], t2o = P[o.uxc[2] + x], a3o = P[o.uxc[3] + x];
        const float b1o = P[o.qxc[0] + x], b2o = P[o.qxc[1] + x], r2o = P[o.qxc[2] + x];
        float a1 = P[o.uxo[0] + x], t2 = P[o.uxo[2] + x], a3 = P[o.uxo[3] + x];
        float b1 = P[o.qxo[0] + x], r2 = P[o.qxo[2] + x], a2, b2;
        const float s1 = fa<E>(d1<E>(U, 1, a.c1, dx, a.cx1), d1<E>(Q, 1, a.c1, dx, a.cx1));
        float d, dd, kn, kq, n3;
        if (E) {
            const float vn = fm<E>(v, fsq(fa<E>(1.0f, fm<E>(2.0f, de))));
            const float vx = fm<E>(v, fsq(fa<E>(1.0f, fm<E>(2.0f, ep))));
            const float axis = fm<E>((float)idx, dx), thick = fm<E>((float)(left ? nxl : nxr), dx);
            const float A = fd(fm<E>(3.0f, vx), fm<E>(2.0f, thick));
            d = fm<E>(fm<E>(A, fm<E>(fd(axis, thick), fd(axis, thick))), L);
            dd = fm<E>(fm<E>(A, fd(fm<E>(2.0f, axis), fm<E>(thick, thick))), L);
            kn = fm<E>(fm<E>(vn, vn), fm<E>(dt, dt));
            kq = fm<E>(fs<E>(fm<E>(vx, vx), fm<E>(vn, vn)), fm<E>(dt, dt));
            n3 = fd(fm<E>(fm<E>(fm<E>(v, v), fm<E>(dt, dt)), fm<E>(szu, fm<E>(dz, dz))), fm<E>(dz, dz));
        } else {
            const float k0 = v * v, sv = v * sqrtf(1.0f + 2.0f * ep), fi = (float)idx;
            d = sv * (a.cd[left ? 0 : 1] * (fi * fi));
            dd = sv * (a.cdd[left ? 0 : 1] * fi);
            kn = k0 * (1.0f + 2.0f * de);
            kq = k0 * (2.0f * (ep - de));
            n3 = k0 * szu;
        }
        pml_cell<E>(d, dd, dt, dx, a1, a1o, t2, t2o, a2, a2o, kn, s2, s1);
        a3 = leap<E>(a3o, a3, n3);
        un = fa<E>(fa<E>(a1, a2), a3);
        pml_cell<E>(d, dd, dt, dx, b1, b1o, r2, r2o, b2, b2o, kq, s2, s1);
        qn = fa<E>(b1, b2);
        P[o.uxo[0] + x] = a1; P[o.uxo[1] + x] = a2; P[o.uxo[2] + x] = t2; P[o.uxo[3] + x] = a3;
        P[o.qxo[0] + x] = b1; P[o.qxo[1] + x] = b2; P[o.qxo[2] + x] = r2;
    }
    P[o.uo + g] = un;
    P[o.qo + g] = qn;
    // ---- recording (VM:446-453, 494-501): new u on the receiver row ----
    const int rr = a.rrow[2 * s], low = a.rrow[2 * s + 1];
    if (gj + 1 == rr && gi >= nxl && gi < nxl + a.range && iit <= a.nt && ((!low && iit >= 1) || (low && iit > 1)))
        a.records[((long long)s * a.range + (gi - nxl)) * a.nt + (iit - 1)] = un;
}

// coefficient_2nd / coefficient_1st (VS:1264-1472): a(i,j) = i^p / p! (p = 2j or 2j-1) inverted
// by successive Sherman-Morrison updates of the identity; coefficient(i) = 0.5 inv(a)(1, i)
int coefficients(int order, int first, float* out) {
    const int k = first ? (order + 1) / 2 : order / 2;
    if (k < 1 || k > 8) return SFD_ERR_ARG;
    float a[64], inv[64], temp[8], col[8], outer[64], upd[64];
    for (int i = 1; i <= k; i++)
        for (int j = 1; j <= k; j++) {
            const int pw = first ? 2 * j - 1 : 2 * j;
            float num = 1.0f, fact = 1.0f;
            for (int m = 0; m < pw; m++) num = num * (float)i;
            for (int m = 1; m <= pw; m++) fact = fact * (float)m;
            a[(i - 1) * k + (j - 1)] = num / fact;
        }
    for (int q = 0; q < k * k; q++) inv[q] = 0.0f;
    for (int d = 0; d < k; d++) inv[d * k + d] = 1.0f;
    for (int i = 0; i < k; i++) {
        for (int c = 0; c < k; c++) temp[c] = a[i * k + c];
        temp[i] = temp[i] - 1.0f;
        float den = 0.0f;
        for (int r = 0; r < k; r++) den = den + temp[r] * inv[r * k + i];
        den = den + 1.0f;
        for (int r = 0; r < k; r++) col[r] = inv[r * k + i];
        for (int r = 0; r < k; r++)
            for (int c = 0; c < k; c++) outer[r * k + c] = col[r] * temp[c];
        for (int r = 0; r < k; r++)
            for (int c = 0; c < k; c++) {
                float s = 0.0f;
                for (int m = 0; m < k; m++) s = s + outer[r * k + m] * inv[m * k + c];
                upd[r * k + c] = s / den;
            }
        for (int q = 0; q < k * k; q++) inv[q] = inv[q] - upd[q];
    }
    for (int i = 0; i < k; i++) {
        float s = 0.0f;
        for (int m = 0; m < k; m++) s = s + inv[m] * (m == i ? 0.5f : 0.0f);
        out[i] = s;
    }
    return SFD_OK;
}

VtiOff<unsigned> narrow_offsets(const VtiOff<long long>& w) {
    VtiOff<unsigned> n{};
    n.uc = (unsigned)w.uc; n.uo = (unsigned)w.uo; n.qc = (unsigned)w.qc; n.qo = (unsigned)w.qo;
    n.vz = (unsigned)w.vz; n.ep = (unsigned)w.ep; n.de = (unsigned)w.de;
    for (int k = 0; k < 4; k++) {
        n.uxc[k] = (unsigned)w.uxc[k]; n.uxo[k] = (unsigned)w.uxo[k];
        n.uzc[k] = (unsigned)w.uzc[k]; n.uzo[k] = (unsigned)w.uzo[k];
        if (k < 3) { n.qxc[k] = (unsigned)w.qxc[k]; n.qxo[k] = (unsigned)w.qxo[k]; }
    }
    return n;
}

template <class T>
struct DevBuf {
    T* p = nullptr;
    ~DevBuf() { if (p) cudaFree(p); }
    cudaError_t alloc(size_t n) { return cudaMalloc(&p, std::max<size_t>(1, n) * sizeof(T)); }
};

}  // namespace

extern "C" {

int sfd_vti_coefficients(int order, int first, float* out) {
    if (!out) return SFD_ERR_ARG;
    return coefficients(order, first, out);
}

int sfd_vti_forward(const sfd_vti_par* par, const float* vz, const float* epsilon, const float* delta, int nshot,
                    const sfd_vti_shot* shots, int device, float* records, sfd_timing* timing) {
    const auto t_start = std::chrono::steady_clock::now();
    if (!par || !vz || !epsilon || !delta || !shots || !records || nshot < 1) return SFD_ERR_ARG;
    const sfd_vti_par& c = *par;
    if (c.nx_v < 1 || c.nz_v < 1 || c.nt < 1 || !(c.dx > 0) || !(c.dz > 0) || !(c.dt > 0)) return SFD_ERR_ARG;
    if (c.order_explicit != 10 || c.order_pml_2nd != 10 || (c.order_pml_1st != 9 && c.order_pml_1st != 10))
        return SFD_ERR_UNSUPPORTED;  // the stencils are written out with five coefficients (VS:511-551)
    if (c.nx_bound_l < 0 || c.nz_bound_u < 0 || c.nx_bound_r < 2 || c.nz_bound_d < 2) return SFD_ERR_ARG;
    const int range = shots[0].xmax - shots[0].xmin + 1;
    if (range < 1) return SFD_ERR_ARG;
    for (int s = 0; s < nshot; s++)
        if (shots[s].xmax - shots[s].xmin + 1 != range) return SFD_ERR_ARG;  // one grid for the batch
    const int nxl = c.nx_bound_l, nxr = c.nx_bound_r, nzu = c.nz_bound_u, nzd = c.nz_bound_d;
    const int nx = range + nxl + nxr - 2, nz = c.nz_v + nzu + nzd - 2;  // VM:248-249
    if (nx <= 10 || nz <= 10) return SFD_ERR_ARG;

    VtiDev a{};
    a.nx = nx; a.nz = nz; a.nxl = nxl; a.nxr = nxr; a.nzu = nzu; a.nzd = nzd; a.range = range; a.nt = c.nt;
    a.dx = c.dx; a.dz = c.dz; a.dt = c.dt;
    a.L = std::log(1.0f / 1.0e-3f);  // log(1/R), R = 1.0E-3 (VS:14)
    if (coefficients(10, 0, a.cE) || coefficients(c.order_pml_1st, 1, a.c1))
        return SFD_ERR_ARG;
    const int ntx = (nx + kTX - 1) / kTX;
    a.pitch = (ntx * kTX + 2 * kGX + 31) / 32 * 32;
    a.field = (long long)a.pitch * (nz + 2 * kH);
    a.xs = (long long)(nxl + nxr) * nz;
    a.zs = (long long)nx * (nzu + nzd);
    const double dt2 = (double)c.dt * c.dt, gx = dt2 / ((double)c.dx * c.dx), gz = dt2 / ((double)c.dz * c.dz);
    a.cx[0] = (float)gx;
    a.cx[1] = (float)(gx - a.cx[0]);
    a.cz[0] = (float)gz;
    a.cz[1] = (float)(gz - a.cz[0]);
    a.cx1 = (float)(dt2 / c.dx);
    const int pn[4] = {nxl, nxr, nzu, nzd};
    for (int k = 0; k < 4; k++) {
        const double h = k < 2 ? c.dx : c.dz, n3 = (double)std::max(pn[k], 1) * std::max(pn[k], 1) * std::max(pn[k], 1);
        a.cd[k] = (float)(1.5 * (double)a.L / (n3 * h));
        a.cdd[k] = (float)(3.0 * (double)a.L / (n3 * h * h));
    }
    a.shot_stride = 7 * a.field + 14 * a.xs + 8 * a.zs;
    a.shot_stride = (a.shot_stride + 31) / 32 * 32;

    // the values that enter a shot's window (vti_window_kernel) must be usable: vz in its columns, and
    // epsilon and delta there below the zeroed rows.  Per model column: vz valid, last bad row
    std::vector<char> vz_ok(c.nx_v, 1);
    std::vector<int> bad(c.nx_v, 0);  // 1-based row
    for (int i = 0; i < c.nx_v; i++)
        for (int j = 0; j < c.nz_v; j++) {
            const size_t m = (size_t)i * c.nz_v + j;
            if (!(vz[m] > 0.0f) || !std::isfinite(vz[m])) vz_ok[i] = 0;
            if (!std::isfinite(epsilon[m]) || !std::isfinite(delta[m]) || !(1.0f + 2.0f * epsilon[m] >= 0.0f) ||
                !(1.0f + 2.0f * delta[m] >= 0.0f))
                bad[i] = j + 1;
        }
    std::vector<int> src(2 * nshot), rrow(2 * nshot), win(3 * nshot), cols(nshot);
    for (int s = 0; s < nshot; s++) {
        const sfd_vti_shot& sh = shots[s];
        const long long lo = (long long)sh.xmin + 1, hi = (long long)sh.xmin + range;  // 1-based columns, then clamped
        const int c0 = (int)std::min<long long>(std::max<long long>(lo, 1), c.nx_v) - 1;
        const int c1 = (int)std::min<long long>(std::max<long long>(hi, 1), c.nx_v) - 1;
        for (int i = c0; i <= c1; i++)
            if (!vz_ok[i] || bad[i] > sh.nsz0 + 6) return SFD_ERR_ARG;
        win[3 * s] = sh.xmin;
        win[3 * s + 1] = sh.nsz0;
        win[3 * s + 2] = c0;
        cols[s] = c1 - c0 + 1;
        src[2 * s] = sh.nsx - sh.xmin + nxl;  // VS:294-295
        src[2 * s + 1] = sh.nsz0 + nzu;
        if (src[2 * s] < 1 || src[2 * s] > nx || src[2 * s + 1] < 1 || src[2 * s + 1] > nz) return SFD_ERR_ARG;
        const int r = sh.nrz0 + nzu;
        rrow[2 * s] = r >= 6 ? r : 6;
        rrow[2 * s + 1] = r >= 6 ? 0 : 1;
        if (rrow[2 * s] > nz) return SFD_ERR_ARG;
    }

    // source samples (VM:420-424): exp(-(pi f0 (it - 0.07/dt) dt)^2) (1 - 2 (...)^2), it <= nwt
    const int nwt = (int)std::lround((double)((2.0f * 0.07f) / c.dt)) + 1;
    const int half = (int)std::lround((double)(nwt - 1) / 2.0);
    const int NT = c.nt + half;
    std::vector<float> w(nwt + 1, 0.0f);
    for (int it = 1; it <= nwt; it++) {
        const float b = ((3.1415926f * c.f0) * ((float)it - (0.07f / c.dt))) * c.dt;
        w[it] = std::exp(-(b * b)) * (1.0f - 2.0f * (b * b));
    }

    if (cudaSetDevice(device) != cudaSuccess) return SFD_ERR_CUDA;
    cudaStream_t st = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return SFD_ERR_CUDA;
    struct StreamGuard { cudaStream_t s; ~StreamGuard() { cudaStreamDestroy(s); } } sg{st};
    DevBuf<float> state, recs, model;
    DevBuf<int> dsrc, drow, dwin, derr;
    const size_t total = (size_t)nshot * a.shot_stride;
    const size_t rec_n = (size_t)nshot * range * c.nt, nm = (size_t)c.nx_v * c.nz_v;
    if (state.alloc(total) != cudaSuccess || recs.alloc(rec_n) != cudaSuccess || dsrc.alloc(2 * nshot) != cudaSuccess ||
        drow.alloc(2 * nshot) != cudaSuccess || dwin.alloc(3 * nshot) != cudaSuccess || derr.alloc(1) != cudaSuccess) {
        cudaGetLastError();
        return SFD_ERR_NOMEM;
    }
    // One copy of the model for all windows; where it does not fit beside the fields, every shot's columns go to
    // its own u and q slots, which are cleared again after the windows are built.
    const bool shared = model.alloc(3 * nm) == cudaSuccess;
    if (!shared) cudaGetLastError();
    long long h2d = 0;
    if (cudaMemsetAsync(state.p, 0, total * sizeof(float), st) != cudaSuccess ||
        cudaMemsetAsync(recs.p, 0, rec_n * sizeof(float), st) != cudaSuccess ||
        cudaMemsetAsync(derr.p, 0, sizeof(int), st) != cudaSuccess)
        return SFD_ERR_CUDA;
    const float* model_host[3] = {vz, epsilon, delta};
    if (shared) std::fill(cols.begin(), cols.end(), c.nx_v);
    for (int s = 0; s < (shared ? 1 : nshot); s++) {
        const size_t n = (size_t)cols[s] * c.nz_v, first = shared ? 0 : (size_t)win[3 * s + 2] * c.nz_v;
        for (int k = 0; k < 3; k++) {
            float* dst = shared ? model.p + k * nm : state.p + (size_t)s * a.shot_stride + k * a.field;
            if (cudaMemcpyAsync(dst, model_host[k] + first, n * sizeof(float), cudaMemcpyHostToDevice, st) != cudaSuccess)
                return SFD_ERR_CUDA;
            h2d += (long long)(n * sizeof(float));
        }
    }
    for (int s = 0; shared && s < nshot; s++) win[3 * s + 2] = 0;
    if (cudaMemcpyAsync(dsrc.p, src.data(), 2 * nshot * sizeof(int), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(drow.p, rrow.data(), 2 * nshot * sizeof(int), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(dwin.p, win.data(), 3 * nshot * sizeof(int), cudaMemcpyHostToDevice, st) != cudaSuccess)
        return SFD_ERR_CUDA;
    a.base = state.p; a.src = dsrc.p; a.rrow = drow.p; a.records = recs.p; a.err_flag = derr.p;
    VtiOff<long long> off[2] = {};  // by the current slot
    for (int b = 0; b < 2; b++) {
        VtiOff<long long>& f = off[b];
        const long long F = a.field, X = a.xs, Z = a.zs, c0 = b, o0 = 1 - b;
        f.uc = c0 * F; f.uo = o0 * F; f.qc = (2 + c0) * F; f.qo = (2 + o0) * F;
        f.vz = 4 * F; f.ep = 5 * F; f.de = 6 * F;
        for (int k = 0; k < 4; k++) {
            f.uxc[k] = 7 * F + (2 * k + c0) * X; f.uxo[k] = 7 * F + (2 * k + o0) * X;
            if (k < 3) { f.qxc[k] = 7 * F + (8 + 2 * k + c0) * X; f.qxo[k] = 7 * F + (8 + 2 * k + o0) * X; }
            f.uzc[k] = 7 * F + 14 * X + (2 * k + c0) * Z; f.uzo[k] = 7 * F + 14 * X + (2 * k + o0) * Z;
        }
        const long long rows = nz + 2 * kH;
        if (!sfd::encode_map3(&a.tm_u[b], state.p + f.uc, a.pitch, rows, nshot, a.pitch, a.shot_stride, kSX, kTZ + 2 * kH) ||
            !sfd::encode_map3(&a.tm_q[b], state.p + f.qc, a.pitch, rows, nshot, a.pitch, a.shot_stride, kSX, kTZ))
            return SFD_ERR_CUDA;
    }
    const bool wide = a.shot_stride > 0xffffffffLL;
    VtiOff<unsigned> narrow[2] = {narrow_offsets(off[0]), narrow_offsets(off[1])};  // unused if wide
    vti_window_kernel<<<dim3((nx + 127) / 128, std::min(nz, kGridY), nshot), 128, 0, st>>>(
        a, shared ? model.p : state.p, shared ? 0 : a.shot_stride, shared ? (long long)nm : a.field, dwin.p, c.nx_v, c.nz_v);
    if (cudaGetLastError() != cudaSuccess) return SFD_ERR_CUDA;
    for (int s = 0; !shared && s < nshot; s++)
        if (cudaMemsetAsync(state.p + (size_t)s * a.shot_stride, 0, 4 * a.field * sizeof(float), st) != cudaSuccess)
            return SFD_ERR_CUDA;

    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const bool exact = (c.flags & SFD_EXACT) != 0;
    const int rows = (nz + kTZ - 1) / kTZ;
    const void* step = wide ? (exact ? (const void*)vti_step_kernel<true, long long>
                                     : (const void*)vti_step_kernel<false, long long>)
                            : (exact ? (const void*)vti_step_kernel<true, unsigned>
                                     : (const void*)vti_step_kernel<false, unsigned>);
    cudaError_t err = cudaSuccess;
    long long launches = 0;
    cudaEventRecord(e0, st);
    for (int it = 1; it <= NT && err == cudaSuccess; it++) {
        int cu = (it % 2 == 1) ? 1 : 0, iit = it - half;  // odd steps: u2 / q2 current (VM:417-505)
        // The chain of programmatic dependents begins after its first kernel, an inject kernel (nwt >= 1): the
        // steps read the model before their acquire(), which would not wait for vti_window_kernel but only for
        // the kernel before them.
        if (it <= nwt) {
            void* args[] = {&a, &off[cu].uc, &w[it]};
            err = sfd::tile::launch((const void*)vti_inject_kernel, dim3(nshot), 32, 0, st, args, it > 1);
            launches++;
        }
        // a cell reads the current slots and writes the old ones, so a step may be several launches
        for (int row0 = 0; row0 < rows && err == cudaSuccess; row0 += kGridY) {
            off[cu].row0 = narrow[cu].row0 = row0;
            void* args[] = {&a, wide ? (void*)&off[cu] : (void*)&narrow[cu], &cu, &iit};
            err = sfd::tile::launch(step, dim3(ntx, std::min(rows - row0, kGridY), nshot), kThreads, 0, st, args);
            launches++;
        }
    }
    cudaEventRecord(e1, st);
    if (err == cudaSuccess) err = cudaGetLastError();
    if (err == cudaSuccess)
        err = cudaMemcpyAsync(records, recs.p, rec_n * sizeof(float), cudaMemcpyDeviceToHost, st);
    if (err == cudaSuccess) err = cudaStreamSynchronize(st);
    float ms = 0.0f;
    if (err == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (err != cudaSuccess) return SFD_ERR_CUDA;
    int late = 0;
    if (cudaMemcpy(&late, derr.p, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return SFD_ERR_CUDA;
    if (late) return SFD_ERR_TIMEOUT;
    if (timing) {
        std::memset(timing, 0, sizeof(*timing));
        timing->loop_ms = ms;
        timing->device_ms = ms;
        timing->total_ms =
            std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count();
        timing->point_updates = (double)nx * nz * NT * nshot;
        timing->launches = launches;
        timing->h2d_bytes = h2d;
        timing->d2h_bytes = (long long)(rec_n * sizeof(float));
        timing->graph = 0;
        timing->kernel_variant = exact ? 71 : 70;
    }
    return SFD_OK;
}

}  // extern "C"
