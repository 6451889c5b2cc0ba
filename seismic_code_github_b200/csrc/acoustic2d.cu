// Dispatch of the 2-D acoustic velocity-pressure step of
// forward/Acoustic_FD_by_ss/src/Acoustic_1order_FD.cpp (AFD:237-380), batched over shots, and the
// injection of the first source sample.
//
// One launch = one time step of every active shot: Vx and Vz (AFD:255-286), P from the undamped new
// velocities (AFD:289-314), the sponge, receiver extraction (AFD:376-377) and the source injection of the
// next step (AFD:247-251).  Velocities are stored *before* the sponge multiply.  AFD multiplies Vx1 (and
// its copy Vx2) by absorb after P has been computed (AFD:329-336), so the next step's Vx2 equals stored *
// absorb, which the kernels evaluate with the same single rounding.  SFD_EXACT keeps AFD's operation order
// (no FMA contraction, double-precision scale factors) and reproduces the reference bit for bit
// (acoustic2d_small.cu); the default kernels (acoustic2d_march.cu, acoustic2d_fma.cu,
// acoustic2d_small.cu) use FMA and agree with one another bit for bit.
#include <cuda_runtime.h>

#include <algorithm>

#include "sfd_internal.h"

namespace sfd {
namespace {

// Step-0 source injection into the zeroed P(0): P2[src] = 0 - ((dt*DEN)*Vp)*signal[0].
__global__ void inject0_kernel(const __grid_constant__ Acou2DArgs a, int nshot, bool exact) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nshot) return;
    const ShotDev sd = a.shots[s];
    const float w = a.wavelets[sd.wav_off];
    const long long c = (long long)s * a.L.shot_stride + (long long)(sd.sx + a.L.gx) * a.L.pitch + a.L.gz + sd.sz;
    a.p_out[c] = exact ? __fsub_rn(0.0f, __fmul_rn(sd.inj_scale, w)) : -(sd.inj_scale * w);
}

__global__ void buoyancy_kernel(const float* __restrict__ den, float c, float* __restrict__ out, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = __fdiv_rn(c, den[i]);
}

}  // namespace

cudaError_t launch_buoyancy(const float* den, float c, float* out, long long n, cudaStream_t st) {
    buoyancy_kernel<<<(unsigned)std::min<long long>((n + 255) / 256, 148 * 16), 256, 0, st>>>(den, c, out, n);
    return cudaGetLastError();
}

bool acoustic2d_plan(int radius, Acou2DPlan* plan) {
    if (radius != 1 && radius != 2 && radius != 4 && radius != 5 && radius != 8) return false;
    *plan = Acou2DPlan{};
    plan->radius = radius;
    plan->tx = kTileX;
    plan->tz = kTileZ;
    plan->gz = acoustic2d_fma_gz(radius);
    plan->stages = 1;
    return true;
}

cudaError_t acoustic2d_launch_step(const Acou2DPlan& plan, const Acou2DArgs& a, int active, bool exact,
                                   bool varden, cudaStream_t st) {
    if (exact) return acoustic2d_exact_launch(plan.radius, a, active, varden, st);
    return acoustic2d_fwd_launch(plan, plan.radius, a, active, varden, st);
}

cudaError_t acoustic2d_launch_inject0(const Acou2DArgs& a, int nshot, bool exact, cudaStream_t st) {
    inject0_kernel<<<(nshot + 127) / 128, 128, 0, st>>>(a, nshot, exact);
    return cudaGetLastError();
}

}  // namespace sfd
