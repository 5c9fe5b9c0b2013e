// force_direct.cu -- the force of a few thousand bodies in one launch.
//
// What bounds small systems is latency: the launches, the first loads, the
// hand-over between kernels; 1,000 bodies are half a microsecond of
// arithmetic for the whole GPU.  Here every CTA stages all bodies in shared
// memory (packed in pairs) and sums up a few targets from all of them: no
// pieces, no second kernel.  A warp has kLanes target lanes with KT targets
// each, so that its 32 / kLanes lane groups and the 16 warps share the sources
// 64 or 128 ways.  Both bodies of a pair are evaluated (12 packed operations
// for two interactions where pairs take 16 for four), so that it ends where
// the arithmetic outweighs the hand-over.
//
// A call in a graph, against the pair and reduction kernels: 64 bodies 4.1 ->
// 1.6 us, 1,000: 5.7 -> 2.5, 2,048: 7.0 -> 4.1, 3,000: 9.4 -> 6.3, 4,096:
// 11.0 -> 9.9, 4,864: 14.2 -> 11.4; one launch instead of two from the host:
// 13.7 -> 8.6 us.  A step of the reference integrator: 1,000 bodies 6.7 ->
// 3.9 us, 4,096: 12.0 -> 11.2; an FP64 step 8.2 -> 4.1 and 14.2 -> 11.9 (with
// the integrator's early launch).
// Errors against 64 bits: 3.3e-8 to 8.7e-8 of the forces' rms from 600 bodies
// on, 0.25 to 0.70 of the one-sided kernel's.  What is added up in plain FP32 is
// at most 304 sources (chains of 38 in each half of a pair, then a tree); the
// one-sided kernel's folds are 256 in chains of 128.
#include <cuda_runtime.h>

#include "nbgb_device.cuh"
#include "nbgb_integrate.cuh"
#include "nbgb_internal.h"
#include "nbody_gb300.h"

namespace nbgb {
namespace {

constexpr int kWarps = 16, kThreads = 32 * kWarps;

struct DirectParams {
    const float4 *pm;
    float4 *__restrict__ force;
    unsigned *__restrict__ status;  // not null: refuse masses < 0
    int n, np;  // bodies; pairs of sources, a multiple of every kSub
    float eps2;
};

// Dynamic shared memory: {x, y} of the pairs, then {z, m}.
size_t direct_smem(int np) { return (size_t)np * 32; }
int pairs_of(size_t n) { return (int)((n + 15) / 16 * 8); }

template <int kLanes, int KT>
__global__ void __launch_bounds__(kThreads, 1)
    direct_kernel(const __grid_constant__ DirectParams P) {
    extern __shared__ __align__(128) float4 pairs[];
    __shared__ float red[kWarps][3][KT * kLanes];
    constexpr int kSub = 32 / kLanes, kShares = kWarps * kSub;  // of the sources
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int at = lane & (kLanes - 1), sub = lane / kLanes;
    float4 *const xy = pairs, *const zm = pairs + P.np;
    grid_dependents_launch();
    grid_dependency_wait();
    f2 nx[KT], ny[KT], nz[KT], ax[KT], ay[KT], az[KT];
    float4 t[KT];
#pragma unroll
    for (int k = 0; k < KT; k++) {
        const int i = blockIdx.x * (KT * kLanes) + k * kLanes + at;
        t[k] = P.pm[min(i, P.n - 1)];
    }
    for (int q = tid; q < P.np; q += kThreads) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 a = 2 * q < P.n ? P.pm[2 * q] : zero, b = 2 * q + 1 < P.n ? P.pm[2 * q + 1] : zero;
        if (P.status && jstream_log_slot(q)) {
            // refused where a log-domain j-stream would hold log2 m: NaN,
            // which every body's sum then meets
            if (!(a.w >= 0.f) || !(b.w >= 0.f)) {
                atomicOr(P.status, NBGB_STATUS_NEGATIVE_MASS);
                a.w = __int_as_float(0x7fc00000);
            }
        }
        xy[q] = make_float4(a.x, b.x, a.y, b.y);
        zm[q] = make_float4(a.z, b.z, a.w, b.w);
    }
#pragma unroll
    for (int k = 0; k < KT; k++) {
        nx[k] = f2_pack(-t[k].x, -t[k].x);
        ny[k] = f2_pack(-t[k].y, -t[k].y);
        nz[k] = f2_pack(-t[k].z, -t[k].z);
        ax[k] = ay[k] = az[k] = 0;
    }
    const f2 eps2p = f2_pack(P.eps2, P.eps2);
    __syncthreads();
    const ulonglong2 *a = reinterpret_cast<const ulonglong2 *>(xy) + warp * kSub + sub;
    const ulonglong2 *b = reinterpret_cast<const ulonglong2 *>(zm) + warp * kSub + sub;
#pragma unroll(KT > 3 ? 1 : 2)
    for (int q = warp * kSub; q < P.np; q += kShares, a += kShares, b += kShares) {
        const ulonglong2 u = *a, v = *b;
#pragma unroll
        for (int k = 0; k < KT; k++)
            pair_interact2(u.x, u.y, v.x, v.y, nx[k], ny[k], nz[k], eps2p, ax[k], ay[k], az[k]);
    }
#pragma unroll
    for (int k = 0; k < KT; k++) {
        const f2 acc[3] = {ax[k], ay[k], az[k]};
#pragma unroll
        for (int c = 0; c < 3; c++) {
            float l, h;
            f2_unpack(acc[c], l, h);
            float s = l + h;
#pragma unroll
            for (int o = kLanes; o < 32; o *= 2)
                s += __shfl_xor_sync(0xffffffffu, s, o);
            if (sub == 0)
                red[warp][c][k * kLanes + at] = s;
        }
    }
    __syncthreads();
    // the warps' sums, in order; four threads a body
    if (tid < 4 * KT * kLanes) {
        const int j = tid >> 2, c = tid & 3, i = blockIdx.x * (KT * kLanes) + j;
        float hi = 0.f, lo = 0.f;
        if (c < 3) {
#pragma unroll
            for (int w = 0; w < kWarps; w++)
                comp_add(hi, lo, red[w][c][j]);
        }
        if (i < P.n)
            reinterpret_cast<float *>(P.force)[4 * i + c] = round_force(hi, lo);
    }
}

// The reference integrator after it (the force kernel's CTAs all read
// positions to the end of their staging).
__global__ void __launch_bounds__(128)
    direct_integrate_kernel(const float4 *force, FusedIntegrate fi, int n) {
    grid_dependents_launch();
    grid_dependency_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const float4 f = force[i], p = fi.pm[i];
    fused_integrate(fi, i, fi.vel[i], p.x, p.y, p.z, p.w, f.x, f.y, f.z);
}

template <int kLanes, int KT>
cudaError_t launch_kt(const DirectParams &P, cudaStream_t st) {
    const unsigned blocks = (unsigned)((P.n + KT * kLanes - 1) / (KT * kLanes));
    return launch_dependent(direct_kernel<kLanes, KT>, blocks, kThreads, direct_smem(P.np), st, P);
}
template <int kLanes, int KT>
bool prepare_kt() {
    return cudaFuncSetAttribute(direct_kernel<kLanes, KT>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)direct_smem(pairs_of(kMaxDirect))) == cudaSuccess;
}

}  // namespace

// Targets of a CTA, in fours: as many as give each SM one CTA, in eights above
// 16.  Four lanes below 16 (more shares of the sources: 1,000 bodies 2.5 us,
// 2.9 with eight), eight from there on (2,432 bodies 4.5 us; four lanes 4.7).
// 20 and 28 targets on four lanes save 4 and 2 % of a call but take all
// registers of an SM: the integrator's blocks, which start early, were then
// all on the two or so SMs without a CTA, and an FP64 step of 3,000 bodies
// took 11.3 us instead of 8.
int direct_targets(size_t n, int sms) {
    const size_t fours = (n + (size_t)sms * 4 - 1) / ((size_t)sms * 4);
    return n <= kMaxDirect && fours <= 8 ? (int)(fours > 4 ? (fours + 1) / 2 * 2 : fours) : 0;
}

int direct_prepare() {
    return prepare_kt<4, 1>() && prepare_kt<4, 2>() && prepare_kt<4, 3>() && prepare_kt<8, 2>() &&
                   prepare_kt<8, 3>() && prepare_kt<8, 4>()
               ? NBGB_OK
               : NBGB_ERR_CUDA;
}

int launch_direct(size_t n, int targets, unsigned *status, float4 *force, const float4 *posMass,
                  float eps2, cudaStream_t st, const FusedIntegrate *fi) {
    DirectParams P;
    P.pm = posMass;
    P.force = force;
    P.status = status;
    P.n = (int)n;
    P.np = pairs_of(n);
    P.eps2 = eps2;
    cudaError_t e = cudaErrorInvalidValue;
    switch (targets) {
    case 1: e = launch_kt<4, 1>(P, st); break;
    case 2: e = launch_kt<4, 2>(P, st); break;
    case 3: e = launch_kt<4, 3>(P, st); break;
    case 4: e = launch_kt<8, 2>(P, st); break;
    case 6: e = launch_kt<8, 3>(P, st); break;
    case 8: e = launch_kt<8, 4>(P, st); break;
    }
    if (e != cudaSuccess)
        return NBGB_ERR_CUDA;
    if (!fi || !fi->vel)
        return NBGB_OK;
    FusedIntegrate f = *fi;
    f.js = nullptr;
    return launch_dependent_n(direct_integrate_kernel, (unsigned)((n + 127) / 128), 128, 0, st,
                              force, f, (int)n) == cudaSuccess
               ? NBGB_OK
               : NBGB_ERR_CUDA;
}

}  // namespace nbgb
