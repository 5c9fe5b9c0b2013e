// pair_potential.cu -- the potential energy's sums with each pair evaluated
// once: for every body i
//     phi_i = -(2 sum_{j in later rows} m_j / r_ij + sum_{j != i in i's row} m_j / r_ij),
// r_ij^2 = |p_j - p_i|^2 + eps2, so that sum_i m_i phi_i / 2 is the potential
// energy: a pair of different rows counts once, twice, instead of from both
// sides, and nothing has to be added to the other body.
//
// What bounds it: 7 packed FP32 operations and two MUFU rsqrt for two pairs
// (one-sided, with the force: 13 and two for two interactions), so the MUFU
// pipe (16 cycles of it, 14 of the FMA pipe).  Rows of 1,024 targets (8 a
// lane) against sets of 128 sources read rotated from shared memory, cut into
// equal stretches of steps, three resident CTAs per SM, as in force_pair.cu.
// Diagnostics of 262,144 bodies, with all that is around this kernel: 26.5 ms
// from the one-sided force-and-potential kernel, 8.0 ms from here (4.3e12
// pairs/s; the MUFU pipe alone allows 4.7e12); 65,536: 1,780 and 570 us;
// 20,000: 288 and 119; 8,192: 128 and 117; 4,096: 108 and 106; 1,000: 104 and 97.
// A stretch's sums carry the remainders of their rounding, which equal masses
// have in common: without them 165,639 bodies are 7.2e-9 off, not 5.5e-9.
// Against 64 bits both are off by 5.5e-9 of the energy at 262,144 (the MUFU
// rsqrt's mean error), and where the self pair weighs (eps2 = 0.01, N = 20,000)
// 2.8e-8 there and 5e-9 here.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "nbgb_internal.h"
#include "nbgb_pair.cuh"
#include "nbody_gb300.h"

namespace nbgb {
namespace {

typedef pair::Geo<4, 8, 2, 3> PG;
constexpr int kFoldSets = 2;  // 256 sources between folds
// From so many steps a CTA on, 12 % of the work is left to late CTAs, which fill
// the SMs as their first CTAs end (force_pair.cu): 262,144 bodies 8,350 us
// without, 8,240 with 4 %, 8,120 with 8, 7,990 with 12, 8,020 with 16, 8,045
// with 20; 65,536: 591 and 570.
constexpr int kLateSteps = 240;
constexpr int kMinSteps = 16;  // of a CTA; with 8, 4,096 bodies take longer (more pieces)

struct PotParams {
    const float4 *__restrict__ pm;
    float *__restrict__ tsum;  // [row + CTA][sums, remainders][kRow]
    int n, nsets, rows, ncta, slots;
    // The first `slots` CTAs take the first `early` steps, the late ones the
    // rest: q[] steps each, one more for the first r[] of them
    unsigned early, q[2], r[2];
    float eps2;
};

__device__ __forceinline__ unsigned first_step(const PotParams &P, int c) {
    const int w = c > P.slots;
    const unsigned k = (unsigned)(c - (w ? P.slots : 0));
    return (w ? P.early : 0u) + k * P.q[w] + min(k, P.r[w]);
}

// the CTA that takes step s
__device__ __forceinline__ int holder(const PotParams &P, unsigned s) {
    const int w = s >= P.early;
    s -= w ? P.early : 0u;
    const unsigned longer = P.r[w] * (P.q[w] + 1);
    return (w ? P.slots : 0) +
           (int)(s < longer ? s / (P.q[w] + 1) : P.r[w] + (s - longer) / P.q[w]);
}

__global__ void __launch_bounds__(PG::kThreads, PG::kCtas)
    potential_kernel(const __grid_constant__ PotParams P) {
    constexpr int KI = PG::KI, NC = PG::NC, kSet = PG::kSet;
    __shared__ __align__(128) float src_buf[2 * PG::kSource];
    __shared__ float4 raw[kSet];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = blockIdx.x;
    unsigned s = first_step(P, cta);
    const unsigned s_end = first_step(P, cta + 1);
    int b;
    {  // the row that holds meeting s / 32
        int lo = 0, hi = P.rows - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (pair::meetings_before<PG>(mid, P.nsets) <= (long long)(s >> 5))
                lo = mid;
            else
                hi = mid - 1;
        }
        b = lo;
    }
    auto fetch = [&](int set) {
        const int j = set * kSet + tid;
        async_g2s_16(raw + tid, P.pm + (j < P.n ? j : 0), j < P.n ? 16u : 0u);
    };
    static_assert(PG::kThreads == kSet, "one thread stages one source");
    const f2 eps2p = f2_pack(P.eps2, P.eps2);
    for (; s < s_end; b++) {
        const unsigned row_step = (unsigned)(pair::meetings_before<PG>(b, P.nsets) << 5);
        const int row_set = b * PG::kRowSets;
        const unsigned seg_end =
            min(s_end, row_step + ((unsigned)(P.nsets - row_set) << 5));
        f2 nx[KI], ny[KI], nz[KI], ap[KI];
        float hi[KI], lo[KI];
#pragma unroll
        for (int k = 0; k < KI; k++) {
            const int i = b * PG::kRow + warp * 32 * KI + lane + 32 * k;
            const float4 v = i < P.n ? P.pm[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            nx[k] = f2_pack(-v.x, -v.x);
            ny[k] = f2_pack(-v.y, -v.y);
            nz[k] = f2_pack(-v.z, -v.z);
            ap[k] = 0;
            hi[k] = lo[k] = 0.f;
        }
        int set = row_set + (int)((s - row_step) >> 5), buf = 0, pending = 0;
        __syncthreads();  // the previous row's buffers are no longer read
        fetch(set);
        async_wait_all();
        pair::store_source<PG>(src_buf, tid, raw[tid]);
        __syncthreads();
        while (s < seg_end) {
            const int t0 = (int)(s & 31u);
            const int t1 = min(32, t0 + (int)(seg_end - s));
            s += (unsigned)(t1 - t0);
            const bool more = s < seg_end;
            if (more)
                fetch(set + 1);
            const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(src_buf) +
                                    (size_t)buf * 2 * NC * 64 + lane;
#pragma unroll 2
            for (int t = t0; t < t1; t++) {
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    const ulonglong2 xy = src[128 * c + t], zm = src[128 * c + 64 + t];
#pragma unroll
                    for (int k = 0; k < KI; k++) {
                        const f2 dx = f2_add(xy.x, nx[k]);
                        const f2 dy = f2_add(xy.y, ny[k]);
                        const f2 dz = f2_add(zm.x, nz[k]);
                        f2 d2 = f2_fma(dx, dx, eps2p);
                        d2 = f2_fma(dy, dy, d2);
                        d2 = f2_fma(dz, dz, d2);
                        float l, h;
                        f2_unpack(d2, l, h);
                        ap[k] = f2_fma(zm.y, f2_pack(rsqrt_mufu(l), rsqrt_mufu(h)), ap[k]);
                    }
                }
            }
            // own-row pairs are met from both sides: half
            const bool own = set < row_set + PG::kRowSets;
            const bool last_own = set + 1 == row_set + PG::kRowSets;
            if (++pending == kFoldSets || last_own || !more) {
                const float scale = own ? 0.5f : 1.f;
#pragma unroll
                for (int k = 0; k < KI; k++) {
                    float l, h;
                    f2_unpack(ap[k], l, h);
                    comp_add(hi[k], lo[k], (l + h) * scale);
                    ap[k] = 0;
                }
                pending = 0;
            }
            if (more) {
                async_wait_all();
                pair::store_source<PG>(src_buf + (buf ^ 1) * PG::kSource, tid, raw[tid]);
            }
            __syncthreads();
            set++;
            buf ^= 1;
        }
        float *out = P.tsum + ((size_t)b + cta) * 2 * PG::kRow + warp * 32 * KI + lane;
#pragma unroll
        for (int k = 0; k < KI; k++) {
            float sum, rest;
            two_sum(hi[k], lo[k], sum, rest);
            out[32 * k] = sum;
            out[PG::kRow + 32 * k] = rest;
        }
    }
}

// Body i's pieces in stretch order, minus the self pair, times -2 into
// phi[i].w.
__global__ void __launch_bounds__(256)
    potential_reduce_kernel(const __grid_constant__ PotParams P, float4 *__restrict__ phi) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n)
        return;
    const int b = i / PG::kRow;
    const unsigned a = (unsigned)(pair::meetings_before<PG>(b, P.nsets) << 5);
    const unsigned e = (unsigned)(pair::meetings_before<PG>(b + 1, P.nsets) << 5);
    const int c0 = holder(P, a), c1 = holder(P, e - 1);
    const float *piece = P.tsum + ((size_t)b + c0) * 2 * PG::kRow + (i - b * PG::kRow);
    float hi = 0.f, lo = 0.f;
#pragma unroll 8
    for (int c = 2 * c0; c <= 2 * c1 + 1; c++, piece += PG::kRow)
        comp_add(hi, lo, *piece);
    // the self pair, its product rounded (the loop adds it unrounded): an error
    // common to bodies of one mass, up to 5e-9 of the energy of 836 of them and
    // below 1e-9 from a few thousand on
    comp_add(hi, lo, -0.5f * (P.pm[i].w * rsqrt_mufu(P.eps2)));
    phi[i].w = -2.f * (hi + lo);
}

PotParams params(size_t n, int sms) {
    PotParams P = {};
    P.n = (int)n;
    P.nsets = (int)((n + PG::kSet - 1) / PG::kSet);
    P.rows = (int)((n + PG::kRow - 1) / PG::kRow);
    const long long steps = 32 * pair::meetings_before<PG>(P.rows, P.nsets);
    P.ncta = P.slots = (int)std::max<long long>(
        1, std::min<long long>((long long)sms * PG::kCtas, steps / kMinSteps));
    long long part[2] = {steps, 0};
    if (steps >= (long long)P.slots * kLateSteps) {
        part[0] = steps * 88 / 100;
        part[1] = steps - part[0];
        P.ncta = 2 * P.slots;
    }
    P.early = (unsigned)part[0];
    for (int w = 0; w < 2; w++) {
        P.q[w] = (unsigned)(part[w] / P.slots);
        P.r[w] = (unsigned)(part[w] % P.slots);
    }
    return P;
}

}  // namespace

size_t potential_workspace_bytes(size_t n, int sms) {
    const PotParams P = params(n, sms);
    return (size_t)(P.rows + P.ncta) * 2 * PG::kRow * 4;
}

int launch_potential(size_t n, int sms, const float4 *posMass, float eps2, void *workspace,
                     float4 *phi, cudaStream_t st) {
    PotParams P = params(n, sms);
    P.pm = posMass;
    P.tsum = (float *)workspace;
    P.eps2 = eps2;
    potential_kernel<<<P.ncta, PG::kThreads, 0, st>>>(P);
    potential_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(P, phi);
    return cudaGetLastError() == cudaSuccess ? NBGB_OK : NBGB_ERR_CUDA;
}

}  // namespace nbgb
