// nbgb_pair.cuh -- a row of targets against sets of sources, every pair
// evaluated once (force_pair.cu has the scheme; ensemble.cu uses the same).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "nbgb_device.cuh"

namespace nbgb {
namespace pair {

template <int W_, int KI_, int NC_, int CTAS_>
struct Geo {
    static constexpr int W = W_, KI = KI_, NC = NC_;
    static constexpr int kThreads = 32 * W;
    static constexpr int kCtas = CTAS_;           // resident CTAs per SM
    static constexpr int kRow = 32 * W * KI;      // targets per row
    static constexpr int kSet = 64 * NC;          // sources per set
    static constexpr int kRowSets = kRow / kSet;
    static_assert(kRow % kSet == 0, "a row is whole sets");
    // steps between folds of the targets' sums: 256 sources
    // (128 where narrow rows serve few bodies: the largest error of the
    // near-cancelling ones falls by a third for 1 % of the time)
    static constexpr int kFoldSteps = KI > 4 ? 128 / NC : 64 / NC;
    static constexpr int kHop = 16;  // steps a reaction travels between adds
    // dynamic shared memory: hi/lo sums, reactions of two pieces, two
    // sets in pairs, the next set as it comes from memory
    static constexpr int kHl = 6 * KI * kThreads;             // floats
    static constexpr int kRed = 2 * W * 3 * kSet;             // floats
    static constexpr int kSource = (2 * NC) * 64 * 4;         // one staged set, floats
    static constexpr int kSrc = 2 * kSource;                  // floats
    static constexpr int kRaw = kSet * 4;                     // floats
    static constexpr size_t kSmem = (size_t)(kHl + kRed + kSrc + kRaw) * 4;
};
typedef Geo<4, 8, 2, 2> Wide;
typedef Geo<4, 4, 2, 2> Narrow;

constexpr float kRange = 1.0995116e12f;  // 2^40

enum : int { kFar = 1, kMixed = 2 };  // set flags: out of range, masses differ

// eps2 within 2^+-80
__host__ __device__ inline int eps2_short_ok(float eps2) {
    return eps2 >= 8.3e-25f && eps2 <= 1.2e24f;
}

// (row, set) meetings of the rows before b, counted from row 0.
template <class G>
__host__ __device__ inline long long meetings_before(int b, int nsets) {
    return (long long)b * nsets - (long long)G::kRowSets * b * (b - 1) / 2;
}

enum : int { kEqual = 0, kShort = 1, kWide = 2, kOneSided = 3 };

// Steps t0 .. t1-1 of one meeting.  src: this lane's first source pair; rw:
// the warp's reaction sums [3][kSet] (overwritten), times rs.  The travelling
// reactions are added to them every kHop steps: chains of kHop KI terms
// instead of 32 KI, so that they are no longer than the targets' chains.
template <class G, int MODE>
__device__ __forceinline__ void
meet(const ulonglong2 *src, int t0, int t1, const f2 (&nx)[G::KI], const f2 (&ny)[G::KI],
     const f2 (&nz)[G::KI], const f2 (&nm)[G::KI], f2 (&ax)[G::KI], f2 (&ay)[G::KI],
     f2 (&az)[G::KI], f2 eps2p, int lane, float *rw, float rs) {
    constexpr int KI = G::KI, NC = G::NC;
    const int from = (lane + 1) & 31;
    f2 sx[NC], sy[NC], sz[NC], sm[NC];
    src += t0;
#pragma unroll
    for (int c = 0; c < NC; c++) {
        const ulonglong2 a = src[128 * c], b = src[128 * c + 64];
        sx[c] = a.x;
        sy[c] = a.y;
        sz[c] = b.x;
        sm[c] = b.y;
    }
#pragma unroll 1
    for (int ta = t0; ta < t1; ta += G::kHop) {
        const int tb = min(ta + G::kHop, t1);
        f2 rx[NC], ry[NC], rz[NC];
#pragma unroll
        for (int c = 0; c < NC; c++)
            rx[c] = ry[c] = rz[c] = 0;
#pragma unroll 2
        for (int t = ta; t < tb; t++) {
            src++;
#pragma unroll
            for (int c = 0; c < NC; c++) {
#pragma unroll
                for (int k = 0; k < KI; k++) {
                    const f2 dx = f2_add(sx[c], nx[k]);
                    const f2 dy = f2_add(sy[c], ny[k]);
                    const f2 dz = f2_add(sz[c], nz[k]);
                    f2 d2 = f2_fma(dx, dx, eps2p);
                    d2 = f2_fma(dy, dy, d2);
                    d2 = f2_fma(dz, dz, d2);
                    float l, h;
                    f2_unpack(d2, l, h);
                    const f2 inv = f2_pack(rsqrt_mufu(l), rsqrt_mufu(h));
                    const f2 inv2 = f2_mul(inv, inv);
                    f2 wi, wj;
                    if constexpr (MODE == kEqual) {
                        wi = wj = f2_mul(inv, inv2);
                    } else if constexpr (MODE == kShort) {
                        const f2 s = f2_mul(inv, inv2);
                        wi = f2_mul(sm[c], s);
                        wj = f2_mul(nm[k], s);
                    } else {
                        wi = f2_mul(f2_mul(sm[c], inv), inv2);
                        if constexpr (MODE == kWide)
                            wj = f2_mul(f2_mul(nm[k], inv), inv2);
                    }
                    ax[k] = f2_fma(dx, wi, ax[k]);
                    ay[k] = f2_fma(dy, wi, ay[k]);
                    az[k] = f2_fma(dz, wi, az[k]);
                    if constexpr (MODE != kOneSided) {
                        rx[c] = f2_fma(dx, wj, rx[c]);
                        ry[c] = f2_fma(dy, wj, ry[c]);
                        rz[c] = f2_fma(dz, wj, rz[c]);
                    }
                }
                const ulonglong2 a = src[128 * c], b = src[128 * c + 64];
                sx[c] = a.x;
                sy[c] = a.y;
                sz[c] = b.x;
                sm[c] = b.y;
                if constexpr (MODE != kOneSided) {
                    rx[c] = __shfl_sync(0xffffffffu, rx[c], from);
                    ry[c] = __shfl_sync(0xffffffffu, ry[c], from);
                    rz[c] = __shfl_sync(0xffffffffu, rz[c], from);
                }
            }
        }
        if constexpr (MODE != kOneSided) {
#pragma unroll
            for (int c = 0; c < NC; c++) {
                const int p = 32 * c + ((lane + tb) & 31);
                const f2 r[3] = {rx[c], ry[c], rz[c]};
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    float2 *d = reinterpret_cast<float2 *>(rw + q * G::kSet + 2 * p);
                    float l, h;
                    f2_unpack(r[q], l, h);
                    float2 v = make_float2(l * rs, h * rs);
                    if (ta > t0) {
                        v.x += d->x;
                        v.y += d->y;
                    }
                    *d = v;
                }
            }
            __syncwarp();
        }
    }
}

// Source j of a set into its staged form: pairs {x0,x1,y0,y1}, {z0,z1,m0,m1},
// each list twice in a row.
template <class G>
__device__ __forceinline__ void store_source(float *buf, int j, float4 v) {
    const int pr = j >> 1, c = pr >> 5;
    float *p = buf + ((2 * c) * 64 + (pr & 31)) * 4 + (j & 1);
    p[0] = p[128] = v.x;
    p[2] = p[130] = v.y;
    p[256] = p[384] = v.z;
    p[258] = p[386] = v.w;
}

// Steps s .. s_end-1 of row b, counted from any whole meeting, the first in its
// meeting with `set`, by the whole CTA.  smem: G::kSmem bytes.  The step loops
// need every register, so what they do not use is asked of io where it is
// needed: pm(), n(), eps2(), short_ok() (eps2 in the short forms' range),
// status() (not null: refuse masses < 0), react(s) (the piece of step s's
// meeting, not asked for one-sided ones), tsum() (the targets' piece, 3 x
// kRow), remainder() (whether what rounding the piece to one float leaves out
// follows it; not asked for where a stretch is 256 sources at most, which the
// one-sided kernel too adds up in one float).  SHARE: the last row may fill only some warps' targets; it meets only
// its own sets, one-sided, and warps without targets of their own then take a
// share of the others' steps (one or two full warps: 4 or 2 shares).
template <class G, bool SHARE, class Io>
__device__ __forceinline__ void row_stretch(const Io &io, float *smem, int b, int set,
                                            unsigned s, unsigned s_end) {
    constexpr int KI = G::KI, NC = G::NC, NT = G::kThreads, kSet = G::kSet;
    float *src_buf = smem;                     // [2][2 NC][64] float4
    float *red = smem + G::kSrc;               // [2][W][3][kSet]
    float *hl = smem + G::kSrc + G::kRed;      // [6 KI][NT]
    float4 *raw = reinterpret_cast<float4 *>(smem + G::kSrc + G::kRed + G::kHl);  // [kSet]
    __shared__ int flags[2][G::W];
    __shared__ float mass[2][G::W];            // a warp's (first) mass of each set
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const f2 eps2p = f2_pack(io.eps2(), io.eps2());
    const f2 zero2 = f2_pack(0.f, 0.f);
    const int row_set = b * G::kRowSets;
    int buf = 0;
    const int full =
        SHARE ? min(G::W, (io.n() - b * G::kRow + 32 * KI - 1) / (32 * KI)) : G::W;
    const int shares = SHARE ? G::W / full : 1;
    const int tile = SHARE ? warp % full : warp;
    const int share = SHARE ? warp / full : 0;  // share >= shares: idle

    // A plan that refuses negative masses refuses them where a log-domain
    // j-stream would hold log2 m (jstream_log_slot): it turns them into NaN,
    // which every body's sum then meets.
    auto checked = [&](float4 v, int i) {
        if (io.status() && jstream_log_slot(i >> 1) && !(v.w >= 0.f)) {
            atomicOr(io.status(), NBGB_STATUS_NEGATIVE_MASS);
            v.w = __int_as_float(0x7fc00000);
        }
        return v;
    };
    // one set: staged by store_source; the flags say which forms it allows.
    // The bodies come asynchronously (no registers held), each read by the thread that
    // asked for it; bodies beyond n are zeros.
    auto fetch = [&](int set) {
        const int j = set * kSet + tid;
        if (tid < kSet)
            async_g2s_16(raw + tid, io.pm() + (j < io.n() ? j : 0), j < io.n() ? 16u : 0u);
    };
    auto stage = [&](int buf) {
        async_wait_all();
        if (tid >= kSet)
            return;
        const float4 v = checked(raw[tid], tid);  // sets are whole groups of pairs
        const float m0 = __shfl_sync(0xffffffffu, v.w, 0);
        const bool far = !(fabsf(v.x) < kRange && fabsf(v.y) < kRange && fabsf(v.z) < kRange);
        const bool mixed = !(v.w == m0 && fabsf(m0) < 1e30f);
        store_source<G>(src_buf + buf * G::kSource, tid, v);
        const bool any_far = __any_sync(0xffffffffu, far);
        const bool any_mixed = __any_sync(0xffffffffu, mixed);
        if (lane == 0) {
            flags[buf][warp] = (any_far ? kFar : 0) | (any_mixed ? kMixed : 0);
            mass[buf][warp] = m0;
        }
    };
    static_assert(kSet % 32 == 0, "whole warps stage");
    static_assert(NT >= kSet, "one thread stages one source");


    f2 nx[KI], ny[KI], nz[KI], nm[KI], ax[KI], ay[KI], az[KI];
    bool tfar = false, tmixed = false;
    float tm0 = 0.f;
#pragma unroll
    for (int k = 0; k < KI; k++) {
        const int i = b * G::kRow + tile * 32 * KI + lane + 32 * k;
        const float4 v =
            i < io.n() ? checked(io.pm()[i], i) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (k == 0)
            tm0 = __shfl_sync(0xffffffffu, v.w, 0);
        tfar |= !(fabsf(v.x) < kRange && fabsf(v.y) < kRange && fabsf(v.z) < kRange);
        tmixed |= !(v.w == tm0 && fabsf(tm0) < 1e30f);
        nx[k] = f2_pack(-v.x, -v.x);
        ny[k] = f2_pack(-v.y, -v.y);
        nz[k] = f2_pack(-v.z, -v.z);
        nm[k] = f2_pack(-v.w, -v.w);
        ax[k] = ay[k] = az[k] = zero2;
#pragma unroll
        for (int c = 0; c < 6; c++)
            hl[(6 * k + c) * NT + tid] = 0.f;
    }
    const bool short_ok = io.short_ok() && !__any_sync(0xffffffffu, tfar);
    const bool tequal = !__any_sync(0xffffffffu, tmixed);
    int folded_steps = 0;
    float scale = 1.f;
    // the targets' sums since the last fold -> compensated sums
    auto fold = [&]() {
#pragma unroll
        for (int k = 0; k < KI; k++) {
            f2 *a[3] = {&ax[k], &ay[k], &az[k]};
#pragma unroll
            for (int c = 0; c < 3; c++) {
                float l, h;
                f2_unpack(*a[c], l, h);
                float hi = hl[(6 * k + c) * NT + tid], lo = hl[(6 * k + 3 + c) * NT + tid];
                comp_add(hi, lo, (l + h) * scale);
                hl[(6 * k + c) * NT + tid] = hi;
                hl[(6 * k + 3 + c) * NT + tid] = lo;
                *a[c] = zero2;
            }
        }
        folded_steps = 0;
    };

    fetch(set);
    stage(buf);
    __syncthreads();
    while (s < s_end) {
        const int t0 = (int)(s & 31u);
        const int t1 = min(32, t0 + (int)(s_end - s));
        const unsigned s_next = s + (unsigned)(t1 - t0);
        const bool more = s_next < s_end;  // then t1 == 32
        if (more)
            fetch(set + 1);
        const float sm0 = mass[buf][0];
        int fl = 0;
#pragma unroll
        for (int w = 0; w < kSet / 32; w++)
            fl |= flags[buf][w] | (mass[buf][w] == sm0 ? 0 : kMixed);
        const bool one_sided = set < row_set + G::kRowSets;
        const bool in_range = short_ok && !(fl & kFar);
        const bool equal = in_range && tequal && !(fl & kMixed) && !one_sided;
        const float new_scale = equal ? sm0 : 1.f;
        if (new_scale != scale) {
            if (folded_steps)
                fold();
            scale = new_scale;
        }
        const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(src_buf) +
                                (size_t)buf * 2 * NC * 64 + lane;
        float *rb = red + (size_t)(buf * G::W) * 3 * kSet;
        float *rw = rb + (size_t)warp * 3 * kSet;
        const float rs = equal ? -tm0 : 1.f;
        if (equal)
            meet<G, kEqual>(src, t0, t1, nx, ny, nz, nm, ax, ay, az, eps2p, lane, rw, rs);
        else if (one_sided)
            meet<G, kOneSided>(
                src,
                SHARE ? (share < shares ? t0 + (t1 - t0) * share / shares : t1) : t0,
                SHARE ? (share < shares ? t0 + (t1 - t0) * (share + 1) / shares : t1) : t1, nx,
                ny, nz, nm, ax, ay, az, eps2p, lane, rw, rs);
        else if (in_range)
            meet<G, kShort>(src, t0, t1, nx, ny, nz, nm, ax, ay, az, eps2p, lane, rw, rs);
        else
            meet<G, kWide>(src, t0, t1, nx, ny, nz, nm, ax, ay, az, eps2p, lane, rw, rs);
        folded_steps += t1 - t0;
        if (folded_steps + 32 > G::kFoldSteps)
            fold();
        if (more)
            stage(buf ^ 1);
        __syncthreads();
        if (!one_sided) {
            float *out = io.react(s);
#pragma unroll
            for (int q = tid; q < 3 * kSet; q += NT) {
                float t = rb[q];
#pragma unroll
                for (int w = 1; w < G::W; w++)
                    t += rb[w * 3 * kSet + q];
                out[q] = t;
            }
        }
        s = s_next;
        set++;
        buf ^= 1;
    }
    if (folded_steps)
        fold();
    if (SHARE && shares > 1)
        __syncthreads();
    float *out = io.tsum() + tile * 32 * KI + lane;
    auto total = [&](int k, int c, float &hi, float &lo) {
        hi = hl[(6 * k + c) * NT + tid];
        lo = hl[(6 * k + 3 + c) * NT + tid];
        for (int q = 1; q < shares; q++) {
            comp_add(hi, lo, hl[(6 * k + c) * NT + tid + 32 * full * q]);
            lo += hl[(6 * k + 3 + c) * NT + tid + 32 * full * q];
        }
    };
    if (share == 0) {
#pragma unroll
        for (int k = 0; k < KI; k++)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                float hi, lo;
                total(k, c, hi, lo);
                out[c * G::kRow + 32 * k] = __fadd_rn(hi, lo);
            }
        // (a loop of its own: a condition on each store cost all rows 4 %)
        if (io.remainder()) {
#pragma unroll
            for (int k = 0; k < KI; k++)
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    float hi, lo, sum, rest;
                    total(k, c, hi, lo);
                    two_sum(hi, lo, sum, rest);
                    out[(3 + c) * G::kRow + 32 * k] = rest;
                }
        }
    }
    // the next row's staging reuses buffers others may still be reading
    __syncthreads();
}

}  // namespace pair
}  // namespace nbgb
