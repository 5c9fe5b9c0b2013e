// ensemble.cu -- many independent systems of uneven N on one GPU.
//
// The reference evaluates one system per call (its algorithms take one
// posMass array, src/nbody.h:68); running thousands of small systems that way
// costs a launch (and a host round trip) per system per step and leaves most
// of the GPU idle.  Here every active system's state is resident in one arena
// and a tick advances all of them by one FP64 kick-drift-kick step.
//
// Pair systems (the default plan): every pair of bodies evaluated once, in
// three launches chained by programmatic dependence:
//
//   ens_drift      v += a dt/2; x += v dt (FP64) for moving systems, FP32
//                  posMass of every active system; one body per thread, 32
//                  bodies of one system per warp
//   ens_pair       persistent CTAs take (system, row, chunk of source sets)
//                  items from a device queue, largest first, and evaluate
//                  them as force_pair.cu does; every partial sum has a place
//                  of its own in the scratch arena.  Small systems are tasks
//                  of single warps instead, four to an item: 128 targets
//                  against all sources, one-sided, with the closing kick
//   ens_reduce     adds each body's partial sums in a fixed order, writes the
//                  FP32 acceleration and applies the closing v += a dt/2
//
// The items and the places of a system's sums depend only on its N.  Systems
// whose scratch together exceeds the arena are evaluated in groups, one
// ens_pair and ens_reduce each.
//
// Systems with an explicit bucket plan, and those too large for the arena, use
// the one-sided work queue with three launches of its own:
//
//   ens_kick_drift   v += a dt/2; x += v dt (FP64) for moving systems, and
//                    rewrite every active system's FP32 posMass and j-stream
//   ens_force        ONE persistent launch: CTAs take work items (system,
//                    i-block, j-split) from a device queue with an atomic
//                    counter, largest items first, and evaluate them with the
//                    same TMA ring, f32x2 pair interaction (every fourth
//                    source pair in the log domain for systems whose masses
//                    are all >= 0) and TwoSum accumulation as the
//                    single-system kernel; a system whose
//                    j-range is split combines its partials in fixed order
//                    (last item of the i-block, atomic counter)
//   ens_kick         v += a dt/2 for moving systems
//
// Newton-3 systems (opt-in, nbgb_ensemble_set_newton3_min): systems of at
// least that many bodies are pair systems whatever their bucket's plan, and
// move in pass 0 of each tick only.  Those too large for the scratch arena are
// evaluated with block pairs and FP64 sums (force_sym.cu), whose results
// repeat to FP64 rounding order (not bit for bit).
//
// Sub-cycling: a system may take up to kMaxSub steps per tick (its `sub`).
// A tick then runs passes p = 0 .. max sub - 1, each the three launches above
// over the systems whose effective sub (min(sub, steps left)) exceeds p, so
// small systems advance several steps while large ones advance one.  Pass p's
// work items are a suffix of one list sorted by effective sub (ascending),
// then cost (descending).
//
// A system's decomposition (kernel variant, tile size, j-split) depends only
// on its own N, so its result is bit-identical whether it runs alone or in
// any mix (with any sub).  Newly admitted systems spend their first tick in the force pass
// only (their initial accelerations); systems whose steps are done leave the
// tick.  While the membership is unchanged the tick is replayed from a CUDA
// graph.  Admission is bounded by a slot count and a device-memory budget.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "nbgb_device.cuh"
#include "nbgb_internal.h"
#include "nbgb_snapshot.h"
#include "nbgb_pair.cuh"
#include "nbody_gb300.h"

namespace nbgb {
namespace ens {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kStages = 3;
constexpr int kMaxJT = 1024;  // largest tile (bodies); ring stage = 16 KiB
constexpr uint32_t kStageBytes = kMaxJT * 16u;

// kLogMass: j-stream pairs q % 4 == 0 (system-local) hold log2 masses and
// are evaluated in the log domain (set when every mass is >= 0).
enum : int { kMove = 1, kInForce = 2, kLogMass = 4 };
constexpr int kMaxSub = 8;  // steps per tick of one system, at most

// Device descriptor of one system slot.
struct Desc {
    int n;         // bodies
    int body_off;  // into the body arrays
    int js_off;    // into the j-stream arena (float4 units, even)
    int ntiles;
    int jt;        // bodies per tile
    int variant;   // targets/thread and unroll: 0 (1, 8), 1 (2, 4), 2 (1, 4), 3 (2, 8)
    int nsplit;
    int nblocks;
    long long part_off;  // into the partial arena (float4 units); lo follows hi
    int cnt_off;         // into the counter arena
    int ni_pad;          // nblocks * block bodies
    int flags;           // kMove | kInForce | kLogMass
    int sub;             // passes of this tick the system moves in (1..kMaxSub)
    float eps2;
    double dt;
    // pair systems
    int pair;            // 0 no, 1 narrow rows, 2 wide rows, 3 warp tasks
    int nsets;           // source sets
    int ch;              // sets per item
    int target_pieces;   // of an item: its targets' sums, and their remainders
    long long react_off, tsum_off;  // into the scratch arena (floats)
};

struct Params {
    const Desc *desc;
    const int4 *items;  // {system, i-block, split, 0}
    int n_items;
    unsigned *head;     // queue counter (zeroed before the launch)
    const float4 *pm;   // all bodies
    const float4 *js;   // all j-streams
    float4 *acc;        // all bodies
    float4 *part;       // partial arena
    unsigned *cnt;      // counter arena
};

// One work item with K targets per thread.  tile_base: tiles this CTA has
// streamed through its ring before this item (keeps stage phases continuous
// across items).  Returns false if a bounded wait ran out.
template <int K, int UNROLL, bool LOGM>
__device__ bool process_item(const Params &P, const Desc &d, int ib, int r, unsigned tile_base,
                             float4 *ring, uint64_t *full, unsigned *released, int *stage_tile,
                             int *abort_flag, int *s_last) {
    constexpr int BI = kThreads * K;
    const int tid = threadIdx.x, lane = tid & 31;
    const int t_begin = (int)(((long long)r * d.ntiles) / d.nsplit);
    const int t_end = (int)(((long long)(r + 1) * d.ntiles) / d.nsplit);
    const int nt = t_end - t_begin;
    const int jt = d.jt;
    const uint32_t tile_bytes = (uint32_t)jt * 16u;
    const float4 *js = P.js + d.js_off;

    if (tid == 0) {
        // the previous item read these stages through the generic proxy
        fence_proxy_async_shared();
        for (int u = 0; u < kStages && u < nt; u++) {
            const unsigned g = tile_base + (unsigned)u;
            const int s = (int)(g % kStages);
            mbar_expect_tx(&full[s], tile_bytes);
            bulk_g2s(ring + (size_t)s * kMaxJT, js + (size_t)(t_begin + u) * jt, tile_bytes,
                     &full[s]);
            stage_tile[s] = (int)g;
        }
    }

    f2 nx[K], ny[K], nz[K];
    float hx[K], hy[K], hz[K], lx[K], ly[K], lz[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int i = ib * BI + k * kThreads + tid;
        const float4 b = (i < d.n) ? P.pm[d.body_off + i] : make_float4(0.f, 0.f, 0.f, 0.f);
        nx[k] = f2_pack(-b.x, -b.x);
        ny[k] = f2_pack(-b.y, -b.y);
        nz[k] = f2_pack(-b.z, -b.z);
        hx[k] = hy[k] = hz[k] = lx[k] = ly[k] = lz[k] = 0.f;
    }
    const f2 eps2p = f2_pack(d.eps2, d.eps2);
    const f2 zero2 = f2_pack(0.f, 0.f);
    const f2 m15 = f2_pack(-1.5f, -1.5f);

    bool failed = false;
    for (int t = 0; t < nt; t++) {
        const unsigned g = tile_base + (unsigned)t;
        const int s = (int)(g % kStages);
        const uint32_t parity = (g / kStages) & 1u;
        if (__any_sync(0xffffffffu, *(volatile int *)abort_flag != 0)) {
            failed = true;
            break;
        }
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(&full[s], parity))) {
            if (lane == 0)
                *(volatile int *)abort_flag = 1;
            failed = true;
            break;
        }
        const ulonglong2 *tp = reinterpret_cast<const ulonglong2 *>(ring + (size_t)s * kMaxJT);
        f2 ax[K], ay[K], az[K];
        // fold into the compensated sum every 256 sources (or per tile)
        const int fpairs = jt / 2 < 128 ? jt / 2 : 128;
        for (int q0 = 0; q0 < jt / 2; q0 += fpairs) {
#pragma unroll
            for (int k = 0; k < K; k++)
                ax[k] = ay[k] = az[k] = zero2;
            if constexpr (LOGM) {  // groups of 4 pairs, the first in the log domain
                constexpr int GROUPS = UNROLL >= 4 ? UNROLL / 4 : 1;
#pragma unroll GROUPS
                for (int q = q0; q < q0 + fpairs; q += 4) {
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const ulonglong2 a = tp[2 * (q + u)];
                        const ulonglong2 b = tp[2 * (q + u) + 1];
#pragma unroll
                        for (int k = 0; k < K; k++) {
                            if (u == 0)
                                pair_interact2_log(a.x, a.y, b.x, b.y, nx[k], ny[k], nz[k], eps2p,
                                                   m15, ax[k], ay[k], az[k]);
                            else
                                pair_interact2(a.x, a.y, b.x, b.y, nx[k], ny[k], nz[k], eps2p,
                                               ax[k], ay[k], az[k]);
                        }
                    }
                }
            } else {
#pragma unroll UNROLL
                for (int q = q0; q < q0 + fpairs; q++) {
                    const ulonglong2 a = tp[2 * q];
                    const ulonglong2 b = tp[2 * q + 1];
#pragma unroll
                    for (int k = 0; k < K; k++)
                        pair_interact2(a.x, a.y, b.x, b.y, nx[k], ny[k], nz[k], eps2p, ax[k],
                                       ay[k], az[k]);
                }
            }
#pragma unroll
            for (int k = 0; k < K; k++) {
                float l, h;
                f2_unpack(ax[k], l, h);
                comp_add(hx[k], lx[k], l + h);
                f2_unpack(ay[k], l, h);
                comp_add(hy[k], ly[k], l + h);
                f2_unpack(az[k], l, h);
                comp_add(hz[k], lz[k], l + h);
            }
        }
        __syncwarp();
        if (lane == 0) {
            const unsigned round = g / kStages + 1u;
            const unsigned prev = atom_add_acqrel_shared(&released[s], 1u);
            if (prev == round * kWarps - 1u && t + kStages < nt) {
                fence_proxy_async_shared();
                mbar_expect_tx(&full[s], tile_bytes);
                bulk_g2s(ring + (size_t)s * kMaxJT, js + (size_t)(t_begin + t + kStages) * jt,
                         tile_bytes, &full[s]);
                stage_tile[s] = (int)(g + kStages);
            }
        }
    }
    if (__syncthreads_or(failed))
        return false;

    float4 *out = P.acc + d.body_off;
    if (d.nsplit == 1) {
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int i = ib * BI + k * kThreads + tid;
            if (i < d.n)
                out[i] = make_float4(hx[k] + lx[k], hy[k] + ly[k], hz[k] + lz[k], 0.f);
        }
        return true;
    }
    float4 *hi = P.part + d.part_off;
    float4 *lo = hi + (size_t)d.nsplit * d.ni_pad;
#pragma unroll
    for (int k = 0; k < K; k++) {
        const size_t o = (size_t)r * d.ni_pad + (size_t)(ib * BI + k * kThreads + tid);
        hi[o] = make_float4(hx[k], hy[k], hz[k], 0.f);
        lo[o] = make_float4(lx[k], ly[k], lz[k], 0.f);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        unsigned *c = P.cnt + d.cnt_off + ib;
        const unsigned prev = atomicAdd(c, 1u);
        *s_last = (prev == (unsigned)(d.nsplit - 1));
        if (*s_last)
            *c = 0u;
    }
    __syncthreads();
    if (!*s_last)
        return true;
    __threadfence();
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int i = ib * BI + k * kThreads + tid;
        if (i >= d.n)
            continue;
        float Hx = 0.f, Hy = 0.f, Hz = 0.f, Lx = 0.f, Ly = 0.f, Lz = 0.f;
        for (int rr = 0; rr < d.nsplit; rr++) {
            float4 h, l;
            if (rr == r) {
                h = make_float4(hx[k], hy[k], hz[k], 0.f);
                l = make_float4(lx[k], ly[k], lz[k], 0.f);
            } else {
                const size_t o = (size_t)rr * d.ni_pad + (size_t)i;
                h = __ldcg(hi + o);
                l = __ldcg(lo + o);
            }
            comp_add(Hx, Lx, h.x);
            comp_add(Hy, Ly, h.y);
            comp_add(Hz, Lz, h.z);
            Lx += l.x;
            Ly += l.y;
            Lz += l.z;
        }
        out[i] = make_float4(Hx + Lx, Hy + Ly, Hz + Lz, 0.f);
    }
    return true;
}

__global__ void __launch_bounds__(kThreads, 2) ens_force_kernel(Params P) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float4 *ring = reinterpret_cast<float4 *>(smem_raw);
    __shared__ __align__(8) uint64_t full[kStages];
    __shared__ unsigned released[kStages];
    __shared__ int stage_tile[kStages];
    __shared__ int abort_flag, s_last, s_item;
    const int tid = threadIdx.x;
    if (tid == 0) {
        for (int s = 0; s < kStages; s++) {
            mbar_init(&full[s], 1);
            released[s] = 0u;
            stage_tile[s] = -1;
        }
        abort_flag = 0;
        fence_mbar_init();
    }
    unsigned tile_base = 0;
    bool ok = true;
    for (;;) {
        __syncthreads();  // previous item fully consumed; ring free
        if (tid == 0)
            s_item = (int)atomicAdd(P.head, 1u);
        __syncthreads();
        const int it = s_item;
        if (it >= P.n_items)
            break;
        const int4 item = P.items[it];
        const Desc d = P.desc[item.x];
        const bool lg = (d.flags & kLogMass) != 0;
#define NBGB_ENS_ITEM(K, U)                                                                \
    (lg ? process_item<K, U, true>(P, d, item.y, item.z, tile_base, ring, full, released,  \
                                   stage_tile, &abort_flag, &s_last)                       \
        : process_item<K, U, false>(P, d, item.y, item.z, tile_base, ring, full, released, \
                                    stage_tile, &abort_flag, &s_last))
        switch (d.variant) {
        case 0:
            ok = NBGB_ENS_ITEM(1, 8);
            break;
        case 1:
            ok = NBGB_ENS_ITEM(2, 4);
            break;
        case 2:
            ok = NBGB_ENS_ITEM(1, 4);
            break;
        default:
            ok = NBGB_ENS_ITEM(2, 8);
            break;
        }
#undef NBGB_ENS_ITEM
        if (!ok)
            break;
        const int t_begin = (int)(((long long)item.z * d.ntiles) / d.nsplit);
        const int t_end = (int)(((long long)(item.z + 1) * d.ntiles) / d.nsplit);
        tile_base += (unsigned)(t_end - t_begin);
    }
    if (!ok && tid == 0)
        for (int s = 0; s < kStages; s++)
            if (stage_tile[s] >= 0)
                (void)mbar_wait_bounded(&full[s], (uint32_t)((stage_tile[s] / kStages) & 1),
                                        100000000ull);
}

// Thread q owns j-stream pair slot q (bodies 2p, 2p+1 of system slot_sys[q]).
// mode 0: kick half + drift for moving systems, then write posMass and the
// j-stream of every active system; mode 1: kick half only.  pass > 0: only
// moving systems with sub > pass take part.
__global__ void ens_kdk_kernel(const Desc *__restrict__ desc, const int *__restrict__ slot_sys,
                               int n_slots, double *__restrict__ x64, size_t stride,
                               const float *__restrict__ mass, const float4 *__restrict__ acc,
                               float4 *__restrict__ pm, float4 *__restrict__ js, int mode,
                               int pass) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_slots)
        return;
    const int sys = slot_sys[q];
    if (sys < 0)
        return;
    const Desc d = desc[sys];
    if (!(d.flags & kInForce))
        return;
    if (pass > 0 && (!(d.flags & kMove) || d.sub <= pass))
        return;
    const bool move = (d.flags & kMove) != 0;
    const int lp = q - d.js_off / 2;
    float4 out[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int b = 2 * lp + h;
        if (b < d.n) {
            const size_t i = (size_t)d.body_off + b;
            double x = x64[i], y = x64[stride + i], z = x64[2 * stride + i];
            if (move) {
                const float4 a = acc[i];
                const double kdt = 0.5 * d.dt;
                // conversions on the integer pipe: GB300's FP64 pipe is narrow
                double u = fma(widen_f32(a.x), kdt, x64[3 * stride + i]);
                double v = fma(widen_f32(a.y), kdt, x64[4 * stride + i]);
                double w = fma(widen_f32(a.z), kdt, x64[5 * stride + i]);
                x64[3 * stride + i] = u;
                x64[4 * stride + i] = v;
                x64[5 * stride + i] = w;
                if (mode == 0) {
                    x = fma(u, d.dt, x);
                    y = fma(v, d.dt, y);
                    z = fma(w, d.dt, z);
                    x64[i] = x;
                    x64[stride + i] = y;
                    x64[2 * stride + i] = z;
                }
            }
            out[h] = make_float4(narrow_f64(x), narrow_f64(y), narrow_f64(z), mass[i]);
            if (mode == 0)
                pm[i] = out[h];
        } else {
            out[h] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    if (mode == 0) {
        if ((d.flags & kLogMass) && (lp & 3) == 0) {  // log-domain pair (padding: -inf)
            out[0].w = jstream_log_mass(out[0].w);
            out[1].w = jstream_log_mass(out[1].w);
        }
        js[2 * q] = make_float4(out[0].x, out[1].x, out[0].y, out[1].y);
        js[2 * q + 1] = make_float4(out[0].z, out[1].z, out[0].w, out[1].w);
    }
}

// ---------------------------------------------------------------------------
// Pair systems
// ---------------------------------------------------------------------------
typedef pair::Narrow Narrow;
typedef pair::Wide Wide;
constexpr int kPairCtaThreads = Narrow::kThreads;
static_assert(Wide::kThreads == Narrow::kThreads && Wide::kSet == Narrow::kSet,
              "one persistent kernel for both geometries");
constexpr size_t kPairSmem = Wide::kSmem > Narrow::kSmem ? Wide::kSmem : Narrow::kSmem;
constexpr int kBodyBlock = 64;  // bodies of one entry of the block map, two a reduction thread

struct PairParams {
    const Desc *desc;
    const int4 *items;  // {system, row, chunk, 0} or {-1, first task, warps a task, 0}
    const int2 *tasks;  // {system, tile}, 4 / warps to an item ({-1, 0}: none)
    int n_items, pass;
    unsigned *head;                  // zeroed by ens_drift
    const float4 *pm;
    float *scratch;
    float4 *acc;
    double *x64;
    size_t stride;
};

// Entry e of the block map: bodies kBodyBlock blk and on of one pair system.
__device__ __forceinline__ bool takes_part(const Desc &d, int pass) {
    return (d.flags & kInForce) && (pass == 0 || ((d.flags & kMove) && d.sub > pass));
}

// Bodies 128 tile .. 128 tile + 127 of a small system by one warp, or by two or
// four of a CTA that share its sets out: forces from
// all its sources, acceleration and closing half kick.  smem: the CTA's shared
// memory.  A system of up to kTaskBelow - 1 bodies is too
// small for rows: most of a row's targets would be padding and its items
// short (1,024 systems a tick, GB300, against rows and the one-sided queue:
// see kTaskBelow).  The sets' sums are added in set order either way, so the
// result does not depend on which it is.
constexpr int kTaskBodies = 32 * Narrow::KI;
constexpr int kTaskSets = 8;  // of a system, at most
static_assert((4 * Narrow::kSource + 2 * kTaskSets * 3 * kTaskBodies) * 4 <= kPairSmem,
              "sources of four warps and the sums of two tasks");

template <int WARPS>
__device__ __forceinline__ void warp_task(const PairParams &P, const Desc &d, int tile,
                                          float *smem) {
    constexpr int KI = Narrow::KI, kSet = Narrow::kSet;
    static_assert(kSet == kTaskBodies, "a lane stages as many sources as it has targets");
    static_assert(KI % WARPS == 0, "a warp finishes 32 KI / WARPS bodies");
    const int lane = threadIdx.x & 31, share = (threadIdx.x >> 5) % WARPS;
    float *buf = smem + (threadIdx.x >> 5) * Narrow::kSource;
    // WARPS > 1: the task's sums, [set][3][KI][32]
    float *part = smem + 4 * Narrow::kSource +
                  (threadIdx.x >> 5) / WARPS * (kTaskSets * 3 * KI * 32);
    const int each = (d.nsets + WARPS - 1) / WARPS;
    const int set0 = share * each, set1 = min(set0 + each, d.nsets);
    const float4 *pm = P.pm + d.body_off;
    const f2 eps2p = f2_pack(d.eps2, d.eps2), zero2 = f2_pack(0.f, 0.f);
    f2 nx[KI], ny[KI], nz[KI], nm[KI], ax[KI], ay[KI], az[KI];
    float hi[3][KI], lo[3][KI];
    float4 next[KI];
#pragma unroll
    for (int k = 0; k < KI; k++) {
        const int i = tile * kTaskBodies + lane + 32 * k, j = set0 * kSet + lane + 32 * k;
        const float4 v = i < d.n ? pm[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        next[k] = j < d.n ? pm[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        nx[k] = f2_pack(-v.x, -v.x);
        ny[k] = f2_pack(-v.y, -v.y);
        nz[k] = f2_pack(-v.z, -v.z);
        nm[k] = zero2;
        ax[k] = ay[k] = az[k] = zero2;
#pragma unroll
        for (int c = 0; c < 3; c++)
            hi[c][k] = lo[c][k] = 0.f;
    }
    for (int set = set0; set < set1; set++) {
        __syncwarp();
#pragma unroll
        for (int k = 0; k < KI; k++) {
            pair::store_source<Narrow>(buf, lane + 32 * k, next[k]);
            const int j = (set + 1) * kSet + lane + 32 * k;
            next[k] = j < d.n ? pm[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncwarp();
        pair::meet<Narrow, pair::kOneSided>(reinterpret_cast<const ulonglong2 *>(buf) + lane, 0,
                                            32, nx, ny, nz, nm, ax, ay, az, eps2p, lane, nullptr,
                                            1.f);
#pragma unroll
        for (int k = 0; k < KI; k++) {
            const f2 a[3] = {ax[k], ay[k], az[k]};
#pragma unroll
            for (int c = 0; c < 3; c++) {
                float l, h;
                f2_unpack(a[c], l, h);
                if (WARPS > 1)
                    part[((set * 3 + c) * KI + k) * 32 + lane] = l + h;
                else
                    comp_add(hi[c][k], lo[c][k], l + h);
            }
            ax[k] = ay[k] = az[k] = zero2;
        }
    }
    constexpr int kMine = KI / WARPS;  // body groups this warp finishes
    if (WARPS > 1) {
        if (WARPS == 4 || threadIdx.x < 32 * WARPS)  // the task's warps only
            asm volatile("bar.sync 1, %0;" ::"n"(32 * WARPS) : "memory");
        else
            asm volatile("bar.sync 2, %0;" ::"n"(32 * WARPS) : "memory");
        for (int set = 0; set < d.nsets; set++)
#pragma unroll
            for (int k = 0; k < kMine; k++)
#pragma unroll
                for (int c = 0; c < 3; c++)
                    comp_add(hi[c][k], lo[c][k],
                             part[((set * 3 + c) * KI + share * kMine + k) * 32 + lane]);
    }
    const double kdt = 0.5 * d.dt;
#pragma unroll
    for (int k = 0; k < kMine; k++) {
        const int b = tile * kTaskBodies + lane + 32 * (share * kMine + k);
        if (b >= d.n)
            continue;
        const size_t i = (size_t)d.body_off + b;
        const float a[3] = {round_force(hi[0][k], lo[0][k]), round_force(hi[1][k], lo[1][k]),
                            round_force(hi[2][k], lo[2][k])};
        P.acc[i] = make_float4(a[0], a[1], a[2], 0.f);
        if (d.flags & kMove)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                double *v = P.x64 + (3 + c) * P.stride + i;
                *v = fma(widen_f32(a[c]), kdt, *v);
            }
    }
}

// Target piece of a row's first item: every row has at most one item more than
// its meetings / ch, so the places of two rows never overlap.
template <class G>
__device__ __forceinline__ long long row_piece(int row, int nsets, int ch) {
    return pair::meetings_before<G>(row, nsets) / ch + row;
}

// One item, in shared memory (row_stretch asks for its parts).
struct Item {
    const float4 *pm_;
    float *react_, *tsum_;
    int n_, row, set, nset, kind;
    // kind: the system's Desc::pair, or 3: tasks from `row` on, `set` warps each
    float eps2_;
    int pieces;  // (last: where it stood before eps2_ the wide rows took 2 % longer)
    __device__ __forceinline__ const float4 *pm() const { return pm_; }
    __device__ __forceinline__ int n() const { return n_; }
    __device__ __forceinline__ float eps2() const { return eps2_; }
    __device__ __forceinline__ int short_ok() const { return pair::eps2_short_ok(eps2_); }
    __device__ __forceinline__ unsigned *status() const { return nullptr; }
    __device__ __forceinline__ float *react(unsigned s) const {
        return react_ + (size_t)(s >> 5) * (3 * Narrow::kSet);
    }
    __device__ __forceinline__ float *tsum() const { return tsum_; }
    __device__ __forceinline__ bool remainder() const { return pieces > 1; }
};

template <class G>
__device__ __forceinline__ void set_item(Item &t, const PairParams &P, const Desc &d, int row,
                                         int chunk) {
    const int set = row * G::kRowSets + chunk * d.ch;
    const long long g = pair::meetings_before<G>(row, d.nsets) + chunk * d.ch;
    t.pm_ = P.pm + d.body_off;
    t.react_ = P.scratch + d.react_off + g * (3 * G::kSet);
    t.tsum_ = P.scratch + d.tsum_off +
              (row_piece<G>(row, d.nsets, d.ch) + chunk) * (d.target_pieces * 3 * G::kRow);
    t.pieces = d.target_pieces;
    t.n_ = d.n;
    t.row = row;
    t.set = set;
    t.nset = min(d.ch, d.nsets - set);
    t.kind = d.pair;
    t.eps2_ = d.eps2;
}

__global__ void __launch_bounds__(kPairCtaThreads, 2) ens_pair_kernel(PairParams P) {
    extern __shared__ __align__(128) float smem_f[];
    __shared__ Item item;
    __shared__ int s_next[2];
    grid_dependents_launch();
    grid_dependency_wait();
    for (int it = blockIdx.x, k = 0; it < P.n_items; it = s_next[k], k ^= 1) {
        if (threadIdx.x == 0) {
            const int next = (int)(atomicAdd(P.head, 1u) + gridDim.x);
            const int4 v = P.items[it];
            if (v.x < 0) {
                item.kind = 3;
                item.row = v.y;
                item.set = v.z;
            } else if (P.desc[v.x].pair == 1) {
                set_item<Narrow>(item, P, P.desc[v.x], v.y, v.z);
            } else {
                set_item<Wide>(item, P, P.desc[v.x], v.y, v.z);
            }
            s_next[k] = next;
        }
        __syncthreads();
        if (item.kind == 3) {
            const int warps = item.set;
            const int2 t = P.tasks[item.row + (int)(threadIdx.x >> 5) / warps];
            if (t.x >= 0 && takes_part(P.desc[t.x], P.pass)) {
                if (warps == 1)
                    warp_task<1>(P, P.desc[t.x], t.y, smem_f);
                else if (warps == 2)
                    warp_task<2>(P, P.desc[t.x], t.y, smem_f);
                else
                    warp_task<4>(P, P.desc[t.x], t.y, smem_f);
            }
            __syncthreads();
        } else if (item.kind == 1) {
            pair::row_stretch<Narrow, true>(item, smem_f, item.row, item.set, 0u,
                                            32u * (unsigned)item.nset);
        } else {
            pair::row_stretch<Wide, false>(item, smem_f, item.row, item.set, 0u,
                                           32u * (unsigned)item.nset);
        }
    }
}

// Opening half kick and drift of moving systems, FP32 positions of all;
// zeroes the item queues.
__global__ void __launch_bounds__(256)
    ens_drift_kernel(const Desc *desc, const int2 *blocks, int n_blocks,
                     double *__restrict__ x64, size_t stride, const float *mass,
                     const float4 *acc, float4 *__restrict__ pm,
                     unsigned *__restrict__ heads, int n_heads, int pass) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    grid_dependents_launch();
    grid_dependency_wait();
    if (q < n_heads)
        heads[q] = 0u;
    const int e = q / kBodyBlock;
    if (e >= n_blocks)
        return;
    const int2 blk = blocks[e];
    const Desc &d = desc[blk.x];
    const int b = blk.y * kBodyBlock + q % kBodyBlock;
    if (!takes_part(d, pass) || b >= d.n)
        return;
    const size_t i = (size_t)d.body_off + b;
    double x = x64[i], y = x64[stride + i], z = x64[2 * stride + i];
    const float m = mass[i];
    if (d.flags & kMove) {
        double u = x64[3 * stride + i], v = x64[4 * stride + i], w = x64[5 * stride + i];
        const float4 a = acc[i];
        const double dt = d.dt, kdt = 0.5 * dt;
        u = fma(widen_f32(a.x), kdt, u);
        v = fma(widen_f32(a.y), kdt, v);
        w = fma(widen_f32(a.z), kdt, w);
        x = fma(u, dt, x);
        y = fma(v, dt, y);
        z = fma(w, dt, z);
        x64[i] = x;
        x64[stride + i] = y;
        x64[2 * stride + i] = z;
        x64[3 * stride + i] = u;
        x64[4 * stride + i] = v;
        x64[5 * stride + i] = w;
    }
    pm[i] = make_float4(narrow_f64(x), narrow_f64(y), narrow_f64(z), m);
}

// One block per entry: kReduceGroups x 3 (components) threads for two bodies
// add their reaction pieces (rows before their own, in row order) and their
// row's target pieces, eight loads in flight; then the acceleration and the
// closing half kick, whose velocities are loaded beside the pieces.  Bound by
// the latency of one block (the entry, its system, the pieces), times the
// blocks that follow one another on an SM: with one body and four groups a
// thread, 3.9 thousand blocks for 64 systems of 64 to 7,205 bodies and 172 us
// a tick; with two bodies 169, and two groups 165; 8 systems of 8,701 to
// 58,144: 3,089 -> 3,051 us.
constexpr int kReduceGroups = 2;
constexpr int kReduceThreads = 3 * 32 * kReduceGroups;

template <class G>
__device__ __forceinline__ void reduce_entry(const Desc &d, int blk, const float *scratch,
                                             double *x64, size_t stride, float4 *acc) {
    constexpr int kB = kBodyBlock, kSet = G::kSet;
    __shared__ __align__(8) float part[kReduceGroups - 1][2][3][kB], out[3][kB];
    static_assert(kB == 64, "two bodies a lane");
    const int tid = threadIdx.x, group = tid / (3 * 32), comp = (tid / 32) % 3, j = 2 * (tid & 31);
    const int i = blk * kB + j, set = blk * kB / kSet, b = set / G::kRowSets;
    const int nt = (d.nsets - b * G::kRowSets + d.ch - 1) / d.ch * d.target_pieces;
    const int total = b + nt;
    const int q0 = total * group / kReduceGroups, q1 = total * (group + 1) / kReduceGroups;
    const float *react = scratch + d.react_off + (size_t)comp * kSet + (i - set * kSet);
    const float *tsum = scratch + d.tsum_off + (size_t)comp * G::kRow + (i - b * G::kRow) +
                        row_piece<G>(b, d.nsets, d.ch) * (d.target_pieces * 3 * G::kRow);
    auto piece = [&](int q) {
        return q < b ? react + (pair::meetings_before<G>(q, d.nsets) + set - q * G::kRowSets) *
                                   (3 * kSet)
                     : tsum + (long long)(q - b) * (3 * G::kRow);
    };
    // the group that kicks has its velocities in flight beside the pieces
    const bool kick = group == 0 && (d.flags & kMove);
    double *vel = x64 + (3 + comp) * stride + d.body_off + i;
    const double v0 = kick && i < d.n ? vel[0] : 0.0, v1 = kick && i + 1 < d.n ? vel[1] : 0.0;
    float2 hi = make_float2(0.f, 0.f), lo = hi;
    for (int q = q0; q < q1; q += 8) {
        float2 v[8];
#pragma unroll
        for (int u = 0; u < 8; u++)
            v[u] = q + u < q1 ? __ldcs((const float2 *)piece(q + u)) : make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 8; u++) {
            comp_add(hi.x, lo.x, v[u].x);
            comp_add(hi.y, lo.y, v[u].y);
        }
    }
    if (group) {
        *(float2 *)&part[group - 1][0][comp][j] = hi;
        *(float2 *)&part[group - 1][1][comp][j] = lo;
    }
    __syncthreads();
    if (group == 0) {
#pragma unroll
        for (int q = 0; q < kReduceGroups - 1; q++) {
            const float2 h = *(const float2 *)&part[q][0][comp][j];
            const float2 l = *(const float2 *)&part[q][1][comp][j];
            comp_add(hi.x, lo.x, h.x);
            lo.x += l.x;
            comp_add(hi.y, lo.y, h.y);
            lo.y += l.y;
        }
        const float2 a = make_float2(round_force(hi.x, lo.x), round_force(hi.y, lo.y));
        *(float2 *)&out[comp][j] = a;
        if (kick && i < d.n)
            vel[0] = fma(widen_f32(a.x), 0.5 * d.dt, v0);
        if (kick && i + 1 < d.n)
            vel[1] = fma(widen_f32(a.y), 0.5 * d.dt, v1);
    }
    __syncthreads();
    const int ib = blk * kB + tid;
    if (tid < kB && ib < d.n)
        acc[(size_t)d.body_off + ib] = make_float4(out[0][tid], out[1][tid], out[2][tid], 0.f);
}

__global__ void __launch_bounds__(kReduceThreads)
    ens_reduce_kernel(const Desc *desc, const int2 *blocks, const float *scratch, double *__restrict__ x64, size_t stride,
                      float4 *__restrict__ acc, int pass) {
    grid_dependents_launch();
    grid_dependency_wait();
    const int2 blk = blocks[blockIdx.x];
    const Desc &d = desc[blk.x];
    if (!takes_part(d, pass))
        return;
    if (d.pair == 1)
        reduce_entry<Narrow>(d, blk.y, scratch, x64, stride, acc);
    else
        reduce_entry<Wide>(d, blk.y, scratch, x64, stride, acc);
}

static NBGB_STATUS_READER(read_status_ens)

}  // namespace ens

int read_status_ensemble(unsigned *bits) { return ens::read_status_ens(bits); }
const unsigned *status_address_ensemble() { return status_address(); }

}  // namespace nbgb

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
using nbgb::ens::Desc;

namespace {

// First-fit allocator over [0, capacity) in abstract units.
struct RangeAlloc {
    struct R {
        size_t off, len;
    };
    size_t capacity = 0;
    std::vector<R> free_list;
    void init(size_t cap) {
        capacity = cap;
        free_list.assign(1, R{0, cap});
    }
    bool alloc(size_t len, size_t align, size_t &off) {
        if (len == 0) {
            off = 0;
            return true;
        }
        for (size_t k = 0; k < free_list.size(); k++) {
            R &f = free_list[k];
            const size_t a = (f.off + align - 1) / align * align;
            if (a + len <= f.off + f.len) {
                const size_t tail = f.off + f.len - (a + len);
                const size_t head = a - f.off;
                off = a;
                if (head && tail) {
                    f.len = head;
                    free_list.insert(free_list.begin() + k + 1, R{a + len, tail});
                } else if (head) {
                    f.len = head;
                } else if (tail) {
                    f.off = a + len;
                    f.len = tail;
                } else {
                    free_list.erase(free_list.begin() + k);
                }
                return true;
            }
        }
        return false;
    }
    void release(size_t off, size_t len) {
        if (len == 0)
            return;
        R r{off, len};
        auto it = std::lower_bound(free_list.begin(), free_list.end(), r,
                                   [](const R &a, const R &b) { return a.off < b.off; });
        it = free_list.insert(it, r);
        // merge with neighbours
        if (it + 1 != free_list.end() && it->off + it->len == (it + 1)->off) {
            it->len += (it + 1)->len;
            free_list.erase(it + 1);
        }
        if (it != free_list.begin() && (it - 1)->off + (it - 1)->len == it->off) {
            (it - 1)->len += it->len;
            free_list.erase(it);
        }
    }
};

struct HostSys {
    bool used = false;
    int n = 0;
    size_t body_off = 0, js_off = 0, part_off = 0, cnt_off = 0;
    size_t body_len = 0, js_len = 0, part_len = 0, cnt_len = 0;
    int variant = 1, jt = 256, nsplit = 1, nblocks = 0, ntiles = 0, ni_pad = 0;
    double dt = 0.0;
    long long steps_left = 0;
    bool started = false;  // has initial accelerations
    long long steps_done = 0;
    bool log_mass = false;  // every mass >= 0: log-domain pairs (kLogMass)
    int sub = 1;            // steps per tick (1..kMaxSub)
    bool n3 = false;        // Newton-3 system
    bool sym = false;       // Newton-3 system too large for pair items
    int pair = 0;           // pair system: 1 narrow rows, 2 wide rows, 3 warp tasks
    int nsets = 0, ch = 0, rows = 0, target_pieces = 1;
    size_t react_len = 0, scratch_len = 0;  // floats
    size_t scratch_off = 0;                 // within its group's scratch
    size_t acc_off = 0, acc_len = 0;  // its FP64 sums ([3][npad] doubles)
};

// Steps a system takes in the coming tick (0 before its initial forces).
inline int sub_eff(const HostSys &h) {
    if (!h.started || h.n3)
        return 1;  // the initial-force pass; Newton-3 systems run in pass 0 only
    return (int)std::min<long long>(h.sub, h.steps_left);
}

// Items of a pair system are whole source sets of one row: few enough that an
// item's start-up (2-3 us) is small beside its steps (11 us a set with narrow
// rows, 30 us with wide ones), many enough that one system alone fills the
// GPU.  Up to two sets the targets' sums need no remainders: with four below
// 2,048 bodies 200 systems of 1,100 take 142 us a tick instead of 131, 249 of
// 1,497 256 instead of 244, one system 39 instead of 25.  Depends on n only, as does the geometry: rows of 512 targets below
// 8,192 bodies (more, smaller items, less padding), 1,024 above.
int sets_per_item(size_t n) {
    if (n < 8192)
        return 2;
    int ch = 1;
    for (size_t m = 16384; m <= n && ch < 32; m *= 2)
        ch *= 2;
    return ch;
}

template <class G>
void pair_shape(size_t n, int ch, HostSys &h) {
    h.nsets = (int)((n + G::kSet - 1) / G::kSet);
    h.rows = (int)((n + G::kRow - 1) / G::kRow);
    h.ch = ch;
    const size_t meetings = (size_t)nbgb::pair::meetings_before<G>(h.rows, h.nsets);
    h.react_len = meetings * 3 * G::kSet;
    // up to 256 sources are one float here as in the one-sided queue
    h.target_pieces = h.ch * G::kSet > 256 ? 2 : 1;
    h.scratch_len = h.react_len +
                    (meetings / h.ch + h.rows) * h.target_pieces * 3 * G::kRow;  // row_piece
}

// Sizes evaluated by warp tasks.  Microseconds a tick of 1,024 systems (one
// system), tasks / rows / the one-sided queue's tuned plan: N = 91 29 / 52 /
// 46 (17 / 19 / 21), 362 104 / 166 / 124 (26 / 19 / 32), 724 304 / 403 / 309
// (38 / 20 / 43), 1,100 635 / 595 / 1,003 (49 / 39 / 106), 1,280 746 / 694 /
// 1,010 (53 / 40 / 106), and of 953 systems of 1,448 1,011 / 882 / 925.
constexpr size_t kTaskBelow = 1024;

// Warp tasks (longest first) that take a warp each, out of `tasks` with `warps`
// resident; the others share their sets out among several warps (task_warps),
// for between a tenth of the GPU's CTA slots and a few rounds it is the last
// tasks that decide: one warp alone takes 47 us for the eight sets of 1,000
// bodies, 77 beside another CTA's.  Where the sets divide evenly (four and eight
// by four warps, six by two) sharing costs nothing: all but whole rounds less
// one.  Where they do not, idle warps cost more than a nearly full round does:
// all but whole rounds, and not the rest either from three quarters of a round
// on.  `sets`: of the longest task after whole rounds.  Microseconds a tick, a
// warp a task / as here / the one-sided queue's tuned plan: 32 systems of 1,000
// bodies 76 / 26 / 50, 128 79 / 71 / 83, 512 264 / 240 / 253, 1,024 472 / 466 /
// 488; of 800 160 71 / 73 / 100, 200 128 / 91 / 116, 1,024 362 / 369 / 464; of
// 700 64 61 / 37 / 44, 128 63 / 55 / 56, 256 114 / 85 / 93; of 512 64 45 / 18 /
// 37, 384 84 / 63 / 72; of 300 24 26 / 14 / 42, 384 41 / 41 / 56.
size_t alone_tasks(size_t tasks, size_t warps, int sets) {
    const size_t full = tasks / warps * warps;
    if (sets % 4 == 0 || sets == 6)
        return full > 0 ? full - warps : 0;
    return 4 * (tasks - full) > 3 * warps ? tasks : full;
}
// Two warps where four would wait for the one with two sets of five or six,
// unless what is left after whole rounds of them are few enough tasks for a CTA
// each.
size_t late_tasks(size_t tasks, size_t ctas) {
    const size_t rest = tasks % (2 * ctas);
    return rest <= ctas ? rest : 0;
}
int task_warps(int nsets, bool late) {
    if (nsets <= 2)
        return 1;
    return !late && (nsets == 5 || nsets == 6) ? 2 : 4;
}

// The pair plan of n bodies if its scratch is at most max_floats.  Where it
// would be more, items of up to kMaxItemSets sets: the places for the
// targets' sums are one to every item, and those for the reactions, 6 N^2 /
// 1,024 bytes, then set the limit.  (With 32 sets at most, systems of 250,000
// bodies did not fit and those of 265,000 did.)
constexpr int kMaxItemSets = 128;
void pair_shape(size_t n, int ch, HostSys &h) {
    if (n < 8192)
        pair_shape<nbgb::ens::Narrow>(n, ch, h);
    else
        pair_shape<nbgb::ens::Wide>(n, ch, h);
}
bool pair_plan(size_t n, size_t max_floats, HostSys &h) {
    HostSys t;
    if (n < kTaskBelow) {
        h.pair = 3;
        h.nsets = (int)((n + nbgb::ens::Narrow::kSet - 1) / nbgb::ens::Narrow::kSet);
        return true;
    }
    int ch = sets_per_item(n);
    pair_shape(n, ch, t);
    while (t.scratch_len > max_floats && ch < kMaxItemSets)
        pair_shape(n, ch *= 2, t);
    if (t.scratch_len > max_floats)
        return false;
    h.pair = n < 8192 ? 1 : 2;
    h.nsets = t.nsets;
    h.rows = t.rows;
    h.ch = t.ch;
    h.target_pieces = t.target_pieces;
    h.react_len = t.react_len;
    h.scratch_len = t.scratch_len;
    return true;
}

// Scratch arena (floats): what the largest pair system of max_bodies needs with
// sets_per_item's items, at most `limit` (larger items fit into it).  Systems
// that need more than the limit are not pair
// systems: a rule on n alone.
constexpr size_t kPairScratch = ((size_t)512 << 20) / 4;     // to 283,008 bodies
constexpr size_t kPairScratchN3 = ((size_t)1 << 30) / 4;     // Newton-3: to 401,152
size_t scratch_for(size_t max_bodies, size_t limit) {
    size_t most = 0;
    for (size_t n : {(size_t)8191, (size_t)16383, (size_t)32767, (size_t)65535,
                     (size_t)131071, (size_t)262143, max_bodies}) {
        HostSys h;
        n = std::min(n, max_bodies);
        if (n >= kTaskBelow) {
            pair_shape(n, sets_per_item(n), h);
            most = std::max(most, h.scratch_len);
        }
    }
    return std::min(most, limit);
}

// Pair systems evaluated together: their items and body blocks, and the
// first item of each pass (items sorted by sub).
struct PairGroup {
    int first = 0, n = 0;
    int block0 = 0, nblocks = 0;
    int pass_first[nbgb::ens::kMaxSub];
};

// Per-N-bucket plan: bucket b covers N in [2^b, 2^(b+1)).
struct BucketPlan {
    int variant = -1, jt = 0, nsplit = 0;  // -1: default rule
};

}  // namespace

struct nbgb_ensemble {
    int device = 0;
    cudaStream_t stream = nullptr;
    float eps2 = 1e-4f;
    int max_systems = 0;
    size_t max_bodies = 0, js_cap = 0, part_cap = 0, cnt_cap = 0;
    // device arena
    double *x64 = nullptr;  // 6 * max_bodies
    float *mass = nullptr;
    float4 *pm = nullptr, *acc = nullptr, *js = nullptr, *part = nullptr;
    unsigned *cnt = nullptr, *head = nullptr;
    Desc *d_desc = nullptr;
    int4 *d_items = nullptr;
    int *d_slot_sys = nullptr;
    size_t items_cap = 0;
    // pinned host mirrors for uploads
    Desc *h_desc = nullptr;
    int4 *h_items = nullptr;
    int *h_slot_sys = nullptr;
    // host bookkeeping
    std::vector<HostSys> sys;
    RangeAlloc a_body, a_js, a_part, a_cnt;
    BucketPlan bucket[32];
    int n_items = 0, n_slots = 0;
    int n_pass = 1;                       // passes per tick (max effective sub)
    // Newton-3 systems
    size_t n3_min = 0;                    // 0: off
    double *acc64 = nullptr;              // FP64 sums arena (allocated when enabled)
    size_t acc64_cap = 0;
    RangeAlloc a_acc;
    nbgb::SymSystem *d_sym = nullptr, *h_sym = nullptr;
    int n_sym = 0;
    // pair systems
    float *scratch = nullptr;             // partial sums of one group
    size_t scratch_cap = 0, scratch_limit = kPairScratch;  // floats
    char *d_lists = nullptr, *h_lists = nullptr;  // items, tasks, blocks
    int4 *d_pitems = nullptr, *h_pitems = nullptr;
    size_t pitems_cap = 0;
    int2 *d_blocks = nullptr, *h_blocks = nullptr;
    size_t blocks_cap = 0;
    unsigned *heads = nullptr;            // one queue per group
    int2 *d_tasks = nullptr, *h_tasks = nullptr;
    size_t tasks_cap = 0;
    int n_blocks = 0, n_tasks = 0;
    std::vector<PairGroup> groups;
    int pass_first[nbgb::ens::kMaxSub];   // first item of pass p (items sorted by sub)
    bool dirty = true;
    cudaGraphExec_t graph = nullptr;
    bool use_graph = true;
    int stable_ticks = 0;  // ticks since the membership last changed
    int grid = 0;      // CTAs of the persistent force launch
    int grid_max = 0;  // SMs x resident CTAs per SM
    size_t bytes_total = 0;
    long long ticks = 0;
    nbgb::Snapshot snap;
};

namespace {

int bucket_of(int n) {
    int b = 0;
    while ((2 << b) <= n && b < 31)
        b++;
    return b;
}

// Default per-bucket rule: pair systems (pair_plan); the ones too large for
// its scratch 2 targets per thread and 512-body tiles.
void choose_plan(nbgb_ensemble *e, int n, HostSys &h) {
    const BucketPlan &bp = e->bucket[bucket_of(n)];
    int variant = bp.variant, jt = bp.jt, nsplit = bp.nsplit;
    if (variant < 0) {
        variant = 1;
        jt = 512;
        nsplit = 1;
    }
    const int bi = nbgb::ens::kThreads * ((variant == 0 || variant == 2) ? 1 : 2);
    h.variant = variant;
    h.jt = jt;
    h.nblocks = (n + bi - 1) / bi;
    h.ntiles = (n + jt - 1) / jt;
    h.nsplit = std::max(1, std::min(std::min(nsplit, 4), h.ntiles));
    h.ni_pad = h.nblocks * bi;
}

void fill_desc(nbgb_ensemble *e, int slot, Desc &d) {
    const HostSys &h = e->sys[slot];
    d.n = h.n;
    d.body_off = (int)h.body_off;
    d.js_off = (int)h.js_off;
    d.ntiles = h.ntiles;
    d.jt = h.jt;
    d.variant = h.variant;
    d.nsplit = h.nsplit;
    d.nblocks = h.nblocks;
    d.part_off = (long long)h.part_off;
    d.cnt_off = (int)h.cnt_off;
    d.ni_pad = h.ni_pad;
    d.flags = h.used ? (nbgb::ens::kInForce | (h.started && h.steps_left > 0 ? nbgb::ens::kMove : 0) |
                        (h.log_mass ? nbgb::ens::kLogMass : 0))
                     : 0;
    d.sub = h.used ? sub_eff(h) : 1;
    d.eps2 = e->eps2;
    d.dt = h.dt;
    d.pair = h.pair;
    d.nsets = h.nsets;
    d.ch = h.ch;
    d.target_pieces = h.target_pieces;
    d.react_off = (long long)h.scratch_off;
    d.tsum_off = (long long)(h.scratch_off + h.react_len);
}

// Groups, items and body blocks of this tick's pair systems (before the
// descriptors are filled: scratch places are set here).
int rebuild_pairs(nbgb_ensemble *e) {
    struct It {
        int4 v;
        int cost, sub;
    };
    std::vector<It> items;
    size_t used = 0, n_items = 0;
    e->n_blocks = 0;
    e->groups.clear();
    auto close_group = [&]() -> int {
        PairGroup &g = e->groups.back();
        std::stable_sort(items.begin(), items.end(), [](const It &a, const It &b) {
            return a.sub != b.sub ? a.sub < b.sub : a.cost > b.cost;
        });
        if (n_items + items.size() > e->pitems_cap)
            return NBGB_ERR_NO_MEMORY;
        g.first = (int)n_items;
        g.n = (int)items.size();
        g.nblocks = e->n_blocks - g.block0;
        for (const It &it : items)
            e->h_pitems[n_items++] = it.v;
        int k = 0;
        for (int p = 0; p < nbgb::ens::kMaxSub; p++) {
            while (p > 0 && k < g.n && items[k].sub <= p)
                k++;
            g.pass_first[p] = k;
        }
        for (const It &it : items)
            e->n_pass = std::max(e->n_pass, it.sub);
        items.clear();
        used = 0;
        return NBGB_OK;
    };
    auto add_blocks = [&](int s) {
        const int nblk = (e->sys[s].n + nbgb::ens::kBodyBlock - 1) / nbgb::ens::kBodyBlock;
        if ((size_t)(e->n_blocks + nblk) > e->blocks_cap)
            return false;
        for (int k = 0; k < nblk; k++)
            e->h_blocks[e->n_blocks++] = make_int2(s, k);
        return true;
    };
    // warp tasks, four of one sub and like length to an item, or fewer that
    // have several warps, in the first group; their bodies need no reduction
    std::vector<It> tasks;
    for (int s = 0; s < e->max_systems; s++) {
        const HostSys &h = e->sys[s];
        if (!h.used || h.pair != 3 || !(h.steps_left > 0 || !h.started))
            continue;
        for (int t = 0; t < h.nsets; t++)  // as many tiles as sets
            tasks.push_back(It{make_int4(s, t, 0, 0), h.nsets, sub_eff(h)});
        if (!add_blocks(s))
            return NBGB_ERR_NO_MEMORY;
    }
    std::stable_sort(tasks.begin(), tasks.end(), [](const It &a, const It &b) {
        return a.sub != b.sub ? a.sub < b.sub : a.cost > b.cost;
    });
    e->n_tasks = 0;
    if (!tasks.empty()) {
        e->groups.emplace_back();
        e->groups.back().block0 = e->n_blocks;
    }
    size_t alone_end = 0;
    size_t late = 0;
    for (size_t k = 0; k < tasks.size();) {
        const int sub = tasks[k].sub;
        if (k == 0 || sub != tasks[k - 1].sub) {
            size_t end = k;
            while (end < tasks.size() && tasks[end].sub == sub)
                end++;
            const size_t slots = 4 * (size_t)e->grid;
            const size_t rest = std::min(k + (end - k) / slots * slots, end - 1);
            alone_end = k + alone_tasks(end - k, slots, tasks[rest].cost);
            late = end - late_tasks(end - alone_end, (size_t)e->grid);
        }
        auto warps_of = [&](size_t t) {
            return t < alone_end ? 1 : task_warps(tasks[t].cost, t >= late);
        };
        const int warps = warps_of(k);
        if ((size_t)e->n_tasks + 4 / warps > e->tasks_cap)
            return NBGB_ERR_NO_MEMORY;
        // a one-sided step of four warps costs three quarters of one of a row
        const int sets = (tasks[k].cost + warps - 1) / warps;
        items.push_back(It{make_int4(-1, e->n_tasks, warps, 0),
                           (sets * nbgb::ens::Narrow::KI * 3 + 3) / 4, sub});
        for (int q = 0; q < 4 / warps; q++, e->n_tasks++) {
            const bool have = k < tasks.size() && tasks[k].sub == sub && warps_of(k) == warps;
            e->h_tasks[e->n_tasks] =
                have ? make_int2(tasks[k].v.x, tasks[k].v.y) : make_int2(-1, 0);
            k += have;
        }
    }
    for (int s = 0; s < e->max_systems; s++) {
        HostSys &h = e->sys[s];
        if (!h.used || !h.pair || h.pair == 3 || !(h.steps_left > 0 || !h.started))
            continue;
        if (e->groups.empty() || used + h.scratch_len > e->scratch_cap) {
            if (!e->groups.empty() && close_group() != NBGB_OK)
                return NBGB_ERR_NO_MEMORY;
            e->groups.emplace_back();
            e->groups.back().block0 = e->n_blocks;
        }
        h.scratch_off = used;
        used += (h.scratch_len + 63) / 64 * 64;
        const int row_sets = h.pair == 1 ? nbgb::ens::Narrow::kRowSets : nbgb::ens::Wide::kRowSets;
        const int ki = h.pair == 1 ? nbgb::ens::Narrow::KI : nbgb::ens::Wide::KI;
        for (int row = 0; row < h.rows; row++)
            for (int set = row * row_sets, c = 0; set < h.nsets; set += h.ch, c++)
                items.push_back(It{make_int4(s, row, c, 0),
                                   std::min(h.ch, h.nsets - set) * ki, sub_eff(h)});
        if (!add_blocks(s))
            return NBGB_ERR_NO_MEMORY;
    }
    if (!e->groups.empty() && close_group() != NBGB_OK)
        return NBGB_ERR_NO_MEMORY;
    return NBGB_OK;
}

// Rebuild descriptors, the j-stream slot map and the largest-first item list.
// The pinned staging buffers are re-filled, so uploads (and ticks) still queued
// from an earlier rebuild must have run first: synchronise the stream.
int rebuild(nbgb_ensemble *e) {
    if (cudaStreamSynchronize(e->stream) != cudaSuccess)
        return NBGB_ERR_CUDA;
    struct It {
        int4 v;
        double cost;
        int sub;
    };
    std::vector<It> items;
    e->n_pass = 1;
    const int prc = rebuild_pairs(e);
    if (prc != NBGB_OK)
        return prc;
    for (int s = 0; s < e->max_systems; s++) {
        fill_desc(e, s, e->h_desc[s]);
        const HostSys &h = e->sys[s];
        if (!h.used)
            continue;
        const bool in_force = h.steps_left > 0 || !h.started;
        if (!in_force) {
            e->h_desc[s].flags = 0;
            continue;
        }
        if (h.sym || h.pair)
            continue;  // evaluated by launches of their own
        const int bi = nbgb::ens::kThreads * ((h.variant == 0 || h.variant == 2) ? 1 : 2);
        for (int b = 0; b < h.nblocks; b++)
            for (int r = 0; r < h.nsplit; r++) {
                const int tb = (int)(((long long)r * h.ntiles) / h.nsplit);
                const int te = (int)(((long long)(r + 1) * h.ntiles) / h.nsplit);
                items.push_back(It{make_int4(s, b, r, 0),
                                   (double)(te - tb) * h.jt * bi + 4096.0, sub_eff(h)});
            }
    }
    // by effective sub (ascending), then largest first: pass p's items are
    // the suffix of systems with sub > p
    std::stable_sort(items.begin(), items.end(), [](const It &a, const It &b) {
        return a.sub != b.sub ? a.sub < b.sub : a.cost > b.cost;
    });
    if (items.size() > e->items_cap)
        return NBGB_ERR_NO_MEMORY;
    for (size_t k = 0; k < items.size(); k++)
        e->h_items[k] = items[k].v;
    e->n_items = (int)items.size();
    for (const It &it : items)
        e->n_pass = std::max(e->n_pass, it.sub);
    for (int p = 0; p < nbgb::ens::kMaxSub; p++) {
        int k = 0;
        while (k < e->n_items && items[k].sub <= p)
            k++;
        e->pass_first[p] = p == 0 ? 0 : k;
    }
    // slot map over the used part of the j-stream arena (pairs)
    size_t end = 0;
    for (int s = 0; s < e->max_systems; s++)
        if (e->sys[s].used)
            end = std::max(end, (e->sys[s].js_off + e->sys[s].js_len) / 2);
    const int n_pairs = (int)end;
    std::fill(e->h_slot_sys, e->h_slot_sys + n_pairs, -1);
    for (int s = 0; s < e->max_systems; s++) {
        const HostSys &h = e->sys[s];
        if (!h.used)
            continue;
        for (size_t q = h.js_off / 2; q < (h.js_off + h.js_len) / 2; q++)
            e->h_slot_sys[q] = s;
    }
    e->n_slots = n_pairs;
    // Newton-3 systems of this tick, with their block-pair prefix counts
    e->n_sym = 0;
    long long pairs = 0;
    const int sb = nbgb::sym_block_bodies();
    for (int s = 0; s < e->max_systems; s++) {
        const HostSys &h = e->sys[s];
        if (!h.used || !h.sym || !(h.steps_left > 0 || !h.started))
            continue;
        nbgb::SymSystem &t = e->h_sym[e->n_sym++];
        t.pm = e->pm + h.body_off;
        t.js = e->js + h.js_off;
        t.acc = e->acc64 + h.acc_off;
        t.out = e->acc + h.body_off;
        t.n = h.n;
        t.npad = (int)(h.js_len);
        t.nblocks = (int)(h.js_len / sb);
        t.eps2 = e->eps2;
        t.pair_begin = pairs;
        pairs += (long long)t.nblocks * (t.nblocks + 1) / 2;
    }
    cudaStream_t st = e->stream;
    if (!e->groups.empty() &&
        (cudaMemcpyAsync(e->d_pitems, e->h_pitems,
                         sizeof(int4) * (e->groups.back().first + e->groups.back().n),
                         cudaMemcpyHostToDevice, st) != cudaSuccess ||
         (e->n_tasks && cudaMemcpyAsync(e->d_tasks, e->h_tasks, sizeof(int2) * e->n_tasks,
                                        cudaMemcpyHostToDevice, st) != cudaSuccess) ||
         cudaMemcpyAsync(e->d_blocks, e->h_blocks, sizeof(int2) * e->n_blocks,
                         cudaMemcpyHostToDevice, st) != cudaSuccess))
        return NBGB_ERR_CUDA;
    if (e->n_sym && cudaMemcpyAsync(e->d_sym, e->h_sym, sizeof(nbgb::SymSystem) * e->n_sym,
                                    cudaMemcpyHostToDevice, st) != cudaSuccess)
        return NBGB_ERR_CUDA;
    if (cudaMemcpyAsync(e->d_desc, e->h_desc, sizeof(Desc) * e->max_systems,
                        cudaMemcpyHostToDevice, st) != cudaSuccess ||
        (e->n_items &&
         cudaMemcpyAsync(e->d_items, e->h_items, sizeof(int4) * e->n_items, cudaMemcpyHostToDevice,
                         st) != cudaSuccess) ||
        (n_pairs && cudaMemcpyAsync(e->d_slot_sys, e->h_slot_sys, sizeof(int) * n_pairs,
                                    cudaMemcpyHostToDevice, st) != cudaSuccess))
        return NBGB_ERR_CUDA;
    if (e->graph) {
        cudaGraphExecDestroy(e->graph);
        e->graph = nullptr;
    }
    e->dirty = false;
    return NBGB_OK;
}

// The pair systems that move in this pass (all of them in pass 0).
int launch_pair_pass(nbgb_ensemble *e, int pass) {
    cudaStream_t st = e->stream;
    const int n_groups = (int)e->groups.size();
    const int work = std::max(e->n_blocks * nbgb::ens::kBodyBlock, n_groups);
    bool ok = nbgb::launch_dependent_n(nbgb::ens::ens_drift_kernel, (work + 255) / 256, 256, 0, st,
                                       e->d_desc, e->d_blocks, e->n_blocks, e->x64, e->max_bodies,
                                       e->mass, e->acc, e->pm, e->heads, n_groups,
                                       pass) == cudaSuccess;
    for (int k = 0; k < n_groups && ok; k++) {
        const PairGroup &g = e->groups[k];
        const int first = g.pass_first[pass], n = g.n - first;
        if (n <= 0)
            continue;
        nbgb::ens::PairParams P;
        P.desc = e->d_desc;
        P.items = e->d_pitems + g.first + first;
        P.tasks = e->d_tasks;
        P.n_items = n;
        P.pass = pass;
        P.head = e->heads + k;
        P.pm = e->pm;
        P.scratch = e->scratch;
        P.acc = e->acc;
        P.x64 = e->x64;
        P.stride = e->max_bodies;
        ok = nbgb::launch_dependent_n(nbgb::ens::ens_pair_kernel, std::min(e->grid, n),
                                      nbgb::ens::kPairCtaThreads, nbgb::ens::kPairSmem, st,
                                      P) == cudaSuccess &&
             (g.nblocks == 0 ||
              nbgb::launch_dependent_n(nbgb::ens::ens_reduce_kernel, g.nblocks,
                                       nbgb::ens::kReduceThreads, 0, st, e->d_desc,
                                       e->d_blocks + g.block0, e->scratch, e->x64, e->max_bodies,
                                       e->acc, pass) == cudaSuccess);
    }
    return ok ? NBGB_OK : NBGB_ERR_CUDA;
}

int launch_tick(nbgb_ensemble *e) {
    cudaStream_t st = e->stream;
    const int tb = 256;
    const int nb = std::max(1, (e->n_slots + tb - 1) / tb);
    for (int pass = 0; pass < e->n_pass; pass++) {
        if (!e->groups.empty()) {
            const int rc = launch_pair_pass(e, pass);
            if (rc != NBGB_OK)
                return rc;
        }
        const int first = e->pass_first[pass];
        const int n_items = e->n_items - first;
        if (n_items <= 0 && (pass > 0 || e->n_sym == 0))
            continue;
        nbgb::ens::ens_kdk_kernel<<<nb, tb, 0, st>>>(e->d_desc, e->d_slot_sys, e->n_slots,
                                                     e->x64, e->max_bodies, e->mass, e->acc,
                                                     e->pm, e->js, 0, pass);
        if (cudaMemsetAsync(e->head, 0, sizeof(unsigned), st) != cudaSuccess)
            return NBGB_ERR_CUDA;
        nbgb::ens::Params P;
        P.desc = e->d_desc;
        P.items = e->d_items + first;
        P.n_items = n_items;
        P.head = e->head;
        P.pm = e->pm;
        P.js = e->js;
        P.acc = e->acc;
        P.part = e->part;
        P.cnt = e->cnt;
        if (n_items > 0)
            nbgb::ens::ens_force_kernel<<<e->grid, nbgb::ens::kThreads,
                                          nbgb::ens::kStages * nbgb::ens::kStageBytes, st>>>(P);
        if (pass == 0 && e->n_sym > 0) {
            const int rc = nbgb::launch_sym_systems(e->d_sym, e->h_sym, e->n_sym, st);
            if (rc != NBGB_OK)
                return rc;
        }
        nbgb::ens::ens_kdk_kernel<<<nb, tb, 0, st>>>(e->d_desc, e->d_slot_sys, e->n_slots,
                                                     e->x64, e->max_bodies, e->mass, e->acc,
                                                     e->pm, e->js, 1, pass);
    }
    return cudaGetLastError() == cudaSuccess ? NBGB_OK : NBGB_ERR_CUDA;
}

void free_ens(nbgb_ensemble *e) {
    if (e->graph)
        cudaGraphExecDestroy(e->graph);
    cudaFree(e->x64);
    cudaFree(e->mass);
    cudaFree(e->pm);
    cudaFree(e->acc);
    cudaFree(e->js);
    cudaFree(e->part);
    cudaFree(e->cnt);
    cudaFree(e->head);
    cudaFree(e->d_desc);
    cudaFree(e->d_items);
    cudaFree(e->d_slot_sys);
    cudaFree(e->acc64);
    cudaFree(e->scratch);
    cudaFree(e->d_lists);
    cudaFree(e->heads);
    cudaFreeHost(e->h_lists);
    cudaFree(e->d_sym);
    cudaFreeHost(e->h_sym);
    cudaFreeHost(e->h_desc);
    cudaFreeHost(e->h_items);
    cudaFreeHost(e->h_slot_sys);
    e->snap.destroy();
    if (e->stream)
        cudaStreamDestroy(e->stream);
}

}  // namespace

extern "C" {

// How a system of N bodies is evaluated by the default plan (newton3: one
// admitted at or above set_newton3_min's size): kind 3 warp tasks, 1 and 2 rows
// of pairs (512 and 1,024 bodies), 0 neither (one-sided queue; Newton-3: block
// pairs); sets_per_item and scratch_bytes of kinds 1 and 2.  No GPU needed.
NBGB_API int nbgb_ensemble_kind(size_t N, int newton3, int *kind, int *sets_per_item,
                                size_t *scratch_bytes) {
    if (N == 0 || N > nbgb::kMaxBodies)
        return NBGB_ERR_INVALID_ARGUMENT;
    HostSys h;
    pair_plan(N, newton3 ? kPairScratchN3 : kPairScratch, h);
    if (kind)
        *kind = h.pair;
    if (sets_per_item)
        *sets_per_item = h.ch;
    if (scratch_bytes)
        *scratch_bytes = h.scratch_len * 4;
    return NBGB_OK;
}

// Capacity: max_bodies bodies in total, max_systems concurrent systems.  The
// device arena is allocated once here (about 250 B per body of capacity plus
// the pair systems' scratch, up to 512 MiB,
// including partials for j-splits of up to 4); admission never allocates.
NBGB_API nbgb_ensemble *nbgb_ensemble_create(size_t max_bodies, int max_systems,
                                             float softeningSquared) {
    if (max_bodies == 0 || max_bodies > ((size_t)1 << 30) || max_systems <= 0)
        return nullptr;
    nbgb_ensemble *e = new (std::nothrow) nbgb_ensemble();
    if (!e)
        return nullptr;
    e->eps2 = softeningSquared;
    e->max_systems = max_systems;
    e->max_bodies = max_bodies;
    // j-stream: bodies rounded up to tiles (<= 1024 per system) or to
    // Newton-3 blocks, and to pairs
    e->js_cap = max_bodies +
                (size_t)max_systems * std::max(nbgb::ens::kMaxJT, nbgb::sym_block_bodies());
    e->js_cap += e->js_cap & 1;
    // split partials: hi + lo for up to 4-way j-splits of every body (plus
    // block padding); counters and items for up to 4 splits of 256-body blocks
    e->part_cap = 8 * (max_bodies + (size_t)max_systems * 512);
    e->cnt_cap = max_bodies / 256 + (size_t)max_systems + 1;
    e->items_cap = 4 * (max_bodies / 256 + (size_t)max_systems) + 64;
    // pair items (at most 0.067 a body, where sets_per_item is about to grow,
    // and four for the smallest systems) and 64-body blocks
    e->scratch_cap = scratch_for(max_bodies, kPairScratch);
    e->pitems_cap = max_bodies / 12 + 4 * (size_t)max_systems + 64;
    e->tasks_cap = max_bodies / nbgb::ens::kTaskBodies + (size_t)max_systems +
                   4 * (size_t)nbgb::ens::kMaxSub;
    e->blocks_cap = max_bodies / nbgb::ens::kBodyBlock + (size_t)max_systems + 1;
    e->sys.assign(max_systems, HostSys());
    e->a_body.init(max_bodies);
    e->a_js.init(e->js_cap);
    e->a_part.init(e->part_cap);
    e->a_cnt.init(e->cnt_cap);
    cudaGetDevice(&e->device);
    bool ok = cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking) == cudaSuccess;
    ok = ok && cudaMalloc(&e->x64, 6 * max_bodies * sizeof(double)) == cudaSuccess;
    ok = ok && cudaMalloc(&e->mass, max_bodies * sizeof(float)) == cudaSuccess;
    ok = ok && cudaMalloc(&e->pm, max_bodies * 16) == cudaSuccess;
    ok = ok && cudaMalloc(&e->acc, max_bodies * 16) == cudaSuccess;
    ok = ok && cudaMalloc(&e->js, e->js_cap * 16) == cudaSuccess;
    ok = ok && cudaMalloc(&e->part, e->part_cap * 16) == cudaSuccess;
    ok = ok && cudaMalloc(&e->cnt, e->cnt_cap * 4) == cudaSuccess;
    ok = ok && cudaMalloc(&e->head, 256) == cudaSuccess;
    ok = ok && cudaMalloc(&e->d_desc, sizeof(Desc) * max_systems) == cudaSuccess;
    ok = ok && cudaMalloc(&e->d_items, sizeof(int4) * e->items_cap) == cudaSuccess;
    ok = ok && cudaMalloc(&e->d_slot_sys, sizeof(int) * (e->js_cap / 2)) == cudaSuccess;
    ok = ok && cudaMalloc(&e->scratch, e->scratch_cap * 4) == cudaSuccess;
    const size_t off_tasks = sizeof(int4) * e->pitems_cap;
    const size_t off_blocks = off_tasks + sizeof(int2) * e->tasks_cap;
    const size_t list_bytes = off_blocks + sizeof(int2) * e->blocks_cap;
    ok = ok && cudaMalloc(&e->d_lists, list_bytes) == cudaSuccess;
    ok = ok && cudaMallocHost(&e->h_lists, list_bytes) == cudaSuccess;
    e->d_pitems = (int4 *)e->d_lists;
    e->h_pitems = (int4 *)e->h_lists;
    e->d_tasks = (int2 *)(e->d_lists + off_tasks);
    e->h_tasks = (int2 *)(e->h_lists + off_tasks);
    e->d_blocks = (int2 *)(e->d_lists + off_blocks);
    e->h_blocks = (int2 *)(e->h_lists + off_blocks);
    ok = ok && cudaMalloc(&e->heads, 4 * ((size_t)max_systems + 1)) == cudaSuccess;
    ok = ok && cudaFuncSetAttribute(nbgb::ens::ens_pair_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)nbgb::ens::kPairSmem) == cudaSuccess;
    ok = ok && cudaMallocHost(&e->h_desc, sizeof(Desc) * max_systems) == cudaSuccess;
    ok = ok && cudaMallocHost(&e->h_items, sizeof(int4) * e->items_cap) == cudaSuccess;
    ok = ok && cudaMallocHost(&e->h_slot_sys, sizeof(int) * (e->js_cap / 2)) == cudaSuccess;
    ok = ok && cudaMalloc(&e->d_sym, sizeof(nbgb::SymSystem) * max_systems) == cudaSuccess;
    ok = ok && cudaMallocHost(&e->h_sym, sizeof(nbgb::SymSystem) * max_systems) == cudaSuccess;
    ok = ok && cudaMemsetAsync(e->cnt, 0, e->cnt_cap * 4, e->stream) == cudaSuccess;
    ok = ok && cudaMemsetAsync(e->js, 0, e->js_cap * 16, e->stream) == cudaSuccess;
    ok = ok && cudaFuncSetAttribute(nbgb::ens::ens_force_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    nbgb::ens::kStages * nbgb::ens::kStageBytes) == cudaSuccess;
    const unsigned *status = nbgb::status_address_ensemble();
    ok = ok && status && e->snap.create(max_bodies, &status, 1) == NBGB_OK;
    int occ = 0, sms = 0;
    ok = ok && cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                   &occ, nbgb::ens::ens_force_kernel, nbgb::ens::kThreads,
                   nbgb::ens::kStages * nbgb::ens::kStageBytes) == cudaSuccess;
    ok = ok && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device) ==
                   cudaSuccess;
    ok = ok && cudaStreamSynchronize(e->stream) == cudaSuccess && occ > 0;
    if (!ok) {
        free_ens(e);
        delete e;
        return nullptr;
    }
    e->grid = sms * occ;
    e->grid_max = e->grid;
    e->bytes_total = max_bodies * (6 * 8 + 4 + 16 + 16) + e->js_cap * 16 + e->part_cap * 16 +
                     e->cnt_cap * 4 + e->scratch_cap * 4;
    return e;
}

NBGB_API void nbgb_ensemble_destroy(nbgb_ensemble *e) {
    if (!e)
        return;
    cudaStreamSynchronize(e->stream);
    free_ens(e);
    delete e;
}

NBGB_API size_t nbgb_ensemble_device_bytes(nbgb_ensemble *e) { return e ? e->bytes_total : 0; }

// Per-bucket plan (bucket b: N in [2^b, 2^(b+1))): variant 0..3 (targets per
// thread and unroll: (1,8) (2,4) (1,4) (2,8)), tile a power of two in
// 16..1024 bodies, j-split 1..4; variant -1 restores the default rule.
// Applies to systems admitted afterwards.
NBGB_API int nbgb_ensemble_set_bucket_plan(nbgb_ensemble *e, int bucket, int variant, int jt,
                                           int nsplit) {
    if (!e || bucket < 0 || bucket >= 32 || variant < -1 || variant > 3)
        return NBGB_ERR_INVALID_ARGUMENT;
    if (variant >= 0 &&
        (jt < 16 || jt > nbgb::ens::kMaxJT || (jt & (jt - 1)) || nsplit < 1 || nsplit > 4))
        return NBGB_ERR_INVALID_ARGUMENT;
    e->bucket[bucket].variant = variant;
    e->bucket[bucket].jt = jt;
    e->bucket[bucket].nsplit = nsplit;
    return NBGB_OK;
}

// Admit one system: HOST FP64 positions/velocities double[n][3], float masses.
// Returns NBGB_ERR_NO_MEMORY when no slot or not enough arena is free (the
// caller retries after systems retire).  *slot receives the system's slot.
NBGB_API int nbgb_ensemble_add(nbgb_ensemble *e, const double *pos3, const double *vel3,
                               const float *mass, size_t n, double dt, long long steps,
                               int *slot) {
    if (!e || !pos3 || !vel3 || !mass || !slot || n == 0 || n > e->max_bodies || steps < 0)
        return NBGB_ERR_INVALID_ARGUMENT;
    int s = -1;
    for (int k = 0; k < e->max_systems; k++)
        if (!e->sys[k].used) {
            s = k;
            break;
        }
    if (s < 0)
        return NBGB_ERR_NO_MEMORY;
    HostSys h;
    h.n = (int)n;
    choose_plan(e, (int)n, h);
    h.body_len = n;
    h.n3 = e->n3_min > 0 && n >= e->n3_min;
    if (h.n3 || e->bucket[bucket_of((int)n)].variant < 0)
        pair_plan(n, h.n3 ? kPairScratchN3 : kPairScratch, h);
    h.sym = h.n3 && !h.pair;
    if (h.pair) {  // scratch is placed tick by tick
        h.js_len = h.part_len = h.cnt_len = 0;
    } else if (h.sym) {  // j-stream padded to whole Newton-3 blocks, FP64 sums
        const size_t sb = (size_t)nbgb::sym_block_bodies();
        h.js_len = (n + sb - 1) / sb * sb;
        h.acc_len = 3 * h.js_len;
        h.part_len = h.cnt_len = 0;
    } else {
        h.js_len = (size_t)h.ntiles * h.jt;
        h.js_len += h.js_len & 1;
        h.part_len = h.nsplit > 1 ? 2 * (size_t)h.nsplit * h.ni_pad : 0;
        h.cnt_len = h.nsplit > 1 ? (size_t)h.nblocks : 0;
    }
    size_t ob, oj, op = 0, oc = 0, oa = 0;
    if (h.acc_len && !e->a_acc.alloc(h.acc_len, 32, oa))
        return NBGB_ERR_NO_MEMORY;
    if (!e->a_body.alloc(h.body_len, 1, ob)) {
        if (h.acc_len)
            e->a_acc.release(oa, h.acc_len);
        return NBGB_ERR_NO_MEMORY;
    }
    if (!e->a_js.alloc(h.js_len, 2, oj)) {
        e->a_body.release(ob, h.body_len);
        if (h.acc_len)
            e->a_acc.release(oa, h.acc_len);
        return NBGB_ERR_NO_MEMORY;
    }
    if (h.part_len && !e->a_part.alloc(h.part_len, 2, op)) {
        e->a_body.release(ob, h.body_len);
        e->a_js.release(oj, h.js_len);
        return NBGB_ERR_NO_MEMORY;
    }
    if (h.cnt_len && !e->a_cnt.alloc(h.cnt_len, 1, oc)) {
        e->a_body.release(ob, h.body_len);
        e->a_js.release(oj, h.js_len);
        if (h.part_len)
            e->a_part.release(op, h.part_len);
        return NBGB_ERR_NO_MEMORY;
    }
    h.acc_off = oa;
    h.body_off = ob;
    h.js_off = oj;
    h.part_off = op;
    h.cnt_off = oc;
    h.dt = dt;
    h.steps_left = steps;
    h.used = true;
    h.log_mass = !h.sym && !h.pair;  // the other kernels read plain masses
    for (size_t i = 0; i < n && h.log_mass; i++)
        h.log_mass = mass[i] >= 0.f;
    // upload state (SoA FP64, masses), zero the j-stream range
    cudaStream_t st = e->stream;
    nbgb::UploadJob job;
    job.n = n;
    job.pos3 = pos3;
    job.vel3 = vel3;
    job.mass = mass;
    job.x64 = e->x64 + ob;
    job.ld = e->max_bodies;
    job.mass_out = e->mass + ob;
    if ((h.js_len && cudaMemsetAsync(e->js + oj, 0, h.js_len * 16, st) != cudaSuccess) ||
        (h.acc_len &&
         cudaMemsetAsync(e->acc64 + oa, 0, h.acc_len * sizeof(double), st) != cudaSuccess) ||
        e->snap.upload(job, st) != NBGB_OK)
        return NBGB_ERR_CUDA;
    e->sys[s] = h;
    e->dirty = true;
    *slot = s;
    return NBGB_OK;
}

// One tick: every admitted system either gets its initial accelerations (its
// first tick) or advances one FP64 KDK step.  Asynchronous.
NBGB_API int nbgb_ensemble_tick(nbgb_ensemble *e, int nticks) {
    if (!e || nticks < 0)
        return NBGB_ERR_INVALID_ARGUMENT;
    for (int k = 0; k < nticks; k++) {
        if (e->dirty) {
            int rc = rebuild(e);
            if (rc != NBGB_OK)
                return rc;
            e->stable_ticks = 0;
        }
        // A graph pays off only when it is replayed: capture it once the
        // membership has been unchanged for two ticks, launch eagerly before.
        if (e->use_graph && e->stable_ticks >= 2) {
            if (!e->graph) {
                cudaGraph_t g = nullptr;
                if (cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal) !=
                    cudaSuccess)
                    return NBGB_ERR_CUDA;
                int rc = launch_tick(e);
                cudaError_t ce = cudaStreamEndCapture(e->stream, &g);
                if (rc != NBGB_OK || ce != cudaSuccess) {
                    if (g)
                        cudaGraphDestroy(g);
                    return NBGB_ERR_CUDA;
                }
                ce = cudaGraphInstantiate(&e->graph, g, 0);
                cudaGraphDestroy(g);
                if (ce != cudaSuccess)
                    return NBGB_ERR_CUDA;
            }
            if (cudaGraphLaunch(e->graph, e->stream) != cudaSuccess)
                return NBGB_ERR_CUDA;
        } else {
            int rc = launch_tick(e);
            if (rc != NBGB_OK)
                return rc;
        }
        e->stable_ticks++;
        e->ticks++;
        // host bookkeeping of this tick
        for (auto &h : e->sys) {
            if (!h.used)
                continue;
            if (!h.started) {
                h.started = true;
                e->dirty = true;  // moves from the next tick on
            } else if (h.steps_left > 0) {
                const int k = sub_eff(h);
                h.steps_left -= k;
                h.steps_done += k;
                if (h.steps_left < h.sub)
                    e->dirty = true;  // leaves the tick, or fewer steps next tick
            }
        }
    }
    return NBGB_OK;
}

// CTAs of the persistent force launch (1 .. SMs x resident CTAs; 0 = all).
// Two ensembles on one GPU can run side by side when their grids together
// fit the GPU's resident CTA slots.
NBGB_API int nbgb_ensemble_set_grid(nbgb_ensemble *e, int ctas) {
    if (!e || ctas < 0 || ctas > e->grid_max)
        return NBGB_ERR_INVALID_ARGUMENT;
    const int g = ctas == 0 ? e->grid_max : ctas;
    if (g != e->grid) {
        e->grid = g;
        if (e->graph) {  // the captured tick launches the old grid
            cudaGraphExecDestroy(e->graph);
            e->graph = nullptr;
        }
    }
    return NBGB_OK;
}

// Resident CTA slots of the persistent force launch on this device.
NBGB_API int nbgb_ensemble_max_grid(nbgb_ensemble *e) { return e ? e->grid_max : 0; }

NBGB_API int nbgb_ensemble_set_graph(nbgb_ensemble *e, int enable) {
    if (!e)
        return NBGB_ERR_INVALID_ARGUMENT;
    e->use_graph = enable != 0;
    return NBGB_OK;
}

NBGB_API int nbgb_ensemble_synchronize(nbgb_ensemble *e) {
    if (!e)
        return NBGB_ERR_INVALID_ARGUMENT;
    unsigned bits = 0;
    if (e->snap.run(nbgb::SnapshotJob(), e->stream, &bits) != NBGB_OK ||
        (bits && nbgb::read_status_ensemble(&bits) != NBGB_OK))
        return NBGB_ERR_CUDA;
    return bits ? NBGB_ERR_DEVICE : NBGB_OK;
}

// Slots whose steps are all done (state synchronised in time), up to max.
NBGB_API int nbgb_ensemble_finished(nbgb_ensemble *e, int *slots, int max) {
    if (!e || (max > 0 && !slots))
        return NBGB_ERR_INVALID_ARGUMENT;
    int k = 0;
    for (int s = 0; s < e->max_systems && k < max; s++)
        if (e->sys[s].used && e->sys[s].started && e->sys[s].steps_left == 0)
            slots[k++] = s;
    return k;
}

// State of a slot (HOST double[n][3]); synchronises the stream first.
NBGB_API int nbgb_ensemble_get_state(nbgb_ensemble *e, int slot, double *pos3, double *vel3,
                                     float *acc4) {
    if (!e || slot < 0 || slot >= e->max_systems || !e->sys[slot].used)
        return NBGB_ERR_INVALID_ARGUMENT;
    const HostSys &h = e->sys[slot];
    nbgb::SnapshotJob job;
    job.n = (size_t)h.n;
    job.vec[0] = e->acc + h.body_off;
    job.out[0] = acc4;
    job.x64 = e->x64 + h.body_off;
    job.ld = e->max_bodies;
    job.pos3 = pos3;
    job.vel3 = vel3;
    unsigned bits = 0;
    return e->snap.run(job, e->stream, &bits);  // (synchronize() reports the status)
}

// Slot info: bodies, steps done, steps left, plan (variant, tile, split).
NBGB_API int nbgb_ensemble_slot_info(nbgb_ensemble *e, int slot, long long *info6) {
    if (!e || slot < 0 || slot >= e->max_systems || !info6)
        return NBGB_ERR_INVALID_ARGUMENT;
    const HostSys &h = e->sys[slot];
    info6[0] = h.used ? h.n : 0;
    info6[1] = h.steps_done;
    info6[2] = h.steps_left;
    info6[3] = h.pair ? -1 : h.variant;  // pair systems: variant -1, no tile
    info6[4] = h.pair ? 0 : h.jt;
    info6[5] = h.pair ? 1 : h.nsplit;
    return NBGB_OK;
}

// Steps per tick of one system (1..8); takes effect from the next tick.
NBGB_API int nbgb_ensemble_set_substeps(nbgb_ensemble *e, int slot, int sub) {
    if (!e || slot < 0 || slot >= e->max_systems || !e->sys[slot].used || sub < 1 ||
        sub > nbgb::ens::kMaxSub)
        return NBGB_ERR_INVALID_ARGUMENT;
    if (e->sys[slot].sub != sub) {
        e->sys[slot].sub = sub;
        e->dirty = true;
    }
    return NBGB_OK;
}

// Stream priority of the ensemble's work: high = the device's greatest
// priority, so that its CTAs are dispatched ahead of other streams' pending
// CTAs as SMs free up (an ensemble beside a busier one).  Recreates the
// stream (after draining it).
NBGB_API int nbgb_ensemble_set_priority(nbgb_ensemble *e, int high) {
    if (!e)
        return NBGB_ERR_INVALID_ARGUMENT;
    int lo = 0, hi = 0;
    if (cudaDeviceGetStreamPriorityRange(&lo, &hi) != cudaSuccess ||
        cudaStreamSynchronize(e->stream) != cudaSuccess)
        return NBGB_ERR_CUDA;
    cudaStream_t st = nullptr;
    if (cudaStreamCreateWithPriority(&st, cudaStreamNonBlocking, high ? hi : lo) != cudaSuccess)
        return NBGB_ERR_CUDA;
    if (e->graph) {
        cudaGraphExecDestroy(e->graph);
        e->graph = nullptr;
    }
    cudaStreamDestroy(e->stream);
    e->stream = st;
    return NBGB_OK;
}

// Systems admitted from now on with at least nmin bodies are pair systems
// whatever their bucket's plan (0: none).  The first nonzero call grows the
// scratch arena, and where a system could still exceed it allocates the FP64
// sums arena of the block-pair kernel (24 B per body of capacity).
NBGB_API int nbgb_ensemble_set_newton3_min(nbgb_ensemble *e, size_t nmin) {
    if (!e)
        return NBGB_ERR_INVALID_ARGUMENT;
    const size_t need = scratch_for(e->max_bodies, kPairScratchN3);
    if (nmin > 0 && need > e->scratch_cap) {  // larger pair systems
        float *p = nullptr;
        if (cudaStreamSynchronize(e->stream) != cudaSuccess)
            return NBGB_ERR_CUDA;
        if (cudaMalloc(&p, need * 4) != cudaSuccess)
            return NBGB_ERR_NO_MEMORY;
        cudaFree(e->scratch);
        e->bytes_total += (need - e->scratch_cap) * 4;
        e->scratch = p;
        e->scratch_cap = need;
        e->dirty = true;  // the captured tick holds the old arena
    }
    HostSys largest;
    if (nmin > 0 && !e->acc64 && !pair_plan(e->max_bodies, kPairScratchN3, largest)) {
        const size_t cap = 3 * (e->max_bodies + (size_t)e->max_systems *
                                                    (size_t)nbgb::sym_block_bodies());
        if (cudaMalloc(&e->acc64, cap * sizeof(double)) != cudaSuccess) {
            e->acc64 = nullptr;
            return NBGB_ERR_NO_MEMORY;
        }
        e->acc64_cap = cap;
        e->a_acc.init(cap);
        e->bytes_total += cap * sizeof(double);
    }
    e->n3_min = nmin;
    return NBGB_OK;
}

// Retire a slot: its arena ranges and slot become free for admission.
NBGB_API int nbgb_ensemble_remove(nbgb_ensemble *e, int slot) {
    if (!e || slot < 0 || slot >= e->max_systems || !e->sys[slot].used)
        return NBGB_ERR_INVALID_ARGUMENT;
    HostSys &h = e->sys[slot];
    // the stream may still run a tick that reads this slot's ranges
    if (cudaStreamSynchronize(e->stream) != cudaSuccess)
        return NBGB_ERR_CUDA;
    e->a_body.release(h.body_off, h.body_len);
    e->a_js.release(h.js_off, h.js_len);
    if (h.part_len)
        e->a_part.release(h.part_off, h.part_len);
    if (h.cnt_len)
        e->a_cnt.release(h.cnt_off, h.cnt_len);
    if (h.acc_len)
        e->a_acc.release(h.acc_off, h.acc_len);
    h = HostSys();
    e->dirty = true;
    return NBGB_OK;
}

NBGB_API int nbgb_ensemble_active(nbgb_ensemble *e) {
    if (!e)
        return 0;
    int k = 0;
    for (auto &h : e->sys)
        k += h.used ? 1 : 0;
    return k;
}

NBGB_API void *nbgb_ensemble_stream(nbgb_ensemble *e) { return e ? e->stream : nullptr; }

}  // extern "C"
