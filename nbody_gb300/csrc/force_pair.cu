// force_pair.cu -- the all-pairs force with every pair of bodies evaluated
// once and applied to both (Newton's third law), deterministic: no atomics,
// every partial sum is written once and added in a fixed order.
//
// What bounds it: the FP32 (FMA) pipe and the registers that feed it.  Two
// pairs cost 16 packed FP32 operations for their four interactions (14 when
// the masses involved are equal), against 23 to 24 of the one-sided
// kernel.  ncu: FMA pipe 79 % busy; the rest are dispatch stalls of
// three-operand instructions (six of the 16) and the other instructions' issue.
// GB300, N = 131,072: 4,267 us with mixed masses (4.03e12 interactions/s),
// 3,897 us with equal ones (4.41e12), against 4,830 us for 8 sources and 8
// targets a lane with all source registers shuffled and FP64 atomics, and
// 5,820 us one-sided.
//
// Work.  Targets are taken in rows of kRow bodies (one CTA: W warps x 32
// lanes x KI bodies held in registers), sources in sets of kSet = 64 NC
// bodies.  Row b meets its own sets one-sided (every ordered pair, the self
// pair contributing 0) and every later set both ways.  A warp meets a set in
// 32 steps: at step t lane L evaluates its KI targets against the NC source
// pairs (L + t) & 31 (f32x2: two sources an instruction), whose reaction sums
// then move to the next lane by shuffle; positions and masses are not
// shuffled but read from shared memory (two 128-bit loads instead of eight
// shuffles a source pair; each set is stored twice in a row, so lane L + t
// needs no wrap).  Every instruction beside the FMA-pipe ones costs about as
// much issue time as one of them, which asks for a tile wide in targets; but
// the own-row meetings, the pieces and the folds grow with it.  At N = 16,384 /
// 131,072 / 1,048,576, in us and ms, mixed and equal masses: 11 targets a lane
// 83.2, 79.7 / 4,415, 4,102 / 280.8, 258.3; 9: 81.7, 77.0 / 4,433, 4,013; 8:
// 80.8, 77.5 / 4,427, 4,037 / 282.3, 255.0; 7: 81.6, 76.1 / 4,556, 4,147 (all
// before the late stretches below).  The next set
// comes by cp.async, which holds no registers.
//
// Narrow rows (512 bodies, 4 targets a lane) serve n below kNarrowBelow, where
// rows of 1,024 are too few pieces of work: 12,500 bodies take 52.7 us narrow
// and 51.2 us wide (equal masses 50.1 and 50.4), 13,000 56.8 and 54.6, 8,192
// 26.5 and 26.6, 10,007 36.8 and 37.1 (before pieces had remainders, which
// cost both 0.6 to 1 us).
//
// Split.  The steps of all (row, set) meetings form one line, and the host
// cuts it into equal stretches of cost, one per resident CTA, and, where there
// is more work, as many short late ones (stretch_cost).  A stretch may begin and end inside a set or a row.
// Pieces: the reactions of one stretch's part of one (row, set) meeting
// (kSet x 3 floats, slot = meeting index + CTA index) and the targets' sums
// of its part of one row (kRow x 3 floats, and as many for what rounding them
// leaves out where stretches exceed 256 sources, slot = row + CTA index); both
// numberings grow strictly along the line, so no two pieces share a slot.
// The reduce kernel adds each body's pieces in a fixed order with compensated
// FP32 sums and writes the force (and integrates, when asked).  Both kernels
// are launched with programmatic dependence: their CTAs start as the previous
// kernel's leave and wait for it only before they touch its results.
//
// Phases.  The reaction pieces of all rows take N^2/(2 kRow) x 12 B; rows are
// processed in as many phases as the workspace needs.  Bodies of the rows
// done are final after their phase and no later phase reads them; the sums
// of later bodies are carried over in the workspace.
//
// Ranges.  (|d|^2 + eps2)^-3/2 alone leaves the binary32 range beyond
// distances of 2^42 although m times it may not.  Warps whose targets and set
// lie within 2^40 of the origin (eps2 within 2^+-80) take the short forms;
// others multiply by the mass first, as the one-sided kernel does.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "nbgb_device.cuh"
#include "nbgb_integrate.cuh"
#include "nbgb_internal.h"
#include "nbgb_pair.cuh"
#include "nbody_gb300.h"

namespace nbgb {
namespace pair {

// The bodies of the system.
struct Source {
    const float4 *pm;               // (may be where the forces go)
    int n;
    float eps2;
    int short_ok;                   // eps2 in the short forms' range
    unsigned *__restrict__ status;  // not null: refuse masses < 0
};

struct Params {
    Source src;
    float *__restrict__ react;  // [slot][3][kSet]
    float *__restrict__ tsum;   // [slot][3 pieces][kRow]
    int nsets, row0, row1;      // rows of this phase
    int ncta, parts;                // parts > 0: stretches are parts of meetings
    int pieces;                     // the targets' sums of a stretch; 2: and remainders
    unsigned step[kMaxPairCtas + 1];  // first step of each CTA's stretch
};

// Row b's part of this CTA's stretch (row_stretch asks for it).
template <class G>
struct StretchIo {
    const Params &P;
    const int b;
    __device__ __forceinline__ const float4 *pm() const { return P.src.pm; }
    __device__ __forceinline__ int n() const { return P.src.n; }
    __device__ __forceinline__ float eps2() const { return P.src.eps2; }
    __device__ __forceinline__ int short_ok() const { return P.src.short_ok; }
    __device__ __forceinline__ unsigned *status() const { return P.src.status; }
    __device__ __forceinline__ float *react(unsigned s) const {
        return P.react + ((size_t)(s >> 5) + blockIdx.x) * 3 * G::kSet;
    }
    __device__ __forceinline__ float *tsum() const {
        return P.tsum +
               ((size_t)(b - P.row0) + blockIdx.x) * P.pieces * 3 * G::kRow;
    }
    __device__ __forceinline__ bool remainder() const { return P.pieces > 1; }
};

template <class G>
__global__ void __launch_bounds__(G::kThreads, G::kCtas)
    pair_kernel(const __grid_constant__ Params P) {
    extern __shared__ __align__(128) float smem[];
    const int cta = blockIdx.x;
    unsigned s = P.step[cta];
    const unsigned s_end = P.step[cta + 1];
    const long long g0 = meetings_before<G>(P.row0, P.nsets);
    int b;
    {  // the row that holds meeting s / 32
        const long long g = g0 + (s >> 5);
        int lo = P.row0, hi = P.row1 - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (meetings_before<G>(mid, P.nsets) <= g)
                lo = mid;
            else
                hi = mid - 1;
        }
        b = lo;
    }
    grid_dependents_launch();
    grid_dependency_wait();
    for (; s < s_end; b++) {
        const int gb = (int)(meetings_before<G>(b, P.nsets) - g0);  // row b's first meeting
        const int row_set = b * G::kRowSets;
        const unsigned seg_end = min(s_end, (unsigned)(gb + (P.nsets - row_set)) << 5);
        row_stretch<G, false>(StretchIo<G>{P, b}, smem, b, row_set + ((int)(s >> 5) - gb), s,
                              seg_end);
        s = seg_end;
    }
}

struct ReduceParams {
    Params p;
    float *__restrict__ carry;  // [6][npad]: sums of bodies whose rows come later
    size_t npad;
    float4 *force;
    FusedIntegrate fi;  // fi.vel == nullptr: forces only
};

// 32 kEach bodies a block, kGroups x 3 (components) threads for kEach bodies:
// the block's reaction pieces (one list, from the phase's earlier rows in row
// order) and then its row's target pieces form one sequence; each group adds
// a contiguous part of it, eight loads in flight, and the parts are added in
// order.  A latency problem, not a bandwidth one: at N = 3,000 about 50 pieces
// a body and 9,000 sums, where four groups took 4 us more than with few
// pieces.
template <int kEach>
struct alignas(4 * kEach) Bodies {  // one component of a thread's bodies
    float v[kEach];
};
__device__ __forceinline__ Bodies<1> load_once(const Bodies<1> *p) {
    return {{__ldcs(&p->v[0])}};
}
__device__ __forceinline__ Bodies<2> load_once(const Bodies<2> *p) {
    const float2 a = __ldcs(reinterpret_cast<const float2 *>(p));
    return {{a.x, a.y}};
}

template <class G, int kGroups, int kEach>
__global__ void __launch_bounds__(3 * 32 * kGroups)
    pair_reduce_kernel(const __grid_constant__ ReduceParams R) {
    typedef Bodies<kEach> V;
    constexpr int kSet = G::kSet, kB = 32 * kEach, kPart = kSet / kB;
    static_assert(kSet % kB == 0, "blocks are parts of a set");
    __shared__ int list[kMaxPairRows + kMaxPairCtas];
    __shared__ int n_list, t_first, t_count;
    __shared__ V part[kGroups - 1][2][3][32], out[3][32];
    const Params &P = R.p;
    const int tid = threadIdx.x, group = tid / (3 * 32), comp = (tid / 32) % 3;
    const int lane = tid & 31, j = kEach * lane;
    const int set = P.row0 * G::kRowSets + blockIdx.x / kPart;
    const int sub = blockIdx.x % kPart;  // part of the set
    const int b = set / G::kRowSets;
    if (tid < 32) {  // one warp finds the pieces
        const long long g0 = meetings_before<G>(P.row0, P.nsets);
        // CTAs f..l (inclusive) whose stretches touch steps [a, e); no stretch
        // is empty
        auto ctas = [&](unsigned a, unsigned e, int &f, int &l) {
            if (P.parts) {
                f = (int)(a >> 5) * P.parts;
                l = (int)(e >> 5) * P.parts - 1;
                return;
            }
            int lo = 0, hi = P.ncta - 1;  // last c with step[c] <= a
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (P.step[mid] <= a)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            f = lo;
            while (lo + 1 < P.ncta && P.step[lo + 1] < e)
                lo++;
            l = lo;
        };
        const int nrow = min(b, P.row1) - P.row0;  // earlier rows of this phase
        int base = 0;
        for (int r0 = 0; r0 < nrow; r0 += 32) {  // list of slots, in row order
            const int row = P.row0 + r0 + tid;
            int slot = 0, c = 0;
            if (r0 + tid < nrow) {
                const int g = (int)(meetings_before<G>(row, P.nsets) - g0) +
                              (set - row * G::kRowSets);
                int f, l;
                ctas((unsigned)g << 5, ((unsigned)g << 5) + 32, f, l);
                slot = g + f;
                c = l - f + 1;
            }
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (tid >= o)
                    incl += v;
            }
            for (int q = 0; q < c; q++)
                list[base + incl - c + q] = slot + q;
            base += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (tid == 0) {
            int tf = 0, tl = -1;
            if (b < P.row1)
                ctas((unsigned)((meetings_before<G>(b, P.nsets) - g0) << 5),
                     (unsigned)((meetings_before<G>(b + 1, P.nsets) - g0) << 5), tf, tl);
            n_list = base;
            t_first = tf;
            t_count = (tl - tf + 1) * P.pieces;
        }
    }
    __syncthreads();
    const bool final = b < P.row1;  // else rows to come add to these bodies
    const int nr = n_list, tf = t_first, total = nr + t_count;
    const int q0 = total * group / kGroups, q1 = total * (group + 1) / kGroups;
    const float *react = P.react + (size_t)comp * kSet + sub * kB + j;
    const int i = set * kSet + sub * kB + j;
    const float *tsum = P.tsum + (size_t)comp * G::kRow + (i - b * G::kRow) +
                        (size_t)(b - P.row0 + tf) * P.pieces * 3 * G::kRow;
    auto piece = [&](int q) {
        return q < nr ? react + (size_t)list[q] * 3 * kSet
                      : tsum + (size_t)(q - nr) * 3 * G::kRow;
    };
    grid_dependents_launch();
    grid_dependency_wait();
    const int ib = set * kSet + sub * kB + tid;
    const bool writes = final && tid < kB && ib < P.src.n;
    V hi = {}, lo = {};
    auto carry = [&](int part) {
        return reinterpret_cast<V *>(R.carry + (3 * part + comp) * R.npad + i);
    };
    if (P.row0 > 0 && group == 0) {
        hi = *carry(0);
        lo = *carry(1);
    }
    int q = q0;
    for (; q + 8 <= q1; q += 8) {
        V v[8];
#pragma unroll
        for (int u = 0; u < 8; u++)
            v[u] = load_once(reinterpret_cast<const V *>(piece(q + u)));
#pragma unroll
        for (int u = 0; u < 8; u++)
#pragma unroll
            for (int k = 0; k < kEach; k++)
                comp_add(hi.v[k], lo.v[k], v[u].v[k]);
    }
    if (q < q1) {
        V v[8];
#pragma unroll
        for (int u = 0; u < 8; u++)
            v[u] = q + u < q1 ? load_once(reinterpret_cast<const V *>(piece(q + u))) : V{};
#pragma unroll
        for (int u = 0; u < 8; u++)
#pragma unroll
            for (int k = 0; k < kEach; k++)
                comp_add(hi.v[k], lo.v[k], v[u].v[k]);
    }
    if (group) {
        part[group - 1][0][comp][lane] = hi;
        part[group - 1][1][comp][lane] = lo;
    }
    __syncthreads();
    if (group == 0) {
#pragma unroll
        for (int q = 0; q < kGroups - 1; q++)
#pragma unroll
            for (int k = 0; k < kEach; k++) {
                comp_add(hi.v[k], lo.v[k], part[q][0][comp][lane].v[k]);
                lo.v[k] += part[q][1][comp][lane].v[k];
            }
        if (!final) {
            *carry(0) = hi;
            *carry(1) = lo;
        }
#pragma unroll
        for (int k = 0; k < kEach; k++)
            out[comp][lane].v[k] = round_force(hi.v[k], lo.v[k]);
    }
    if (!final)
        return;
    __syncthreads();
    if (writes) {
        const float fx = out[0][tid / kEach].v[tid % kEach];
        const float fy = out[1][tid / kEach].v[tid % kEach];
        const float fz = out[2][tid / kEach].v[tid % kEach];
        R.force[ib] = make_float4(fx, fy, fz, 0.f);
        if (R.fi.vel) {
            const float4 pos = P.src.pm[ib], vel = R.fi.vel[ib];
            fused_integrate(R.fi, ib, vel, pos.x, pos.y, pos.z, pos.w, fx, fy, fz);
        }
    }
}

// Cost of a step: both ways against one-sided (measured 4 : 3); a stretch has
// at least kMinCost (no stretch is empty, and few pieces at small N), a part
// of a meeting at least kMinPartSteps steps.
constexpr int kCostBoth = 4, kCostOne = 3, kMinCost = 32, kMinPartSteps = 4;
constexpr int kShortSteps = 64;  // 256 sources
constexpr size_t kLoneSmem = 120 * 1024;  // one CTA an SM

template <class G>
static int sets_of(size_t n) { return (int)((n + G::kSet - 1) / G::kSet); }
template <class G>
static int rows_of(size_t n) { return (int)((n + G::kRow - 1) / G::kRow); }

// Cost of the rows before b, from row 0 (meetings x 32 steps).
template <class G>
static long long cost_before(int b, int nsets) {
    return 32 * (kCostBoth * meetings_before<G>(b, nsets) -
                 (long long)(kCostBoth - kCostOne) * std::min((long long)G::kRowSets * b,
                                                              (long long)nsets));
}

// Late stretches.  Of the CTAs that share an SM one runs ahead of the other
// (the scheduler's choice; with equal stretches the SMs held 6.2 of 8 warps on
// average), and the one left runs alone at four fifths of their rate.  So where
// there is enough work the resident CTAs' stretches are 92 % of it, and as
// many short ones start as the first of them end.  N = 131,072, mixed and
// equal masses: all of it at once 4,424 and 4,037 us; 96 % 4,340, 3,920;
// 94 % 4,297, 3,879; 92 % 4,256, 3,884; 90 % 4,266, 3,893; 88 % 4,275, 4,116;
// two or three equal stretches a CTA 4,351, 3,973 and 4,329, 3,957; a third
// wave 4,267, 3,890.  40,000 bodies 429 -> 415 us, 24,576 167.2 -> 165.8, but
// 20,000 115.7 -> 117.6: the line is at 240 steps a CTA (about 24,000 bodies).
constexpr int kLateSteps = 240;

// Cost of the first c of ncta stretches, the first `slots` of them resident.
static long long stretch_cost(long long total, int c, int ncta, int slots) {
    if (ncta <= slots)
        return total * c / ncta;
    const long long early = total * 23 / 25;
    return c <= slots ? early * c / slots
                      : early + (total - early) * (c - slots) / (ncta - slots);
}

// First steps of ncta stretches over rows row0..row1-1, and the end.  parts >
// 0: every meeting is cut into that many stretches of its own.
template <class G>
static void cut_steps(int row0, int row1, int nsets, int ncta, int slots, int parts,
                      unsigned *step) {
    const unsigned end = (unsigned)((meetings_before<G>(row1, nsets) -
                                     meetings_before<G>(row0, nsets))
                                    << 5);
    if (parts > 0) {
        for (int c = 0; c <= ncta; c++)
            step[c] = (unsigned)(c / parts * 32 + c % parts * 32 / parts);
        return;
    }
    const long long c0 = cost_before<G>(row0, nsets), total = cost_before<G>(row1, nsets) - c0;
    int row = row0;
    long long steps = 0;                          // before the row
    long long begin = 0;                          // the row's first cost
    long long next = cost_before<G>(row + 1, nsets) - c0;
    for (int c = 0; c < ncta; c++) {
        const long long at = stretch_cost(total, c, ncta, slots);
        while (at >= next && row + 1 < row1) {
            steps += 32LL * (nsets - row * G::kRowSets);
            row++;
            begin = next;
            next = cost_before<G>(row + 1, nsets) - c0;
        }
        const long long off = at - begin;
        const long long own = 32LL * kCostOne * std::min(G::kRowSets, nsets - row * G::kRowSets);
        step[c] = (unsigned)(steps + (off <= own ? (off + kCostOne - 1) / kCostOne
                                                 : own / kCostOne +
                                                       (off - own + kCostBoth - 1) / kCostBoth));
    }
    step[ncta] = end;
}

}  // namespace pair

static size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// Reaction pieces of one phase of rows [row0, row1).
template <class G>
static size_t react_bytes(int row0, int row1, int nsets, int ncta) {
    const long long g = pair::meetings_before<G>(row1, nsets) - pair::meetings_before<G>(row0, nsets);
    return (size_t)(g + ncta) * 3 * G::kSet * 4;
}

// Rows of the phase that starts at `row`: as many as fit (0: not even one).
template <class G>
static int phase_end(int row, int rows, int nsets, int ncta, int max_rows, size_t room) {
    int end = row;
    while (end < rows && end - row < max_rows &&
           react_bytes<G>(row, end + 1, nsets, ncta) <= room)
        end++;
    return end;
}

template <class G>
static bool plan_geometry(size_t n, int sms, size_t max_bytes, PairPlan &pl) {
    const int nsets = pair::sets_of<G>(n), rows = pair::rows_of<G>(n);
    // Stretches of equal cost, or, for small n, every meeting in `parts` equal
    // parts of its own, so that no stretch has two pieces.  Estimated in
    // microseconds (narrow rows): a step takes 0.21 where a CTA has its SM to
    // itself and 0.34 for two, a body's target piece 0.05 of the reduction, a
    // second piece of a stretch 1.2.
    const int slots = std::min(sms * G::kCtas, kMaxPairCtas);
    const long long cost = pair::cost_before<G>(rows, nsets);
    const long long meetings = pair::meetings_before<G>(rows, nsets);
    auto estimate = [&](double steps, long long ncta) {
        return steps * (ncta <= sms ? 0.21 : 0.34) + 0.05 * (double)ncta / rows;
    };
    pl.ncta = (int)std::min<long long>(slots, cost / pair::kMinCost);
    double best = estimate((double)cost / pl.ncta / pair::kCostBoth, pl.ncta) + 1.2;
    for (int parts = 1; parts <= 32 / pair::kMinPartSteps && meetings * parts <= slots; parts++) {
        const double t = estimate((32 + parts - 1) / parts, meetings * parts);
        if (rows <= kMaxPairRows && t < best) {
            best = t;
            pl.parts = parts;
        }
    }
    if (pl.parts)
        pl.ncta = (int)meetings * pl.parts;
    // CTAs of this kernel start while the previous one still holds some SMs;
    // more shared memory than two can have keeps them from sharing an SM when
    // there is one for each
    pl.lone = pl.ncta <= sms;
    if (pl.parts) {
        // eight reduction threads a body where it has many pieces (N = 6,000,
        // 31: 16.5 us against 17.5 with four); two bodies a thread where the
        // blocks of one would not be resident together
        pl.groups8 = pl.ncta / rows + rows / 2 >= 28 && rows <= 16;
        pl.each = (long long)nsets * (G::kSet / 32) > sms * (pl.groups8 ? 2LL : 5LL) ? 2 : 1;
    } else {
        // with remainders to add, two bodies a thread throughout, and eight
        // threads for them where few rows share the CTAs' pieces.  us a call,
        // eight and four threads: N = 5,000 15.5, 16.2; 8,192 27.0, 27.5; 9,000
        // 31.4, 31.8; 10,007 (20 rows) 37.5, 37.4; 16,384 81.2, 81.5; 18,000
        // 95.8, 96.2; 20,000 (20 rows) 119.5, 116.8; one body a thread: 16,384
        // 81.2, 82.4, 10,007 37.5, 37.7
        pl.groups8 = rows <= 18;
        pl.each = 2;
    }
    pl.slots = pl.ncta;
    if (!max_bytes && cost >= (long long)slots * pair::kLateSteps * pair::kCostBoth)
        pl.ncta = std::min(2 * slots, kMaxPairCtas);
    // stretches of one-sided steps only hold most of them
    pl.pieces = pl.parts || cost <= (long long)pl.ncta * pair::kShortSteps * pair::kCostOne ? 1 : 2;
    // (a small workspace holds few rows' pieces at a time, which need few
    // places for the targets' sums)
    pl.max_rows = max_bytes ? 64 : kMaxPairRows;
    const size_t tsum = align256((size_t)(std::min(rows, pl.max_rows) + pl.ncta) *
                                 (3 * pl.pieces) * G::kRow * 4);
    const size_t carry = align256((size_t)nsets * G::kSet * 6 * 4);
    const size_t all = align256(react_bytes<G>(0, rows, nsets, pl.ncta));
    // a phase of 256 MiB of pieces is about 16 ms of work; always at least
    // four rows
    size_t room = std::max((size_t)256 << 20, (size_t)4 * (nsets + pl.ncta) * 3 * G::kSet * 4);
    if (max_bytes) {
        if (rows <= pl.max_rows && all + tsum <= max_bytes)
            room = std::min(room, max_bytes - tsum);
        else if (max_bytes > tsum + carry)
            room = std::min(room, (max_bytes - tsum - carry) & ~(size_t)255);
        else
            return false;
    }
    const bool one = rows <= pl.max_rows && all <= room;
    if (!one && (pl.pieces == 1 || phase_end<G>(0, rows, nsets, pl.ncta, pl.max_rows, room) == 0))
        return false;  // (short stretches are few pieces, always one phase)
    pl.react_bytes = one ? all : room;
    pl.off_react = 0;
    pl.off_tsum = align256(pl.react_bytes);
    pl.off_carry = pl.off_tsum + tsum;
    pl.workspace_bytes = pl.off_carry + (one ? 0 : carry);
    return !max_bytes || pl.workspace_bytes <= max_bytes;
}

template <class G>
static cudaError_t launch_reduce(const PairPlan &pl, const pair::ReduceParams &R, int sets,
                                 cudaStream_t st) {
    const unsigned blocks = (unsigned)(sets * (G::kSet / 32 / pl.each));
    if (pl.each == 1)
        return pl.groups8 ? launch_dependent(pair::pair_reduce_kernel<G, 8, 1>, blocks, 768, 0, st, R)
                          : launch_dependent(pair::pair_reduce_kernel<G, 4, 1>, blocks, 384, 0, st, R);
    return pl.groups8 ? launch_dependent(pair::pair_reduce_kernel<G, 8, 2>, blocks, 768, 0, st, R)
                      : launch_dependent(pair::pair_reduce_kernel<G, 4, 2>, blocks, 384, 0, st, R);
}

template <class G>
static int launch_geometry(const PairPlan &pl, float4 *force, const float4 *posMass, float eps2,
                           void *workspace, cudaStream_t st, const FusedIntegrate *fi) {
    static_assert(sizeof(pair::ReduceParams) <= 4096, "kernel parameters");
    const int nsets = pair::sets_of<G>(pl.n), rows = pair::rows_of<G>(pl.n);
    char *ws = (char *)workspace;
    pair::ReduceParams R;
    pair::Params &P = R.p;
    P.src.pm = posMass;
    P.react = (float *)(ws + pl.off_react);
    P.tsum = (float *)(ws + pl.off_tsum);
    P.src.n = (int)pl.n;
    P.nsets = nsets;
    P.src.eps2 = eps2;
    P.src.status = pl.status;
    P.src.short_ok = pair::eps2_short_ok(eps2);
    R.carry = (float *)(ws + pl.off_carry);
    R.npad = (size_t)nsets * G::kSet;
    R.force = force;
    R.fi = fi ? *fi : FusedIntegrate{};
    R.fi.js = nullptr;
    for (P.row0 = 0; P.row0 < rows; P.row0 = P.row1) {
        P.row1 = phase_end<G>(P.row0, rows, nsets, pl.ncta, pl.max_rows, pl.react_bytes);
        if (P.row1 == P.row0)
            return NBGB_ERR_WORKSPACE;
        const long long total =
            pair::cost_before<G>(P.row1, nsets) - pair::cost_before<G>(P.row0, nsets);
        const bool late = total >= (long long)pl.slots * pair::kLateSteps * pair::kCostBoth;
        P.ncta = (int)std::min<long long>(late ? pl.ncta : pl.slots, total / pair::kMinCost);
        P.parts = pl.parts;
        P.pieces = pl.pieces;
        if (pl.parts)
            P.ncta = pl.ncta;
        pair::cut_steps<G>(P.row0, P.row1, nsets, P.ncta, pl.slots, pl.parts, P.step);
        const size_t smem = pl.lone ? pair::kLoneSmem : G::kSmem;
        if (launch_dependent(pair::pair_kernel<G>, P.ncta, G::kThreads, smem, st, P) !=
                cudaSuccess ||
            launch_reduce<G>(pl, R, nsets - P.row0 * G::kRowSets, st) != cudaSuccess)
            return NBGB_ERR_CUDA;
    }
    return NBGB_OK;
}

template <class G>
static int launches_geometry(const PairPlan &pl) {
    const int nsets = pair::sets_of<G>(pl.n), rows = pair::rows_of<G>(pl.n);
    int k = 0;
    for (int row = 0; row < rows; k++) {
        const int end = phase_end<G>(row, rows, nsets, pl.ncta, pl.max_rows, pl.react_bytes);
        if (end == row)
            break;
        row = end;
    }
    return 2 * k;
}

template <class G>
static cudaError_t prepare_geometry() {
    return cudaFuncSetAttribute(pair::pair_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)std::max(G::kSmem, pair::kLoneSmem));
}

bool plan_pair(size_t n, int sms, size_t max_bytes, PairPlan &pl) {
    if (n == 0 || n > kMaxBodies || sms <= 0)
        return false;
    pl = PairPlan{};
    pl.n = n;
    pl.narrow = n < kNarrowBelow;
    return pl.narrow ? plan_geometry<pair::Narrow>(n, sms, max_bytes, pl)
                     : plan_geometry<pair::Wide>(n, sms, max_bytes, pl);
}

int launch_pair(const PairPlan &pl, float4 *force, const float4 *posMass, float eps2,
                void *workspace, cudaStream_t st, const FusedIntegrate *fi) {
    return pl.narrow
               ? launch_geometry<pair::Narrow>(pl, force, posMass, eps2, workspace, st, fi)
               : launch_geometry<pair::Wide>(pl, force, posMass, eps2, workspace, st, fi);
}

int pair_launches(const PairPlan &pl) {
    return pl.narrow ? launches_geometry<pair::Narrow>(pl) : launches_geometry<pair::Wide>(pl);
}

int pair_prepare() {
    return prepare_geometry<pair::Narrow>() == cudaSuccess &&
                   prepare_geometry<pair::Wide>() == cudaSuccess
               ? NBGB_OK
               : NBGB_ERR_CUDA;
}

}  // namespace nbgb
