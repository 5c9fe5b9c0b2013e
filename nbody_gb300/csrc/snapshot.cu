// snapshot.cu -- device state to host arrays, and back.
//
// What bounds a download of a few thousand bodies is the number of its
// copies: one into pageable memory holds the host for 8 to 15 us, a system's
// FP64 state was six of them or more, the status words three, and the
// components were put side by side on the host.  Here a kernel writes the
// arrays in their final order.  Small ones go, with the status words, into
// pinned memory, from where the host copies them on; with more, that second
// copy (13 GB/s into fresh pages) costs more than the calls, and the arrays
// are put in order in device memory, a chunk at a time, and copied straight
// to the caller's.  Uploads go the same way back.
//
// One slot of an ensemble (FP64 state and accelerations): 1,000 bodies 80 ->
// 27 us, 8,192: 117 -> 51, 25,000: 177 -> 58, 65,536: 1,900 -> 71 into
// resident arrays and 324 into fresh ones.  A reference system's float4 state: 1,000 bodies 57 -> 19 us,
// 8,192: 64 -> 32, 65,536: 105 -> 48; synchronise 29 -> 11 us.
// Admission of one system: 1,000 bodies 80 -> 25 us, 65,536: 365 -> 71; FP64
// state into a system of 262,144 bodies: 1,870 -> 264 us.
#include "nbgb_snapshot.h"

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cerrno>
#include <cstdint>
#include <cstring>

#include "nbody_gb300.h"

namespace nbgb {
namespace {

// Jobs up to this size go through pinned memory: 512 KiB of an ensemble's
// slot take 51 us there and 46 through device memory, 256 KiB 35 and 40.
constexpr size_t kPinned = 512 << 10;
constexpr size_t kScratch = 8 << 20;   // device memory for arrays put in order
constexpr size_t kBodyBytes = 64;      // the most a body takes (FP64 state and acceleration)
constexpr size_t kOrderedBytes = 56;   // ... of it put in order, 8-byte multiple

struct ChunkParams {
    const float4 *vec[2];
    float4 *out[2];
    const double *x64;
    size_t ld;
    double *pos3, *vel3;
    const float *mass;
    float4 *velinv;
    size_t count;
    const unsigned *status[3];
    unsigned *bits;  // null: no status yet
};

__global__ void __launch_bounds__(256) snapshot_kernel(const __grid_constant__ ChunkParams P) {
    const size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (P.x64 && o < 3 * P.count) {
        const size_t i = o / 3, c = o - 3 * i;
        if (P.pos3)
            P.pos3[o] = P.x64[c * P.ld + i];
        if (P.vel3)
            P.vel3[o] = P.x64[(3 + c) * P.ld + i];
    }
    if (o < P.count) {
#pragma unroll
        for (int k = 0; k < 2; k++)
            if (P.out[k])
                P.out[k][o] = P.vec[k][o];
        if (P.velinv) {
            const double *v = P.x64 + 3 * P.ld + o;
            P.velinv[o] = make_float4((float)v[0], (float)v[P.ld], (float)v[2 * P.ld],
                                      __fdiv_rn(1.0f, P.mass[o]));
        }
    }
    if (o == 0 && P.bits) {
        unsigned b = 0;
#pragma unroll
        for (int k = 0; k < 3; k++)
            if (P.status[k])
                b |= *P.status[k];
        *P.bits = b;
    }
}

struct UploadParams {
    const double *pos3, *vel3;
    const float *mass;
    const float4 *posMass, *velInvMass;
    double *x64;
    size_t ld, count, pad;
    float *mass_out;
    float4 *pm;
};

__global__ void __launch_bounds__(256) upload_kernel(const __grid_constant__ UploadParams P) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.count + P.pad)
        return;
    double x[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (i < P.count) {
        float4 pm;
        if (P.pos3) {
#pragma unroll
            for (int c = 0; c < 3; c++) {
                x[c] = P.pos3[3 * i + c];
                x[3 + c] = P.vel3[3 * i + c];
            }
            pm = make_float4((float)x[0], (float)x[1], (float)x[2], P.mass[i]);
        } else {
            pm = P.posMass[i];
            const float4 v = P.velInvMass[i];
            x[0] = pm.x;
            x[1] = pm.y;
            x[2] = pm.z;
            x[3] = v.x;
            x[4] = v.y;
            x[5] = v.z;
        }
        P.mass_out[i] = pm.w;
        if (P.pm)
            P.pm[i] = pm;
    }
#pragma unroll
    for (int c = 0; c < 6; c++)
        P.x64[c * P.ld + i] = x[c];
}

// Have the pages of an array present before the device writes to them: the
// device's first touch of one takes about 1 us, this a tenth.  FP64 state into
// fresh arrays, without and with it: 16,384 bodies 329 and 97 us, 262,144:
// 1,090 and 593, 1,048,576: 22,700 and 2,230; into resident ones 448 and 466.
// Contents stay; where the call is not known, the copy does it all.
void populate(char *dst, size_t bytes) {
#ifdef MADV_POPULATE_WRITE
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    const uintptr_t a = (uintptr_t)dst & ~(page - 1);
    const uintptr_t e = ((uintptr_t)dst + bytes + page - 1) & ~(page - 1);
    const int saved = errno;
    madvise((void *)a, e - a, MADV_POPULATE_WRITE);
    errno = saved;
#else
    (void)dst, (void)bytes;
#endif
}

}  // namespace

int launch_status(const unsigned *const *status, int n, unsigned *out, cudaStream_t st) {
    ChunkParams p = {};
    for (int k = 0; k < n && k < 3; k++)
        p.status[k] = status[k];
    p.bits = out;
    snapshot_kernel<<<1, 32, 0, st>>>(p);
    return cudaGetLastError() == cudaSuccess ? NBGB_OK : NBGB_ERR_CUDA;
}

int Snapshot::create(size_t bodies, const unsigned *const *status, int nstatus) {
    for (int k = 0; k < nstatus && k < 3; k++)
        status_[k] = status[k];
    const size_t job = bodies * kBodyBytes;
    const size_t pinned = std::min(kPinned, (job + 255) / 256 * 256);
    scratch_bytes_ = job > kPinned ? std::min(kScratch, (bodies + 1) * kOrderedBytes) : 0;
    void *p = nullptr;
    if (cudaHostAlloc(&p, 64 + pinned + 64, cudaHostAllocDefault) != cudaSuccess)
        return NBGB_ERR_NO_MEMORY;
    word_ = (unsigned *)p;
    if (scratch_bytes_ && cudaMalloc(&scratch_, scratch_bytes_) != cudaSuccess)
        return NBGB_ERR_NO_MEMORY;
    return NBGB_OK;
}

void Snapshot::destroy() {
    cudaFreeHost(word_);
    cudaFree(scratch_);
    word_ = nullptr;
    scratch_ = nullptr;
}

int Snapshot::run(const SnapshotJob &job, cudaStream_t st, unsigned *bits) {
    std::lock_guard<std::mutex> hold(lock_);
    struct Part {
        char *dst;
        size_t bytes;  // of a body
    };
    const Part part[5] = {{(char *)job.out[0], 16}, {(char *)job.out[1], 16},
                          {(char *)job.velinv, 16}, {(char *)job.pos3, 24},
                          {(char *)job.vel3, 24}};
    size_t body = 0, ordered = 0;
    for (int k = 0; k < 5; k++) {
        body += part[k].dst ? part[k].bytes : 0;
        ordered += part[k].dst && k >= 2 ? part[k].bytes : 0;
    }
    const bool pinned = body * job.n <= kPinned;
    char *const buf = pinned ? (char *)word_ + 64 : (char *)scratch_;
    const int first_part = pinned ? 0 : 2;  // plain arrays need no scratch
    const size_t of_buf = pinned ? body : ordered;
    // (even counts in parts of chunks: every array starts on 16 bytes)
    const size_t room = pinned || !ordered ? job.n : scratch_bytes_ / ordered / 2 * 2;
    const size_t per = std::min(job.n + (job.n & 1), room + (room & 1));
    bool ok = true;
    for (int k = 0; !pinned && k < 5; k++)
        if (part[k].dst)
            populate(part[k].dst, part[k].bytes * job.n);
    if (!pinned)
        for (int k = 0; k < 2; k++)
            if (job.out[k])
                ok = ok && cudaMemcpyAsync(job.out[k], job.vec[k], job.n * 16,
                                           cudaMemcpyDeviceToHost, st) == cudaSuccess;
    if (!of_buf)
        ok = ok && launch_status(status_, 3, word_, st) == NBGB_OK;
    for (size_t first = 0; ok && of_buf && first < job.n; first += per) {
        const size_t count = std::min(per, job.n - first);
        char *at[5], *next = buf;
        for (int k = 0; k < 5; k++) {
            at[k] = part[k].dst && k >= first_part ? next : nullptr;
            next += at[k] ? part[k].bytes * per : 0;
        }
        ChunkParams p = {};
        for (int k = 0; k < 2; k++) {
            p.out[k] = (float4 *)at[k];
            p.vec[k] = job.vec[k];
        }
        p.velinv = (float4 *)at[2];
        p.pos3 = (double *)at[3];
        p.vel3 = (double *)at[4];
        p.x64 = job.x64 ? job.x64 + first : nullptr;
        p.ld = job.ld;
        p.mass = job.mass ? job.mass + first : nullptr;
        p.count = count;
        for (int k = 0; k < 3; k++)
            p.status[k] = status_[k];
        p.bits = first == 0 ? word_ : nullptr;
        const size_t work = p.pos3 || p.vel3 ? 3 * count : count;
        snapshot_kernel<<<(unsigned)((work + 255) / 256), 256, 0, st>>>(p);
        ok = cudaGetLastError() == cudaSuccess;
        for (int k = 2; ok && !pinned && k < 5; k++)
            if (at[k])
                ok = cudaMemcpyAsync(part[k].dst + first * part[k].bytes, at[k],
                                     count * part[k].bytes, cudaMemcpyDeviceToHost,
                                     st) == cudaSuccess;
    }
    // (also after an error: nothing may still write to the buffers)
    if (cudaStreamSynchronize(st) != cudaSuccess || !ok)
        return NBGB_ERR_CUDA;
    if (pinned) {
        const char *src = buf;
        for (const Part &q : part)
            if (q.dst) {
                std::memcpy(q.dst, src, job.n * q.bytes);
                src += q.bytes * per;
            }
    }
    *bits = *(volatile unsigned *)word_;
    return NBGB_OK;
}

int Snapshot::upload(const UploadJob &job, cudaStream_t st) {
    std::lock_guard<std::mutex> hold(lock_);
    struct Part {
        const char *src;
        size_t bytes;  // of a body
    };
    const Part part[5] = {{(const char *)job.posMass, 16}, {(const char *)job.velInvMass, 16},
                          {(const char *)job.pos3, 24}, {(const char *)job.vel3, 24},
                          {(const char *)job.mass, 4}};
    size_t body = 0;
    for (const Part &q : part)
        body += q.src ? q.bytes : 0;
    const bool pinned = body * job.n <= kPinned;
    char *const buf = pinned ? (char *)word_ + 64 : (char *)scratch_;
    const size_t room = pinned ? job.n + (job.n & 1) : scratch_bytes_ / body / 2 * 2;
    const size_t per = std::min(job.n + (job.n & 1), room);
    bool ok = true;
    for (size_t first = 0; ok && first < job.n; first += per) {
        const size_t count = std::min(per, job.n - first);
        char *at[5], *next = buf;
        for (int k = 0; ok && k < 5; k++) {
            at[k] = part[k].src ? next : nullptr;
            if (!at[k])
                continue;
            const char *src = part[k].src + first * part[k].bytes;
            if (pinned)
                std::memcpy(at[k], src, count * part[k].bytes);
            else
                ok = cudaMemcpyAsync(at[k], src, count * part[k].bytes, cudaMemcpyHostToDevice,
                                     st) == cudaSuccess;
            next += part[k].bytes * per;
        }
        if (!ok)
            break;
        UploadParams p = {};
        p.posMass = (const float4 *)at[0];
        p.velInvMass = (const float4 *)at[1];
        p.pos3 = (const double *)at[2];
        p.vel3 = (const double *)at[3];
        p.mass = (const float *)at[4];
        p.x64 = job.x64 + first;
        p.ld = job.ld;
        p.count = count;
        p.pad = first + count == job.n ? job.pad : 0;
        p.mass_out = job.mass_out + first;
        p.pm = job.pm ? job.pm + first : nullptr;
        upload_kernel<<<(unsigned)((count + p.pad + 255) / 256), 256, 0, st>>>(p);
        ok = cudaGetLastError() == cudaSuccess;
    }
    // the caller's arrays and the buffers are free again
    return cudaStreamSynchronize(st) == cudaSuccess && ok ? NBGB_OK : NBGB_ERR_CUDA;
}

}  // namespace nbgb
