// nbgb_snapshot.h -- device state to host arrays (snapshot.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>

namespace nbgb {

// What to download: sources of n bodies on the device and the host arrays
// they go to (null: not wanted).
struct SnapshotJob {
    size_t n = 0;
    const float4 *vec[2] = {nullptr, nullptr};  // to out[k], as they are
    float *out[2] = {nullptr, nullptr};
    const double *x64 = nullptr;  // px,py,pz,vx,vy,vz, ld apart, to [n][3]
    size_t ld = 0;
    double *pos3 = nullptr, *vel3 = nullptr;
    const float *mass = nullptr;  // with x64: {(float)v, 1/m} to velinv
    float *velinv = nullptr;
};

// What to upload into FP64 components: n bodies as {pos3, vel3, mass} or as
// {posMass, velInvMass} from the host, to the device arrays.
struct UploadJob {
    size_t n = 0;
    const double *pos3 = nullptr, *vel3 = nullptr;
    const float *mass = nullptr;
    const float *posMass = nullptr, *velInvMass = nullptr;
    double *x64 = nullptr;  // px,py,pz,vx,vy,vz, ld apart
    size_t ld = 0, pad = 0;  // bodies n .. n + pad - 1 become zeros
    float *mass_out = nullptr;
    float4 *pm = nullptr;  // FP32 {x,y,z,m}, if not null
};

// A path between host arrays and device state: pinned memory for small jobs,
// device memory in which larger ones are put in order, and the status words
// of the translation units.  Belongs to one object and its stream; calls from several threads
// take turns.
class Snapshot {
  public:
    // bodies: the most of a job (bounds the buffers of small objects)
    int create(size_t bodies, const unsigned *const *status, int nstatus);
    void destroy();
    // Everything queued on the stream, then the job, then *bits = the status
    // words' OR (not cleared).  Synchronises the stream.
    int run(const SnapshotJob &job, cudaStream_t st, unsigned *bits);
    // Uploads, and synchronises the stream.
    int upload(const UploadJob &job, cudaStream_t st);

  private:
    std::mutex lock_;
    unsigned *word_ = nullptr;  // status, then (64 bytes on) the pinned buffer
    void *scratch_ = nullptr;
    size_t scratch_bytes_ = 0;
    const unsigned *status_[3] = {nullptr, nullptr, nullptr};
};

// status[k], k < n, OR-ed into *out (pinned host memory) on the stream
int launch_status(const unsigned *const *status, int n, unsigned *out, cudaStream_t st);

}  // namespace nbgb
