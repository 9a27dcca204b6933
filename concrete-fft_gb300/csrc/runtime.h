// runtime.h -- host runtime helpers shared by the CUDA translation units.
#pragma once
#include <cuda_runtime.h>

#include <cstdio>
#include <string>

#include "cfft_internal.h"

#define CFFT_CUDA_TRY(expr)                                                                  \
  do {                                                                                       \
    cudaError_t err__ = (expr);                                                              \
    if (err__ != cudaSuccess) {                                                              \
      ::cfft::set_error(std::string(#expr) + ": " + cudaGetErrorString(err__));              \
      return err__ == cudaErrorMemoryAllocation ? CFFT_ERR_OUT_OF_MEMORY : CFFT_ERR_CUDA;    \
    }                                                                                        \
  } while (0)

#define CFFT_CHECK_LAUNCH()                                                                  \
  do {                                                                                       \
    cudaError_t err__ = cudaGetLastError();                                                  \
    if (err__ != cudaSuccess) {                                                              \
      ::cfft::set_error(std::string("kernel launch: ") + cudaGetErrorString(err__));         \
      return CFFT_ERR_CUDA;                                                                  \
    }                                                                                        \
  } while (0)

namespace cfft {

inline cfft_status fail(cfft_status s, const std::string& msg) {
  set_error(msg);
  return s;
}

// Device-resident copy of a host table.
template <class T>
cfft_status upload(const T* host, size_t count, T** dev) {
  *dev = nullptr;
  if (count == 0) return CFFT_OK;
  CFFT_CUDA_TRY(cudaMalloc((void**)dev, count * sizeof(T)));
  CFFT_CUDA_TRY(cudaMemcpy(*dev, host, count * sizeof(T), cudaMemcpyHostToDevice));
  return CFFT_OK;
}

int sm_count();
// Whether a launch of `ctas` CTAs, whose passes have `butterflies` butterflies each, runs
// them as half butterflies, two threads each, with every addition on the FP64 pipe.  With
// about one warp per SM sub-partition a pass is one warp's dependent chain: halves shorten
// it (one 1024-point forward on Dif4, 4 CTAs: 5.3 us against 7.4 with whole butterflies).
// With more warps the pipes bind, and whole butterflies with most additions on the integer
// pipes win (batch 96: 9.1 us against 9.9; batch 256: 14.8 against 19.4).
inline bool half_butterflies(long ctas, size_t butterflies) {
  return ctas * (long)((butterflies + 31) / 32) * 4 < 5L * 4 * sm_count();
}

// Which instance of a kernel a plan's launch takes: additions on the FP64 pipe (true) or
// most of them on the integer pipes.  int_adds: the plan's cfft_*_set_int_adds, or
// kIntAddsAuto; few: the launch's own choice, as half_butterflies or one like it gives it.
constexpr int kIntAddsAuto = -1;
constexpr int kIntAddsShare = 6;  // eighths that the integer instances move (kAddsBatch)
inline bool fp64_additions(int int_adds, bool few) { return int_adds == kIntAddsAuto ? few : int_adds == 0; }
inline int int_adds_of(int int_adds) { return int_adds == kIntAddsAuto ? kIntAddsShare : int_adds; }

// Launch a kernel through its pointer, raising its dynamic shared-memory limit
// the first time it is used with more than 48 KiB.  `pdl`: programmatic stream
// serialization (the kernel may start while the previous one drains; it must
// call grid_dependency_wait() before its first global access).
cfft_status launch_kernel(const void* fn, int grid, int block, void** args, size_t smem, cudaStream_t stream,
                          bool pdl = false);
// Raises a kernel's dynamic shared-memory limit to `smem` on the current
// device, once (thread-safe); a no-op up to 48 KiB.
cfft_status ensure_smem(const void* fn, size_t smem);
// The same with a thread-block cluster of `cluster` CTAs (grid a multiple of it).
cfft_status launch_kernel_cluster(const void* fn, int grid, int block, int cluster, void** args, size_t smem,
                                  cudaStream_t stream, bool pdl = false);
int max_blocks_per_sm(const void* fn, int block, size_t smem);
// Dynamic shared memory for a launch that spreads a one-wave grid evenly over
// the SMs (ceil(grid / SMs) CTAs per SM); `smem` itself when the grid takes
// several waves, already spreads, or the padded shape would not hold it.
size_t spread_smem(const void* fn, int grid, int block, int cluster, size_t smem);
// Clusters of 9-16 CTAs (non-portable sizes) for fn; launch_kernel_cluster calls it.
cfft_status allow_cluster16(const void* fn);
// Clusters of `cluster` CTAs of fn with this shape resident at once
// (cudaOccupancyMaxActiveClusters, kept per device, kernel and shape).
int cluster_count(const void* fn, int block, int cluster, size_t smem);
// Whether one cluster of `cluster` CTAs of fn with this shape can be resident.
bool cluster_fits(const void* fn, int block, int cluster, size_t smem);
// Clusters of `cluster` CTAs of fn resident at once with one CTA per SM (dynamic
// shared memory padded to the per-block limit).  A 16-CTA cluster needs 16 SMs of
// one GPC: a 152-SM GB300 holds 7 such clusters, and 15 of 8 CTAs.
int spread_clusters(const void* fn, int block, int cluster);

// kernel<<<grid, block, smem, stream>>>(args...) as a programmatic dependent
// launch (the kernel calls grid_dependency_wait() before its first global access).
template <typename... Params, typename... Args>
cudaError_t launch_dependent(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t stream,
                             Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// Persistent scratch for the *_host convenience entry points (one per thread).
cfft_status host_staging(size_t bytes, void** dev_ptr, cudaStream_t* stream);
// Page-locked, device-mapped bounce buffer of the calling thread (at most
// kHostBounceMax bytes) for small host calls on pageable memory: host address
// and the address kernels use.
constexpr size_t kHostBounceMax = size_t(4) << 20;
cfft_status host_bounce(size_t bytes, void** host_ptr, void** dev_ptr);

// Copy/compute pipeline of the *_host product entry points: `nslots` device
// buffers of `bytes` each, one stream per slot (per thread, grown on demand).
struct PipeSlot {
  void* dev;
  cudaStream_t stream;
};
cfft_status host_pipeline(int nslots, size_t bytes, PipeSlot* slots);
// The schedule of the host product entry points' pipeline (cfft_diag_set_host_chunks):
// `chunks` equal chunks on `slots` streams, after a first chunk of `first` products and
// before a last one of `last` (0: none).
struct HostChunks {
  int chunks, slots, first, last;
};
HostChunks host_chunks();

// The device address of `bytes` of page-locked host memory starting at p, or
// nullptr when the range is not one page-locked, device-mapped allocation
// (pageable memory, device memory).  Kernels then write results there
// directly: on a Grace host they cross NVLink-C2C as the kernel stores them.
void* mapped_host_range(const void* p, size_t bytes);
// Stream-ordered workspaces of the product entry points, from a pool of the library's own
// per device.  CUDA's default pool gives its memory back at every synchronisation, so that
// a caller that waits for each product paid a device allocation per call (one launch with a
// 128 KiB workspace, waited for: 114 us, 13 us from this pool).  At most
// kWorkspaceKeep bytes stay in the pool across synchronisations, and none after the last
// product plan is destroyed.  Safe with several streams and threads, and under stream
// capture, as cudaMallocAsync is.  A plan holds a WorkspaceUser; cudaFreeAsync frees.
// Larger batches go through parts of kWorkspaceKeep, so that these do not come from the
// device again each time (a pool of 256 MiB under parts of 1 GiB, waited for: 1000 sums of 4
// terms of N = 32768 7.35 ms, 5.63; 9000 u128 products of N = 4096 15.2 ms, 14.4; 6000 u64
// products of N = 32768, all at once before, 15.0 ms, 12.3.  Parts of 256 MiB
// instead took 5.75 and 14.6 ms, and 2.5% more where nothing waits: 1100 u128 products of
// N = 16384 8.34 ms, 8.13).
constexpr unsigned long long kWorkspaceKeep = 1ull << 30;
// The most for calls that have another route.
constexpr unsigned long long kWorkspaceSmall = 256ull << 20;
struct WorkspaceUser {
  WorkspaceUser();  // makes the pool of the current device, the plan's, if there is none
  ~WorkspaceUser();
  // A failure leaves no CUDA error behind: the caller reports it, or runs kernels that need
  // no workspace, whose launch checks would otherwise find it.
  cudaError_t alloc(void** ptr, size_t bytes, cudaStream_t stream) const;
  cudaMemPool_t pool = nullptr;
  WorkspaceUser(const WorkspaceUser&) = delete;
  WorkspaceUser& operator=(const WorkspaceUser&) = delete;
};
// Whether `stream` is being captured.  A workspace allocated there becomes nodes of the
// graph, and CUDA then allows one instance of it at a time and no child graph of it; a call
// that also has kernels without a workspace takes those, and its graph stays unrestricted.
bool stream_capturing(cudaStream_t stream);
// Input for timing candidates (Method::Measure, the batch tuner): 64-bit words, uniform as
// integers, or doubles uniform in [-scale, scale).  Zeros would not do: the butterflies'
// integer path (int_fp64.cuh) leaves them to the FP64 pipe.
cfft_status fill_timing_words(uint64_t* p, size_t count, cudaStream_t stream);
cfft_status fill_timing_doubles(double* p, size_t count, double scale, cudaStream_t stream);
// Transforms are unnormalised, so repeated in-place calls grow their data.  A timed run of
// `bits` bits of growth per call starts at kTimingScale and lasts at most timing_reps_max
// calls, then the data are filled again.
constexpr double kTimingScale = 0x1p-900;
inline int timing_reps_max(int bits) { return 1800 / (bits < 1 ? 1 : bits); }
// Makes the current device's primary context current on the calling thread.
void bind_device_context();

}  // namespace cfft
