// Internal host-side definitions shared by the C-ABI translation units.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <string>

#include "../../include/pocketwind.h"
#include "pw_common.cuh"

namespace pwhost {

void set_error(const char *fmt, ...);
int cuda_status(cudaError_t e, const char *what);  // PW_ERR_OOM / PW_ERR_CUDA with message

#define PW_TRY(call)                                           \
  do {                                                         \
    cudaError_t e_ = (call);                                   \
    if (e_ != cudaSuccess) return pwhost::cuda_status(e_, #call); \
  } while (0)

void domain_dims(const pw_domain *d, uint32_t *nx, uint32_t *ny, uint32_t *nz);

// Read-only view of a domain's device state for kernels outside pw_domain.cu.
struct DomainView {
  void *f;
  const uint32_t *flags;
  uint32_t nx, ny, nz, stride;
  uint64_t steps;
  int storage;
  cudaStream_t stream;
  uint32_t slip;  // free-slip faces (bit 0 y, bit 1 z)
  int device;     // the device the domain was created on
};
DomainView domain_view(const pw_domain *d);
// Load the allocation-free readout's code and fixed array onto the current
// device and look up the array's address (pw_noalloc.cu).  pw_domain_create
// calls it, so that the readout itself never loads a module later, when the
// device's memory may already be taken.  Failures are left for the readout
// to report.
void noalloc_prepare_device();

// What a batch needs of a member domain (pw_batch.cu).
struct MemberView {
  bool split;                // fast build, one cell per thread (plain kernels + edge list)
  bool one_launch;           // its step is one launch
  bool closure;              // a learned closure is attached
  int storage, op, les;
  uint32_t nx, ny, nz;
  uint64_t steps;
  bool ramping;              // inlet ramp still in progress
  bool interpolated;         // interpolated (Bouzidi) walls
  uint32_t slip;             // free-slip faces (bit 0 y, bit 1 z)
  const uint32_t *edges;
  uint32_t edge_count;
  uint32_t *status;
  cudaStream_t stream;
};
MemberView member_view(const pw_domain *d);
// The step parameters of step `step` (1-based) at the domain's full inlet speed.
pw::StepParams member_params(const pw_domain *d, uint64_t step, int write_macro);
// Queue step `step` of a one-launch domain on its own stream, among other domains'
// steps; write_macro and before_macro as in pw_domain.cu's enqueue_step.
void member_enqueue(pw_domain *d, uint64_t step, int write_macro, bool before_macro, bool cleared);
// Count `n` steps run for the domain by a batch.
void member_advance(pw_domain *d, uint64_t n);

// Device-resident packed geometry (the reference's VoxelGrid).
struct Grid {
  uint32_t nx = 0, ny = 0, nz = 0;
  size_t cells = 0;
  void *cell_arrays = nullptr;    // the allocation of flags and qoff
  void *link_arrays = nullptr;    // the allocation of fractions and boundary
  uint32_t *flags = nullptr;      // cells
  uint32_t *qoff = nullptr;       // cells
  float *fractions = nullptr;     // nfrac
  uint32_t *boundary = nullptr;   // nboundary
  size_t nfrac = 0, nboundary = 0;
  pw_grid_stats stats{};
  ~Grid();
};

// Several device arrays in one allocation (an allocation and its release cost 35 and
// 30 to 100 us each, whatever their size).  want() notes an array, alloc() allocates and
// places them all, each on a 256-byte boundary in the order noted.
struct Arena {
  struct Part {
    void **at;
    size_t bytes, offset;
  };
  Part parts[16];
  int n = 0;
  size_t total = 0;
  void want(void **p, size_t bytes) {
    parts[n++] = Part{p, bytes, total};
    total += ((bytes ? bytes : 16) + 255) / 256 * 256;
  }
  cudaError_t alloc(void **base) {
    const cudaError_t e = cudaMalloc(base, total);
    if (e != cudaSuccess) return e;
    for (int k = 0; k < n; k++) *parts[k].at = static_cast<char *>(*base) + parts[k].offset;
    return cudaSuccess;
  }
};

// Sets the device's stream-ordered pool up, once: before the first domain's memory, so that
// the voxelizer's temporaries do not lie behind it (links of a 150x75x61 grid in a process
// whose domain came first 695 us, and 645 so).
void prepare_pool();

// Pinned host slots of kPinnedSlot bytes for a domain's small results, cut from 4 KB
// slabs (a pinned allocation costs 117 us and its release 168).  A slab goes back when
// its last slot does and another empty one is kept: at most one stays behind.
constexpr size_t kPinnedSlot = 64;
void *pinned_acquire();  // NULL when no pinned memory can be had
void pinned_release(void *slot);

}  // namespace pwhost

struct pw_grid : pwhost::Grid {};
