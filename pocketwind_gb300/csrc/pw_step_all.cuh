// One launch per step of the fast build: blocks by role (aa_step_all).  Included by one
// translation unit per storage type.
#pragma once
#define PW_NS pwall
#define PW_STRICT 0
#include "pw_lbm.cuh"

namespace pwall {

// The blocks of a step that are not the plain kernel's, in the order in which they
// start: edge cells, floor layer, seam rows; they fill the grid's first z slices.
struct SideBlocks {
  uint32_t edge, floor, seam, slices;
};

// The roles beside the plain cells, each a function of its own: inlined into the
// kernel they took registers from the plain path (512x256x256 FP16 2.4% slower), and
// the compiler's choice of which products to fuse in the wall model changed with what
// surrounded it: the stored 16-bit codes with it, and the vehicle's binary32 velocity
// after 1,000 steps from 3e-6 to 3e-5 off the reference's path.
template <int ST, int OP, bool LES, bool ODD, int BLOCKS>
__device__ __noinline__ void edge_role(const StepParams &p, const uint32_t *list, uint32_t count, uint32_t b) {
  edge_block<ST, OP, LES, ODD>(p, list, count, b, threadIdx.x + BX * threadIdx.y);
}
template <int ST, int OP, bool LES, bool ODD, int BLOCKS>
__device__ __noinline__ void floor_role(const StepParams &p, uint32_t x, uint32_t y) {
  floor_thread<ST, OP, LES, ODD>(p, x, y);
}
template <int ST, int OP, bool LES, bool PAIRS, int BLOCKS>
__device__ __noinline__ void seam_role(const StepParams &p, uint32_t b) {
  if constexpr (PAIRS) {
    seam_pair_thread<ST, OP, LES>(p, (b % gridDim.x) * (2 * BX) + 2u * threadIdx.x, (b / gridDim.x) * BY + threadIdx.y);
  } else {
    const uint32_t runs = (p.nx + BX - 1u) / BX, row = (b / runs) * BY + threadIdx.y;
    if (row < seam_rows(p.ny, p.nz)) seam_thread<ST, OP, LES>(p, (b % runs) * BX + threadIdx.x, row);
  }
}

// A whole step in one launch.  The first z slices of the grid hold the edge, floor
// and seam blocks (the long ones start first), the others the plain blocks, each
// the same device code as in a kernel of its own.  The cells of the roles are
// disjoint and in the in-place pattern none reads a slot that another writes within
// the step, so they run in any order.
// A small domain's step is bound by its longest chain of instructions (128 edge
// cells: about 9 us) and by launches: three or four of them, forked to a second
// stream and joined, against one here, whose successor is launched while it runs
// (griddepcontrol).  A step in a run of eight, before and now: 64x32x32 20.4 and
// 12.3 us, 128x64x64 23.4 and 15.0 us (FP32, vehicle), 96x48x48 27.5 and 16.2 us
// (FP16, vehicle).
// The plain cells' form: 64-cell runs of a row as cells x and x + 32 a lane (binary32)
// or as cell pairs (16-bit storage, nx even), or pairs over a plane (16-bit, nx odd).
enum Plain { RUNS, PAIRS, LINEAR, LINEAR_NY_ODD };

template <int ST, int OP, bool LES, bool ODD, Plain FORM, int BLOCKS>
__global__ void __launch_bounds__(NTHREADS, BLOCKS) aa_step_all(const __grid_constant__ StepParams p,
                                                               const uint32_t *list, uint32_t count, SideBlocks s) {
  // the next step's blocks may come as soon as this step's last ones have started;
  // they, as these, touch nothing until the step before has ended
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (blockIdx.z < s.slices) {
    if (p.clear_status && (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x | threadIdx.y) == 0u) *p.status = 0u;
    uint32_t b = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    if (b < s.edge) {
      edge_role<ST, OP, LES, ODD, BLOCKS>(p, list, count, b);
      return;
    }
    b -= s.edge;
    if constexpr (FORM == PAIRS) {
      if (b < s.floor) {
        floor_role<ST, OP, LES, ODD, BLOCKS>(p, (b % gridDim.x) * (2 * BX) + 2u * threadIdx.x,
                                     1u + (b / gridDim.x) * BY + threadIdx.y);
        return;
      }
      b -= s.floor;
    }
    if constexpr (ODD) {
      if (b < s.seam) seam_role<ST, OP, LES, FORM == PAIRS, BLOCKS>(p, b);
    }
    return;
  }
  const uint32_t off = ODD ? 1u : 0u, z = blockIdx.z - s.slices + off;
  if constexpr (FORM == LINEAR || FORM == LINEAR_NY_ODD) {
    // the plane's first pair begins in the plane before when the plane starts at an odd cell
    const uint32_t start = (p.nx * p.ny * z) & 1u;
    const uint32_t t = blockIdx.x * NTHREADS + threadIdx.x + BX * threadIdx.y;
    linear_thread<ST, OP, LES, ODD, FORM == LINEAR_NY_ODD>(p, (int32_t)(2u * t) - (int32_t)start, z);
  } else {
    const uint32_t y = blockIdx.y * BY + threadIdx.y + off;
    if (y + off >= p.ny) return;
    if constexpr (FORM == PAIRS) pair_thread<ST, OP, LES, ODD>(p, blockIdx.x * (2 * BX) + 2u * threadIdx.x, y, z);
    else plain_thread<ST, OP, LES, ODD>(p, blockIdx.x * (2 * BX) + threadIdx.x, y, z);
  }
}

namespace {

// Blocks per SM, and with them the registers a thread may have.  Large domains want many
// blocks for the plain cells' loads (for the plane's pairs 8, 64 registers with 100 bytes
// spilled, are 1 to 2% slower than 7 and 6 5% slower at 399x200x200).  A step of fewer
// than 16 plain blocks per SM takes as long as its slowest edge cells, which spill a
// kilobyte at 64 registers and nothing at 128: four per SM (128x64x64 FP32 vehicle 16.6
// and 15.1 us, FP16 18.5 and 16.7; 136x68x68, 22 blocks per SM, 15.6 and 18.7 for the
// FP32 sphere: the line lies between).  With the wall model or interpolated walls in the
// edge cells six blocks are the better ones a while longer: binary32 up to 32 plain blocks
// per SM (160x80x80 25.9 and 25.0 us, interpolated 24.3 and 23.5; 176x88x88 39.4 and
// 40.2), 16-bit pairs up to 48 (160x80x80 22.9 and 21.7, interpolated 24.3 and 21.4,
// 192x96x96 31.8 and 30.4; 208x104x104 44.5 and 46.3).  Domains stepped side by side
// share the SMs and keep the form for large ones.
constexpr int kPairBlocks = 8, kCellBlocks = 7, kLinearBlocks = 7, kFewBlocks = 4, kMidBlocks = 6;
constexpr uint32_t kFewPerSm = 16, kMidPerSmRuns = 32, kMidPerSmPairs = 48;

template <int ST, int OP, bool LES, Plain FORM, int BLOCKS>
void launch_grid(const StepParams &p, bool odd, const uint32_t *list, uint32_t count, const SideBlocks &w, dim3 grid,
                 cudaStream_t s, bool early) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(BX, BY);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  if (odd) cudaLaunchKernelEx(&cfg, aa_step_all<ST, OP, LES, true, FORM, BLOCKS>, p, list, count, w);
  else cudaLaunchKernelEx(&cfg, aa_step_all<ST, OP, LES, false, FORM, BLOCKS>, p, list, count, w);
}

template <int ST, int OP, bool LES, Plain FORM>
void launch4(const StepParams &p, bool odd, const uint32_t *list, uint32_t count, cudaStream_t s, bool early) {
  constexpr bool linear = FORM == LINEAR || FORM == LINEAR_NY_ODD, pairs = FORM == PAIRS;
  const uint32_t off = odd ? 1u : 0u, runs = (p.nx + 2u * BX - 1u) / (2u * BX);
  // pairs of a plane, one more when it starts at an odd cell
  const uint32_t gx = linear ? ((p.nx * p.ny + 2u) / 2u + NTHREADS - 1u) / NTHREADS : runs;
  const uint32_t gy = linear ? 1u : (p.ny - 2u * off + BY - 1u) / BY;
  SideBlocks w{};
  w.edge = (count + NTHREADS - 1u) / NTHREADS;
  if (pairs && p.floor_rows) w.floor = runs * ((p.ny - 2u + BY - 1u) / BY);
  if (odd) w.seam = (pairs ? runs : (p.nx + BX - 1u) / BX) * ((seam_rows(p.ny, p.nz) + BY - 1u) / BY);
  const uint32_t slice = gx * gy;
  w.slices = (w.edge + w.floor + w.seam + slice - 1u) / slice;
  if (p.clear_status && w.slices == 0u) w.slices = 1u;  // its first thread clears the flag
  const dim3 grid(gx, gy, p.nz - 2u * off + w.slices);
  constexpr int kMany = FORM == RUNS ? kCellBlocks : (pairs ? kPairBlocks : kLinearBlocks);
  const uint64_t per_sm = (uint64_t)slice * (p.nz - 2u * off) / pwhost::multiprocessors();
  if (early && per_sm < kFewPerSm) {
    launch_grid<ST, OP, LES, FORM, kFewBlocks>(p, odd, list, count, w, grid, s, early);
    return;
  }
  if constexpr (!linear) {
    if (early && (LES || p.hist) && per_sm < (pairs ? kMidPerSmPairs : kMidPerSmRuns)) {
      launch_grid<ST, OP, LES, FORM, kMidBlocks>(p, odd, list, count, w, grid, s, early);
      return;
    }
  }
  launch_grid<ST, OP, LES, FORM, kMany>(p, odd, list, count, w, grid, s, early);
}

template <int ST, bool LES, Plain FORM>
void launch3(const StepParams &p, int op, bool odd, const uint32_t *list, uint32_t count, cudaStream_t s, bool early) {
  if (op == OP_REG) launch4<ST, OP_REG, LES, FORM>(p, odd, list, count, s, early);
  else launch4<ST, OP_TRT, LES, FORM>(p, odd, list, count, s, early);
}

// The pairs of a plane with LES, the operators that step_all_supported admits.
template <int ST, Plain FORM>
void launch_linear_les(const StepParams &p, int op, bool odd, const uint32_t *list, uint32_t count, cudaStream_t s,
                       bool early) {
  if constexpr (ST == STORE_F16) launch4<ST, OP_REG, true, FORM>(p, odd, list, count, s, early);
  else launch3<ST, true, FORM>(p, op, odd, list, count, s, early);
}

}  // namespace

// The step of one storage type; 16-bit: pairs of a row, or of a plane with nx odd.
template <int ST>
void launch_storage(const StepParams &p, int op, int les, bool odd, const uint32_t *list, uint32_t count,
                    cudaStream_t s, bool early) {
  if constexpr (ST == STORE_F32) {
    if (les) launch3<ST, true, RUNS>(p, op, odd, list, count, s, early);
    else launch3<ST, false, RUNS>(p, op, odd, list, count, s, early);
  } else if ((p.nx & 1u) == 0u) {
    if (les) launch3<ST, true, PAIRS>(p, op, odd, list, count, s, early);
    else launch3<ST, false, PAIRS>(p, op, odd, list, count, s, early);
  } else if (p.ny & 1u) {
    if (!les) launch3<ST, false, LINEAR_NY_ODD>(p, op, odd, list, count, s, early);
    else launch_linear_les<ST, LINEAR_NY_ODD>(p, op, odd, list, count, s, early);
  } else {
    if (!les) launch3<ST, false, LINEAR>(p, op, odd, list, count, s, early);
    else launch_linear_les<ST, LINEAR>(p, op, odd, list, count, s, early);
  }
}

}  // namespace pwall
