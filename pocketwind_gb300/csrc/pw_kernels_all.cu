// One launch per step of the fast build: blocks by role (aa_step_all).
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
template <int ST, int OP, bool LES, bool ODD>
__device__ __noinline__ void edge_role(const StepParams &p, const uint32_t *list, uint32_t count, uint32_t b) {
  edge_block<ST, OP, LES, ODD>(p, list, count, b, threadIdx.x + BX * threadIdx.y);
}
template <int ST, int OP, bool LES, bool ODD>
__device__ __noinline__ void floor_role(const StepParams &p, uint32_t x, uint32_t y) {
  floor_thread<ST, OP, LES, ODD>(p, x, y);
}
template <int ST, int OP, bool LES, bool PAIRS>
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
// 12.8 us, 128x64x64 23.4 and 15.2 us (FP32, vehicle), 96x48x48 27.5 and 16.9 us,
// 256x128x128 73.9 and 71.5 us (FP16, vehicle).
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
      edge_role<ST, OP, LES, ODD>(p, list, count, b);
      return;
    }
    b -= s.edge;
    if constexpr (FORM == PAIRS) {
      if (b < s.floor) {
        floor_role<ST, OP, LES, ODD>(p, (b % gridDim.x) * (2 * BX) + 2u * threadIdx.x,
                                     1u + (b / gridDim.x) * BY + threadIdx.y);
        return;
      }
      b -= s.floor;
    }
    if constexpr (ODD) {
      if (b < s.seam) seam_role<ST, OP, LES, FORM == PAIRS>(p, b);
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

// Blocks per SM.  For the plane's pairs 8 (64 registers, 100 bytes spilled) are 1 to 2%
// slower than 7 and 6 5% slower at 399x200x200.  With 4 to 6 for all, domains below half
// a million cells would gain up to 8% (their edge cells spill less), 256x128x128 lose 5
// to 25%.
constexpr int kPairBlocks = 8, kCellBlocks = 7, kLinearBlocks = 7;

template <int ST, int OP, bool LES, Plain FORM>
void launch4(const StepParams &p, bool odd, const uint32_t *list, uint32_t count, cudaStream_t s, bool early) {
  const bool linear = FORM == LINEAR || FORM == LINEAR_NY_ODD, pairs = FORM == PAIRS;
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
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(gx, gy, p.nz - 2u * off + w.slices);
  cfg.blockDim = dim3(BX, BY);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  constexpr int B = FORM == RUNS ? kCellBlocks : (FORM == PAIRS ? kPairBlocks : kLinearBlocks);
  if (odd) cudaLaunchKernelEx(&cfg, aa_step_all<ST, OP, LES, true, FORM, B>, p, list, count, w);
  else cudaLaunchKernelEx(&cfg, aa_step_all<ST, OP, LES, false, FORM, B>, p, list, count, w);
}

template <int ST, bool LES, Plain FORM>
void launch3(const StepParams &p, int op, bool odd, const uint32_t *list, uint32_t count, cudaStream_t s, bool early) {
  if (op == OP_REG) launch4<ST, OP_REG, LES, FORM>(p, odd, list, count, s, early);
  else launch4<ST, OP_TRT, LES, FORM>(p, odd, list, count, s, early);
}

// 16-bit storage: pairs of a row, or of a plane with nx odd (without LES).
template <int ST>
void launch2(const StepParams &p, int op, int les, bool odd, const uint32_t *list, uint32_t count, cudaStream_t s,
             bool early) {
  if ((p.nx & 1u) == 0u) {
    if (les) launch3<ST, true, PAIRS>(p, op, odd, list, count, s, early);
    else launch3<ST, false, PAIRS>(p, op, odd, list, count, s, early);
  } else if (p.ny & 1u) {
    launch3<ST, false, LINEAR_NY_ODD>(p, op, odd, list, count, s, early);
  } else {
    launch3<ST, false, LINEAR>(p, op, odd, list, count, s, early);
  }
}

}  // namespace

// Whether a domain's steps run in one launch.  Binary32 storage: always (the vehicle
// at 64^2 x 128 23.4 us before and 15.2 now, at 256^2 x 512 795 and 794).  16-bit cell
// pairs: up to 8 M cells (4.2 M: 73.9 us before, 71.5 now; 14 M: 222.8 and 224.9, where
// the side kernels' registers no longer pay), and not beside reflecting seam rows, which
// take one cell a thread.  16-bit storage with nx odd: any size without LES (203x101x67:
// 35.0 and 24.4, 399x200x200: 308 and 266); with LES the seam rows' rounding depends on the kernel around them.
// The side blocks take at most five slices a plane, and a grid has 65,535.
bool step_all_supported(uint32_t nx, uint32_t ny, uint32_t nz, int storage, int les, uint32_t slip) {
  if (nx < 3u || ny < 3u || nz < 3u || nz > 8192u) return false;
  if (storage == STORE_F32) return true;
  if (nx & 1u) return !les && (uint64_t)nx * ny < (1ull << 31) - 2048u;
  return slip == 0u && (uint64_t)nx * ny * nz <= 8ull << 20;
}

void launch_step_all(const StepParams &p, int storage, int op, int les, bool odd, const uint32_t *list, uint32_t count,
                     cudaStream_t s, bool early) {
  if (storage == STORE_F16) launch2<STORE_F16>(p, op, les, odd, list, count, s, early);
  else if (storage == STORE_BF16) launch2<STORE_BF16>(p, op, les, odd, list, count, s, early);
  else if (les) launch3<STORE_F32, true, RUNS>(p, op, odd, list, count, s, early);
  else launch3<STORE_F32, false, RUNS>(p, op, odd, list, count, s, early);
}

}  // namespace pwall
