// The learned subgrid closure (pw_closure_*): training data from the solver's
// own fine-grid fields, hand-written training (forward, backward, Adam), and
// inference fused into a step kernel on the tensor cores.  No counterpart in
// the reference.
//
// Data: a fine run's macros are box-filtered 2x2x2 onto the coarse grid; the
// target is the eddy viscosity that best reproduces the subgrid stress of the
// filtered fields, nu* = max(0, -tau_sgs : S / (2 S : S)), with
// tau_sgs = mean((u - ubar)(u - ubar)) and S the finite-difference strain of the
// filtered velocity, expressed as c* = nu* / nu_smag - 1 (clipped to [-1, 3]),
// nu_smag = (0.1)^2 |S| the Smagorinsky viscosity of the same strain.  Cells
// within two coarse cells of a wall or of the x faces are left out (the wall
// model owns the wall cells).
//
// Inference, periodic faces (closure_pairs): the plain step's two-cell update
// (update_fast2) with a hook between the Smagorinsky relaxation time and the
// reconstruction.  Each thread takes cells x and x + 32 of a row, a block the
// 256 cells of four rows; the hook takes each plain LES cell's strain
// S = -3 Pi_neq / (2 rho tau_s) and its nine inputs, and the block runs the
// network for its cells on the 5th-generation tensor cores as two tiles of
// M = 128 cells: each layer is one tcgen05.mma per tile of N = 32 outputs
// (K = 16 inputs, or two of K = 16 hidden units), bf16 operands in shared
// memory, binary32 accumulators in tensor memory, issued by one thread and
// read back by every thread for its own cells (tcgen05.ld); the update then
// goes on with tau = tau0 + (tau_s - tau0) max(0, 1 + c).  The wall-link cells
// and the floor layer run in blocks of their own in the same launch with plain
// Smagorinsky and the reference's wall model, as in a step without the closure.
// Free-slip faces (closure_step): one cell per thread over every cell, 128
// cells per block, the same network on one tile; for the regularized operator
// the first pass's Smagorinsky post-collision state is corrected in place
// (finish_plain_reg), for TRT the cell goes through the one-cell path again.
#define PW_NS pwclosure
#define PW_STRICT 0
#include <algorithm>
#include <cmath>
#include <vector>

#include "pw_internal.h"
#include "pw_lbm.cuh"
#include "pw_closure.cuh"
#include "pw_launch.h"

using namespace pwhost;
using pw::StepParams;
using namespace pwcl;

namespace {

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t *>(&v);
}

// ---------------------------------------------------------------- tensor-core operands
// K-major operands without swizzle: 8-row x 16-byte core matrices, element
// (row r, k) at byte (r % 8) * 16 + (r / 8) * SBO + (k / 8) * LBO + (k % 8) * 2
// (LBO: the next 8 elements of K; SBO: the next 8 rows).
constexpr uint32_t kLbo = 128;
__host__ __device__ constexpr uint32_t cm_offset(uint32_t r, uint32_t k, uint32_t sbo) {
  return (r & 7u) * 16u + (r >> 3) * sbo + (k >> 3) * kLbo + (k & 7u) * 2u;
}
constexpr uint32_t kSbo1 = 2 * kLbo, kSbo2 = 4 * kLbo;  // K = 16 (layer 1), K = 32 (layer 2)
// The network's image in global memory, copied to shared memory by each block:
// W1 (32 x 16, inputs 9..15 zero) and W2 (32 x 32) as bf16 operands, then b1,
// b2, W3 (bf16-rounded) and b3 as binary32.
constexpr uint32_t kImgW1 = 0, kImgW2 = 1024, kImgB1 = 3072, kImgB2 = kImgB1 + 128, kImgW3 = kImgB2 + 128,
                   kImgB3 = kImgW3 + 128, kImgBytes = kImgB3 + 16;
constexpr uint32_t kFragWords = 48;  // the image's buffer: 32 x 48 words (>= kImgBytes / 4)
static_assert(kImgBytes <= 4 * 32 * kFragWords, "network image does not fit its buffer");

__global__ void build_fragments(const float *w, uint32_t *frag) {
  unsigned char *img = reinterpret_cast<unsigned char *>(frag);
  for (uint32_t i = threadIdx.x; i < 32u * 16u; i += blockDim.x) {
    const uint32_t n = i >> 4, k = i & 15u;
    const float v = k < (uint32_t)kIn ? w[kW1 + n * kIn + k] : 0.0f;
    *reinterpret_cast<__nv_bfloat16 *>(img + kImgW1 + cm_offset(n, k, kSbo1)) = __float2bfloat16_rn(v);
  }
  for (uint32_t i = threadIdx.x; i < 32u * 32u; i += blockDim.x) {
    const uint32_t n = i >> 5, k = i & 31u;
    *reinterpret_cast<__nv_bfloat16 *>(img + kImgW2 + cm_offset(n, k, kSbo2)) =
        __float2bfloat16_rn(w[kW2 + n * kHidden + k]);
  }
  for (uint32_t j = threadIdx.x; j < 32u; j += blockDim.x) {
    reinterpret_cast<float *>(img + kImgB1)[j] = w[kB1 + j];
    reinterpret_cast<float *>(img + kImgB2)[j] = w[kB2 + j];
    reinterpret_cast<float *>(img + kImgW3)[j] = bf16_round(w[kW3 + j]);
  }
  if (threadIdx.x == 0) reinterpret_cast<float *>(img + kImgB3)[0] = w[kB3];
}

// tcgen05 instruction descriptor (kind::f16): binary32 accumulator, bf16 A and
// B, both K-major, N = 32, M = 128.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((32u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ uint32_t smem_u32(const void *ptr) { return (uint32_t)__cvta_generic_to_shared(ptr); }
// Shared-memory matrix descriptor: start, LBO, SBO (each in 16-byte units),
// the fixed version 1 at bit 46, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3fffu) | ((uint64_t)((kLbo >> 4) & 0x3fffu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3fffu) << 32) | ((uint64_t)1 << 46);
}
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
          tmem_d),
      "l"(adesc), "l"(bdesc), "r"(kIdesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tc_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 8 binary32 columns from column col of this thread's TMEM lane (warp w reads
// lanes 32w..32w+31), waited for.
__device__ __forceinline__ void tc_load8(uint32_t taddr, float *v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 8; j++) v[j] = __uint_as_float(r[j]);
}

// Shared state of a block's network evaluation.
struct TcShared {
  __align__(128) unsigned char img[kImgBytes];   // the network image
  __align__(128) unsigned char a1[128 * 32];     // layer-1 operand: 128 cells x 16 inputs, bf16
  __align__(128) unsigned char a2[128 * 64];     // layer-2 operand: 128 cells x 32 hidden units, bf16
  __align__(8) uint64_t bar;                     // MMA completion
  uint32_t tmem;                                 // base of the block's 64 TMEM columns
  uint32_t failed;                               // a completion wait ran out
};

// Bounded wait on the MMA barrier's phase `parity`; false when it ran out
// (the caller then skips the network and keeps plain Smagorinsky, c = 0).
// Before returning false it waits once more, also bounded, so that an MMA
// still in flight can finish before its operands or columns are reused.
__device__ __forceinline__ bool tc_wait_once(uint64_t *bar, uint32_t parity) {
  for (uint32_t it = 0; it < (1u << 22); it++) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok)
                 : "r"(smem_u32(bar)), "r"(parity)
                 : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __noinline__ void tc_drain(uint64_t *bar, uint32_t parity) { tc_wait_once(bar, parity); }
__device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t parity) {
  if (tc_wait_once(bar, parity)) return true;
  tc_drain(bar, parity);  // out of line: the kernels' code stays small for the instruction cache
  return false;
}

// Block start: copy the image, set up the barrier, allocate 64 TMEM columns
// (warp 0).  All 128 threads call it.
template <class Sh>
__device__ void tc_setup(Sh &sh, const uint32_t *frag) {
  const uint32_t tid = threadIdx.x + 32u * threadIdx.y;
  const uint32_t *src = frag;
  uint32_t *dst = reinterpret_cast<uint32_t *>(sh.img);
  for (uint32_t i = tid; i < kImgBytes / 4u; i += 128u) dst[i] = __ldg(&src[i]);
  if (tid == 0) {
    sh.failed = 0u;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh.bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 32u) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 64;" ::"r"(smem_u32(&sh.tmem))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
}

// Block end: free the TMEM columns (warp 0), after every thread's last read.
template <class Sh>
__device__ void tc_teardown(Sh &sh) {
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  if (threadIdx.x + 32u * threadIdx.y < 32u)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 64;" ::"r"(sh.tmem) : "memory");
}

// The network on the block's 128 cells: every thread passes its cell's inputs
// x (zeros for cells without a closure) and gets its c.  `phase` counts the
// barrier's completions (two per call).  Rounding as forward_scalar: inputs,
// weights and hidden activations in bf16, binary32 accumulation.
__device__ float block_mlp(TcShared &sh, const float x[kIn], uint32_t &phase) {
  const uint32_t tid = threadIdx.x + 32u * threadIdx.y, warp = tid >> 5;
  const uint32_t lane_addr = sh.tmem + ((warp * 32u) << 16);
  // layer-1 operand row: inputs 0..7 and 8..15 (9..15 zero) as two 16-byte pieces
  {
    uint4 lo, hi;
    lo.x = pack_bf16(x[0], x[1]); lo.y = pack_bf16(x[2], x[3]); lo.z = pack_bf16(x[4], x[5]);
    lo.w = pack_bf16(x[6], x[7]);
    hi.x = pack_bf16(x[8], 0.0f); hi.y = 0u; hi.z = 0u; hi.w = 0u;
    *reinterpret_cast<uint4 *>(sh.a1 + cm_offset(tid, 0, kSbo1)) = lo;
    *reinterpret_cast<uint4 *>(sh.a1 + cm_offset(tid, 8, kSbo1)) = hi;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  const bool live = sh.failed == 0u;
  if (tid == 0 && live) {
    tc_mma(sh.tmem, smem_desc(smem_u32(sh.a1), kSbo1), smem_desc(smem_u32(sh.img + kImgW1), kSbo1), 0u);
    tc_commit(&sh.bar);
  }
  // each warp reads TMEM only when all its lanes saw the layer complete
  const bool done1 = __all_sync(0xffffffffu, live && tc_wait(&sh.bar, phase & 1u));
  phase++;
  tc_after_sync();
  if (!done1 && live) atomicOr(&sh.failed, 1u);
  const float *b1 = reinterpret_cast<const float *>(sh.img + kImgB1);
#pragma unroll
  for (int k = 0; k < 32; k += 8) {  // eight columns at a time: fewer live registers
    float h[8];
    if (done1) {
      tc_load8(lane_addr + (uint32_t)k, h);
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) h[j] = 0.0f;
    }
    uint4 v;
    v.x = pack_bf16(tanh_fast(h[0] + b1[k]), tanh_fast(h[1] + b1[k + 1]));
    v.y = pack_bf16(tanh_fast(h[2] + b1[k + 2]), tanh_fast(h[3] + b1[k + 3]));
    v.z = pack_bf16(tanh_fast(h[4] + b1[k + 4]), tanh_fast(h[5] + b1[k + 5]));
    v.w = pack_bf16(tanh_fast(h[6] + b1[k + 6]), tanh_fast(h[7] + b1[k + 7]));
    *reinterpret_cast<uint4 *>(sh.a2 + cm_offset(tid, k, kSbo2)) = v;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  const bool live2 = sh.failed == 0u;
  if (tid == 0 && live2) {
    const uint32_t a2 = smem_u32(sh.a2), w2 = smem_u32(sh.img + kImgW2);
    tc_mma(sh.tmem + 32u, smem_desc(a2, kSbo2), smem_desc(w2, kSbo2), 0u);
    tc_mma(sh.tmem + 32u, smem_desc(a2 + 2u * kLbo, kSbo2), smem_desc(w2 + 2u * kLbo, kSbo2), 1u);
    tc_commit(&sh.bar);
  }
  const bool done2 = __all_sync(0xffffffffu, live2 && tc_wait(&sh.bar, phase & 1u));
  phase++;
  tc_after_sync();
  if (!done2) {
    if (live2) atomicOr(&sh.failed, 1u);
    return 0.0f;
  }
  const float *b2 = reinterpret_cast<const float *>(sh.img + kImgB2);
  const float *w3 = reinterpret_cast<const float *>(sh.img + kImgW3);
  float out = 0.0f;
#pragma unroll
  for (int k = 0; k < 32; k += 8) {
    float h[8];
    tc_load8(lane_addr + 32u + (uint32_t)k, h);
#pragma unroll
    for (int j = 0; j < 8; j++) out = fmaf(w3[k + j], bf16_round(tanh_fast(h[j] + b2[k + j])), out);
  }
  return out + reinterpret_cast<const float *>(sh.img + kImgB3)[0];
}

// Records the Smagorinsky state of a cell (first pass).
struct CaptureHook {
  float *s;  // tau_s, rho, ux, uy, uz, pxx, pyy, pzz, pxy, pxz, pyz
  __device__ __forceinline__ float operator()(const StepParams &, float tau_s, float rho, float vx, float vy, float vz,
                                              float pxx, float pyy, float pzz, float pxy, float pxz,
                                              float pyz) const {
    s[0] = tau_s; s[1] = rho; s[2] = vx; s[3] = vy; s[4] = vz;
    s[5] = pxx; s[6] = pyy; s[7] = pzz; s[8] = pxy; s[9] = pxz; s[10] = pyz;
    return tau_s;
  }
};

// Scales the Smagorinsky eddy viscosity by max(0, 1 + c) (second pass).
struct ClosureHook {
  float c;
  __device__ __forceinline__ float operator()(const StepParams &p, float tau_s, float, float, float, float, float,
                                              float, float, float, float, float) const {
    return p.tau0 + (tau_s - p.tau0) * fmaxf(0.0f, 1.0f + c);
  }
};

// Inputs of a cell from its Smagorinsky state (strain from the stress).
__device__ __forceinline__ void cell_inputs(const StepParams &p, const float *st, float wall, float x[kIn]) {
  const float tau_s = st[0], rho = st[1];
  const float k = -1.5f / (rho * tau_s);  // S = -Pi / (2 rho c_s^2 tau), c_s^2 = 1/3
  const float s[6] = {k * st[5], k * st[6], k * st[7], k * st[8], k * st[9], k * st[10]};
  const float nu_s = (tau_s - p.tau0) * (1.0f / 3.0f);
  features(s, rho, st[2], st[3], st[4], wall, p.nu, nu_s, p.u_in, x);
}

// REG collision of a plain cell with the closure's relaxation time, from its
// Smagorinsky post-collision state post (first pass): in the regularized
// operator the relaxation time enters only through (1 - omega) 4.5 w_i Q_i:Pi,
// so the closure's state is post_i + 4.5 (omega_s - omega) w_i Q_i:Pi (Q_i:Pi
// with the trace removed, as update_fast projects it).  Then the cell's
// rounding, stores, macros and outlet plane, as general_cell ends.
template <int ST, bool ODD>
__device__ __forceinline__ void finish_plain_reg(const StepParams &p, uint32_t x, uint32_t y, uint32_t z, uint32_t n,
                                                 const float *st, float c, float *post, bool interior) {
  using S = pw::Store<ST>;
  using T = typename S::T;
  const float tau_s = st[0];
  const float tau = p.tau0 + (tau_s - p.tau0) * fmaxf(0.0f, 1.0f + c);
  const float dc = 4.5f * (__fdividef(1.0f, tau_s) - __fdividef(1.0f, tau));
  const float pxx = st[5], pyy = st[6], pzz = st[7], pxy = st[8], pxz = st[9], pyz = st[10];
  const float tr3 = (pxx + pyy + pzz) * (1.0f / 3.0f);
  const float proj[10] = {-tr3,
                          pxx - tr3,
                          pyy - tr3,
                          pzz - tr3,
                          pxx + pyy + 2.0f * pxy - tr3,
                          pxx + pzz + 2.0f * pxz - tr3,
                          pyy + pzz + 2.0f * pyz - tr3,
                          pxx + pyy - 2.0f * pxy - tr3,
                          pxx + pzz - 2.0f * pxz - tr3,
                          pyy + pzz - 2.0f * pyz - tr3};
  post[0] = fmaf(dc * pw::w_of(0), proj[0], post[0]);
#pragma unroll
  for (int i = 1; i < 19; i++) post[i] = fmaf(dc * pw::w_of(i), proj[(i + 1) / 2], post[i]);
  const float rho = st[1];
  if (p.write_macro && !(rho >= 0.5f && rho <= 1.5f)) atomicOr(p.status, 1u);  // also catches NaN
  T *f = reinterpret_cast<T *>(p.f);
  T code[19];
#pragma unroll
  for (int j = 0; j < 19; j++) code[j] = S::encode(post[j], (uint32_t)j, n);
  if (interior) {
#pragma unroll
    for (int j = 0; j < 19; j++) f[n + p.st[j]] = code[j];
  } else {
    const pwclosure::Nbr b = pwclosure::make_nbr(p, x, y, z);
#pragma unroll
    for (int j = 0; j < 19; j++) f[ODD ? b.push(j, p.stride) : (pw::pidx)pw::opp_of(j) * p.stride + n] = code[j];
  }
  if (p.write_macro) p.macros[n] = make_float4(rho, st[2], st[3], st[4]);
  if (x + 2 == p.nx) p.plane_out[y + p.ny * z] = pwclosure::outlet_velocity_of<ST>(code);
}

// A persistent grid (four blocks per SM): each block sets up the network image
// and its TMEM columns once, then walks tiles of 32 x 4 cells of one z-plane,
// tiles W apart for W blocks.
template <int ST, int OP, bool ODD>
__global__ void __launch_bounds__(128, 4) closure_step(StepParams p, const uint32_t *frag, const uint8_t *wall_dist,
                                                       uint32_t tiles_x, uint32_t tiles_y) {
  using S = pw::Store<ST>;
  using T = typename S::T;
  __shared__ TcShared sh;
  __shared__ float post_s[OP == pw::OP_REG ? 19 : 1][128];  // REG: plain cells' Smagorinsky post-collision state
  tc_setup(sh, frag);
  uint32_t phase = 0;
  const uint32_t tid = threadIdx.x + 32u * threadIdx.y;
  const uint32_t tiles = tiles_x * tiles_y * p.nz;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint32_t bx = tile % tiles_x, by = (tile / tiles_x) % tiles_y, z = tile / (tiles_x * tiles_y);
    const uint32_t x = bx * 32 + threadIdx.x;
    const uint32_t y = by * 4 + threadIdx.y;
    const bool in = x < p.nx && y < p.ny;
    const uint32_t n = in ? x + p.nx * (y + p.ny * z) : 0u;
    const uint32_t flag = in ? __ldg(&p.flags[n]) : (uint32_t)pw::SOLID;
    float xin[kIn], st[11];
#pragma unroll
    for (int k = 0; k < kIn; k++) xin[k] = 0.0f;
    const bool plain = in && flag == pw::FLUID;  // fluid without wall links
    // cells whose neighbours need no periodic wrap take the step's element
    // offsets from the kernel parameters (the wrap arithmetic otherwise)
    const bool interior = x >= 1u && x + 2u <= p.nx && y >= 1u && y + 2u <= p.ny && z >= 1u && z + 2u <= p.nz &&
                          p.slip == 0u;
    if (plain) {
      const T *f = reinterpret_cast<const T *>(p.f);
      float g[19];
      if (interior) {
#pragma unroll
        for (int i = 0; i < 19; i++) g[i] = S::decode(f[n + p.ld[i]]);
      } else {
        const pwclosure::Nbr b = pwclosure::make_nbr(p, x, y, z);
#pragma unroll
        for (int i = 0; i < 19; i++) g[i] = S::decode(f[ODD ? b.pull(i, p.stride) : (pw::pidx)i * p.stride + n]);
      }
      float rho, vx, vy, vz;
      pwclosure::update_fast<OP, true, CaptureHook>(p, g, rho, vx, vy, vz, 1.0f, 1.0f, CaptureHook{st});
      cell_inputs(p, st, (float)wall_dist[n], xin);
      if (OP == pw::OP_REG) {
#pragma unroll
        for (int i = 0; i < 19; i++) post_s[i][tid] = g[i];
      }
    }
    const float c = block_mlp(sh, xin, phase);
    bool any = false;
    double fx = 0.0, fy = 0.0, fz = 0.0;
    if (OP == pw::OP_REG && plain) {
      // single pass: the Smagorinsky state corrected to the closure's relaxation time
      float post[19];
#pragma unroll
      for (int i = 0; i < 19; i++) post[i] = post_s[OP == pw::OP_REG ? i : 0][tid];
      finish_plain_reg<ST, ODD>(p, x, y, z, n, st, c, post, interior);
    } else if (in) {
      pwclosure::general_cell<ST, OP, true, ODD, ClosureHook>(p, x, y, z, n, flag, fx, fy, fz, any, ClosureHook{c});
    }
    // the partial slot of tile (x block, y block, z), as the cell kernels number them
    const size_t slot = tile;
    pwclosure::reduce_force_at(any, fx, fy, fz, p.partials, slot, threadIdx.x + 32 * threadIdx.y);
  }
  if (threadIdx.x == 0 && threadIdx.y == 0 && sh.failed) atomicOr(p.status, 4u);
  tc_teardown(sh);
}

// ---------------------------------------------------------------- cell-pair closure step
// The closure step on the plain step's two-cell arithmetic (update_fast2):
// each thread takes cells x and x + 32 of a 64-cell run, as aa_step_fast does
// for every storage, and a block the 256 cells of four rows, so its network
// runs as two M = 128 tiles, the threads' first cells and their second cells.
// Every row of both parities runs here, the seam rows with their periodic
// wrap as per-row offsets (SeamWrap); the wall-link cells and the floor layer
// run in blocks of their own, with the reference's wall model, as in a step
// without the closure.
struct TcPair {
  __align__(128) unsigned char img[kImgBytes];   // the network image
  // the layer-2 operands of the two tiles (128 x 32 bf16 each); the two
  // layer-1 operands (128 x 16 each) share the first tile's, which layer 1's
  // MMAs have read by the time their outputs come back
  __align__(128) unsigned char a2[2][128 * 64];
  __align__(8) uint64_t bar;                     // MMA completion
  uint32_t tmem;                                 // 64 TMEM columns: tile t's layer output at column 32 t
  uint32_t next[2];                              // the block's next tile, by turns
  uint32_t failed;                               // a completion wait ran out
  __device__ __forceinline__ unsigned char *a1(int t) { return a2[0] + t * (128 * 32); }
};

__device__ __forceinline__ void put_inputs(unsigned char *a1, uint32_t row, const float x[kIn]) {
  uint4 lo, hi;
  lo.x = pack_bf16(x[0], x[1]); lo.y = pack_bf16(x[2], x[3]); lo.z = pack_bf16(x[4], x[5]);
  lo.w = pack_bf16(x[6], x[7]);
  hi.x = pack_bf16(x[8], 0.0f); hi.y = 0u; hi.z = 0u; hi.w = 0u;
  *reinterpret_cast<uint4 *>(a1 + cm_offset(row, 0, kSbo1)) = lo;
  *reinterpret_cast<uint4 *>(a1 + cm_offset(row, 8, kSbo1)) = hi;
}

// block_mlp for the block's two tiles: c of the thread's first (.x) and
// second (.y) cell.  Layer 2 writes the columns layer 1's outputs were read
// from, after the block barrier that follows those reads.  The loops over
// the two tiles stay rolled: the smaller kernel measured 3.7% faster (its
// warps had waited on instruction fetch more than on anything else).
__device__ float2 block_mlp2(TcPair &sh, const float xa[kIn], const float xb[kIn], uint32_t &phase) {
  const uint32_t tid = threadIdx.x + 32u * threadIdx.y, warp = tid >> 5;
  const uint32_t lane_addr = sh.tmem + ((warp * 32u) << 16);
  put_inputs(sh.a1(0), tid, xa);
  put_inputs(sh.a1(1), tid, xb);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  const bool live = sh.failed == 0u;
  if (tid == 0 && live) {
    const uint64_t w1 = smem_desc(smem_u32(sh.img + kImgW1), kSbo1);
    tc_mma(sh.tmem, smem_desc(smem_u32(sh.a1(0)), kSbo1), w1, 0u);
    tc_mma(sh.tmem + 32u, smem_desc(smem_u32(sh.a1(1)), kSbo1), w1, 0u);
    tc_commit(&sh.bar);
  }
  const bool done1 = __all_sync(0xffffffffu, live && tc_wait(&sh.bar, phase & 1u));
  phase++;
  tc_after_sync();
  if (!done1 && live) atomicOr(&sh.failed, 1u);
  const float *b1 = reinterpret_cast<const float *>(sh.img + kImgB1);
#pragma unroll 1
  for (int t = 0; t < 2; t++) {
#pragma unroll
    for (int k = 0; k < 32; k += 8) {
      float h[8];
      if (done1) {
        tc_load8(lane_addr + 32u * t + (uint32_t)k, h);
      } else {
#pragma unroll
        for (int j = 0; j < 8; j++) h[j] = 0.0f;
      }
      uint4 v;
      v.x = pack_bf16(tanh_fast(h[0] + b1[k]), tanh_fast(h[1] + b1[k + 1]));
      v.y = pack_bf16(tanh_fast(h[2] + b1[k + 2]), tanh_fast(h[3] + b1[k + 3]));
      v.z = pack_bf16(tanh_fast(h[4] + b1[k + 4]), tanh_fast(h[5] + b1[k + 5]));
      v.w = pack_bf16(tanh_fast(h[6] + b1[k + 6]), tanh_fast(h[7] + b1[k + 7]));
      *reinterpret_cast<uint4 *>(sh.a2[t] + cm_offset(tid, k, kSbo2)) = v;
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  const bool live2 = sh.failed == 0u;
  if (tid == 0 && live2) {
    const uint32_t w2 = smem_u32(sh.img + kImgW2);
#pragma unroll
    for (int t = 0; t < 2; t++) {
      const uint32_t a2 = smem_u32(sh.a2[t]);
      tc_mma(sh.tmem + 32u * t, smem_desc(a2, kSbo2), smem_desc(w2, kSbo2), 0u);
      tc_mma(sh.tmem + 32u * t, smem_desc(a2 + 2u * kLbo, kSbo2), smem_desc(w2 + 2u * kLbo, kSbo2), 1u);
    }
    tc_commit(&sh.bar);
  }
  const bool done2 = __all_sync(0xffffffffu, live2 && tc_wait(&sh.bar, phase & 1u));
  phase++;
  tc_after_sync();
  if (!done2) {
    if (live2) atomicOr(&sh.failed, 1u);
    return make_float2(0.0f, 0.0f);
  }
  const float *b2 = reinterpret_cast<const float *>(sh.img + kImgB2);
  const float *w3 = reinterpret_cast<const float *>(sh.img + kImgW3);
  float out0 = 0.0f, out1 = 0.0f;
#pragma unroll 1
  for (int t = 0; t < 2; t++) {
    float o = 0.0f;
#pragma unroll
    for (int k = 0; k < 32; k += 8) {
      float h[8];
      tc_load8(lane_addr + 32u * t + (uint32_t)k, h);
#pragma unroll
      for (int j = 0; j < 8; j++) o = fmaf(w3[k + j], bf16_round(tanh_fast(h[j] + b2[k + j])), o);
    }
    if (t == 0) out0 = o; else out1 = o;
  }
  const float b3 = reinterpret_cast<const float *>(sh.img + kImgB3)[0];
  return make_float2(out0 + b3, out1 + b3);
}

// update_fast2's hook: the network's relaxation time for the lanes in live
// (bit 0 .x, bit 1 .y: plain LES cells), the Smagorinsky one for the others.
struct ClosureHook2 {
  TcPair *sh;
  uint32_t *phase;
  float2 wall;
  uint32_t live;
  __device__ __forceinline__ float2 operator()(const StepParams &p, float2 tau_s, float2 rho, float2 vx, float2 vy,
                                               float2 vz, float2 pxx, float2 pyy, float2 pzz, float2 pxy, float2 pxz,
                                               float2 pyz) const {
    float xa[kIn], xb[kIn];
#pragma unroll
    for (int k = 0; k < kIn; k++) xa[k] = xb[k] = 0.0f;
    if (live & 1u) {
      const float st[11] = {tau_s.x, rho.x, vx.x, vy.x, vz.x, pxx.x, pyy.x, pzz.x, pxy.x, pxz.x, pyz.x};
      cell_inputs(p, st, wall.x, xa);
    }
    if (live & 2u) {
      const float st[11] = {tau_s.y, rho.y, vx.y, vy.y, vz.y, pxx.y, pyy.y, pzz.y, pxy.y, pxz.y, pyz.y};
      cell_inputs(p, st, wall.y, xb);
    }
    const float2 c = block_mlp2(*sh, xa, xb, *phase);
    float2 tau = tau_s;
    if (live & 1u) tau.x = p.tau0 + (tau_s.x - p.tau0) * fmaxf(0.0f, 1.0f + c.x);
    if (live & 2u) tau.y = p.tau0 + (tau_s.y - p.tau0) * fmaxf(0.0f, 1.0f + c.y);
    return tau;
  }
};

// The wall-link cells and the floor layer, as functions of their own (see pw_step_all.cuh).
template <int ST, int OP, bool ODD, int BLOCKS>
__device__ __noinline__ void edge_role(const StepParams &p, const uint32_t *list, uint32_t count, uint32_t b) {
  pwclosure::edge_block<ST, OP, true, ODD>(p, list, count, b, threadIdx.x + 32u * threadIdx.y);
}
template <int ST, int OP, bool ODD, int BLOCKS>
__device__ __noinline__ void floor_role(const StepParams &p, uint32_t b, uint32_t runs) {
  pwclosure::floor_thread<ST, OP, true, ODD>(p, (b % runs) * 64u + 2u * threadIdx.x,
                                             1u + (b / runs) * 4u + threadIdx.y);
}

// One launch a step: the first blocks take the wall-link cells and the floor
// layer, the others are a persistent grid: each sets up the network image and
// its TMEM columns once, then walks tiles of 64 x 4 cells of one z-plane, tiles
// W apart for W blocks.  Plain cells and EQ cells without wall links are stored,
// as in aa_step_fast; every thread takes part in each tile's network.
// Eight blocks per SM (64 registers; all 512 TMEM columns): measured 6%
// faster than six (80 registers) and 9% faster than four.
// A block's first tile is its own, the others it takes as it gets to them: blocks
// that start after a side block, or whose cells take longer, take fewer.  The next
// step's blocks set up their networks while this one's last ones run.  A step, before
// (edge and floor kernels beside a static share of the tiles) and now: 96x48x48 FP16
// 31.4 and 26.5 us, 128x64x64 FP32 37.3 and 36.2, 256x128x128 FP32 255 and 238,
// 384x192x192 FP16 658 and 603.
// A step whose blocks all find a place at four per SM runs in the form with their 128
// registers: its time is one tile's and one wall-link cell's, whose spilled registers
// count then (64x32x32 FP32 15.3 and 13.4 us with 64 and 128 registers, FP16 18.2 and
// 14.9; separate kernels 15.9 and 23.8 in short calls).  Long runs of few tiles are captured
// with separate kernels (closure_long_runs_captured).
#ifndef PW_CLOSURE_PAIR_BLOCKS
#define PW_CLOSURE_PAIR_BLOCKS 8
#endif
#define PW_CLOSURE_FEW_BLOCKS 4
static_assert(PW_CLOSURE_PAIR_BLOCKS * 64 <= 512, "the blocks of an SM must fit its 512 TMEM columns");
struct ClosureSide {
  const uint32_t *list;
  uint32_t count, edge, floor;
  uint32_t *taken;  // tiles handed out beyond the blocks' first ones; zero between steps
};
template <int ST, int OP, bool ODD, int BLOCKS>
__global__ void __launch_bounds__(128, BLOCKS) closure_pairs(const __grid_constant__ StepParams p,
                                                                            const uint32_t *frag,
                                                                            const uint8_t *wall_dist, uint32_t runs,
                                                                            uint32_t row_blocks, ClosureSide side) {
  const uint32_t first = side.edge + side.floor;
  if (blockIdx.x < first) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (blockIdx.x < side.edge) {
      edge_role<ST, OP, ODD, BLOCKS>(p, side.list, side.count, blockIdx.x);
    } else {
      if constexpr (ST != pw::STORE_F32) floor_role<ST, OP, ODD, BLOCKS>(p, blockIdx.x - side.edge, runs);
    }
    return;
  }
  using S = pw::Store<ST>;
  using T = typename S::T;
  __shared__ TcPair sh;
  tc_setup(sh, frag);
  // the next step's blocks may come once every block here has its TMEM columns
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const bool leader = (threadIdx.x | threadIdx.y) == 0u;
  if (leader && blockIdx.x == first && p.clear_status) *p.status = 0u;
  uint32_t phase = 0, turn = 0;
  T *f = reinterpret_cast<T *>(p.f);
  const uint32_t tiles = runs * row_blocks * p.nz;
  const bool more = gridDim.x - first < tiles;  // tiles beyond the blocks' first ones
  uint32_t next = tiles;
  for (uint32_t tile = blockIdx.x - first; tile < tiles; tile = next) {
    // the tile after this one, stored once this one's loads are under way; every thread
    // reads it behind the network's barriers.  One is asked for per tile taken, so the
    // count wraps to zero with the step's last.
    uint32_t got = 0;
    if (more && leader) got = atomicInc(side.taken, tiles - 1u);
    const uint32_t run = tile % runs, rest = tile / runs;
    const uint32_t x = run * 64u + threadIdx.x, y = (rest % row_blocks) * 4u + threadIdx.y, z = rest / row_blocks;
    const bool row_in = y < p.ny;
    const uint32_t n = x + p.nx * ((row_in ? y : 0u) + p.ny * z);
    uint32_t ok = 0u, eq = 0u;
    if (row_in) {
#pragma unroll
      for (uint32_t k = 0; k < 2u; k++) {
        const uint32_t xk = x + 32u * k, nk = n + 32u * k;
        if (xk >= p.nx) continue;
        if (!((__ldg(&p.special[nk >> 5]) >> (nk & 31u)) & 1u)) {
          if (pwclosure::is_plain_position(xk, p.nx)) ok |= 1u << k;
        } else if (__ldg(&p.flags[nk]) == pw::EQ) {
          ok |= 1u << k;
          eq |= 1u << k;
        }
      }
    }
    const uint32_t live = ok & ~eq;
    // odd steps pull across the periodic y and z faces on the seam rows (the
    // offsets are zero on the other rows: one code path keeps the kernel small,
    // measured 3.7% faster than a separate path for the seam rows)
    const pwclosure::SeamWrap sw = ODD && row_in ? pwclosure::SeamWrap(p, y, z, 1) : pwclosure::SeamWrap();
    float2 g[19];
    if (row_in) {
#pragma unroll
      for (int i = 0; i < 19; i++) {
        const T *a = f + (n + p.ld[i] + sw.of(i));
        g[i] = make_float2(S::raw(a[0]), S::raw(a[32]));
      }
    } else {
#pragma unroll
      for (int i = 0; i < 19; i++) g[i] = make_float2(0.0f, 0.0f);
    }
    if (more && leader) sh.next[turn & 1u] = gridDim.x - first + got;
    float2 eux = pwclosure::f2(p.u_in), euy = pwclosure::f2(0.f), euz = pwclosure::f2(0.f);
    if (eq) {
      const uint32_t row = y + p.ny * z;
      if ((eq & 1u) && x == p.nx - 1 && x > 0) {
        const float4 u = p.plane_in[row];
        eux.x = u.x; euy.x = u.y; euz.x = u.z;
      }
      if ((eq & 2u) && x + 32u == p.nx - 1) {
        const float4 u = p.plane_in[row];
        eux.y = u.x; euy.y = u.y; euz.y = u.z;
      }
    }
    const float2 wall = make_float2((live & 1u) ? (float)wall_dist[n] : 0.0f, (live & 2u) ? (float)wall_dist[n + 32] : 0.0f);
    float2 rho, vx, vy, vz;
    const float2 om = pwclosure::update_fast2<OP, true, ClosureHook2>(
        p, g, rho, vx, vy, vz, S::kScale, S::kInvScale, eq, eux, euy, euz, ClosureHook2{&sh, &phase, wall, live});
    if (more) next = sh.next[turn & 1u];
    turn++;
    if (!ok) continue;
    if (ST != pw::STORE_F32) {
      // a non-finite state is stored as NaN, as the reference's GPUs store it
      if (!(fabsf(rho.x + om.x) < INFINITY)) {
#pragma unroll
        for (int j = 0; j < 19; j++) g[j].x = __uint_as_float(0x7fc00000u);
      }
      if (!(fabsf(rho.y + om.y) < INFINITY)) {
#pragma unroll
        for (int j = 0; j < 19; j++) g[j].y = __uint_as_float(0x7fc00000u);
      }
    }
    const uint32_t nk = n * 0x9e3779b9u, nk2 = nk + 32u * 0x9e3779b9u;
    const uint32_t xa = x, xb = x + 32u;
#pragma unroll
    for (int j = 0; j < 19; j++) {
      // odd steps: the EQ cell at x = 0 pushes c_x = -1 to x = nx - 1 and the
      // one at x = nx - 1 pushes c_x = +1 to x = 0 (signed element offsets)
      const int cx = pw::cx_of(j);
      const int64_t wa = !ODD ? 0 : (cx < 0 && xa == 0u ? (int64_t)p.nx : (cx > 0 && xa + 1u == p.nx ? -(int64_t)p.nx : 0));
      const int64_t wb = ODD && cx > 0 && xb + 1u == p.nx ? -(int64_t)p.nx : 0;
      T ca, cb;
      pwclosure::encode_two<ST>(g[j], j, nk, nk2, ca, cb);
      T *a = f + (n + p.st[j] + sw.of(pw::opp_of(j)));
      if (ok & 1u) a[wa] = ca;
      if (ok & 2u) a[32 + wb] = cb;
    }
    if (p.write_macro) {
      const bool bad_a = (ok & ~eq & 1u) && !(rho.x >= 0.5f && rho.x <= 1.5f);
      const bool bad_b = (ok & ~eq & 2u) && !(rho.y >= 0.5f && rho.y <= 1.5f);
      if (bad_a || bad_b) atomicOr(p.status, 1u);
      if (ok & 1u) p.macros[n] = make_float4(rho.x, vx.x, vy.x, vz.x);
      if (ok & 2u) p.macros[n + 32] = make_float4(rho.y, vx.y, vy.y, vz.y);
    }
    const bool pub_a = (ok & 1u) && x + 2u == p.nx, pub_b = (ok & 2u) && x + 34u == p.nx;
    if (pub_a || pub_b) {
      // the outlet's upstream plane publishes the velocity of its stored codes
      const uint32_t xo = pub_a ? x : x + 32u, no = n + (xo - x);
      const pwclosure::Nbr b = pwclosure::make_nbr(p, xo, y, z);
      T code[19];
#pragma unroll
      for (int j = 0; j < 19; j++) code[j] = f[pwclosure::slot_of<ODD>(b, j, p.stride, no)];
      p.plane_out[y + p.ny * z] = pwclosure::outlet_velocity_of<ST>(code);
    }
  }
  if (threadIdx.x == 0 && threadIdx.y == 0 && sh.failed) atomicOr(p.status, 4u);
  tc_teardown(sh);
}

// Network outputs for given inputs through the same tensor-core path (tests);
// *status gets bit 0 if a completion wait ran out.
__global__ void __launch_bounds__(128) eval_kernel(const uint32_t *frag, const float *xin, uint32_t count, float *out,
                                                   uint32_t *status) {
  __shared__ TcShared sh;
  tc_setup(sh, frag);
  uint32_t phase = 0;
  const uint32_t i = blockIdx.x * 128 + threadIdx.x;
  float x[kIn];
#pragma unroll
  for (int k = 0; k < kIn; k++) x[k] = i < count ? xin[(size_t)i * kIn + k] : 0.0f;
  const float c = block_mlp(sh, x, phase);
  if (i < count) out[i] = c;
  if (threadIdx.x == 0 && sh.failed) atomicOr(status, 1u);
  tc_teardown(sh);
}

// ---------------------------------------------------------------- wall distance
// Cells to the nearest wall cell (6-neighbour steps, capped at kWallCap): x
// bounded, y and z periodic as the lattice.
__global__ void dist_init(const uint32_t *flags, size_t cells, uint8_t *d) {
  const size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n < cells) d[n] = pw::is_wall_kind(flags[n] & 7u) ? 0 : 255;
}
__global__ void dist_from_solid(const uint8_t *solid, size_t cells, uint8_t *d) {
  const size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n < cells) d[n] = solid[n] ? 0 : 255;
}
__global__ void dist_step(const uint8_t *in, uint8_t *out, uint32_t nx, uint32_t ny, uint32_t nz) {
  const size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= (size_t)nx * ny * nz) return;
  const uint32_t x = (uint32_t)(n % nx), y = (uint32_t)((n / nx) % ny), z = (uint32_t)(n / ((size_t)nx * ny));
  const size_t plane = (size_t)nx * ny;
  uint32_t v = in[n];
  if (x > 0) v = min(v, in[n - 1] + 1u);
  if (x + 1 < nx) v = min(v, in[n + 1] + 1u);
  v = min(v, in[n - (size_t)y * nx + (size_t)((y + ny - 1) % ny) * nx] + 1u);
  v = min(v, in[n - (size_t)y * nx + (size_t)((y + 1) % ny) * nx] + 1u);
  v = min(v, in[n - (size_t)z * plane + (size_t)((z + nz - 1) % nz) * plane] + 1u);
  v = min(v, in[n - (size_t)z * plane + (size_t)((z + 1) % nz) * plane] + 1u);
  out[n] = (uint8_t)min(v, 255u);
}

int wall_distance(uint8_t *d, uint8_t *tmp, uint32_t nx, uint32_t ny, uint32_t nz, cudaStream_t s) {
  const size_t cells = (size_t)nx * ny * nz;
  const unsigned blocks = (unsigned)((cells + 255) / 256);
  for (int k = 0; k < (int)kWallCap; k += 2) {
    dist_step<<<blocks, 256, 0, s>>>(d, tmp, nx, ny, nz);
    dist_step<<<blocks, 256, 0, s>>>(tmp, d, nx, ny, nz);
  }
  PW_TRY(cudaGetLastError());
  return PW_OK;
}

// ---------------------------------------------------------------- training data
// coarse[q][N]: rho, ux, uy, uz and the subgrid stress mean((u - ubar)(u - ubar)):
// xx, yy, zz, xy, xz, yz (taken from the deviations, free of the cancellation
// of mean(u u) - ubar ubar in binary32).
__global__ void coarsen_kernel(const float4 *macros, const uint32_t *flags, uint32_t nx, uint32_t ny, uint32_t nz,
                               float *coarse, uint8_t *solid) {
  const uint32_t cx = nx / 2, cy = ny / 2, cz = nz / 2;
  const size_t nc = (size_t)cx * cy * cz;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const uint32_t X = (uint32_t)(c % cx), Y = (uint32_t)((c / cx) % cy), Z = (uint32_t)(c / ((size_t)cx * cy));
  float4 m[8];
  float mean[4] = {0, 0, 0, 0};
  uint32_t walls = 0;
  for (uint32_t k = 0; k < 8; k++) {
    const size_t n = (2 * X + (k & 1)) + (size_t)nx * ((2 * Y + ((k >> 1) & 1)) + (size_t)ny * (2 * Z + (k >> 2)));
    m[k] = macros[n];
    walls += pw::is_wall_kind(flags[n] & 7u) ? 1u : 0u;
    mean[0] += m[k].x; mean[1] += m[k].y; mean[2] += m[k].z; mean[3] += m[k].w;
  }
  for (int q = 0; q < 4; q++) mean[q] *= 0.125f;
  float t[6] = {0, 0, 0, 0, 0, 0};
  for (uint32_t k = 0; k < 8; k++) {
    const float dx = m[k].y - mean[1], dy = m[k].z - mean[2], dz = m[k].w - mean[3];
    t[0] += dx * dx; t[1] += dy * dy; t[2] += dz * dz; t[3] += dx * dy; t[4] += dx * dz; t[5] += dy * dz;
  }
  for (int q = 0; q < 4; q++) coarse[(size_t)q * nc + c] = mean[q];
  for (int q = 0; q < 6; q++) coarse[(size_t)(4 + q) * nc + c] = 0.125f * t[q];
  solid[c] = walls ? 1 : 0;
}

// Target and inputs of coarse cell c, or false when it is left out.
__device__ __forceinline__ bool coarse_sample(const float *co, const uint8_t *dist, uint32_t cx, uint32_t cy,
                                              uint32_t cz, size_t c, float nu0, float u_in, float x[kIn], float *y) {
  const size_t nc = (size_t)cx * cy * cz;
  const uint32_t X = (uint32_t)(c % cx), Y = (uint32_t)((c / cx) % cy), Z = (uint32_t)(c / ((size_t)cx * cy));
  if (X < 2 || X + 3 > cx || dist[c] < 2) return false;
  const size_t plane = (size_t)cx * cy;
  const size_t xm = c - 1, xp = c + 1;
  const size_t ym = c - (size_t)Y * cx + (size_t)((Y + cy - 1) % cy) * cx, yp = c - (size_t)Y * cx + (size_t)((Y + 1) % cy) * cx;
  const size_t zm = c - (size_t)Z * plane + (size_t)((Z + cz - 1) % cz) * plane;
  const size_t zp = c - (size_t)Z * plane + (size_t)((Z + 1) % cz) * plane;
  auto u = [&](int comp, size_t at) { return co[(size_t)(1 + comp) * nc + at]; };
  float grad[3][3];  // grad[a][b] = d u_b / d x_a
  for (int b = 0; b < 3; b++) {
    grad[0][b] = 0.5f * (u(b, xp) - u(b, xm));
    grad[1][b] = 0.5f * (u(b, yp) - u(b, ym));
    grad[2][b] = 0.5f * (u(b, zp) - u(b, zm));
  }
  const float s[6] = {grad[0][0], grad[1][1], grad[2][2], 0.5f * (grad[0][1] + grad[1][0]),
                      0.5f * (grad[0][2] + grad[2][0]), 0.5f * (grad[1][2] + grad[2][1])};
  const float ux = u(0, c), uy = u(1, c), uz = u(2, c);
  const float tsgs[6] = {co[4 * nc + c], co[5 * nc + c], co[6 * nc + c], co[7 * nc + c], co[8 * nc + c],
                         co[9 * nc + c]};
  const float ss = s[0] * s[0] + s[1] * s[1] + s[2] * s[2] + 2.0f * (s[3] * s[3] + s[4] * s[4] + s[5] * s[5]);
  const float ts = tsgs[0] * s[0] + tsgs[1] * s[1] + tsgs[2] * s[2] + 2.0f * (tsgs[3] * s[3] + tsgs[4] * s[4] + tsgs[5] * s[5]);
  const float nu_s = 0.01f * sqrtf(2.0f * ss);
  if (!(nu_s > 1e-9f)) return false;
  const float nu_t = fmaxf(0.0f, -ts / (2.0f * ss));
  *y = fminf(3.0f, fmaxf(-1.0f, nu_t / nu_s - 1.0f));
  features(s, co[c], ux, uy, uz, (float)dist[c], nu0, nu_s, u_in, x);
  return true;
}

constexpr int kScanBlock = 1024;

__global__ void sample_count(const float *co, const uint8_t *dist, uint32_t cx, uint32_t cy, uint32_t cz, float nu0,
                             float u_in, uint32_t *block_counts) {
  __shared__ uint32_t warp_counts[kScanBlock / 32];
  const size_t c = (size_t)blockIdx.x * kScanBlock + threadIdx.x;
  float x[kIn], y;
  const bool ok = c < (size_t)cx * cy * cz && coarse_sample(co, dist, cx, cy, cz, c, nu0, u_in, x, &y);
  const uint32_t ballot = __ballot_sync(0xffffffffu, ok);
  if ((threadIdx.x & 31) == 0) warp_counts[threadIdx.x >> 5] = __popc(ballot);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kScanBlock / 32; w++) t += warp_counts[w];
    block_counts[blockIdx.x] = t;
  }
}

__global__ void scan_counts(uint32_t *counts, uint32_t nblk, uint32_t *total) {
  __shared__ uint32_t sh[kScanBlock];
  uint32_t carry = 0;
  for (uint32_t base = 0; base < nblk; base += kScanBlock) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < nblk ? counts[i] : 0u;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < kScanBlock; o <<= 1) {
      const uint32_t add = threadIdx.x >= (unsigned)o ? sh[threadIdx.x - o] : 0u;
      __syncthreads();
      sh[threadIdx.x] += add;
      __syncthreads();
    }
    if (i < nblk) counts[i] = carry + sh[threadIdx.x] - v;
    carry += sh[kScanBlock - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

__global__ void sample_write(const float *co, const uint8_t *dist, uint32_t cx, uint32_t cy, uint32_t cz, float nu0,
                             float u_in, const uint32_t *offsets, uint64_t base, uint64_t cap, float *X, float *Y) {
  __shared__ uint32_t warp_base[kScanBlock / 32];
  const size_t c = (size_t)blockIdx.x * kScanBlock + threadIdx.x;
  float x[kIn], y = 0.0f;
  const bool ok = c < (size_t)cx * cy * cz && coarse_sample(co, dist, cx, cy, cz, c, nu0, u_in, x, &y);
  const uint32_t ballot = __ballot_sync(0xffffffffu, ok);
  const uint32_t lane = threadIdx.x & 31;
  if (lane == 0) warp_base[threadIdx.x >> 5] = __popc(ballot);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = offsets[blockIdx.x];
    for (int w = 0; w < kScanBlock / 32; w++) { const uint32_t k = warp_base[w]; warp_base[w] = t; t += k; }
  }
  __syncthreads();
  if (!ok) return;
  const uint64_t at = base + warp_base[threadIdx.x >> 5] + __popc(ballot & ((1u << lane) - 1u));
  if (at >= cap) return;
  for (int k = 0; k < kIn; k++) X[at * kIn + k] = x[k];
  Y[at] = y;
}

// ---------------------------------------------------------------- training
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Forward with the network's rounding, squared error against the target, backward
// (the bf16 roundings pass gradients through unchanged; tanh' = 1 - h^2 of the
// rounded activation), and the block's parameter-gradient sums and loss sum in
// partial[block].
// sample index: explicit list `idx` when given, else mix64(seed + step * 2^32 + i) mod n.
//
// One block of 16 warps an SM.  A warp takes 32 samples at a time, one a lane, and
// needs no block barrier until its last: weights are broadcast from shared memory
// four at a time, a lane's activations go to its row of the warp's own buffers
// (36 words a row: rows and columns both free of bank conflicts as 16-byte pieces),
// and the gradients are products over the 32 rows with an 8 x 4 tile of dW2 and a
// row of dW1 in each lane's registers, kept there over all of the warp's samples.
// With 65,536 samples a warp has one group, and the pass is its chain of shared-memory
// loads and multiply-adds with four warps a scheduler (LSU 34%, FMA 30% busy).
// 65,536 samples: 26 us; 145 us with a sample a thread, rows of 32 words (every
// column access 32 ways in conflict) and a thread a parameter for the sums.
constexpr int kTrainWarps = 16, kTrainThreads = 32 * kTrainWarps;
constexpr int kRow = 36, kXRow = 12;
struct TrainWarp {
  float a[32 * kRow];   // hidden layer 2 (h2, then d2), then d1; at the end the warp's sums
  float b[32 * kRow];   // hidden layer 1
  float x[32 * kXRow];  // inputs, 9..11 zero
};
struct TrainShared {
  float w1[kHidden * kXRow], w2[kHidden * kHidden], w3[kHidden], b1[kHidden], b2[kHidden];
  TrainWarp warp[kTrainWarps];
};
static_assert(2 * 32 * kRow >= kParams + 1, "a warp's sums fit its row buffers");

__global__ void __launch_bounds__(kTrainThreads, 1) train_block(const float *w, const float *X, const float *Y,
                                                               uint64_t n, uint32_t batch, uint64_t seed,
                                                               const uint32_t *step, const uint32_t *idx,
                                                               float *partial) {
  extern __shared__ __align__(16) unsigned char train_smem_raw[];
  TrainShared &sh = *reinterpret_cast<TrainShared *>(train_smem_raw);
  const uint32_t tid = threadIdx.x, lane = tid & 31u, wib = tid >> 5;
  for (int k = tid; k < kHidden * kXRow; k += kTrainThreads)
    sh.w1[k] = k % kXRow < kIn ? bf16_round(w[kW1 + k / kXRow * kIn + k % kXRow]) : 0.0f;
  for (int k = tid; k < kHidden * kHidden; k += kTrainThreads) sh.w2[k] = bf16_round(w[kW2 + k]);
  if (tid < kHidden) {
    sh.w3[tid] = bf16_round(w[kW3 + tid]);
    sh.b1[tid] = w[kB1 + tid];
    sh.b2[tid] = w[kB2 + tid];
  }
  const float b3 = w[kB3];
  __syncthreads();
  TrainWarp &my = sh.warp[wib];
  float *arow = my.a + lane * kRow, *brow = my.b + lane * kRow, *xrow = my.x + lane * kXRow;
  const float4 *w1v = reinterpret_cast<const float4 *>(sh.w1), *w2v = reinterpret_cast<const float4 *>(sh.w2);
  const float4 *w3v = reinterpret_cast<const float4 *>(sh.w3);
  const uint32_t groups = (batch + 31u) / 32u;  // group g: block g mod grid, its warp g / grid mod 16
  const uint32_t j0 = (lane >> 3) * 8u, k0 = (lane & 7u) * 4u;  // this lane's tile of dW2
  float g2[8][4], g1[kIn], gb1 = 0.0f, gb2 = 0.0f, g3 = 0.0f, gb3 = 0.0f, loss = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; j++)
#pragma unroll
    for (int k = 0; k < 4; k++) g2[j][k] = 0.0f;
#pragma unroll
  for (int k = 0; k < kIn; k++) g1[k] = 0.0f;
  for (uint32_t g = blockIdx.x + gridDim.x * wib; g < groups; g += gridDim.x * kTrainWarps) {
    const uint32_t i = g * 32u + lane;
    const bool live = i < batch;
    uint64_t s = 0;
    if (live) s = idx ? idx[i] : mix64(seed + ((uint64_t)*step << 32) + i) % n;
    const float target = live ? Y[s] : 0.0f;
    float x[kXRow];
#pragma unroll
    for (int k = 0; k < kXRow; k++) x[k] = live && k < kIn ? bf16_round(X[s * kIn + k]) : 0.0f;
#pragma unroll
    for (int k = 0; k < kXRow; k += 4)
      *reinterpret_cast<float4 *>(xrow + k) = make_float4(x[k], x[k + 1], x[k + 2], x[k + 3]);
    // layer 1, four units at a time
#pragma unroll 1
    for (int j = 0; j < kHidden; j += 4) {
      float h[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float4 wa = w1v[3 * (j + q)], wb = w1v[3 * (j + q) + 1];
        float acc = fmaf(wa.x, x[0], 0.0f);
        acc = fmaf(wa.y, x[1], acc);
        acc = fmaf(wa.z, x[2], acc);
        acc = fmaf(wa.w, x[3], acc);
        acc = fmaf(wb.x, x[4], acc);
        acc = fmaf(wb.y, x[5], acc);
        acc = fmaf(wb.z, x[6], acc);
        acc = fmaf(wb.w, x[7], acc);
        acc = fmaf(sh.w1[kXRow * (j + q) + 8], x[8], acc);
        h[q] = bf16_round(tanh_fast(acc + sh.b1[j + q]));
      }
      *reinterpret_cast<float4 *>(brow + j) = make_float4(h[0], h[1], h[2], h[3]);
    }
    float out = 0.0f;
    {
      float h1[kHidden];
#pragma unroll
      for (int k = 0; k < kHidden; k += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(brow + k);
        h1[k] = v.x; h1[k + 1] = v.y; h1[k + 2] = v.z; h1[k + 3] = v.w;
      }
#pragma unroll 1
      for (int j = 0; j < kHidden; j += 4) {
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int k = 0; k < kHidden; k += 4) {
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const float4 v = w2v[(j + q) * (kHidden / 4) + k / 4];
            acc[q] = fmaf(v.x, h1[k], acc[q]);
            acc[q] = fmaf(v.y, h1[k + 1], acc[q]);
            acc[q] = fmaf(v.z, h1[k + 2], acc[q]);
            acc[q] = fmaf(v.w, h1[k + 3], acc[q]);
          }
        }
        const float4 w3 = w3v[j / 4];
        float4 h;
        h.x = bf16_round(tanh_fast(acc[0] + sh.b2[j]));
        h.y = bf16_round(tanh_fast(acc[1] + sh.b2[j + 1]));
        h.z = bf16_round(tanh_fast(acc[2] + sh.b2[j + 2]));
        h.w = bf16_round(tanh_fast(acc[3] + sh.b2[j + 3]));
        out = fmaf(w3.x, h.x, out);
        out = fmaf(w3.y, h.y, out);
        out = fmaf(w3.z, h.z, out);
        out = fmaf(w3.w, h.w, out);
        *reinterpret_cast<float4 *>(arow + j) = h;
      }
    }
    out += b3;
    const float err = live ? out - target : 0.0f;
    const float d3 = live ? 2.0f * err / (float)batch : 0.0f;
    loss += err * err;
    gb3 += d3;
    __syncwarp();
    // dW3: lane j sums d3 h2[j] over the warp's samples
#pragma unroll 8
    for (int r = 0; r < 32; r++) g3 = fmaf(__shfl_sync(0xffffffffu, d3, r), my.a[r * kRow + lane], g3);
    __syncwarp();
    // d2 over h2, and d1 = (W2^T d2) (1 - h1^2) in registers
    float d1[kHidden];
#pragma unroll
    for (int k = 0; k < kHidden; k++) d1[k] = 0.0f;
#pragma unroll 1
    for (int j = 0; j < kHidden; j += 4) {
      const float4 h = *reinterpret_cast<const float4 *>(arow + j), w3 = w3v[j / 4];
      float d2[4];
      d2[0] = d3 * w3.x * (1.0f - h.x * h.x);
      d2[1] = d3 * w3.y * (1.0f - h.y * h.y);
      d2[2] = d3 * w3.z * (1.0f - h.z * h.z);
      d2[3] = d3 * w3.w * (1.0f - h.w * h.w);
      *reinterpret_cast<float4 *>(arow + j) = make_float4(d2[0], d2[1], d2[2], d2[3]);
#pragma unroll
      for (int q = 0; q < 4; q++) {
#pragma unroll
        for (int k = 0; k < kHidden; k += 4) {
          const float4 v = w2v[(j + q) * (kHidden / 4) + k / 4];
          d1[k] = fmaf(d2[q], v.x, d1[k]);
          d1[k + 1] = fmaf(d2[q], v.y, d1[k + 1]);
          d1[k + 2] = fmaf(d2[q], v.z, d1[k + 2]);
          d1[k + 3] = fmaf(d2[q], v.w, d1[k + 3]);
        }
      }
    }
    __syncwarp();
    // dW2 over the 32 rows of d2 and h1; db2 with it
#pragma unroll 4
    for (int r = 0; r < 32; r++) {
      const float4 da = *reinterpret_cast<const float4 *>(my.a + r * kRow + j0);
      const float4 db = *reinterpret_cast<const float4 *>(my.a + r * kRow + j0 + 4);
      const float4 h = *reinterpret_cast<const float4 *>(my.b + r * kRow + k0);
      const float d[8] = {da.x, da.y, da.z, da.w, db.x, db.y, db.z, db.w};
#pragma unroll
      for (int j = 0; j < 8; j++) {
        g2[j][0] = fmaf(d[j], h.x, g2[j][0]);
        g2[j][1] = fmaf(d[j], h.y, g2[j][1]);
        g2[j][2] = fmaf(d[j], h.z, g2[j][2]);
        g2[j][3] = fmaf(d[j], h.w, g2[j][3]);
      }
      gb2 += my.a[r * kRow + lane];
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kHidden; k += 4) {
      const float4 h = *reinterpret_cast<const float4 *>(brow + k);
      *reinterpret_cast<float4 *>(arow + k) =
          make_float4(d1[k] * (1.0f - h.x * h.x), d1[k + 1] * (1.0f - h.y * h.y), d1[k + 2] * (1.0f - h.z * h.z),
                      d1[k + 3] * (1.0f - h.w * h.w));
    }
    __syncwarp();
    // dW1: lane j over the rows of d1 and x; db1 with it
#pragma unroll 4
    for (int r = 0; r < 32; r++) {
      const float d = my.a[r * kRow + lane];
      const float4 xa = *reinterpret_cast<const float4 *>(my.x + r * kXRow);
      const float4 xb = *reinterpret_cast<const float4 *>(my.x + r * kXRow + 4);
      const float xc = my.x[r * kXRow + 8];
      g1[0] = fmaf(d, xa.x, g1[0]); g1[1] = fmaf(d, xa.y, g1[1]); g1[2] = fmaf(d, xa.z, g1[2]);
      g1[3] = fmaf(d, xa.w, g1[3]); g1[4] = fmaf(d, xb.x, g1[4]); g1[5] = fmaf(d, xb.y, g1[5]);
      g1[6] = fmaf(d, xb.z, g1[6]); g1[7] = fmaf(d, xb.w, g1[7]); g1[8] = fmaf(d, xc, g1[8]);
      gb1 += d;
    }
    __syncwarp();  // the buffers are free again
  }
  // the warp's sums into its own buffers, then over the block's warps in order
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    loss += __shfl_down_sync(0xffffffffu, loss, o);
    gb3 += __shfl_down_sync(0xffffffffu, gb3, o);
  }
  float *sum = reinterpret_cast<float *>(&my);  // a and b
#pragma unroll
  for (int k = 0; k < kIn; k++) sum[kW1 + lane * kIn + k] = g1[k];
  sum[kB1 + lane] = gb1;
#pragma unroll
  for (int j = 0; j < 8; j++)
    *reinterpret_cast<float4 *>(sum + kW2 + (j0 + j) * kHidden + k0) =
        make_float4(g2[j][0], g2[j][1], g2[j][2], g2[j][3]);
  sum[kB2 + lane] = gb2;
  sum[kW3 + lane] = g3;
  if (lane == 0) {
    sum[kB3] = gb3;
    sum[kParams] = loss;
  }
  __syncthreads();
  // warps past the last group hold zeros: leave them out
  const uint32_t own = groups > blockIdx.x ? (groups - blockIdx.x + gridDim.x - 1u) / gridDim.x : 0u;
  const uint32_t warps = min(own, (uint32_t)kTrainWarps);
  float *out_p = partial + (size_t)blockIdx.x * (kParams + 1);
  for (int q = tid; q < kParams + 1; q += kTrainThreads) {
    float acc = 0.0f;
    for (uint32_t v = 0; v < warps; v++) acc += reinterpret_cast<const float *>(&sh.warp[v])[q];
    out_p[q] = acc;
  }
}

// The block partials' sums, grad[q] for q < kParams and grad[kParams] the loss sum, in
// an order that the block count alone sets: 16 threads a parameter, each every 16th
// block, then those 16 in order.  With w also Adam (beta1 0.9, beta2 0.999, eps 1e-8)
// on the binary32 master weights, the batch loss, and, by the last block to come
// here, the step counter (the other blocks have read it by then).  6.4 us with 152
// partials; six blocks of a thread a parameter over 512 partials, and Adam in a
// launch of its own, took 28 us.
constexpr int kReduceParams = 32, kReduceSplit = 16;
constexpr int kReduceBlocks = (kParams + 1 + kReduceParams - 1) / kReduceParams;
__global__ void __launch_bounds__(kReduceParams * kReduceSplit) train_reduce(const float *partial, uint32_t blocks,
                                                                            float *grad, float *w, float *m, float *v,
                                                                            uint32_t *step, uint32_t *ticket, float lr,
                                                                            uint32_t batch, float *loss) {
  __shared__ float part[kReduceSplit][kReduceParams];
  const uint32_t c = threadIdx.x % kReduceParams, r = threadIdx.x / kReduceParams;
  const uint32_t q = blockIdx.x * kReduceParams + c;
  float acc = 0.0f;
  if (q <= (uint32_t)kParams)
    for (uint32_t b = r; b < blocks; b += kReduceSplit) acc += partial[(size_t)b * (kParams + 1) + q];
  part[r][c] = acc;
  const uint32_t t = w ? *step + 1u : 0u;
  __syncthreads();
  if (r == 0 && q <= (uint32_t)kParams) {
    acc = part[0][c];
#pragma unroll
    for (int k = 1; k < kReduceSplit; k++) acc += part[k][c];
    grad[q] = acc;
    if (w && q < (uint32_t)kParams) {
      const float c1 = 1.0f - powf(0.9f, (float)t), c2 = 1.0f - powf(0.999f, (float)t);
      const float mq = 0.9f * m[q] + 0.1f * acc;
      const float vq = 0.999f * v[q] + 0.001f * acc * acc;
      m[q] = mq;
      v[q] = vq;
      w[q] -= lr * (mq / c1) / (sqrtf(vq / c2) + 1e-8f);
    } else if (w) {
      *loss = acc / (float)batch;
    }
  }
  if (w && threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(ticket, 1u) + 1u == gridDim.x) {
      *ticket = 0u;
      *step = t;
    }
  }
}

}  // namespace

struct pw_closure {
  float *w = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr, *partial = nullptr, *loss = nullptr;
  uint32_t *frag = nullptr, *step = nullptr;  // step[0]: steps taken; step[1]: the reducing blocks' ticket
  float *X = nullptr, *Y = nullptr;
  uint64_t n = 0, cap = 0;
  uint32_t partial_blocks = 0;
  cudaStream_t stream = nullptr;
};

namespace {

// Blocks of a training pass: one an SM, fewer for a batch of fewer groups of 32.
uint32_t train_blocks(uint32_t batch) {
  return std::min((batch + 31u) / 32u, multiprocessors());
}

int ensure_partials(pw_closure *c, uint32_t blocks) {
  if (blocks <= c->partial_blocks) return PW_OK;
  cudaFree(c->partial);
  c->partial = nullptr;
  c->partial_blocks = 0;
  PW_TRY(cudaMalloc(&c->partial, (size_t)blocks * (kParams + 1) * sizeof(float)));
  c->partial_blocks = blocks;
  return PW_OK;
}

int refresh_fragments(pw_closure *c) {
  build_fragments<<<1, 1024, 0, c->stream>>>(c->w, c->frag);
  PW_TRY(cudaGetLastError());
  return PW_OK;
}

}  // namespace

namespace pwclosure_host {
// The closure step for a domain with an attached closure (pw_domain.cu).
void launch_closure_step(const StepParams &p, int storage, int op, bool odd, dim3 grid, const uint32_t *frag,
                         const uint8_t *wall, cudaStream_t s) {
  const dim3 blk(32, 4);
  const uint32_t tiles = grid.x * grid.y * grid.z;
  const unsigned g = (unsigned)std::min<uint32_t>(tiles, 4u * multiprocessors());
#define PW_CL_LAUNCH(ST, OPV)                                                                  \
  do {                                                                                        \
    if (odd) closure_step<ST, OPV, true><<<g, blk, 0, s>>>(p, frag, wall, grid.x, grid.y);    \
    else closure_step<ST, OPV, false><<<g, blk, 0, s>>>(p, frag, wall, grid.x, grid.y);       \
  } while (0)
  if (op == pw::OP_REG) {
    if (storage == pw::STORE_F16) PW_CL_LAUNCH(pw::STORE_F16, pw::OP_REG);
    else if (storage == pw::STORE_BF16) PW_CL_LAUNCH(pw::STORE_BF16, pw::OP_REG);
    else PW_CL_LAUNCH(pw::STORE_F32, pw::OP_REG);
  } else {
    if (storage == pw::STORE_F16) PW_CL_LAUNCH(pw::STORE_F16, pw::OP_TRT);
    else if (storage == pw::STORE_BF16) PW_CL_LAUNCH(pw::STORE_BF16, pw::OP_TRT);
    else PW_CL_LAUNCH(pw::STORE_F32, pw::OP_TRT);
  }
#undef PW_CL_LAUNCH
}

template <int ST, int OP, bool ODD, int BLOCKS>
static void closure_pairs_step(const StepParams &p, const uint32_t *frag, const uint8_t *wall, uint32_t runs,
                               uint32_t row_blocks, const ClosureSide &side, bool early, cudaStream_t s) {
  // the blocks that fit at once: the launch bound's count per SM (registers; 20 KB of
  // shared memory and 64 TMEM columns a block leave room for more)
  const uint32_t tiles = runs * row_blocks * p.nz, walk = std::min(tiles, (uint32_t)BLOCKS * multiprocessors());
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(side.edge + side.floor + walk);
  cfg.blockDim = dim3(32, 4);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&cfg, closure_pairs<ST, OP, ODD, BLOCKS>, p, frag, wall, runs, row_blocks, side);
}

template <int ST, int OP, bool ODD>
static void closure_pairs_step(const StepParams &p, const uint32_t *frag, const uint8_t *wall, const uint32_t *list,
                               uint32_t count, uint32_t *taken, bool early, cudaStream_t s,
                               const pwfast::SideStream *beside) {
  const uint32_t runs = (p.nx + 63u) / 64u, row_blocks = (p.ny + 3u) / 4u;
  if (beside) {
    if constexpr (ST != pw::STORE_F32) {
      if (p.floor_rows && p.ny >= 3u)
        pwclosure::aa_step_floor<ST, OP, true, ODD>
            <<<dim3(runs, (p.ny - 2u + pwclosure::BY - 1u) / pwclosure::BY), dim3(pwclosure::BX, pwclosure::BY), 0,
               beside->stream>>>(p);
    }
    if (count)
      pwclosure::aa_step_edges<ST, OP, true, ODD>
          <<<(count + pwclosure::NTHREADS - 1) / pwclosure::NTHREADS, pwclosure::NTHREADS, 0, beside->stream>>>(p, list,
                                                                                                             count);
    const ClosureSide none{list, 0u, 0u, 0u, taken};
    closure_pairs_step<ST, OP, ODD, PW_CLOSURE_PAIR_BLOCKS>(p, frag, wall, runs, row_blocks, none, false, s);
    return;
  }
  ClosureSide side{list, count, (count + pwclosure::NTHREADS - 1) / pwclosure::NTHREADS, 0u, taken};
  if (ST != pw::STORE_F32 && p.floor_rows && p.ny >= 3u) side.floor = runs * ((p.ny - 2u + 3u) / 4u);
  if ((uint64_t)runs * row_blocks * p.nz + side.edge + side.floor <= (uint64_t)PW_CLOSURE_FEW_BLOCKS * multiprocessors())
    closure_pairs_step<ST, OP, ODD, PW_CLOSURE_FEW_BLOCKS>(p, frag, wall, runs, row_blocks, side, early, s);
  else
    closure_pairs_step<ST, OP, ODD, PW_CLOSURE_PAIR_BLOCKS>(p, frag, wall, runs, row_blocks, side, early, s);
}

// The line between a long run's two forms.  A step of few tiles is as long as one tile or one
// edge cell, and captured steps follow one another closer than early launches; more tiles
// fill the GPU, and blocks that take tiles as they come win.  A step in a run of 256, early
// launches and captured: FP32 REG with a floor 64x32x32 13.7 and 12.4 us, 33x17x17 13.1 and
// 10.9, 66x33x33 15.7 and 15.1, 72x36x36 (648 tiles) 15.4 and 16.4; FP16 with nx odd and a
// floor 33x17x17 15.0 and 11.7, 65x33x33 18.1 and 15.9, 73x37x37 16.9 and 17.5.  With few
// edge cells the line is later (a sphere without a floor, FP16: 72x36x36 18.5 and 15.8,
// 73x37x37 18.7 and 16.8, 88x44x44 18.0 and 19.7).  With the floor layer in a kernel of its
// own the early launches are the faster ones at any size (FP16 64x32x32 16.1 and 16.3).
// FP32 TRT with many edge cells (a floor) is faster captured again once the tiles fill the
// GPU: 97x49x49 29.0 and 28.4, 104x52x52 31.6 and 30.0, 128x64x64 42.1 and 41.0, 160x80x80
// 81.5 and 77.0; REG is not (97x49x49 24.0 and 24.7, 128x64x64 34.5 and 35.9).
bool closure_long_runs_captured(uint32_t nx, uint32_t ny, uint32_t nz, int storage, int op, int floor_rows,
                                uint32_t count) {
  if (floor_rows && ny >= 3u) return false;
  const uint64_t tiles = (uint64_t)((nx + 63u) / 64u) * ((ny + 3u) / 4u) * nz, sms = (uint64_t)multiprocessors();
  const uint64_t edge = (count + pwclosure::NTHREADS - 1) / pwclosure::NTHREADS;
  const bool many = 8u * edge >= sms;
  return 5u * tiles <= (many ? 21u : 25u) * sms ||
         (storage == pw::STORE_F32 && op == pw::OP_TRT && many && tiles >= 8u * sms);
}

void launch_closure_pairs(const StepParams &p, int storage, int op, bool odd, const uint32_t *frag,
                          const uint8_t *wall, const uint32_t *list, uint32_t count, uint32_t *taken,
                          bool early, cudaStream_t s, const pwfast::SideStream *side) {
  if (side) {
    cudaEventRecord(side->fork, s);
    cudaStreamWaitEvent(side->stream, side->fork, 0);
  }
#define PW_CLP(ST, OPV)                                                                            \
  do {                                                                                             \
    if (odd) closure_pairs_step<ST, OPV, true>(p, frag, wall, list, count, taken, early, s, side); \
    else closure_pairs_step<ST, OPV, false>(p, frag, wall, list, count, taken, early, s, side);    \
  } while (0)
  if (op == pw::OP_REG) {
    if (storage == pw::STORE_F16) PW_CLP(pw::STORE_F16, pw::OP_REG);
    else if (storage == pw::STORE_BF16) PW_CLP(pw::STORE_BF16, pw::OP_REG);
    else PW_CLP(pw::STORE_F32, pw::OP_REG);
  } else {
    if (storage == pw::STORE_F16) PW_CLP(pw::STORE_F16, pw::OP_TRT);
    else if (storage == pw::STORE_BF16) PW_CLP(pw::STORE_BF16, pw::OP_TRT);
    else PW_CLP(pw::STORE_F32, pw::OP_TRT);
  }
#undef PW_CLP
  if (side) {
    cudaEventRecord(side->join, side->stream);
    cudaStreamWaitEvent(s, side->join, 0);
  }
}

int wall_distance_of(const uint32_t *flags, uint32_t nx, uint32_t ny, uint32_t nz, uint8_t *out, cudaStream_t s) {
  const size_t cells = (size_t)nx * ny * nz;
  uint8_t *tmp = nullptr;
  PW_TRY(cudaMalloc(&tmp, cells));
  dist_init<<<(unsigned)((cells + 255) / 256), 256, 0, s>>>(flags, cells, out);
  int rc = wall_distance(out, tmp, nx, ny, nz, s);
  cudaStreamSynchronize(s);
  cudaFree(tmp);
  return rc;
}

const uint32_t *fragments(const pw_closure *c) { return c->frag; }
}  // namespace pwclosure_host

extern "C" {

int pw_closure_create(uint64_t seed, pw_closure **out) {
  if (!out) { set_error("NULL argument"); return PW_ERR_INVALID; }
  *out = nullptr;
  pw_closure *c = new pw_closure();
  cudaError_t e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc(&c->w, kParams * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&c->m, kParams * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&c->v, kParams * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&c->grad, (kParams + 1) * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&c->loss, 2 * sizeof(float));  // the latest step's, a call's first
  if (e == cudaSuccess) e = cudaMalloc(&c->frag, 32 * kFragWords * sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMalloc(&c->step, 2 * sizeof(uint32_t));
  if (e != cudaSuccess) {
    int rc = cuda_status(e, "pw_closure_create");
    pw_closure_destroy(c);
    return rc;
  }
  // Glorot-uniform hidden layers (seeded), zero biases, zero output layer: the
  // untrained network outputs c = 0, plain Smagorinsky.
  std::vector<float> w(kParams, 0.0f);
  uint64_t state = seed;
  auto uniform = [&]() {
    state += 0x9E3779B97F4A7C15ull;
    uint64_t z = state;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
  };
  const double a1 = std::sqrt(6.0 / (kIn + kHidden)), a2 = std::sqrt(6.0 / (2 * kHidden));
  for (int k = 0; k < kHidden * kIn; k++) w[kW1 + k] = (float)(a1 * uniform());
  for (int k = 0; k < kHidden * kHidden; k++) w[kW2 + k] = (float)(a2 * uniform());
  e = cudaMemcpy(c->w, w.data(), kParams * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(c->m, 0, kParams * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(c->v, 0, kParams * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(c->step, 0, 2 * sizeof(uint32_t));
  if (e != cudaSuccess) {
    int rc = cuda_status(e, "pw_closure_create");
    pw_closure_destroy(c);
    return rc;
  }
  int rc = refresh_fragments(c);
  if (rc == PW_OK) rc = cudaStreamSynchronize(c->stream) == cudaSuccess ? PW_OK : PW_ERR_CUDA;
  if (rc != PW_OK) { pw_closure_destroy(c); return rc; }
  *out = c;
  return PW_OK;
}

void pw_closure_destroy(pw_closure *c) {
  if (!c) return;
  if (c->stream) cudaStreamSynchronize(c->stream);
  cudaFree(c->w); cudaFree(c->m); cudaFree(c->v); cudaFree(c->grad); cudaFree(c->loss);
  cudaFree(c->frag); cudaFree(c->step); cudaFree(c->partial); cudaFree(c->X); cudaFree(c->Y);
  if (c->stream) cudaStreamDestroy(c->stream);
  cudaGetLastError();
  delete c;
}

int pw_closure_get_params(pw_closure *c, float *out) {
  if (!c || !out) { set_error("NULL argument"); return PW_ERR_INVALID; }
  PW_TRY(cudaMemcpyAsync(out, c->w, kParams * sizeof(float), cudaMemcpyDeviceToHost, c->stream));
  PW_TRY(cudaStreamSynchronize(c->stream));
  return PW_OK;
}

int pw_closure_set_params(pw_closure *c, const float *in) {
  if (!c || !in) { set_error("NULL argument"); return PW_ERR_INVALID; }
  for (int k = 0; k < kParams; k++)
    if (!std::isfinite(in[k])) { set_error("Closure parameters must be finite."); return PW_ERR_INVALID; }
  PW_TRY(cudaMemcpyAsync(c->w, in, kParams * sizeof(float), cudaMemcpyHostToDevice, c->stream));
  PW_TRY(cudaMemsetAsync(c->m, 0, kParams * sizeof(float), c->stream));
  PW_TRY(cudaMemsetAsync(c->v, 0, kParams * sizeof(float), c->stream));
  PW_TRY(cudaMemsetAsync(c->step, 0, sizeof(uint32_t), c->stream));
  int rc = refresh_fragments(c);
  if (rc != PW_OK) return rc;
  PW_TRY(cudaStreamSynchronize(c->stream));
  return PW_OK;
}

int pw_closure_eval(pw_closure *c, const float *x, uint32_t count, float *out) {
  if (!c || (!x && count) || (!out && count)) { set_error("NULL argument"); return PW_ERR_INVALID; }
  if (!count) return PW_OK;
  float *dx = nullptr, *dy = nullptr;
  uint32_t *dstatus = nullptr, status = 0;
  PW_TRY(cudaMalloc(&dx, (size_t)count * kIn * sizeof(float)));
  cudaError_t e = cudaMalloc(&dy, (size_t)count * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&dstatus, sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMemsetAsync(dstatus, 0, sizeof(uint32_t), c->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dx, x, (size_t)count * kIn * sizeof(float), cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) {
    eval_kernel<<<(count + 127) / 128, 128, 0, c->stream>>>(c->frag, dx, count, dy, dstatus);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, dy, (size_t)count * sizeof(float), cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&status, dstatus, sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  cudaFree(dx);
  cudaFree(dy);
  cudaFree(dstatus);
  if (e != cudaSuccess) return cuda_status(e, "pw_closure_eval");
  if (status) {
    set_error("pw_closure_eval: a tensor-core layer did not complete in time");
    return PW_ERR_TIMEOUT;
  }
  return PW_OK;
}

int pw_closure_gradients(pw_closure *c, const float *x, const float *y, uint32_t count, float *grad, float *loss) {
  if (!c || !x || !y || !grad || count == 0) { set_error("NULL argument or no samples"); return PW_ERR_INVALID; }
  float *dx = nullptr, *dy = nullptr;
  uint32_t *idx = nullptr;
  const uint32_t blocks = train_blocks(count);
  int rc = ensure_partials(c, blocks);
  if (rc != PW_OK) return rc;
  PW_TRY(cudaFuncSetAttribute(train_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainShared)));
  cudaError_t e = cudaMalloc(&dx, (size_t)count * kIn * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&dy, (size_t)count * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&idx, (size_t)count * sizeof(uint32_t));
  std::vector<uint32_t> seq(count);
  for (uint32_t i = 0; i < count; i++) seq[i] = i;
  if (e == cudaSuccess) e = cudaMemcpyAsync(dx, x, (size_t)count * kIn * sizeof(float), cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dy, y, (size_t)count * sizeof(float), cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(idx, seq.data(), (size_t)count * sizeof(uint32_t), cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) {
    train_block<<<blocks, kTrainThreads, sizeof(TrainShared), c->stream>>>(c->w, dx, dy, count, count, 0, c->step, idx,
                                                                           c->partial);
    train_reduce<<<kReduceBlocks, kReduceParams * kReduceSplit, 0, c->stream>>>(
        c->partial, blocks, c->grad, nullptr, nullptr, nullptr, nullptr, nullptr, 0.0f, count, nullptr);
    e = cudaGetLastError();
  }
  std::vector<float> h(kParams + 1);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), c->grad, (kParams + 1) * sizeof(float), cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  cudaFree(dx); cudaFree(dy); cudaFree(idx);
  if (e != cudaSuccess) return cuda_status(e, "pw_closure_gradients");
  std::copy(h.begin(), h.begin() + kParams, grad);
  if (loss) *loss = h[kParams] / (float)count;
  return PW_OK;
}

int pw_closure_dataset_clear(pw_closure *c) {
  if (!c) { set_error("NULL argument"); return PW_ERR_INVALID; }
  c->n = 0;
  return PW_OK;
}

int pw_closure_dataset_reserve(pw_closure *c, uint64_t capacity) {
  if (!c) { set_error("NULL argument"); return PW_ERR_INVALID; }
  if (capacity <= c->cap) return PW_OK;
  float *nx = nullptr, *ny = nullptr;
  PW_TRY(cudaMalloc(&nx, capacity * kIn * sizeof(float)));
  cudaError_t e = cudaMalloc(&ny, capacity * sizeof(float));
  if (e == cudaSuccess && c->n) e = cudaMemcpy(nx, c->X, c->n * kIn * sizeof(float), cudaMemcpyDeviceToDevice);
  if (e == cudaSuccess && c->n) e = cudaMemcpy(ny, c->Y, c->n * sizeof(float), cudaMemcpyDeviceToDevice);
  if (e != cudaSuccess) { cudaFree(nx); cudaFree(ny); return cuda_status(e, "pw_closure_dataset_reserve"); }
  cudaFree(c->X); cudaFree(c->Y);
  c->X = nx; c->Y = ny; c->cap = capacity;
  return PW_OK;
}

int pw_closure_dataset_write(pw_closure *c, const float *x, const float *y, uint64_t count) {
  if (!c || (count && (!x || !y))) { set_error("NULL argument"); return PW_ERR_INVALID; }
  int rc = pw_closure_dataset_reserve(c, count ? count : 1);
  if (rc != PW_OK) return rc;
  if (count) {
    PW_TRY(cudaMemcpy(c->X, x, count * kIn * sizeof(float), cudaMemcpyHostToDevice));
    PW_TRY(cudaMemcpy(c->Y, y, count * sizeof(float), cudaMemcpyHostToDevice));
  }
  c->n = count;
  return PW_OK;
}

int pw_closure_dataset_size(const pw_closure *c, uint64_t *n) {
  if (!c || !n) { set_error("NULL argument"); return PW_ERR_INVALID; }
  *n = c->n;
  return PW_OK;
}

int pw_closure_dataset_read(pw_closure *c, uint64_t first, uint64_t count, float *x, float *y) {
  if (!c || (count && (!x || !y))) { set_error("NULL argument"); return PW_ERR_INVALID; }
  if (first + count > c->n) { set_error("Dataset range beyond its %llu samples.", (unsigned long long)c->n); return PW_ERR_INVALID; }
  if (!count) return PW_OK;
  PW_TRY(cudaMemcpy(x, c->X + first * kIn, count * kIn * sizeof(float), cudaMemcpyDeviceToHost));
  PW_TRY(cudaMemcpy(y, c->Y + first, count * sizeof(float), cudaMemcpyDeviceToHost));
  return PW_OK;
}

// Append the samples of a fine domain's latest macros (the last step must have
// written them) at the given coarse molecular viscosity.
int pw_closure_dataset_add(pw_closure *c, pw_domain *fine, double nu0_coarse, uint64_t *added) {
  if (!c || !fine) { set_error("NULL argument"); return PW_ERR_INVALID; }
  uint32_t nx, ny, nz;
  domain_dims(fine, &nx, &ny, &nz);
  if (nx % 2 || ny % 2 || nz % 2 || nx < 10 || ny < 4 || nz < 4) {
    set_error("The fine grid must have even dimensions of at least 10 x 4 x 4.");
    return PW_ERR_INVALID;
  }
  if (!(nu0_coarse > 0.0) || !std::isfinite(nu0_coarse)) { set_error("The coarse viscosity must be positive."); return PW_ERR_INVALID; }
  void *macros = nullptr, *flags = nullptr, *stream = nullptr;
  int rc = pw_domain_buffers(fine, &macros, &flags, &stream);
  if (rc != PW_OK) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  const uint32_t cx = nx / 2, cy = ny / 2, cz = nz / 2;
  const size_t nc = (size_t)cx * cy * cz;
  float *co = nullptr;
  uint8_t *solid = nullptr, *dist = nullptr, *tmp = nullptr;
  uint32_t *counts = nullptr;
  const uint32_t nblk = (uint32_t)((nc + kScanBlock - 1) / kScanBlock);
  cudaError_t e = cudaMalloc(&co, 10 * nc * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&solid, nc);
  if (e == cudaSuccess) e = cudaMalloc(&dist, nc);
  if (e == cudaSuccess) e = cudaMalloc(&tmp, nc);
  if (e == cudaSuccess) e = cudaMalloc(&counts, (nblk + 1) * sizeof(uint32_t));
  uint32_t total = 0;
  float u_in = 0.0f;
  if (e == cudaSuccess) {
    pw::StepParams p = member_params(fine, 2, 0);
    u_in = p.u_in;
    coarsen_kernel<<<(unsigned)((nc + 255) / 256), 256, 0, s>>>((const float4 *)macros, (const uint32_t *)flags, nx, ny,
                                                                 nz, co, solid);
    dist_from_solid<<<(unsigned)((nc + 255) / 256), 256, 0, s>>>(solid, nc, dist);
    rc = wall_distance(dist, tmp, cx, cy, cz, s);
    sample_count<<<nblk, kScanBlock, 0, s>>>(co, dist, cx, cy, cz, (float)nu0_coarse, u_in, counts);
    scan_counts<<<1, kScanBlock, 0, s>>>(counts, nblk, counts + nblk);
    e = cudaMemcpyAsync(&total, counts + nblk, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  if (e == cudaSuccess && rc == PW_OK) {
    const uint64_t need = c->n + total;
    if (need > c->cap) rc = pw_closure_dataset_reserve(c, std::max<uint64_t>(need, c->cap * 2));
  }
  if (e == cudaSuccess && rc == PW_OK) {
    sample_write<<<nblk, kScanBlock, 0, s>>>(co, dist, cx, cy, cz, (float)nu0_coarse, u_in, counts, c->n, c->cap,
                                             c->X, c->Y);
    e = cudaStreamSynchronize(s);
  }
  cudaFree(co); cudaFree(solid); cudaFree(dist); cudaFree(tmp); cudaFree(counts);
  if (e != cudaSuccess) return cuda_status(e, "pw_closure_dataset_add");
  if (rc != PW_OK) return rc;
  c->n += total;
  if (added) *added = total;
  return PW_OK;
}

// Adam over `steps` minibatches of `batch` samples drawn by a seeded hash from
// the dataset; first and last batch losses (mean squared error of c).
int pw_closure_train(pw_closure *c, uint32_t steps, uint32_t batch, float lr, uint64_t seed, float *loss_first,
                     float *loss_last) {
  if (!c || steps == 0 || batch == 0 || !(lr > 0.0f)) { set_error("Training needs steps, a batch and a positive rate."); return PW_ERR_INVALID; }
  if (c->n == 0) { set_error("The closure dataset is empty."); return PW_ERR_INVALID; }
  const uint32_t blocks = train_blocks(batch);
  int rc = ensure_partials(c, blocks);
  if (rc != PW_OK) return rc;
  PW_TRY(cudaFuncSetAttribute(train_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainShared)));
  auto one = [&](cudaStream_t s) {
    train_block<<<blocks, kTrainThreads, sizeof(TrainShared), s>>>(c->w, c->X, c->Y, c->n, batch, seed, c->step,
                                                                   nullptr, c->partial);
    train_reduce<<<kReduceBlocks, kReduceParams * kReduceSplit, 0, s>>>(c->partial, blocks, c->grad, c->w, c->m, c->v,
                                                                        c->step, c->step + 1, lr, batch, c->loss);
  };
  one(c->stream);
  PW_TRY(cudaGetLastError());
  // kept on the device until the end: a copy to the host here would hold back the launches
  PW_TRY(cudaMemcpyAsync(c->loss + 1, c->loss, sizeof(float), cudaMemcpyDeviceToDevice, c->stream));
  // the rest as replays of a captured 100-step graph
  uint32_t done = 1;
  const uint32_t chunk = 100;
  cudaGraphExec_t exec = nullptr;
  if (steps - done >= chunk) {
    cudaStream_t cap;
    PW_TRY(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
    cudaGraph_t graph = nullptr;
    if (cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
      for (uint32_t k = 0; k < chunk; k++) one(cap);
      if (cudaStreamEndCapture(cap, &graph) == cudaSuccess && graph) {
        if (cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) exec = nullptr;
        cudaGraphDestroy(graph);
      }
    }
    cudaStreamDestroy(cap);
    cudaGetLastError();
  }
  while (exec && steps - done >= chunk) {
    if (cudaGraphLaunch(exec, c->stream) != cudaSuccess) break;
    done += chunk;
  }
  if (exec) cudaGraphExecDestroy(exec);
  for (; done < steps; done++) one(c->stream);
  PW_TRY(cudaGetLastError());
  rc = refresh_fragments(c);
  if (rc != PW_OK) return rc;
  float losses[2];
  PW_TRY(cudaMemcpyAsync(losses, c->loss, sizeof losses, cudaMemcpyDeviceToHost, c->stream));
  PW_TRY(cudaStreamSynchronize(c->stream));
  if (loss_last) *loss_last = losses[0];
  if (loss_first) *loss_first = losses[1];
  return PW_OK;
}

}  // extern "C"
