// The one-launch step's host side and its binary32 kernels (pw_step_all.cuh).
#include "pw_step_all.cuh"

namespace pwall {

extern template void launch_storage<STORE_F16>(const StepParams &, int, int, bool, const uint32_t *, uint32_t,
                                               cudaStream_t, bool);
extern template void launch_storage<STORE_BF16>(const StepParams &, int, int, bool, const uint32_t *, uint32_t,
                                                cudaStream_t, bool);

// Whether a domain's steps may run in one launch.  Binary32 storage: always (the vehicle
// at 64^2 x 128 23.4 us before and 15.0 now; a large domain of the regularized operator that
// steps on its own is split, pw_domain.cu's split_in_one).  16-bit cell
// pairs up to 3.7 M cells with LES, 2.6 M without (split and one launch, by eight steps:
// FP16 REG LES 224x112x112 55.5 and 54.3 us, 240x120x120 64.1 and 63.5, 256x128x128 74.3
// and 74.2, BF16 there 73.0 and 74.1, 320x160x160 136.2 and 139.6; FP16 TRT 224x112x112
// 53.3 and 54.5, 300x150x150 113.6 and 119.3): past that the side kernels' own register
// counts pay more than the launches cost; and not beside reflecting seam rows, which take
// one cell a thread (with nx even only the split step is built and measured for them: a
// free-slip FP16 TRT sphere 96x48x48 20.1 us a step in calls of 8, 14.2 in captured runs).  16-bit storage with nx odd: any size (203x101x67 without LES
// 35.0 and 24.4, 399x200x200 308 and 266; FP16 REG with LES 97x48x48 25.4 and 15.9,
// 203x101x101 48.5 and 37.2, 399x199x199 299 and 266; free-slip BF16 97x48x48 59 and
// 17), but FP16 TRT with LES: the compiler rounds that seam's rows differently in this
// kernel than in aa_step_seam, in the last bit, and the stored codes with it.
// The side blocks take at most five slices a plane, and a grid has 65,535.
bool step_all_supported(uint32_t nx, uint32_t ny, uint32_t nz, int storage, int op, int les, uint32_t slip) {
  if (nx < 3u || ny < 3u || nz < 3u || nz > 8192u) return false;
  if (storage == STORE_F32) return true;
  if (nx & 1u) return !(les && op == OP_TRT && storage == STORE_F16) && (uint64_t)nx * ny < (1ull << 31) - 2048u;
  return slip == 0u && (uint64_t)nx * ny * nz <= (les ? 7ull : 5ull) << 19;
}

void launch_step_all(const StepParams &p, int storage, int op, int les, bool odd, const uint32_t *list, uint32_t count,
                     cudaStream_t s, bool early) {
  if (storage == STORE_F16) launch_storage<STORE_F16>(p, op, les, odd, list, count, s, early);
  else if (storage == STORE_BF16) launch_storage<STORE_BF16>(p, op, les, odd, list, count, s, early);
  else launch_storage<STORE_F32>(p, op, les, odd, list, count, s, early);
}

}  // namespace pwall
