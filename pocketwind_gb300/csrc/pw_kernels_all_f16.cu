// The one-launch step's FP16 kernels (pw_step_all.cuh).
#include "pw_step_all.cuh"

namespace pwall {
template void launch_storage<STORE_F16>(const StepParams &, int, int, bool, const uint32_t *, uint32_t, cudaStream_t,
                                       bool);
}
