// fjb_launches.h -- what launches share: the process-wide count of them, and the shared memory
// that a kernel may ask for.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace fjb {

// Called next to every kernel launch of the render path; read through
// fjb_kernel_launches().
void count_launch();

// Lets `kernel` be launched with `need` bytes of dynamic shared memory, besides `own` bytes of
// static arrays. The limit belongs to the function, not to a launch: a host thread that set its
// own call's size could lower it between another thread's setting and launch, which is then
// refused. So it is only ever set to the largest size, 227 KB (what a CTA can have on sm_100)
// less the static arrays; up to 48 KB needs no setting.
template <typename Kernel>
inline cudaError_t allow_dynamic_smem(Kernel* kernel, size_t need, size_t own = 0) {
    constexpr size_t kLargest = 227 * 1024, kAlways = 48 * 1024;
    if (need + own <= kAlways) return cudaSuccess;
    if (need + own > kLargest) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kLargest - own));
}

} // namespace fjb
