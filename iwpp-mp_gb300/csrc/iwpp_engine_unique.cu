// iwpp_engine_unique.cu -- the engine's kernels of the unique queue.
#include "iwpp_engine_kernel.cuh"

namespace iwpp {
template void* kernel_for<VAR_UNIQUE>(int, int, int, int);
}
