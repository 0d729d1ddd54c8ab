// iwpp_engine_double.cu -- the engine's kernels of the double queue.
#include "iwpp_engine_kernel.cuh"

namespace iwpp {
template void* kernel_for<VAR_DOUBLE>(int, int, int, int);
}
