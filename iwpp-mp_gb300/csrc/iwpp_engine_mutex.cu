// iwpp_engine_mutex.cu -- the engine's kernels of the mutex queue.
#include "iwpp_engine_kernel.cuh"

namespace iwpp {
template void* kernel_for<VAR_MUTEX>(int, int, int, int);
}
