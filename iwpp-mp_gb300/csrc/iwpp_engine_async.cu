// iwpp_engine_async.cu -- the engine's kernels of the async queue.
#include "iwpp_engine_kernel.cuh"

namespace iwpp {
template void* kernel_for<VAR_ASYNC>(int, int, int, int);
}
