// iwpp_engine.cu -- job initialisation, queue self-test and the host side of
// the persistent tile engine.
#include <algorithm>
#include <atomic>
#include <cstdio>

#include "iwpp_engine_kernel.cuh"

namespace iwpp {

// Job initialisation: every tile DIRTY; round 0 (double / unique) is the
// virtual list of all tiles; the mutex stack holds every tile so that the
// first pops come out in raster order (IWPP MP/src/globalQueue.cu:83-97,
// initFillGlobalQueue).  After the front stage (or a seed check alone) the
// check has set the tile states and listed the tiles to start from: the
// mutex stack and the first round's read queue are that list, the async
// ring starts from it; the stage's error word and top-pixel count stand.  A
// list that is longer than the double queue holds is left for the virtual
// list of all tiles, as after an overflow: tiles that are not DIRTY are
// released unvisited.
__global__ void engine_init_kernel(EngineArgs a, int variant) {
    const unsigned stride = gridDim.x * blockDim.x;
    const bool seeded = a.init_list != nullptr;
    unsigned n0 = a.G;
    if (seeded) n0 = min(*(const volatile unsigned*)a.init_count, a.G);
    for (unsigned g = blockIdx.x * blockDim.x + threadIdx.x; g < a.G; g += stride) {
        if (!seeded && !a.states_set) a.state[g] = ST_DIRTY | ST_SIDES;
        if (variant == VAR_MUTEX && g < a.cap) a.q0[g] = seeded ? (g < n0 ? a.init_list[g] : 0u) : a.G - 1u - g;
        if ((variant == VAR_DOUBLE || variant == VAR_UNIQUE) && seeded && g < n0 && g < a.cap) a.q0[g] = a.init_list[g];
    }
    if (variant == VAR_ASYNC)
        for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < a.cap; i += stride) a.q0[i] = 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        Ctrl* c = a.ctrl;
        const bool listed = seeded && !(variant == VAR_DOUBLE && n0 > a.cap);
        c->rn = listed ? n0 : a.G;
        c->wn = 0u;
        c->rcur = 0u;
        c->qsel = 0u;
        c->vfull = listed ? 0u : 1u;
        c->done = n0 == 0u && !a.phantom ? 1u : 0u;
        c->overflow = n0 > a.cap && variant == VAR_MUTEX ? 1u : 0u;
        c->restarts = 0u;
        c->rounds = 0u;
        c->bar_count = 0u;
        c->bar_gen = 0u;
        if (!a.front) c->error = 0u;  // else the seed check's job keeps its error word
        c->lock_next = 0u;
        // the mutex stack's first entries: a slice per CTA taken without the
        // lock when the kernel starts (at most half a CTA buffer each), the
        // rest stacked
        const unsigned stacked = n0 < a.cap ? n0 : a.cap;
        const unsigned ctas = a.grid > 0 ? (unsigned)a.grid : 1u;
        unsigned pf = variant == VAR_MUTEX ? stacked / ctas : 0u;
        if (pf > (unsigned)kMutexPrefill) pf = (unsigned)kMutexPrefill;
        c->prefill = pf;
        c->prefill_base = stacked - pf * ctas;
        c->lock_word = (unsigned long long)(stacked - pf * ctas) << 32;  // ticket 0 served
        c->pending = (int)(n0 < a.cap ? n0 : a.cap);
        c->progress = 0u;
        c->idle = 0u;
        c->ahead = 0u;
        c->atail = n0;
        c->ninit = n0;
        if (variant == VAR_ASYNC) c->pending = (int)n0;
        // test hook: one pending entry that nobody inserts or finishes, so
        // the waiting warps never see the job end and their bounded waits
        // run out (the round-based queues stall at their barrier instead)
        if (a.phantom) c->pending += 1;
        c->visits = 0ull;
        c->sweeps = 0ull;
        c->pushes = 0ull;
        c->row_steps = 0ull;
        for (int i = 0; i < 5; ++i) c->phase[i] = 0ull;
        if (!a.front) c->top_pixels = 0ull;  // else the top-level stage's count stands
        if (!a.front_gated) c->front_gate = a.front_ran ? 1u : 0u;  // else the device's decision stands
    }
}

// ------------------------------------------------------- queue self-test
// The counterpart of the reference's queue test (IWPP MP DQ/src/
// globalQueue.cu:161-253: fill a 128 x 128 tile-id queue several times, read
// it back, check every id's count): all warps insert every tile id `copies`
// times at once through the variant's own insertion path (push_entries:
// mutex stack, warp-aggregated write-queue reservations, async ring; the
// unique queue deduplicates through the tile state word as notify does),
// then the queue's contents are counted per id.
struct QueueTest {
    unsigned* hist;          // G counters
    unsigned long long* out;  // [0] entries found, [1] ids with a wrong count, [2] smallest such id
};

__global__ void queue_test_init_kernel(EngineArgs a, QueueTest t) {
    const unsigned stride = gridDim.x * blockDim.x;
    for (unsigned g = blockIdx.x * blockDim.x + threadIdx.x; g < a.G; g += stride) {
        a.state[g] = 0u;
        t.hist[g] = 0u;
    }
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < a.cap; i += stride) {
        a.q0[i] = 0u;
        a.q1[i] = 0u;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        Ctrl* c = a.ctrl;
        c->wn = 0u;
        c->overflow = 0u;
        c->error = 0u;
        c->lock_next = 0u;
        c->lock_word = 0ull;
        c->pending = 0;
        c->atail = a.G;  // ring positions below G are the (absent) initial tiles
        t.out[0] = 0ull;
        t.out[1] = 0ull;
        t.out[2] = ~0ull;
    }
}

template <int VAR>
__global__ void queue_test_insert_kernel(EngineArgs a, int copies) {
    const int lane = threadIdx.x & 31;
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned nwarps = (gridDim.x * blockDim.x) >> 5;
    const unsigned total = a.G * (unsigned)copies;
    for (unsigned base = warp * 32u; base < total; base += nwarps * 32u) {
        const unsigned idx = base + (unsigned)lane;
        bool want = idx < total;
        const unsigned g = want ? idx % a.G : 0u;
        if (VAR == VAR_UNIQUE && want) want = (atomicOr(&a.state[g], ST_DIRTY) & ST_DIRTY) == 0u;
        push_entries<VAR>(a, want, g, lane, a.q1);
        if (ld_volatile(&a.ctrl->error) != 0u) return;
    }
}

__global__ void queue_test_count_kernel(EngineArgs a, int variant, QueueTest t) {
    const Ctrl* c = a.ctrl;
    unsigned n;
    if (variant == VAR_MUTEX) n = (unsigned)stack_top(c);
    else if (variant == VAR_ASYNC) n = c->atail - a.G;
    else n = c->wn;
    if (n > a.cap) n = a.cap;
    if (blockIdx.x == 0 && threadIdx.x == 0) t.out[0] = n;
    const unsigned stride = gridDim.x * blockDim.x;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        unsigned e = variant == VAR_MUTEX ? a.q0[i] : variant == VAR_ASYNC ? a.q0[i] - 1u : a.q1[i];
        if (e < a.G) atomicAdd(&t.hist[e], 1u);
    }
}

__global__ void queue_test_check_kernel(EngineArgs a, QueueTest t, unsigned expect) {
    const unsigned stride = gridDim.x * blockDim.x;
    for (unsigned g = blockIdx.x * blockDim.x + threadIdx.x; g < a.G; g += stride) {
        if (t.hist[g] != expect) {
            atomicAdd(&t.out[1], 1ull);
            atomicMin(&t.out[2], (unsigned long long)g);
        }
    }
}

cudaError_t queue_selftest(const EngineArgs& a, int variant, int copies, unsigned* hist, unsigned long long* out,
                           int device, cudaStream_t s) {
    int sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    QueueTest t{hist, out};
    const unsigned blocks = (unsigned)sms * 4u;
    queue_test_init_kernel<<<blocks, 256, 0, s>>>(a, t);
    switch (variant) {
        case VAR_MUTEX: queue_test_insert_kernel<VAR_MUTEX><<<blocks, 128, 0, s>>>(a, copies); break;
        case VAR_DOUBLE: queue_test_insert_kernel<VAR_DOUBLE><<<blocks, 128, 0, s>>>(a, copies); break;
        case VAR_UNIQUE: queue_test_insert_kernel<VAR_UNIQUE><<<blocks, 128, 0, s>>>(a, copies); break;
        default: queue_test_insert_kernel<VAR_ASYNC><<<blocks, 128, 0, s>>>(a, copies); break;
    }
    queue_test_count_kernel<<<blocks, 256, 0, s>>>(a, variant, t);
    queue_test_check_kernel<<<blocks, 256, 0, s>>>(a, t, variant == VAR_UNIQUE ? 1u : (unsigned)copies);
    return cudaGetLastError();
}

// ------------------------------------------------------------ host side
// The engine's kernel shapes: tile height, and warps per tile for the passes or
// one of the alternative in-tile solvers.
enum Shape : int { T32_W4, T64_W8, T64_W4, T64_W2, T32_SWEEPS, T64_SWEEPS, T32_PQ, T64_PQ, SHAPES };

// Shape of a job's kernel.  solver: iwpp_config.solver (0 and 2 are the
// passes, 1 the row sweeps, 3 the pixel queue).  Warps per tile:
// the fewer tiles an SM has, the more warps work on one, since only a part
// of a job's tiles can be visited at any time and a visit's length then sets
// the pace; with many tiles the warps that wait for others of their tile cost
// more.  Measured on h-dome images, 8 / 4 / 2 warps per 64-row tile, us:
//   tiles per SM   0.8 (1024^2 u8)  68 / 76 / 86
//                  3.4 (2048^2 u8)  88 / 90 / 99
//                  7.6 (3072^2 u8)  126 / 113 / 116
//                 13.5 (4096^2 u8)  195 / 152 / 144, 8-connected 366 / 331 / 322
//                 30   (6144^2 u8)  400 / 298 / 256
//                 54   (8192^2 u8)  791 / 561 / 453
// A grid that the caller limits (grid_ctas > 0) works on that many tiles at
// most, with as many warps per tile as leave that many CTAs resident.  4096^2 u8
// 8-connected h-domes, us, by the rule for the tiles alone / so: 8 CTAs 13132 /
// 9158, 38 2990 / 2082, 304 488 / 394.
static Shape select_shape(int tile_rows, int solver, long long tiles, int grid_ctas, int sms) {
    if (solver == 1) return tile_rows == 32 ? T32_SWEEPS : T64_SWEEPS;
    if (solver == 3) return tile_rows == 32 ? T32_PQ : T64_PQ;
    if (tile_rows == 32) return T32_W4;
    if (4 * tiles <= 27ll * sms || (grid_ctas > 0 && grid_ctas <= 3ll * sms)) return T64_W8;
    return 2 * tiles <= 25ll * sms || (grid_ctas > 0 && grid_ctas <= 6ll * sms) ? T64_W4 : T64_W2;
}

struct Kernel {
    void* fn;
    int threads;
    size_t smem;
    int workers;  // tiles that a CTA works on at a time
};
static Kernel kernel_of(int variant, Shape shape, int conn) {
    constexpr size_t slack = 128;
    auto fn = [&](int tile_rows, int warps, int solve) {
        switch (variant) {
            case VAR_MUTEX: return kernel_for<VAR_MUTEX>(tile_rows, warps, solve, conn);
            case VAR_DOUBLE: return kernel_for<VAR_DOUBLE>(tile_rows, warps, solve, conn);
            case VAR_ASYNC: return kernel_for<VAR_ASYNC>(tile_rows, warps, solve, conn);
            default: return kernel_for<VAR_UNIQUE>(tile_rows, warps, solve, conn);
        }
    };
    auto passes = [&](int tile_rows, int warps, size_t tile) {
        return Kernel{fn(tile_rows, warps, SOLVE_PASSES), 32 * warps, slack + tile, 1};
    };
    auto alt = [&](int tile_rows, int solve, size_t tile) {
        return Kernel{fn(tile_rows, 1, solve), 32 * kAltWorkers, slack + kAltWorkers * tile, kAltWorkers};
    };
    switch (shape) {
        case T32_W4: return passes(32, 4, sizeof(TileSmemPasses<32, 4>));
        case T64_W8: return passes(64, 8, sizeof(TileSmemPasses<64, 8>));
        case T64_W4: return passes(64, 4, sizeof(TileSmemPasses<64, 4>));
        case T64_W2: return passes(64, 2, sizeof(TileSmemPasses<64, 2>));
        case T32_SWEEPS: return alt(32, SOLVE_SWEEPS, sizeof(TileSmem<32>));
        case T64_SWEEPS: return alt(64, SOLVE_SWEEPS, sizeof(TileSmem<64>));
        case T32_PQ: return alt(32, SOLVE_PQ, sizeof(TileSmemPq<32>));
        default: return alt(64, SOLVE_PQ, sizeof(TileSmemPq<64>));
    }
}

// Multiprocessors of a device (asked once), 0 when it cannot be asked.
int engine_sm_count(int device) {
    static std::atomic<int> cache[64];
    if (device < 0 || device >= 64) return 0;
    int n = cache[device].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        cache[device].store(n, std::memory_order_relaxed);
    }
    return n;
}

// CTAs of a kernel that a multiprocessor keeps resident, asked (and the kernel
// loaded) once.
static cudaError_t resident_ctas(int variant, Shape shape, int conn, int device, int* per_sm) {
    static std::atomic<int> cache[64][4][SHAPES][3];
    std::atomic<int>& cached = cache[device][variant][shape][conn / 4];
    *per_sm = cached.load(std::memory_order_relaxed);
    if (*per_sm != 0) return cudaSuccess;
    const Kernel k = kernel_of(variant, shape, conn);
    cudaFuncAttributes attr;
    cudaError_t e = cudaFuncGetAttributes(&attr, k.fn);  // (loads it where kernels are loaded on demand)
    if (e == cudaSuccess && k.smem > 48 * 1024)
        e = cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k.fn, k.threads, k.smem);
    if (e == cudaSuccess) cached.store(*per_sm, std::memory_order_relaxed);
    return e;
}

cudaError_t engine_prepare(int variant, int tile_rows, int solver, int conn, long long tiles, int grid_ctas,
                           int device, LaunchInfo* li) {
    const int sms = engine_sm_count(device);
    if (sms <= 0 || variant < 0 || variant > 3 || conn < 0 || conn > 8) return cudaErrorInvalidValue;
    const Shape shape = select_shape(tile_rows, solver, tiles, grid_ctas, sms);
    int per_sm = 0;
    const cudaError_t e = resident_ctas(variant, shape, conn, device, &per_sm);
    if (e != cudaSuccess) return e;
    // CTAs of the mutex queue take turns at its lock, and past a few per SM the
    // longer line costs more than the visits beside one another gain.  Where that
    // is depends on the image; two is a compromise that is seldom far off, not
    // the best for each (8-connected, h = 40, likes three).  1 / 2 / 3 / all
    // that fit (10, 5 or 3) per SM, us: 4096^2 u8 h-domes, 4-connected, h = 10
    // 757 / 843 / 905 / 2062, h = 100 1726 / 1260 / 1288 / 3054, 8-connected, h = 40
    // 2600 / 2259 / 1540 / 3137; 6000 x 5000 u8 2530 / 1550 / 2388 / 2450; 2048 x 1500
    // u16 600 / 757 / 1856 / 1855; sparse seeds 4096^2 u8 4120 / 3680 / 3266 / 3180,
    // 5000^2 i32 19900 / 21100 / 21400 / 30300.  CTAs of four workers, row sweeps,
    // 1 / 2 / 3: 4096^2 u8 4-connected 1181 / 1705 / 1574, 8-connected 3403 / 3090 /
    // 3031, sparse 3911 / 4514 / 6403, 8192^2 sparse 13132 / 13672 / 14395; pixel
    // queue 1100 / 1682 / 2245, 3348 / 2357 / 2866, 5459 / 4930 / 5348, 20713 / 15843 /
    // 15093.
    if (variant == VAR_MUTEX) per_sm = std::min(per_sm, 2);
    li->grid = per_sm * sms;
    li->workers = kernel_of(variant, shape, conn).workers;
    li->shape = shape;
    li->conn = conn;
    return li->grid > 0 ? cudaSuccess : cudaErrorInvalidConfiguration;
}

cudaError_t engine_load(int variant, int tile_rows, int device) {
    if (engine_sm_count(device) <= 0 || variant < 0 || variant > 3) return cudaErrorInvalidValue;
    cudaError_t e = cudaSuccess;
    for (int conn : {4, 8})
        for (Shape shape : {T32_W4, T64_W8, T64_W4, T64_W2}) {
            int per_sm = 0;
            if ((shape == T32_W4) == (tile_rows == 32) && e == cudaSuccess)
                e = resident_ctas(variant, shape, conn, device, &per_sm);
        }
    return e;
}

cudaError_t engine_launch_init(const EngineArgs& a, int variant, cudaStream_t s) {
    unsigned blocks = (a.G + 255u) / 256u;
    if (blocks == 0u) blocks = 1u;
    if (blocks > 4096u) blocks = 4096u;
    engine_init_kernel<<<blocks, 256, 0, s>>>(a, variant);
    return cudaGetLastError();
}

cudaError_t engine_launch(const EngineArgs& a, int variant, const LaunchInfo& li, int grid, cudaStream_t s) {
    const Kernel k = kernel_of(variant, static_cast<Shape>(li.shape), li.conn);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)k.threads);
    cfg.dynamicSmemBytes = k.smem;
    cfg.stream = s;
    // The round queues' grid barrier and the mutex queue's initial slices need
    // every CTA resident.  With the async queue any CTA can do any entry, so
    // its launch may start with part of its CTAs beside another job's.
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = variant == VAR_ASYNC ? 0 : 1;
    EngineArgs args = a;
    void* params[] = {&args};
    return cudaLaunchKernelExC(&cfg, k.fn, params);
}

}  // namespace iwpp
