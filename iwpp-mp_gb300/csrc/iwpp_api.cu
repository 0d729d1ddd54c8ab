// iwpp_api.cu -- host side of libiwpp.so: argument checks, workspaces,
// staging of unaligned images, launch sequencing, CUDA-graph plans and the
// reference-compatible entry points.  Declarations: include/iwpp.h.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "iwpp.h"
#include "iwpp_engine.cuh"
#include "iwpp_top.cuh"
#include "iwpp_tune.h"

using namespace iwpp;

namespace {

std::atomic<int> g_last_status{IWPP_OK};

int set_last(int s) {
    g_last_status.store(s);
    return s;
}

int bpp_of(int dtype) { return dtype == IWPP_U8 ? 1 : dtype == IWPP_U16 ? 2 : 4; }
int ppw_of(int dtype) { return dtype == IWPP_U8 ? 4 : dtype == IWPP_U16 ? 2 : 1; }

int resolve_variant(int variant) {
    if (variant == IWPP_QUEUE_MUTEX || variant == IWPP_QUEUE_DOUBLE || variant == IWPP_QUEUE_UNIQUE ||
        variant == IWPP_QUEUE_ASYNC)
        return variant;
    const char* e = std::getenv("IWPP_QUEUE_VARIANT");
    if (e) {
        std::string s(e);
        if (s == "mutex" || s == "mp" || s == "MP") return IWPP_QUEUE_MUTEX;
        if (s == "double" || s == "dq" || s == "DQ") return IWPP_QUEUE_DOUBLE;
        if (s == "unique" || s == "uq" || s == "UQ") return IWPP_QUEUE_UNIQUE;
        if (s == "async") return IWPP_QUEUE_ASYNC;
    }
    return IWPP_QUEUE_ASYNC;
}

struct Config {
    int tile_rows;
    long long queue_capacity;  // < 0: that multiple of the job's tile count
    int init_passes;
    int grid_ctas;
    int max_restarts;
    int timeout_ms;
    int clip_marker;
    int plain_loads;
    int solver;
    int front_passes;  // 0 default, 1 always, 2 never
    int phantom_work;
    // fields the caller left at their defaults (the tuning table may fill them)
    bool dflt_tile, dflt_queue, dflt_init, dflt_solver, dflt_front;
};

Config resolve_config(const iwpp_config* c) {
    Config r;
    r.tile_rows = c && (c->tile_rows == 32 || c->tile_rows == 64) ? c->tile_rows : 0;
    r.queue_capacity = c && c->queue_capacity != 0 ? c->queue_capacity : 0;
    r.init_passes = c && c->init_passes >= 0 ? c->init_passes : 0;
    r.grid_ctas = c && c->grid_ctas > 0 ? c->grid_ctas : 0;
    r.max_restarts = c && c->max_restarts > 0 ? c->max_restarts : 64;
    r.timeout_ms = c && c->timeout_ms > 0 ? c->timeout_ms : 10000;
    r.clip_marker = c ? c->clip_marker : 0;
    r.plain_loads = c ? c->plain_loads : 0;
    r.solver = c && c->solver >= 0 && c->solver <= 3 ? c->solver : 0;
    r.front_passes = c && c->front_passes >= 0 && c->front_passes <= 4 ? c->front_passes : 0;
    r.phantom_work = c && c->phantom_work == 1 ? 1 : 0;
    r.dflt_tile = r.tile_rows == 0;
    r.dflt_queue = r.queue_capacity == 0;
    r.dflt_init = !c || c->init_passes < 0;
    r.dflt_solver = r.solver == 0;
    r.dflt_front = r.front_passes == 0;
    if (std::getenv("IWPP_PLAIN_LOADS")) r.plain_loads = 1;
    return r;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no
// libcuda link needed).
PFN_cuTensorMapEncodeTiled_v12000 tmap_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        cudaGetLastError();
    });
    return fn;
}

// A 2-D map over the image's bytes (uint8 elements): dims {W * bpp, H},
// row pitch in bytes, box {128 bytes, TH + 2 rows}.  Needs 16-byte aligned
// base and pitch.
bool encode_tmap(CUtensorMap* out, const void* base, int w, int h, size_t pitch, int bpp, int th) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tmap_encoder();
    if (!enc) return false;
    if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0u || (pitch & 15u) != 0u) return false;
    cuuint64_t dims[2] = {(cuuint64_t)w * (cuuint64_t)bpp, (cuuint64_t)h};
    cuuint64_t strides[1] = {(cuuint64_t)pitch};
    cuuint32_t box[2] = {128u, (cuuint32_t)(th + 2)};
    cuuint32_t estr[2] = {1u, 1u};
    CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

bool aligned_for_engine(const void* p, size_t pitch) {
    return (reinterpret_cast<uintptr_t>(p) & 3u) == 0u && (pitch & 3u) == 0u;
}

int check_image(const void* marker, const void* mask, size_t pm, size_t pk, int w, int h, int dtype, int conn) {
    if (dtype != IWPP_U8 && dtype != IWPP_U16 && dtype != IWPP_I32) return IWPP_ERR_INVALID;
    if (conn != 4 && conn != 8) return IWPP_ERR_INVALID;
    if (w < 0 || h < 0 || w > (1 << 28) || h > (1 << 28)) return IWPP_ERR_INVALID;
    if (w == 0 || h == 0) return IWPP_OK;
    if (!marker || !mask) return IWPP_ERR_INVALID;
    const size_t row = (size_t)w * (size_t)bpp_of(dtype);
    if (pm < row || pk < row) return IWPP_ERR_INVALID;
    if ((reinterpret_cast<uintptr_t>(marker) % (uintptr_t)bpp_of(dtype)) != 0u ||
        (reinterpret_cast<uintptr_t>(mask) % (uintptr_t)bpp_of(dtype)) != 0u)
        return IWPP_ERR_INVALID;
    if (pm % (size_t)bpp_of(dtype) != 0u || pk % (size_t)bpp_of(dtype) != 0u) return IWPP_ERR_INVALID;
    return IWPP_OK;
}

int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return IWPP_OK;
    if (e == cudaErrorMemoryAllocation) return IWPP_ERR_OOM;
    return IWPP_ERR_CUDA;
}

long long tiles_of(int w, int h, int dtype, int th) {
    if (w <= 0 || h <= 0) return 0;
    const long long tw = 32ll * ppw_of(dtype);
    return ((w + tw - 1) / tw) * (((long long)h + th - 1) / th);
}

// Tile height for calls that leave it at its default: 64-row tiles (fewer
// tile boundaries to cross, fewer visits), or 32 for jobs with at most one
// 64-row tile per SM, which would leave SMs without one.  Measured on h-dome
// images, 32 rows by four warps / 64 rows by eight, us: 256^2 uint8 41 / 43
// (8-connected 80 / 70), 512^2 8-connected 117 / 132, uint16 98 / 112, int32
// 121 / 123, 1024^2 uint8 73 / 68 (120 / 122); above that 64 rows: 1536^2
// uint8 77 / 66, 1024^2 uint16 124 / 106, 4096^2 uint8 191 / 144 (64 rows by
// two warps).  The mutex queue is bound by its one lock (every take and insert
// is a critical section), so its cost grows with the tile count: 64 rows always.
// The other solvers have one warp per tile: 32 rows below 2.5 64-row tiles per
// warp that the grid keeps resident, 12 per SM.  A grid that the caller limits
// to fewer CTAs than there are 64-row tiles leaves no SM that it uses without one.
int default_tile_rows(int variant, int solver, long long tiles64, int grid_ctas = 0) {
    if (variant == IWPP_QUEUE_MUTEX) return 64;
    int device = -1;
    if (cudaGetDevice(&device) != cudaSuccess) {
        cudaGetLastError();
        return 64;
    }
    const int sms = engine_sm_count(device);
    if (solver == 1 || solver == 3) return tiles64 < 30ll * sms ? 32 : 64;
    return tiles64 <= (grid_ctas > 0 ? std::min(grid_ctas, sms) : sms) ? 32 : 64;
}

long long job_tiles64(const iwpp_image* imgs, int n) {
    long long t = 0;
    for (int i = 0; i < n; ++i) t += tiles_of(imgs[i].width, imgs[i].height, imgs[i].dtype, 64);
    return t;
}

// Device workspace of one job: [Ctrl][ImgDesc x n][state x G][q0][q1].
struct Workspace {
    void* base = nullptr;
    size_t bytes = 0;
};

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct Layout {
    size_t off_imgs, off_tmaps, off_state, off_q0, off_q1, off_sweep, off_list, total;
};

// sweep_bytes: scratch of the whole-image sweeps or the front stage run
// before the engine; seed_list: room for the engine's seed list after a seed
// check
// (G ids and their count)
Layout layout_for(long long n_imgs, long long G, long long cap, bool two_queues, size_t sweep_bytes = 0,
                  bool seed_list = false) {
    Layout l;
    l.off_imgs = align_up(sizeof(Ctrl), 256);
    l.off_tmaps = align_up(l.off_imgs + (size_t)n_imgs * sizeof(ImgDesc), 256);
    l.off_state = align_up(l.off_tmaps + (size_t)n_imgs * 2u * sizeof(CUtensorMap), 256);
    l.off_q0 = align_up(l.off_state + (size_t)G * 4u, 256);
    l.off_q1 = align_up(l.off_q0 + (size_t)cap * 4u, 256);
    l.off_sweep = align_up(l.off_q1 + (two_queues ? (size_t)cap * 4u : 0u), 256);
    l.off_list = align_up(l.off_sweep + sweep_bytes, 256);
    l.total = align_up(l.off_list + (seed_list ? (size_t)(G + 1) * 4u : 0u), 256);
    return l;
}

// Whole-image passes after the top-level stage when the caller asks for the
// stage (front_passes 1) and leaves init_passes at its default.  Jobs decided
// on the device run none: what the passes cover the engine now does sooner
// (16384^2 spirals with 0 / 1 / 2 / 3 passes, ms: uint8 2.57 / 2.85 / 3.03 /
// 3.49, uint16 4.12 / 5.15 / 5.62 / 6.45, 16384 x 12000 int32 5.35 / 6.45 /
// 6.45 / 7.24; 9001 x 9999 uint8 1.11 / 3.37 / 5.56 / 7.86), and without them
// the labelling itself can add the tiles that it raises pixels in to the first
// check's list, which spares the second check over both planes.
constexpr int kFrontFullPasses = 2;
// Untuned jobs whose largest image has at least this many pixels decide on
// the device whether to take the front stage (front_passes 3): the seed
// check over the untouched images measures the initial front, and a small
// one (a few sparse seeds) means long propagation paths, which the tile
// engine alone walks one dependent tile visit at a time (the 16384^2
// spiral: 235 ms alone, 4 ms with the stage) while a large one is
// short-range work the engine does faster alone (16384^2 h-dome: 3.4 ms
// alone, 6.5 ms with the stage).  The check and the skipped launches cost
// about 0.1 ms, too much below this size (six 4096^2 h-dome images take
// 0.24-0.73 ms each).
constexpr long long kFrontDefaultPixels = 1ll << 26;

// The job runs the front stage always (1) or as the device decides (3).
bool job_front(const Config& c) { return c.front_passes == 1 || c.front_passes == 3; }
// The tile engine starts from a seed check's list (the front stage's, or
// the check alone: 4) instead of every tile.
bool job_seeded(const Config& c) { return job_front(c) || c.front_passes == 4; }

// Whole-image raster / anti-raster passes a job runs before the engine.
int job_full_passes(const Config& c) {
    if (c.front_passes == 1 && c.dflt_init) return kFrontFullPasses;
    return c.init_passes;
}

long long queue_capacity_for(int variant, long long G, long long requested) {
    long long cap;
    if (variant == IWPP_QUEUE_ASYNC) {
        cap = std::max<long long>(2 * G, 1024);  // ring: at most G entries outstanding
    } else if (variant == IWPP_QUEUE_UNIQUE) {
        cap = std::max<long long>(G, 1);  // one entry per tile at most
    } else if (requested > 0) {
        cap = variant == IWPP_QUEUE_MUTEX ? std::max(requested, G) : requested;
    } else {
        cap = std::max<long long>(4 * G, 4096);
    }
    return std::min<long long>(cap, 0x7fffffffll);
}

// A job in preparation: descriptors (possibly pointing at staging copies).
struct Staged {
    void* user_marker;
    size_t user_pm;
    const void* user_mask;
    size_t user_pk;
    void* buf_m;  // staging copies (nullptr when the user buffer is used)
    void* buf_k;
    size_t pitch;
    int w, h, dtype;
    bool owned;   // allocated for a plan: copied and freed by the plan
    StageCopy in_m() const { return {user_marker, buf_m, (long long)user_pm, (long long)pitch, row(), h}; }
    StageCopy in_k() const { return {user_mask, buf_k, (long long)user_pk, (long long)pitch, row(), h}; }
    StageCopy out_m() const { return {buf_m, user_marker, (long long)pitch, (long long)user_pm, row(), h}; }
    long long row() const { return (long long)w * bpp_of(dtype); }
};

// Where a handle's direct calls get their staging buffers from: a memory pool
// that keeps up to kStagePoolKeep bytes between calls (the default pool gives
// everything back at each synchronisation, and getting it again cost such a
// call about 300 us, more than the reconstruction of a 6-megapixel image).
// It goes with the handle.
constexpr unsigned long long kStagePoolKeep = 256ull << 20;
struct StagePool {
    cudaMemPool_t pool = nullptr;
    int device = 0;
    cudaError_t alloc(void** out, size_t bytes, cudaStream_t s) {
        if (!pool) {
            cudaMemPoolProps props{};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = device;
            unsigned long long keep = kStagePoolKeep;
            if (cudaMemPoolCreate(&pool, &props) != cudaSuccess ||
                cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
                cudaGetLastError();
                release();
                return cudaMallocAsync(out, bytes, s);
            }
        }
        return cudaMallocFromPoolAsync(out, bytes, pool, s);
    }
    void release() {
        if (pool) cudaMemPoolDestroy(pool);
        pool = nullptr;
    }
};

struct Job {
    std::vector<ImgDesc> descs;
    std::vector<Staged> staged;
    std::vector<CUtensorMap> tmaps;  // two per descriptor (marker, mask)
    std::vector<char> has_tma;
    bool staged_in = false;  // the staging buffers hold the images
    int stage_launches = 0;
    long long G = 0;
    int tile_rows = 64;
    int variant = IWPP_QUEUE_UNIQUE;
    Config cfg;
};

// The connectivity of a job's images, 0 where they mix them.
int job_conn(const Job& job) {
    int conn = 0;
    for (const ImgDesc& d : job.descs) {
        if (conn != 0 && d.conn != conn) return 0;
        conn = d.conn;
    }
    return conn;
}

// Queue entries of a job: the variant's rule applied to the requested
// capacity (negative: that multiple of the job's tiles).
long long job_queue_capacity(const Job& job) {
    const long long req = job.cfg.queue_capacity < 0 ? -job.cfg.queue_capacity * std::max(job.G, 1ll)
                                                     : job.cfg.queue_capacity;
    return queue_capacity_for(job.variant, job.G, req);
}

// The workspace layout of a job (the same for direct calls and plans).
Layout job_layout(const Job& job) {
    const bool two = job.variant == IWPP_QUEUE_DOUBLE || job.variant == IWPP_QUEUE_UNIQUE;
    const bool front = job_front(job.cfg);
    const bool seeded = job_seeded(job.cfg);
    size_t sweep = 0;
    for (const auto& d : job.descs) {
        if (job_full_passes(job.cfg) > 0) {
            ImgDesc dv = d;
            dv.conn = 4;
            sweep = std::max(sweep, sweep_scratch_bytes(dv));
        }
        if (front) sweep = std::max(sweep, top_scratch_bytes(d));
    }
    return layout_for((long long)job.descs.size(), job.G, job_queue_capacity(job), two, sweep, seeded);
}

// How images whose rows are not 4-byte aligned are handled.
enum StageMode { STAGE_REJECT = 0, STAGE_ASYNC = 1, STAGE_OWNED = 2 };

// STAGE_ASYNC: stream-ordered staging buffers (from `pool`, or the device's
// default pool), copied in now and back by finish_staging.  STAGE_OWNED: plain allocations owned by the caller (a
// plan), copies left to the caller.
int build_job(Job& job, const iwpp_image* imgs, int n, int variant, const iwpp_config* cfgp, cudaStream_t s,
              int staging, StagePool* pool, bool use_table = true) {
    job.cfg = resolve_config(cfgp);
    job.variant = resolve_variant(variant);
    if (use_table && n > 0 &&
        (job.cfg.dflt_tile || job.cfg.dflt_queue || job.cfg.dflt_init || job.cfg.dflt_solver || job.cfg.dflt_front)) {
        // fields left at their defaults come from the tuning table, if it
        // has an entry for this workload class
        std::vector<int> dts, cns;
        std::vector<long long> pxs;
        for (int i = 0; i < n; ++i) {
            if (imgs[i].width <= 0 || imgs[i].height <= 0) continue;
            dts.push_back(imgs[i].dtype);
            cns.push_back(imgs[i].connectivity);
            pxs.push_back((long long)imgs[i].width * imgs[i].height);
        }
        TuneEntry e;
        if (!dts.empty() &&
            tune_lookup(tune_key(job.variant, dts.data(), cns.data(), pxs.data(), (int)dts.size()), &e)) {
            if (job.cfg.dflt_tile) job.cfg.tile_rows = e.tile_rows;
            if (job.cfg.dflt_solver) job.cfg.solver = e.solver;
            if (job.cfg.dflt_init) {
                job.cfg.init_passes = e.init_passes;
                job.cfg.dflt_init = false;  // the table's count stands, also with the front stage
            }
            if (job.cfg.dflt_queue && e.queue_mult > 0) job.cfg.queue_capacity = -(long long)e.queue_mult;
            if (job.cfg.dflt_front) job.cfg.front_passes = tune_front_code(e.front_passes);
        }
    }
    if (job.cfg.front_passes == 0) {
        long long largest = 0;
        for (int i = 0; i < n; ++i)
            if (imgs[i].width > 0 && imgs[i].height > 0)
                largest = std::max(largest, (long long)imgs[i].width * imgs[i].height);
        job.cfg.front_passes = largest >= kFrontDefaultPixels ? 3 : 2;
    }
    int th = job.cfg.tile_rows;
    if (th == 0 && n > 0)
        th = default_tile_rows(job.variant, job.cfg.solver, job_tiles64(imgs, n), job.cfg.grid_ctas);
    else if (th == 0)
        th = 64;
    job.tile_rows = th;
    long long G = 0;
    for (int i = 0; i < n; ++i) {
        const iwpp_image& im = imgs[i];
        int rc = check_image(im.marker, im.mask, im.pitch_marker, im.pitch_mask, im.width, im.height, im.dtype,
                             im.connectivity);
        if (rc != IWPP_OK) return rc;
    }
    for (int i = 0; i < n; ++i) {
        const iwpp_image& im = imgs[i];
        if (im.width == 0 || im.height == 0) continue;
        ImgDesc d{};
        d.marker = static_cast<unsigned char*>(im.marker);
        d.mask = static_cast<const unsigned char*>(im.mask);
        d.pitch_m = (long long)im.pitch_marker;
        d.pitch_k = (long long)im.pitch_mask;
        d.W = im.width;
        d.H = im.height;
        d.dtype = im.dtype;
        d.conn = im.connectivity;
        const int tw = 32 * ppw_of(im.dtype);
        d.tiles_x = (im.width + tw - 1) / tw;
        d.tiles_y = (im.height + th - 1) / th;
        d.tile_rows = th;
        d.tile_base = (int)G;
        Staged st{im.marker, im.pitch_marker, im.mask, im.pitch_mask, nullptr, nullptr, 0, im.width, im.height,
                  im.dtype, staging == STAGE_OWNED};
        const bool ok_m = aligned_for_engine(im.marker, im.pitch_marker);
        const bool ok_k = aligned_for_engine(im.mask, im.pitch_mask);
        if (!ok_m || !ok_k) {
            if (staging == STAGE_REJECT) return IWPP_ERR_INVALID;
            // Rows that do not start on a 4-byte boundary: reconstruct in
            // aligned copies and copy the marker back afterwards.
            const size_t row = (size_t)im.width * bpp_of(im.dtype);
            const size_t pitch = align_up(row, 128);
            cudaError_t e;
            if (staging == STAGE_OWNED) {
                e = cudaMalloc(&st.buf_m, pitch * im.height);
                if (e == cudaSuccess) e = cudaMalloc(&st.buf_k, pitch * im.height);
                if (e != cudaSuccess) {
                    if (st.buf_m) cudaFree(st.buf_m);
                    cudaGetLastError();
                    return cuda_status(e);
                }
                st.pitch = pitch;
                job.staged.push_back(st);  // recorded even if a later image fails
                st.buf_m = st.buf_k = nullptr;
                Staged& kept = job.staged.back();
                d.marker = static_cast<unsigned char*>(kept.buf_m);
                d.mask = static_cast<const unsigned char*>(kept.buf_k);
                d.pitch_m = (long long)pitch;
                d.pitch_k = (long long)pitch;
                G += (long long)d.tiles_x * d.tiles_y;
                if (G > 0x7fffffffll) return IWPP_ERR_INVALID;
                CUtensorMap maps2[2];
                std::memset(maps2, 0, sizeof(maps2));
                const bool tma2 = !job.cfg.plain_loads &&
                                  encode_tmap(&maps2[0], d.marker, d.W, d.H, pitch, bpp_of(d.dtype), th) &&
                                  encode_tmap(&maps2[1], d.mask, d.W, d.H, pitch, bpp_of(d.dtype), th);
                job.tmaps.push_back(maps2[0]);
                job.tmaps.push_back(maps2[1]);
                job.has_tma.push_back(tma2 ? 1 : 0);
                job.descs.push_back(d);
                continue;
            }
            auto alloc = [&](void** out) {
                return pool ? pool->alloc(out, pitch * im.height, s) : cudaMallocAsync(out, pitch * im.height, s);
            };
            e = alloc(&st.buf_m);
            if (e == cudaSuccess) e = alloc(&st.buf_k);
            if (e != cudaSuccess) {
                if (st.buf_m) cudaFreeAsync(st.buf_m, s);
                if (st.buf_k) cudaFreeAsync(st.buf_k, s);
                cudaGetLastError();
                return cuda_status(e);
            }
            st.pitch = pitch;
            d.marker = static_cast<unsigned char*>(st.buf_m);
            d.mask = static_cast<const unsigned char*>(st.buf_k);
            d.pitch_m = (long long)pitch;
            d.pitch_k = (long long)pitch;
        }
        G += (long long)d.tiles_x * d.tiles_y;
        if (G > 0x7fffffffll) return IWPP_ERR_INVALID;
        CUtensorMap maps[2];
        std::memset(maps, 0, sizeof(maps));
        bool tma = !job.cfg.plain_loads &&
                   encode_tmap(&maps[0], d.marker, d.W, d.H, (size_t)d.pitch_m, bpp_of(d.dtype), th) &&
                   encode_tmap(&maps[1], d.mask, d.W, d.H, (size_t)d.pitch_k, bpp_of(d.dtype), th);
        job.tmaps.push_back(maps[0]);
        job.tmaps.push_back(maps[1]);
        job.has_tma.push_back(tma ? 1 : 0);
        job.descs.push_back(d);
        job.staged.push_back(st);
    }
    job.G = G;
    if (staging == STAGE_ASYNC) {
        std::vector<StageCopy> copies;
        for (const auto& st : job.staged)
            if (st.buf_m) {
                copies.push_back(st.in_m());
                copies.push_back(st.in_k());
            }
        const int rc = cuda_status(launch_stage_copies(copies, s, &job.stage_launches));
        if (rc != IWPP_OK) return rc;
        job.staged_in = true;
    }
    return IWPP_OK;
}

int finish_staging(Job& job, cudaStream_t s) {
    std::vector<StageCopy> copies;
    if (job.staged_in)
        for (const auto& st : job.staged)
            if (st.buf_m && !st.owned) copies.push_back(st.out_m());
    const cudaError_t e = launch_stage_copies(copies, s, &job.stage_launches);
    for (auto& st : job.staged) {
        if (!st.buf_m || st.owned) continue;
        cudaFreeAsync(st.buf_m, s);
        cudaFreeAsync(st.buf_k, s);
        st.buf_m = st.buf_k = nullptr;
    }
    return cuda_status(e);
}

// Pinned host slots for the descriptor uploads of asynchronous calls: a
// copy from pageable memory makes the driver wait for the stream's earlier
// work first, which would turn every asynchronous call into a synchronous
// one.  Two slots alternate; a slot is reused once its last upload is done.
struct HostStaging {
    void* p[2] = {nullptr, nullptr};
    size_t bytes[2] = {0, 0};
    cudaEvent_t done[2] = {nullptr, nullptr};
    bool pending[2] = {false, false};
    int next = 0;

    char* acquire(size_t need, int* slot) {
        const int k = next;
        next ^= 1;
        if (pending[k]) {
            cudaEventSynchronize(done[k]);
            pending[k] = false;
        }
        if (!done[k] && cudaEventCreateWithFlags(&done[k], cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            done[k] = nullptr;
            return nullptr;
        }
        if (bytes[k] < need) {
            if (p[k]) cudaFreeHost(p[k]);
            p[k] = nullptr;
            bytes[k] = 0;
            const size_t want = std::max<size_t>(need, 64u << 10);
            if (cudaMallocHost(&p[k], want) != cudaSuccess) {
                cudaGetLastError();
                p[k] = nullptr;
                return nullptr;
            }
            bytes[k] = want;
        }
        *slot = k;
        return static_cast<char*>(p[k]);
    }
    void mark(int k, cudaStream_t s) {
        if (cudaEventRecord(done[k], s) == cudaSuccess) pending[k] = true;
    }
    void release() {
        for (int k = 0; k < 2; ++k) {
            if (pending[k]) cudaEventSynchronize(done[k]);
            if (p[k]) cudaFreeHost(p[k]);
            if (done[k]) cudaEventDestroy(done[k]);
            p[k] = nullptr;
            done[k] = nullptr;
            bytes[k] = 0;
            pending[k] = false;
        }
    }
};

}  // namespace

struct iwpp_handle_s {
    int device = 0;
    Workspace ws;
    Ctrl* host_ctrl = nullptr;  // pinned
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    HostStaging staging;
    StagePool stage_pool;
    cudaStream_t last_stream = nullptr;
    long long last_tiles = 0;
    int last_variant = IWPP_QUEUE_UNIQUE;
    int last_launch_status = IWPP_OK;
    int last_launches = 0;
    bool timed = false;
    std::mutex mu;
};

struct iwpp_plan_s {
    iwpp_handle h = nullptr;
    std::vector<Staged> staged;  // owned staging buffers of unaligned images
    Workspace ws;
    Ctrl* host_ctrl = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaStream_t last_stream = nullptr;
    long long tiles = 0;
    int variant = IWPP_QUEUE_UNIQUE;
    int launches = 0;
};

namespace {

int ensure_workspace(Workspace& ws, size_t bytes) {
    if (ws.bytes >= bytes) return IWPP_OK;
    if (ws.base) {
        cudaFree(ws.base);
        ws.base = nullptr;
        ws.bytes = 0;
    }
    cudaError_t e = cudaMalloc(&ws.base, bytes);
    if (e != cudaSuccess) {
        ws.base = nullptr;
        cudaGetLastError();
        return cuda_status(e);
    }
    ws.bytes = bytes;
    return IWPP_OK;
}

int check_device(int device) {
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
        cudaGetLastError();
        return IWPP_ERR_NO_DEVICE;
    }
    if (device < 0 || device >= count) return IWPP_ERR_INVALID;
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return IWPP_ERR_CUDA;
    // The kernels are built for sm_103a only.
    if (!(prop.major == 10 && prop.minor == 3)) return IWPP_ERR_NO_DEVICE;
    return IWPP_OK;
}

// Enqueues a prepared job on `s` into workspace `ws`.
int enqueue_job(const Job& job, Workspace& ws, cudaStream_t s, int device, bool use_events, cudaEvent_t ev0,
                cudaEvent_t ev1, bool upload_descs, HostStaging* hs = nullptr, int* launches = nullptr) {
    int nl = 0;  // kernels launched
    struct Count {
        int* out;
        int* n;
        ~Count() {
            if (out) *out = *n;
        }
    } count_out{launches, &nl};
    const bool two = job.variant == IWPP_QUEUE_DOUBLE || job.variant == IWPP_QUEUE_UNIQUE;
    const long long cap = job_queue_capacity(job);
    const Layout l = job_layout(job);
    int rc = ensure_workspace(ws, l.total);
    if (rc != IWPP_OK) return rc;
    char* base = static_cast<char*>(ws.base);
    EngineArgs a{};
    a.imgs = reinterpret_cast<const ImgDesc*>(base + l.off_imgs);
    a.nimg = (int)job.descs.size();
    if (a.nimg == 1) {
        a.one = job.descs[0];
        a.one_tma = job.has_tma[0];
        std::memcpy(a.one_maps, job.tmaps.data(), sizeof(a.one_maps));
    }
    a.G = (unsigned)job.G;
    a.state = reinterpret_cast<unsigned*>(base + l.off_state);
    a.q0 = reinterpret_cast<unsigned*>(base + l.off_q0);
    a.q1 = two ? reinterpret_cast<unsigned*>(base + l.off_q1) : a.q0;
    a.cap = (unsigned)cap;
    a.ctrl = reinterpret_cast<Ctrl*>(base);
    a.timeout_ns = (long long)job.cfg.timeout_ms * 1000000ll;
    a.max_restarts = job.cfg.max_restarts;
    a.solver = job.cfg.solver;
    a.phantom = job.cfg.phantom_work;
    const bool front = job_front(job.cfg) && job.G > 0;
    const bool seeded = job_seeded(job.cfg) && job.G > 0;
    const bool gated = front && job.cfg.front_passes == 3;
    unsigned* seed_list = reinterpret_cast<unsigned*>(base + l.off_list);
    unsigned* seed_count = seed_list + job.G;
    if (seeded) {
        a.front = 1;
        a.front_ran = front && !gated ? 1 : 0;
        a.front_gated = gated ? 1 : 0;
        if (front) {
            // after the front stage few tiles are left: the engine starts
            // from the list
            a.init_list = seed_list;
            a.init_count = seed_count;
        } else {
            // the check alone: its tile states, the queue in tile order
            // (a list filled by atomics would lose the raster order that
            // lets a tile's upper and left neighbours go first)
            a.states_set = 1;
        }
    }

    cudaError_t e = cudaSuccess;
    if (upload_descs && job.descs.size() > 1) {
        std::vector<ImgDesc> descs = job.descs;
        for (size_t i = 0; i < descs.size(); ++i)
            descs[i].tmaps = job.has_tma[i] ? base + l.off_tmaps + i * 2u * sizeof(CUtensorMap) : nullptr;
        const size_t tb = job.tmaps.size() * sizeof(CUtensorMap), db = descs.size() * sizeof(ImgDesc);
        int slot = -1;
        char* pin = hs ? hs->acquire(tb + db, &slot) : nullptr;
        const void* src_t = job.tmaps.data();
        const void* src_d = descs.data();
        if (pin) {
            std::memcpy(pin, job.tmaps.data(), tb);
            std::memcpy(pin + tb, descs.data(), db);
            src_t = pin;
            src_d = pin + tb;
        }
        e = cudaMemcpyAsync(base + l.off_tmaps, src_t, tb, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(base + l.off_imgs, src_d, db, cudaMemcpyHostToDevice, s);
        if (pin) hs->mark(slot, s);
    }
    if (e != cudaSuccess) return cuda_status(e);
    if (use_events) cudaEventRecord(ev0, s);
    if (job.cfg.clip_marker)
        for (const auto& d : job.descs) {
            e = launch_clip(d, s);
            if (e != cudaSuccess) return cuda_status(e);
            ++nl;
        }
    // the front stage's view of the images: gated by the device's decision
    const int full_passes = job_full_passes(job.cfg);
    // a gated job without passes checks once: the labelling marks what it raises
    const bool marks = gated && full_passes == 0;
    std::vector<ImgDesc> fdescs = job.descs;
    if (gated)
        for (auto& d : fdescs) d.gate = &a.ctrl->front_gate;
    if (front) {
        // The top level of each image first (its connected sets of pixels at
        // the mask's largest value, however long); the whole-image passes and
        // the seed check follow.  The job's error word and top-pixel count
        // are zeroed here: the engine's initialisation keeps them.  A gated
        // job first measures its initial front (a seed check over the
        // untouched images) and decides.
        Ctrl* c = a.ctrl;
        e = cudaMemsetAsync(&c->error, 0, sizeof(c->error), s);
        if (e == cudaSuccess) e = cudaMemsetAsync(&c->top_pixels, 0, sizeof(c->top_pixels), s);
        if (gated) {
            if (e == cudaSuccess) e = cudaMemsetAsync(seed_count, 0, sizeof(unsigned), s);
            if (e == cudaSuccess)
                e = launch_seed_batch(a.imgs, job.descs, nullptr, a.state, seed_list, seed_count, s, &nl);
            if (e == cudaSuccess) e = launch_front_decide(&c->front_gate, seed_count, (unsigned)job.G, !marks, s, &nl);
        }
        for (size_t i = 0; i < fdescs.size() && e == cudaSuccess; ++i)
            e = launch_top(fdescs[i], base + l.off_sweep, &c->top_pixels,
                           marks ? SeedMarks{a.state, seed_list, seed_count} : SeedMarks{}, device, s, &nl);
        if (e != cudaSuccess) return cuda_status(e);
    }
    for (int p = 0; p < full_passes; ++p)
        for (const auto& d : fdescs)
            for (int dir = 0; dir < 4; ++dir) {
                // raster (+X, +Y) then anti-raster (-X, -Y).  The vertical
                // sweeps take the pixel above / below only: a valid update
                // for either connectivity with no shuffle on the column
                // chain; the tile engine completes the diagonals.
                static const int order[4] = {0, 1, 2, 3};
                ImgDesc dv = d;
                dv.conn = 4;
                e = launch_sweep(dv, order[dir], s, base + l.off_sweep, &nl);
                if (e != cudaSuccess) return cuda_status(e);
            }
    if (seeded) {
        // the tile engine starts from the tiles still holding a pixel that a
        // neighbour can raise (a gated job keeps the list of its first check
        // when it left the stage out, or with what the labelling added to it);
        // the error word and top-pixel count of a job without the stage are
        // zeroed here (the engine's initialisation keeps them)
        if (!front) {
            e = cudaMemsetAsync(&a.ctrl->error, 0, sizeof(a.ctrl->error), s);
            if (e == cudaSuccess) e = cudaMemsetAsync(&a.ctrl->top_pixels, 0, sizeof(a.ctrl->top_pixels), s);
        }
        if (!gated && e == cudaSuccess) e = cudaMemsetAsync(seed_count, 0, sizeof(unsigned), s);
        if (e == cudaSuccess && !marks)
            e = launch_seed_batch(a.imgs, job.descs, gated ? &a.ctrl->front_gate : nullptr, a.state, seed_list,
                                  seed_count, s, &nl);
        if (e != cudaSuccess) return cuda_status(e);
    }
    long long grid = 1;
    LaunchInfo li{};
    if (job.G > 0) {
        e = engine_prepare(job.variant, job.tile_rows, job.cfg.solver, job_conn(job), job.G, job.cfg.grid_ctas, device,
                           &li);
        if (e != cudaSuccess) return cuda_status(e);
        grid = li.grid;
        grid = std::min(grid, (job.G + li.workers - 1) / li.workers);
        if (job.cfg.grid_ctas > 0 && job.cfg.grid_ctas < grid) grid = job.cfg.grid_ctas;
        if (grid < 1) grid = 1;
    }
    a.grid = (int)grid;
    e = engine_launch_init(a, job.variant, s);
    if (e != cudaSuccess) return cuda_status(e);
    ++nl;
    if (job.G > 0) {
        e = engine_launch(a, job.variant, li, (int)grid, s);
        if (e != cudaSuccess) return cuda_status(e);
        ++nl;
    }
    if (use_events) cudaEventRecord(ev1, s);
    return IWPP_OK;
}

// Waits for a job and its counters with one synchronisation; ev0 / ev1
// (nullable) were recorded around it.
int read_stats(Ctrl* host_ctrl, const Workspace& ws, cudaStream_t s, long long tiles, int variant,
               iwpp_stats* out, cudaEvent_t ev0 = nullptr, cudaEvent_t ev1 = nullptr, int launches = 0) {
    cudaError_t e = cudaMemcpyAsync(host_ctrl, ws.base, sizeof(Ctrl), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_status(e);
    const int st = status_of_job(host_ctrl->error);
    if (out) {
        out->tiles = tiles;
        out->visits = (long long)host_ctrl->visits;
        out->sweeps = (long long)host_ctrl->sweeps;
        out->pushes = (long long)host_ctrl->pushes;
        out->rounds = (int)host_ctrl->rounds;
        out->restarts = (int)host_ctrl->restarts;
        out->status = st;
        out->variant = variant;
        float ms = 0.f;
        if (ev0 && cudaEventElapsedTime(&ms, ev0, ev1) != cudaSuccess) cudaGetLastError();
        out->device_ms = ms;
        out->row_steps = (long long)host_ctrl->row_steps;
        for (int i = 0; i < 5; ++i) out->phase_cycles[i] = (long long)host_ctrl->phase[i];
        out->launches = launches;
        out->top_pixels = (long long)host_ctrl->top_pixels;
        out->front_stage = host_ctrl->front_gate != 0u ? 1 : 0;
    }
    return st;
}

iwpp_handle default_handle(int* rc_out) {
    static std::mutex mu;
    static iwpp_handle handles[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        *rc_out = IWPP_ERR_NO_DEVICE;
        return nullptr;
    }
    if (dev < 0 || dev >= 64) {
        *rc_out = IWPP_ERR_INVALID;
        return nullptr;
    }
    std::lock_guard<std::mutex> lk(mu);
    if (!handles[dev]) {
        int rc = iwpp_handle_create(&handles[dev], dev);
        if (rc != IWPP_OK) {
            *rc_out = rc;
            return nullptr;
        }
    }
    *rc_out = IWPP_OK;
    return handles[dev];
}

int run_job_sync(iwpp_handle h, const iwpp_image* imgs, int n, int variant, const iwpp_config* cfg,
                 cudaStream_t s, iwpp_stats* stats) {
    int rc = IWPP_OK;
    // Arguments are checked before any device is touched; an all-empty job
    // is complete without one.
    bool any_pixels = false;
    for (int i = 0; i < n; ++i) {
        const iwpp_image& im = imgs[i];
        rc = check_image(im.marker, im.mask, im.pitch_marker, im.pitch_mask, im.width, im.height, im.dtype,
                         im.connectivity);
        if (rc != IWPP_OK) return rc;
        any_pixels |= im.width > 0 && im.height > 0;
    }
    if (!any_pixels) {
        if (stats) *stats = iwpp_stats{};
        return IWPP_OK;
    }
    if (!h) h = default_handle(&rc);
    if (!h) return rc;
    std::lock_guard<std::mutex> lk(h->mu);
    int prev_dev = 0;
    cudaGetDevice(&prev_dev);
    if (prev_dev != h->device) cudaSetDevice(h->device);
    Job job;
    int nl = 0;
    rc = build_job(job, imgs, n, variant, cfg, s, STAGE_ASYNC, &h->stage_pool);
    if (rc == IWPP_OK) rc = enqueue_job(job, h->ws, s, h->device, true, h->ev0, h->ev1, true, &h->staging, &nl);
    const int rc_stage = finish_staging(job, s);
    if (rc == IWPP_OK) {
        rc = read_stats(h->host_ctrl, h->ws, s, job.G, job.variant, stats, h->ev0, h->ev1, nl + job.stage_launches);
    } else {
        cudaStreamSynchronize(s);
    }
    if (rc == IWPP_OK) rc = rc_stage;
    if (prev_dev != h->device) cudaSetDevice(prev_dev);
    return rc;
}

}  // namespace

namespace iwpp {
int resolve_queue_variant(int variant) { return resolve_variant(variant); }

// Grows a handle's workspace ahead of use (the server sizes each lane once).
int handle_reserve(iwpp_handle h, size_t bytes) {
    if (!h) return IWPP_ERR_INVALID;
    std::lock_guard<std::mutex> lk(h->mu);
    int prev = 0;
    cudaGetDevice(&prev);
    if (prev != h->device) cudaSetDevice(h->device);
    const int rc = ensure_workspace(h->ws, bytes);
    if (prev != h->device) cudaSetDevice(prev);
    return rc;
}
}  // namespace iwpp

// ====================================================================== API
extern "C" {

const char* iwpp_status_string(int status) {
    switch (status) {
        case IWPP_OK: return "ok";
        case IWPP_ERR_INVALID: return "invalid argument";
        case IWPP_ERR_OOM: return "out of device memory";
        case IWPP_ERR_TIMEOUT: return "a bounded device-side wait timed out";
        case IWPP_ERR_CUDA: return "CUDA runtime error";
        case IWPP_ERR_OVERFLOW: return "queue overflow restarts exhausted";
        case IWPP_ERR_NO_DEVICE: return "no sm_103 (GB300) CUDA device";
        case IWPP_ERR_BUSY: return "server queue full, shutting down, or request not finished";
        case IWPP_ERR_TOO_LARGE: return "image too large for the no-allocation scratch or the server budget";
        case IWPP_ERR_INTERNAL: return "a device-side consistency check failed";
        default: return "unknown status";
    }
}

int iwpp_version(void) { return 1; }

int iwpp_handle_create(iwpp_handle* out, int device) {
    if (!out) return IWPP_ERR_INVALID;
    *out = nullptr;
    int rc = check_device(device);
    if (rc != IWPP_OK) return rc;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    iwpp_handle h = new (std::nothrow) iwpp_handle_s();
    if (!h) return IWPP_ERR_OOM;
    h->device = h->stage_pool.device = device;
    cudaError_t e = cudaMallocHost(&h->host_ctrl, sizeof(Ctrl));
    if (e == cudaSuccess) e = cudaEventCreate(&h->ev0);
    if (e == cudaSuccess) e = cudaEventCreate(&h->ev1);
    cudaSetDevice(prev);
    if (e != cudaSuccess) {
        iwpp_handle_destroy(h);
        return cuda_status(e);
    }
    *out = h;
    return IWPP_OK;
}

int iwpp_handle_destroy(iwpp_handle h) {
    if (!h) return IWPP_OK;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(h->device);
    cudaDeviceSynchronize();
    h->staging.release();
    h->stage_pool.release();
    if (h->ws.base) cudaFree(h->ws.base);
    if (h->host_ctrl) cudaFreeHost(h->host_ctrl);
    if (h->ev0) cudaEventDestroy(h->ev0);
    if (h->ev1) cudaEventDestroy(h->ev1);
    cudaSetDevice(prev);
    delete h;
    return IWPP_OK;
}

long long iwpp_workspace_bytes(long long tiles, int variant, long long queue_capacity) {
    const int v = resolve_variant(variant);
    const long long cap = queue_capacity_for(v, tiles, queue_capacity < 0 ? -queue_capacity * tiles : queue_capacity);
    return (long long)layout_for(1, tiles, cap, v == IWPP_QUEUE_DOUBLE || v == IWPP_QUEUE_UNIQUE).total;
}

long long iwpp_tile_count(int width, int height, int dtype, int tile_rows) {
    if (dtype != IWPP_U8 && dtype != IWPP_U16 && dtype != IWPP_I32) return -1;
    const int th = tile_rows == 32 || tile_rows == 64
                       ? tile_rows
                       : default_tile_rows(resolve_variant(IWPP_QUEUE_DEFAULT), 0, tiles_of(width, height, dtype, 64));
    return tiles_of(width, height, dtype, th);
}

int iwpp_reconstruct(iwpp_handle h, void* marker, const void* mask, size_t pitch_marker, size_t pitch_mask,
                     int width, int height, int dtype, int connectivity, int variant, const iwpp_config* cfg,
                     void* stream, iwpp_stats* stats) {
    iwpp_image im{marker, mask, pitch_marker, pitch_mask, width, height, dtype, connectivity};
    return set_last(run_job_sync(h, &im, 1, variant, cfg, static_cast<cudaStream_t>(stream), stats));
}

int iwpp_reconstruct_batch(iwpp_handle h, const iwpp_image* images, int n, int variant, const iwpp_config* cfg,
                           void* stream, iwpp_stats* stats) {
    if (n < 0 || (n > 0 && !images)) return set_last(IWPP_ERR_INVALID);
    return set_last(run_job_sync(h, images, n, variant, cfg, static_cast<cudaStream_t>(stream), stats));
}

int iwpp_reconstruct_batch_async(iwpp_handle h, const iwpp_image* images, int n, int variant, const iwpp_config* cfg,
                                 void* stream) {
    if (!h || n < 0 || (n > 0 && !images)) return set_last(IWPP_ERR_INVALID);
    std::lock_guard<std::mutex> lk(h->mu);
    int prev_dev = 0;
    cudaGetDevice(&prev_dev);
    if (prev_dev != h->device) cudaSetDevice(h->device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Job job;
    int nl = 0;
    int rc = build_job(job, images, n, variant, cfg, s, STAGE_ASYNC, &h->stage_pool);
    if (rc == IWPP_OK) rc = enqueue_job(job, h->ws, s, h->device, true, h->ev0, h->ev1, true, &h->staging, &nl);
    const int rc2 = finish_staging(job, s);
    if (rc == IWPP_OK) rc = rc2;
    if (rc == IWPP_OK && h->ws.base) {
        // queue the counters copy behind the job; iwpp_handle_sync waits for it
        cudaError_t e = cudaMemcpyAsync(h->host_ctrl, h->ws.base, sizeof(Ctrl), cudaMemcpyDeviceToHost, s);
        rc = cuda_status(e);
    } else if (rc == IWPP_OK) {
        std::memset(h->host_ctrl, 0, sizeof(Ctrl));
    }
    h->last_stream = s;
    h->last_tiles = job.G;
    h->last_variant = job.variant;
    h->last_launch_status = rc;
    h->last_launches = nl + job.stage_launches;
    h->timed = job.G > 0;
    if (prev_dev != h->device) cudaSetDevice(prev_dev);
    return set_last(rc);
}

int iwpp_reconstruct_async(iwpp_handle h, void* marker, const void* mask, size_t pitch_marker, size_t pitch_mask,
                           int width, int height, int dtype, int connectivity, int variant, const iwpp_config* cfg,
                           void* stream) {
    iwpp_image im{marker, mask, pitch_marker, pitch_mask, width, height, dtype, connectivity};
    return iwpp_reconstruct_batch_async(h, &im, 1, variant, cfg, stream);
}

int iwpp_handle_sync(iwpp_handle h, iwpp_stats* stats) {
    if (!h) return set_last(IWPP_ERR_INVALID);
    std::lock_guard<std::mutex> lk(h->mu);
    if (h->last_launch_status != IWPP_OK) return set_last(h->last_launch_status);
    cudaError_t e = cudaStreamSynchronize(h->last_stream);
    if (e != cudaSuccess) return set_last(cuda_status(e));
    float ms = 0.f;
    if (h->timed) cudaEventElapsedTime(&ms, h->ev0, h->ev1);
    const Ctrl& c = *h->host_ctrl;
    const int st = status_of_job(c.error);
    if (stats) {
        stats->tiles = h->last_tiles;
        stats->visits = (long long)c.visits;
        stats->sweeps = (long long)c.sweeps;
        stats->pushes = (long long)c.pushes;
        stats->rounds = (int)c.rounds;
        stats->restarts = (int)c.restarts;
        stats->status = st;
        stats->variant = h->last_variant;
        stats->device_ms = ms;
        stats->row_steps = (long long)c.row_steps;
        for (int i = 0; i < 5; ++i) stats->phase_cycles[i] = (long long)c.phase[i];
        stats->launches = h->last_launches;
        stats->top_pixels = (long long)c.top_pixels;
        stats->front_stage = c.front_gate != 0u ? 1 : 0;
    }
    return set_last(st);
}

int iwpp_plan_create(iwpp_plan* out, iwpp_handle h, const iwpp_image* images, int n, int variant,
                     const iwpp_config* cfg) {
    if (!out || !h || n < 0 || (n > 0 && !images)) return set_last(IWPP_ERR_INVALID);
    *out = nullptr;
    std::lock_guard<std::mutex> lk(h->mu);
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(h->device);
    iwpp_plan p = new (std::nothrow) iwpp_plan_s();
    if (!p) return set_last(IWPP_ERR_OOM);
    p->h = h;
    Job job;
    cudaStream_t cs = nullptr;
    int rc = build_job(job, images, n, variant, cfg, nullptr, STAGE_OWNED, nullptr);
    for (const auto& st : job.staged)
        if (st.owned && st.buf_m) p->staged.push_back(st);
    cudaError_t e = cudaSuccess;
    if (rc == IWPP_OK) {
        p->tiles = job.G;
        p->variant = job.variant;
        e = cudaMallocHost(&p->host_ctrl, sizeof(Ctrl));
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
        rc = cuda_status(e);
    }
    if (rc == IWPP_OK) {
        // Workspace and descriptors first (outside the graph, once).
        const Layout l = job_layout(job);
        rc = ensure_workspace(p->ws, l.total);
        if (rc == IWPP_OK && job.descs.size() > 1) {
            char* wbase = static_cast<char*>(p->ws.base);
            std::vector<ImgDesc> descs = job.descs;
            for (size_t i = 0; i < descs.size(); ++i)
                descs[i].tmaps = job.has_tma[i] ? wbase + l.off_tmaps + i * 2u * sizeof(CUtensorMap) : nullptr;
            e = cudaMemcpy(wbase + l.off_tmaps, job.tmaps.data(), job.tmaps.size() * sizeof(CUtensorMap),
                           cudaMemcpyHostToDevice);
            if (e == cudaSuccess)
                e = cudaMemcpy(wbase + l.off_imgs, descs.data(), descs.size() * sizeof(ImgDesc),
                               cudaMemcpyHostToDevice);
            rc = cuda_status(e);
        }
        // Warm the kernel attributes before capture.
        LaunchInfo li;
        if (rc == IWPP_OK && job.G > 0)
            rc = cuda_status(
                engine_prepare(job.variant, job.tile_rows, job.cfg.solver, job_conn(job), job.G, job.cfg.grid_ctas,
                               h->device, &li));
    }
    if (rc == IWPP_OK) {
        e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeRelaxed);
        rc = cuda_status(e);
        if (rc == IWPP_OK) {
            // unaligned images: copy into the plan's staging buffers, run, copy back
            std::vector<StageCopy> in, back;
            int copies = 0;
            for (const auto& st : p->staged) {
                in.push_back(st.in_m());
                in.push_back(st.in_k());
                back.push_back(st.out_m());
            }
            e = launch_stage_copies(in, cs, &copies);
            rc = cuda_status(e);
            if (rc == IWPP_OK)
                rc = enqueue_job(job, p->ws, cs, h->device, false, nullptr, nullptr, false, nullptr, &p->launches);
            if (rc == IWPP_OK) rc = cuda_status(launch_stage_copies(back, cs, &copies));
            p->launches += copies;
            cudaError_t e2 = cudaStreamEndCapture(cs, &p->graph);
            if (rc == IWPP_OK) rc = cuda_status(e2);
        }
        if (rc == IWPP_OK) rc = cuda_status(cudaGraphInstantiate(&p->exec, p->graph, 0));
    }
    if (cs) cudaStreamDestroy(cs);
    cudaSetDevice(prev);
    if (rc != IWPP_OK) {
        cudaGetLastError();
        iwpp_plan_destroy(p);
        return set_last(rc);
    }
    *out = p;
    return set_last(IWPP_OK);
}

int iwpp_plan_launch(iwpp_plan p, void* stream) {
    if (!p || !p->exec) return set_last(IWPP_ERR_INVALID);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaGraphLaunch(p->exec, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(p->host_ctrl, p->ws.base, sizeof(Ctrl), cudaMemcpyDeviceToHost, s);
    p->last_stream = s;
    return set_last(cuda_status(e));
}

int iwpp_plan_sync(iwpp_plan p, iwpp_stats* stats) {
    if (!p) return set_last(IWPP_ERR_INVALID);
    cudaError_t e = cudaStreamSynchronize(p->last_stream);
    if (e != cudaSuccess) return set_last(cuda_status(e));
    const Ctrl& c = *p->host_ctrl;
    const int st = status_of_job(c.error);
    if (stats) {
        stats->tiles = p->tiles;
        stats->visits = (long long)c.visits;
        stats->sweeps = (long long)c.sweeps;
        stats->pushes = (long long)c.pushes;
        stats->rounds = (int)c.rounds;
        stats->restarts = (int)c.restarts;
        stats->status = st;
        stats->variant = p->variant;
        stats->device_ms = 0.0;
        stats->row_steps = (long long)c.row_steps;
        for (int i = 0; i < 5; ++i) stats->phase_cycles[i] = (long long)c.phase[i];
        stats->launches = p->launches;
        stats->top_pixels = (long long)c.top_pixels;
        stats->front_stage = c.front_gate != 0u ? 1 : 0;
    }
    return set_last(st);
}

int iwpp_plan_destroy(iwpp_plan p) {
    if (!p) return IWPP_OK;
    if (p->exec) cudaGraphExecDestroy(p->exec);
    if (p->graph) cudaGraphDestroy(p->graph);
    if (p->ws.base) cudaFree(p->ws.base);
    if (p->host_ctrl) cudaFreeHost(p->host_ctrl);
    for (auto& st : p->staged) {
        if (st.buf_m) cudaFree(st.buf_m);
        if (st.buf_k) cudaFree(st.buf_k);
    }
    delete p;
    return IWPP_OK;
}

int iwpp_queue_selftest(int device, int variant, int grid_side, int copies, iwpp_queue_test_result* out) {
    if (grid_side < 1 || grid_side > 4096 || copies < 1 || copies > 16) return set_last(IWPP_ERR_INVALID);
    int rc = check_device(device);
    if (rc != IWPP_OK) return set_last(rc);
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    const int v = resolve_variant(variant);
    const long long G = (long long)grid_side * grid_side;
    const long long cap = v == IWPP_QUEUE_UNIQUE ? G : G * copies;
    const size_t off_state = align_up(sizeof(Ctrl), 256);
    const size_t off_q0 = align_up(off_state + (size_t)G * 4u, 256);
    const size_t off_q1 = align_up(off_q0 + (size_t)cap * 4u, 256);
    const size_t off_hist = align_up(off_q1 + (size_t)cap * 4u, 256);
    const size_t off_out = align_up(off_hist + (size_t)G * 4u, 256);
    const size_t total = off_out + 3 * sizeof(unsigned long long);
    char* base = nullptr;
    cudaStream_t s = nullptr;
    cudaError_t e = cudaMalloc(&base, total);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    unsigned long long res[3] = {0ull, 0ull, ~0ull};
    Ctrl ctrl;
    std::memset(&ctrl, 0, sizeof(ctrl));
    if (e == cudaSuccess) {
        EngineArgs a{};
        a.G = (unsigned)G;
        a.state = reinterpret_cast<unsigned*>(base + off_state);
        a.q0 = reinterpret_cast<unsigned*>(base + off_q0);
        a.q1 = reinterpret_cast<unsigned*>(base + off_q1);
        a.cap = (unsigned)cap;
        a.ctrl = reinterpret_cast<Ctrl*>(base);
        a.timeout_ns = 10ll * 1000000000ll;
        a.max_restarts = 0;
        e = queue_selftest(a, v, copies, reinterpret_cast<unsigned*>(base + off_hist),
                           reinterpret_cast<unsigned long long*>(base + off_out), device, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(res, base + off_out, sizeof(res), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&ctrl, base, sizeof(Ctrl), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    rc = cuda_status(e);
    if (rc == IWPP_OK) rc = status_of_job(ctrl.error);
    if (rc == IWPP_OK && ctrl.overflow != 0u) rc = IWPP_ERR_OVERFLOW;
    if (out) {
        out->entries = (long long)res[0];
        out->expected = v == IWPP_QUEUE_UNIQUE ? G : G * copies;
        out->mismatched = (long long)res[1];
        out->first_bad = res[1] ? (long long)res[2] : -1;
        out->status = rc;
        out->variant = v;
    }
    if (s) cudaStreamDestroy(s);
    if (base) cudaFree(base);
    cudaSetDevice(prev);
    return set_last(rc);
}

int iwpp_autotune(iwpp_handle h, const iwpp_image* images, int n, int variant, int repeats, void* stream,
                  iwpp_tune_result* out) {
    if (!h || n <= 0 || !images || repeats < 0 || repeats > 50) return set_last(IWPP_ERR_INVALID);
    for (int i = 0; i < n; ++i) {
        const iwpp_image& im = images[i];
        const int rc = check_image(im.marker, im.mask, im.pitch_marker, im.pitch_mask, im.width, im.height, im.dtype,
                                   im.connectivity);
        if (rc != IWPP_OK) return set_last(rc);
    }
    if (repeats == 0) repeats = 3;
    std::lock_guard<std::mutex> lk(h->mu);
    int prev_dev = 0;
    cudaGetDevice(&prev_dev);
    if (prev_dev != h->device) cudaSetDevice(h->device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int v = resolve_variant(variant);

    // pristine copies of the markers: every candidate starts from them
    std::vector<void*> saved((size_t)n, nullptr);
    int rc = IWPP_OK;
    for (int i = 0; i < n && rc == IWPP_OK; ++i) {
        const iwpp_image& im = images[i];
        if (im.width == 0 || im.height == 0) continue;
        const size_t row = (size_t)im.width * bpp_of(im.dtype);
        cudaError_t e = cudaMallocAsync(&saved[(size_t)i], row * im.height, s);
        if (e == cudaSuccess)
            e = cudaMemcpy2DAsync(saved[(size_t)i], row, im.marker, im.pitch_marker, row, im.height,
                                  cudaMemcpyDeviceToDevice, s);
        rc = cuda_status(e);
    }
    auto restore = [&]() -> int {
        for (int i = 0; i < n; ++i) {
            const iwpp_image& im = images[i];
            if (!saved[(size_t)i]) continue;
            const size_t row = (size_t)im.width * bpp_of(im.dtype);
            cudaError_t e = cudaMemcpy2DAsync(im.marker, im.pitch_marker, saved[(size_t)i], row, row, im.height,
                                              cudaMemcpyDeviceToDevice, s);
            if (e != cudaSuccess) return cuda_status(e);
        }
        return IWPP_OK;
    };
    // median device time of one configuration, or a negative value when it failed
    int timed = 0;
    auto measure = [&](const iwpp_config& c) -> double {
        std::vector<float> ts;
        for (int r = 0; r < repeats; ++r) {
            if (restore() != IWPP_OK) return -1.0;
            Job job;
            int jrc = build_job(job, images, n, v, &c, s, STAGE_ASYNC, &h->stage_pool, false);
            if (jrc == IWPP_OK) jrc = enqueue_job(job, h->ws, s, h->device, true, h->ev0, h->ev1, true, &h->staging);
            const int src = finish_staging(job, s);
            if (jrc == IWPP_OK) jrc = src;
            if (jrc != IWPP_OK) {
                cudaStreamSynchronize(s);
                return -1.0;
            }
            if (cudaStreamSynchronize(s) != cudaSuccess) return -1.0;
            if (read_stats(h->host_ctrl, h->ws, s, job.G, job.variant, nullptr) != IWPP_OK) return -1.0;
            float ms = 0.f;
            if (job.G > 0) cudaEventElapsedTime(&ms, h->ev0, h->ev1);
            ts.push_back(ms);
        }
        ++timed;
        std::sort(ts.begin(), ts.end());
        return ts[ts.size() / 2];
    };

    iwpp_config best{};
    best.init_passes = 0;
    best.tile_rows = 64;
    double best_ms = -1.0, default_ms = -1.0;
    auto consider = [&](const iwpp_config& c, bool is_default) {
        const double ms = measure(c);
        if (ms < 0.0) return;
        if (is_default) default_ms = ms;
        if (best_ms < 0.0 || ms < best_ms) {
            best_ms = ms;
            best = c;
        }
    };
    if (rc == IWPP_OK) {
        // the untuned default first when it is the front stage (large
        // images), then stage 1: tile height x in-tile solver, no passes
        const int dflt_th = default_tile_rows(v, 0, job_tiles64(images, n));
        long long largest = 0;
        for (int i = 0; i < n; ++i)
            if (images[i].width > 0 && images[i].height > 0)
                largest = std::max(largest, (long long)images[i].width * images[i].height);
        const bool front_default = largest >= kFrontDefaultPixels;
        if (front_default) {
            // (the front stage as the device decides, with its default passes)
            iwpp_config c{};
            c.tile_rows = dflt_th;
            c.init_passes = 0;
            c.front_passes = 3;
            consider(c, true);
        }
        for (int th : {64, 32})
            for (int solver : {0, 1}) {  // (2 is the kernel of 0)
                iwpp_config c{};
                c.tile_rows = th;
                c.solver = solver;
                c.init_passes = 0;
                c.front_passes = 2;
                consider(c, !front_default && th == dflt_th && solver == 0);
            }
        // stage 1b: the best of stage 1 started from a seed check (the tiles
        // holding a pixel a neighbour can raise) instead of every tile
        if (best_ms >= 0.0 && best.front_passes == 2) {
            iwpp_config c = best;
            c.front_passes = 4;
            consider(c, false);
        }
        // stage 2: the front stage (top-level labelling, then 0 / 1 / 2 / 3 / 4 / 8
        // whole-image passes, then the engine from the seed check) with the
        // best tile height and solver; long propagation paths want it
        if (best_ms >= 0.0) {
            const iwpp_config base = best;
            for (int ip : {0, 1, 2, 3, 4, 8}) {
                iwpp_config c = base;
                c.front_passes = 1;
                c.init_passes = ip;
                consider(c, false);
            }
        }
        // stage 3: else a fixed number of initial whole-image raster /
        // anti-raster passes, doubling while they pay (long corridors want
        // one pass per turn of the front), stopping at the first count that
        // does not beat the best
        if (best_ms >= 0.0 && best.front_passes != 1 && best.front_passes != 3) {
            const iwpp_config base = best;
            for (int ip = 1; ip <= 64; ip *= 2) {
                iwpp_config c = base;
                c.init_passes = ip;
                const double before = best_ms;
                consider(c, false);
                if (!(best_ms < before)) break;
            }
        }
        // stage 4: queue capacity, for the queues whose capacity is free
        if (best_ms >= 0.0 && (v == IWPP_QUEUE_MUTEX || v == IWPP_QUEUE_DOUBLE)) {
            const iwpp_config base = best;
            for (int mult : {1, 16}) {
                iwpp_config c = base;
                c.queue_capacity = -mult;
                consider(c, false);
            }
        }
        if (best_ms < 0.0) rc = IWPP_ERR_TIMEOUT;
    }
    if (rc == IWPP_OK) {
        // record the winner for this workload class
        std::vector<int> dts, cns;
        std::vector<long long> pxs;
        for (int i = 0; i < n; ++i) {
            if (images[i].width <= 0 || images[i].height <= 0) continue;
            dts.push_back(images[i].dtype);
            cns.push_back(images[i].connectivity);
            pxs.push_back((long long)images[i].width * images[i].height);
        }
        if (!dts.empty()) {
            TuneEntry e{best.tile_rows, best.solver, best.init_passes,
                        best.queue_capacity < 0 ? (int)-best.queue_capacity : 0, tune_front_store(best.front_passes)};
            tune_store(tune_key(v, dts.data(), cns.data(), pxs.data(), (int)dts.size()), e);
        }
        // leave the images reconstructed (with the winner)
        rc = restore();
        if (rc == IWPP_OK) {
            Job job;
            rc = build_job(job, images, n, v, &best, s, STAGE_ASYNC, &h->stage_pool, false);
            if (rc == IWPP_OK) rc = enqueue_job(job, h->ws, s, h->device, false, h->ev0, h->ev1, true, &h->staging);
            const int src = finish_staging(job, s);
            if (rc == IWPP_OK) rc = src;
            if (cudaStreamSynchronize(s) != cudaSuccess && rc == IWPP_OK) rc = IWPP_ERR_CUDA;
            if (rc == IWPP_OK) rc = read_stats(h->host_ctrl, h->ws, s, job.G, job.variant, nullptr);
        }
    } else {
        restore();  // leave the markers as they came
    }
    for (void* p : saved)
        if (p) cudaFreeAsync(p, s);
    cudaStreamSynchronize(s);
    if (out) {
        out->best = best;
        out->best_ms = best_ms;
        out->default_ms = default_ms;
        out->candidates = timed;
        out->reserved = 0;
    }
    if (prev_dev != h->device) cudaSetDevice(prev_dev);
    return set_last(rc);
}

int iwpp_clip(void* marker, const void* mask, size_t pitch_marker, size_t pitch_mask, int width, int height,
              int dtype, void* stream) {
    int rc = check_image(marker, mask, pitch_marker, pitch_mask, width, height, dtype, 4);
    if (rc != IWPP_OK) return set_last(rc);
    ImgDesc d{};
    d.marker = static_cast<unsigned char*>(marker);
    d.mask = static_cast<const unsigned char*>(mask);
    d.pitch_m = (long long)pitch_marker;
    d.pitch_k = (long long)pitch_mask;
    d.W = width;
    d.H = height;
    d.dtype = dtype;
    d.conn = 4;
    if (!aligned_for_engine(marker, pitch_marker) || !aligned_for_engine(mask, pitch_mask)) {
        // byte-granular rows: one thread per pixel via a pixel-sized view
        // is not needed for correctness here; route through staging
        iwpp_image im{marker, mask, pitch_marker, pitch_mask, width, height, dtype, 4};
        Job job;
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        iwpp_config c{};
        rc = build_job(job, &im, 1, IWPP_QUEUE_UNIQUE, &c, s, STAGE_ASYNC, nullptr);
        if (rc == IWPP_OK && !job.descs.empty()) rc = cuda_status(launch_clip(job.descs[0], s));
        const int rc2 = finish_staging(job, s);
        return set_last(rc == IWPP_OK ? rc2 : rc);
    }
    return set_last(cuda_status(launch_clip(d, static_cast<cudaStream_t>(stream))));
}

int iwpp_fixed_point_violations(const void* result, const void* mask, size_t pitch_result, size_t pitch_mask,
                                int width, int height, int dtype, int connectivity, void* stream,
                                unsigned long long* count) {
    if (!count) return set_last(IWPP_ERR_INVALID);
    *count = 0ull;
    int rc = check_image(result, mask, pitch_result, pitch_mask, width, height, dtype, connectivity);
    if (rc != IWPP_OK || width == 0 || height == 0) return set_last(rc);
    ImgDesc d{};
    d.marker = static_cast<unsigned char*>(const_cast<void*>(result));
    d.mask = static_cast<const unsigned char*>(mask);
    d.pitch_m = (long long)pitch_result;
    d.pitch_k = (long long)pitch_mask;
    d.W = width;
    d.H = height;
    d.dtype = dtype;
    d.conn = connectivity;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    unsigned long long* dc = nullptr;
    cudaError_t e = cudaMallocAsync(&dc, sizeof(unsigned long long), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(dc, 0, sizeof(unsigned long long), s);
    if (e == cudaSuccess) e = launch_fixed_point_check(d, dc, s);
    unsigned long long host = 0ull;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&host, dc, sizeof(host), cudaMemcpyDeviceToHost, s);
    if (dc) cudaFreeAsync(dc, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    *count = host;
    return set_last(cuda_status(e));
}

int iwpp_sweep(void* marker, const void* mask, size_t pitch_marker, size_t pitch_mask, int width, int height,
               int dtype, int connectivity, int direction, void* stream) {
    int rc = check_image(marker, mask, pitch_marker, pitch_mask, width, height, dtype, connectivity);
    if (rc != IWPP_OK) return set_last(rc);
    if (direction < 0 || direction > 3) return set_last(IWPP_ERR_INVALID);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    auto sweep = [&](const ImgDesc& d) {
        void* scratch = nullptr;
        const size_t sb = direction == 1 || direction == 3 ? sweep_scratch_bytes(d) : 0;
        if (sb > 0 && cudaMallocAsync(&scratch, sb, s) != cudaSuccess) {
            cudaGetLastError();
            scratch = nullptr;  // one warp per whole column instead
        }
        const int r = cuda_status(launch_sweep(d, direction, s, scratch));
        if (scratch) cudaFreeAsync(scratch, s);
        return r;
    };
    if (aligned_for_engine(marker, pitch_marker) && aligned_for_engine(mask, pitch_mask)) {
        ImgDesc d{};
        d.marker = static_cast<unsigned char*>(marker);
        d.mask = static_cast<const unsigned char*>(mask);
        d.pitch_m = (long long)pitch_marker;
        d.pitch_k = (long long)pitch_mask;
        d.W = width;
        d.H = height;
        d.dtype = dtype;
        d.conn = connectivity;
        return set_last(width > 0 && height > 0 ? sweep(d) : IWPP_OK);
    }
    iwpp_image im{marker, mask, pitch_marker, pitch_mask, width, height, dtype, connectivity};
    Job job;
    iwpp_config c{};
    rc = build_job(job, &im, 1, IWPP_QUEUE_UNIQUE, &c, s, STAGE_ASYNC, nullptr);
    if (rc == IWPP_OK && !job.descs.empty()) rc = sweep(job.descs[0]);
    const int rc2 = finish_staging(job, s);
    return set_last(rc == IWPP_OK ? rc2 : rc);
}

int iwpp_sweep_timing(void* marker, const void* mask, size_t pitch_marker, size_t pitch_mask, int width,
                      int height, int dtype, int connectivity, float* ms_out) {
    if (!ms_out) return set_last(IWPP_ERR_INVALID);
    int rc = check_image(marker, mask, pitch_marker, pitch_mask, width, height, dtype, connectivity);
    if (rc != IWPP_OK) return set_last(rc);
    for (int dir = 0; dir < 4; ++dir) ms_out[dir] = 0.f;
    if (width == 0 || height == 0) return set_last(IWPP_OK);
    // Prepared once (staging, scratch), then the four kernels alone between
    // events, as the reference times its passes (DQ MR.cu:1077-1178).
    iwpp_image im{marker, mask, pitch_marker, pitch_mask, width, height, dtype, connectivity};
    Job job;
    cudaStream_t s = nullptr;
    iwpp_config c{};
    rc = build_job(job, &im, 1, IWPP_QUEUE_UNIQUE, &c, s, STAGE_ASYNC, nullptr);
    void* scratch = nullptr;
    cudaEvent_t ev[5] = {};
    if (rc == IWPP_OK && !job.descs.empty()) {
        const size_t sb = sweep_scratch_bytes(job.descs[0]);
        if (sb > 0 && cudaMallocAsync(&scratch, sb, s) != cudaSuccess) {
            cudaGetLastError();
            scratch = nullptr;
        }
        for (auto& e : ev) cudaEventCreate(&e);
        cudaEventRecord(ev[0], s);
        for (int dir = 0; dir < 4 && rc == IWPP_OK; ++dir) {
            rc = cuda_status(launch_sweep(job.descs[0], dir, s, scratch));
            cudaEventRecord(ev[dir + 1], s);
        }
        if (rc == IWPP_OK) {
            rc = cuda_status(cudaEventSynchronize(ev[4]));
            for (int dir = 0; dir < 4 && rc == IWPP_OK; ++dir) cudaEventElapsedTime(&ms_out[dir], ev[dir], ev[dir + 1]);
        }
        for (auto& e : ev)
            if (e) cudaEventDestroy(e);
        if (scratch) cudaFreeAsync(scratch, s);
    }
    const int rc2 = finish_staging(job, s);
    cudaStreamSynchronize(s);
    return set_last(rc == IWPP_OK ? rc2 : rc);
}

void MorphologicalReconstruction(unsigned char* marker, unsigned char* mask, size_t pitchMarker, size_t pitchMask,
                                 int size) {
    iwpp_image im{marker, mask, pitchMarker, pitchMask, size, size, IWPP_U8, 4};
    set_last(run_job_sync(nullptr, &im, 1, IWPP_QUEUE_DEFAULT, nullptr, nullptr, nullptr));
}

void configureHeapSize(void) {}

int iwpp_last_status(void) { return g_last_status.load(); }

}  // extern "C"
