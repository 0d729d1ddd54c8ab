// iwpp_device.cuh -- device building blocks of the GB300 reconstruction
// engine: tile visits by a CTA (TMA fetch with halo, vertical and horizontal
// passes to local convergence, write-back, neighbour detection).
//
// Layout: a tile is TH rows x TW pixels with TW * sizeof(pixel) = 128 bytes
// (TW = 128 uint8, 64 uint16, 32 int32).  One CTA owns one tile at a time, a
// warp each block of eight rows.  Shared memory holds the tile plus the halo
// rows above and below as dense 128-byte rows (SMEM row r = image row
// y0 - 1 + r), so one TMA box load per image plane fetches it.  A 32-bit word
// holds PPW = 4 / 2 / 1 pixels.  Vertical propagation walks a block's rows
// with a word column per lane; horizontal propagation is a lane's own chain
// and a scan over eight lanes in the max-min semiring.
//
// Reference counterparts (IWPP MP/src/MorphologicalReconstruction.cu):
//   tile fetch with a one-pixel halo        MR.cu:232-312
//   in-tile directional sweeps to stability MR.cu:34-161, loop MR.cu:320-325
//   write-back + neighbour detection        MR.cu:335-512
// The rule everywhere is MR.cu:43-44: m[c] = max(m[c], min(m[p], mask[c])).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace iwpp {

constexpr unsigned FULL = 0xffffffffu;

enum : int { DT_U8 = 0, DT_U16 = 1, DT_I32 = 2 };

// ------------------------------------------------------------------ pixels
// Pixels are carried as uint32 (zero-extended for the unsigned types, the
// bit pattern for int32); Px<DT> supplies the order and the packing.
template <int DT>
struct Px;

template <>
struct Px<DT_U8> {
    static constexpr int PPW = 4;
    static constexpr int BPP = 1;
    static constexpr uint32_t MINPX = 0u;
    static constexpr uint32_t MINW = 0u;
    static constexpr uint32_t FIRST_MASK = 0x000000ffu, LAST_MASK = 0xff000000u;
    __device__ static __forceinline__ uint32_t mx(uint32_t a, uint32_t b) { return max(a, b); }
    __device__ static __forceinline__ uint32_t mn(uint32_t a, uint32_t b) { return min(a, b); }
    __device__ static __forceinline__ uint32_t mx3(uint32_t a, uint32_t b, uint32_t c) { return __vimax3_u32(a, b, c); }
    __device__ static __forceinline__ bool gt(uint32_t a, uint32_t b) { return a > b; }
    __device__ static __forceinline__ void unpack(uint32_t w, uint32_t (&p)[4]) {
        p[0] = __byte_perm(w, 0u, 0x4440);
        p[1] = __byte_perm(w, 0u, 0x4441);
        p[2] = __byte_perm(w, 0u, 0x4442);
        p[3] = __byte_perm(w, 0u, 0x4443);
    }
    __device__ static __forceinline__ uint32_t pack(const uint32_t (&p)[4]) {
        const uint32_t lo = __byte_perm(p[0], p[1], 0x0040);
        const uint32_t hi = __byte_perm(p[2], p[3], 0x0040);
        return __byte_perm(lo, hi, 0x5410);
    }
    __device__ static __forceinline__ uint32_t ld_px(const unsigned char* p) { return *p; }
    __device__ static __forceinline__ uint32_t ld_px_cg(const unsigned char* p) { return __ldcg(p); }
    __device__ static __forceinline__ void st_px(unsigned char* p, uint32_t v) { *p = (unsigned char)v; }
};

template <>
struct Px<DT_U16> {
    static constexpr int PPW = 2;
    static constexpr int BPP = 2;
    static constexpr uint32_t MINPX = 0u;
    static constexpr uint32_t MINW = 0u;
    static constexpr uint32_t FIRST_MASK = 0x0000ffffu, LAST_MASK = 0xffff0000u;
    __device__ static __forceinline__ uint32_t mx(uint32_t a, uint32_t b) { return max(a, b); }
    __device__ static __forceinline__ uint32_t mn(uint32_t a, uint32_t b) { return min(a, b); }
    __device__ static __forceinline__ uint32_t mx3(uint32_t a, uint32_t b, uint32_t c) { return __vimax3_u32(a, b, c); }
    __device__ static __forceinline__ bool gt(uint32_t a, uint32_t b) { return a > b; }
    __device__ static __forceinline__ void unpack(uint32_t w, uint32_t (&p)[2]) {
        p[0] = w & 0xffffu;
        p[1] = w >> 16;
    }
    __device__ static __forceinline__ uint32_t pack(const uint32_t (&p)[2]) { return __byte_perm(p[0], p[1], 0x5410); }
    __device__ static __forceinline__ uint32_t ld_px(const unsigned char* p) {
        return *reinterpret_cast<const unsigned short*>(p);
    }
    __device__ static __forceinline__ uint32_t ld_px_cg(const unsigned char* p) {
        return __ldcg(reinterpret_cast<const unsigned short*>(p));
    }
    __device__ static __forceinline__ void st_px(unsigned char* p, uint32_t v) {
        *reinterpret_cast<unsigned short*>(p) = (unsigned short)v;
    }
};

template <>
struct Px<DT_I32> {
    static constexpr int PPW = 1;
    static constexpr int BPP = 4;
    static constexpr uint32_t MINPX = 0x80000000u;
    static constexpr uint32_t MINW = 0x80000000u;
    static constexpr uint32_t FIRST_MASK = 0xffffffffu, LAST_MASK = 0xffffffffu;
    __device__ static __forceinline__ uint32_t mx(uint32_t a, uint32_t b) { return (uint32_t)max((int)a, (int)b); }
    __device__ static __forceinline__ uint32_t mn(uint32_t a, uint32_t b) { return (uint32_t)min((int)a, (int)b); }
    __device__ static __forceinline__ uint32_t mx3(uint32_t a, uint32_t b, uint32_t c) {
        return (uint32_t)__vimax3_s32((int)a, (int)b, (int)c);
    }
    __device__ static __forceinline__ bool gt(uint32_t a, uint32_t b) { return (int)a > (int)b; }
    __device__ static __forceinline__ void unpack(uint32_t w, uint32_t (&p)[1]) { p[0] = w; }
    __device__ static __forceinline__ uint32_t pack(const uint32_t (&p)[1]) { return p[0]; }
    __device__ static __forceinline__ uint32_t ld_px(const unsigned char* p) {
        return (uint32_t)*reinterpret_cast<const int*>(p);
    }
    __device__ static __forceinline__ uint32_t ld_px_cg(const unsigned char* p) {
        return (uint32_t)__ldcg(reinterpret_cast<const int*>(p));
    }
    __device__ static __forceinline__ void st_px(unsigned char* p, uint32_t v) { *reinterpret_cast<int*>(p) = (int)v; }
};

// ------------------------------------------------------------ image / tiles
// One image of a (possibly single-image) job.  Pitches are in bytes.
struct ImgDesc {
    unsigned char* marker;
    const unsigned char* mask;
    long long pitch_m;
    long long pitch_k;
    const void* tmaps;  // two CUtensorMap (marker, mask) or nullptr (plain loads)
    int W, H;
    int dtype, conn;
    int tiles_x, tiles_y;
    int tile_base;  // first global tile index of this image
    int tile_rows;  // TH used for this image
    // Nullable.  The front-stage kernels (top-level labelling, whole-image
    // passes, seed check) over this image return at once while *gate is 0:
    // the job decided on the device to leave the image to the tile engine.
    const unsigned* gate;
};

__device__ __forceinline__ bool gated_off(const ImgDesc& d) {
    return d.gate != nullptr && *(const volatile unsigned*)d.gate == 0u;
}

// neighbour direction bits returned by a tile visit
enum : unsigned {
    NB_N = 1u << 0, NB_S = 1u << 1, NB_W = 1u << 2, NB_E = 1u << 3,
    NB_NW = 1u << 4, NB_NE = 1u << 5, NB_SW = 1u << 6, NB_SE = 1u << 7,
    NB_STORED = 1u << 8  // the visit stored pixels
};
__device__ __constant__ static const int kNbDx[8] = {0, 0, -1, 1, -1, 1, -1, 1};
__device__ __constant__ static const int kNbDy[8] = {-1, 1, 0, 0, -1, -1, 1, 1};

// In-tile solvers of a kernel (iwpp_config.solver): passes by several warps; by
// one warp per tile, row sweeps, or revisits by the pixel queue.
enum : int { SOLVE_PASSES = 0, SOLVE_SWEEPS = 1, SOLVE_PQ = 2 };

// A CTA's counters.
struct VisitCount {
    unsigned visits, pushes;
    unsigned sweeps;     // rounds of passes, or sweeps
    unsigned row_steps;  // rows processed
    long long cycles[5];  // queue read, fetch, processing, dump, queue write (the first warp's clock)
};

// A tile's shared memory (128-byte aligned; TMA writes tm / tk densely).
// SMEM row r holds image row y0 - 1 + r: row 0 is the halo above the tile,
// rows 1..TH the tile, row TH+1 the halo below.  hL* / hR* hold the left /
// right halo column pixels of the same rows.
constexpr int kPqCap = 448;  // pixel-queue solver: FIFO entries
template <int TH>
struct __align__(128) TileSmem {
    uint32_t tm[(TH + 2) * 32];
    uint32_t tk[(TH + 2) * 32];
    uint32_t hLm[TH + 2];
    uint32_t hLk[TH + 2];
    uint32_t hRm[TH + 2];
    uint32_t hRk[TH + 2];
    unsigned long long mbar;
    // the visit the CTA's warps work on together; kept here rather than in
    // registers, which the passes need
    ImgDesc d;        // its image
    int tx, ty;       // its place
    unsigned sides;   // NB_* bits: halo sides to look at
    unsigned nb;      // NB_* bits found by the warps
    unsigned go;      // 1 a tile, 0 the job is over
    VisitCount count;  // the first warp's counters
};
// with what the W warps of a visit by passes tell one another
template <int TH, int W>
struct __align__(128) TileSmemPasses : TileSmem<TH> {
    // a row beside a warp's first / last block rose: by the parity of the
    // round, the warp, from above / below
    unsigned mark[2][W][2];
};
// with the pixel-queue solver's FIFO: tile pixel indices r * TW + c
template <int TH>
struct __align__(128) TileSmemPq : TileSmem<TH> {
    unsigned short pq[kPqCap];
};

// ------------------------------------------------------- async-copy helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0u;
}

// 2-D TMA box load: box origin (x bytes, y rows) of the tensor map into smem.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const void* tmap, int x, int y,
                                            unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
            "r"(smem_u32(smem_dst)),
        "l"(tmap), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// One word, global to shared, by the calling thread (4-byte aligned).  Goes
// through L1: an acquire before it (which drops what L1 holds) makes it see
// other SMs' released stores like any load.
__device__ __forceinline__ void cp_async_4(void* smem_dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem_dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// acquire / release fence at GPU scope (cheaper than __threadfence, which is
// sequentially consistent)
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ long long globaltimer_ns() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ------------------------------------------------------ packed-word max
// Per-pixel max of two packed words (uint8: four bytes, uint16: two halves,
// int32: one signed value).
template <int DT>
__device__ __forceinline__ uint32_t word_max(uint32_t a, uint32_t b) {
    if (DT == DT_U8) return __vmaxu4(a, b);
    if (DT == DT_U16) return __vmaxu2(a, b);
    return (uint32_t)max((int)a, (int)b);
}

// ------------------------------------------------ clamp-map scan steps
// Carrying a value x through a run of pixels along the scan direction maps
// it to max(min(x, B), A) (B: the run's least mask, A: the run's last pixel
// without a carry).  One step of the warp's inclusive scan composes a lane's
// map after the map of the lanes d before it:
//   A = max(min(A_prev, B), A),  B = min(B_prev, B).
// A lane with no source at distance d reads its own map back, and a clamp
// map composed with itself is itself, so no lane predicate is needed.
// uint8 / uint16: (A, B) share one word, A in the low half, and a step is
// one shuffle, one 16x2 min and one 16x2 max on the critical path.
template <bool FWD>
__device__ __forceinline__ uint32_t map_step_packed(uint32_t cur, int d) {
    const uint32_t prev = FWD ? __shfl_up_sync(FULL, cur, d) : __shfl_down_sync(FULL, cur, d);
    return __vmaxu2(__vminu2(prev, __byte_perm(cur, 0u, 0x3232)), cur & 0xffffu);
}
// int32: A and B in two words, signed order.
template <bool FWD>
__device__ __forceinline__ void map_step_i32(uint32_t& A, uint32_t& B, int d) {
    const int Ap = FWD ? __shfl_up_sync(FULL, (int)A, d) : __shfl_down_sync(FULL, (int)A, d);
    const int Bp = FWD ? __shfl_up_sync(FULL, (int)B, d) : __shfl_down_sync(FULL, (int)B, d);
    A = (uint32_t)max(min(Ap, (int)B), (int)A);
    B = (uint32_t)min(Bp, (int)B);
}

// ---------------------------------------------------- horizontal warp scan
// Propagates along one row in scan order (FWD: left to right) with `cin` the
// marker value of the halo pixel entering the row at the first lane.  The
// transfer function of a word for the value x entering it is
// f(x) = max(min(x, B), A) with B = min of its mask pixels and A = its exit
// pixel after the in-word pass; these compose associatively:
// (A2,B2) o (A1,B1) = (max(min(A1, B2), A2), min(B1, B2)).
// N: pixels per lane (one 32-bit word by default; the 16-byte-lane sweeps
// hold four words).
template <int DT, bool FWD, int N = Px<DT>::PPW>
__device__ __forceinline__ void hscan(uint32_t (&m)[N], const uint32_t (&k)[N], uint32_t cin, int lane) {
    using P = Px<DT>;
#pragma unroll
    for (int s = 1; s < N; ++s) {
        const int j = FWD ? s : N - 1 - s;
        const int jp = FWD ? j - 1 : j + 1;
        m[j] = P::mx(m[j], P::mn(m[jp], k[j]));
    }
    const int first = FWD ? 0 : N - 1, last = FWD ? N - 1 : 0;
    const int edge_lane = FWD ? 0 : 31;
    uint32_t in_px = FWD ? __shfl_up_sync(FULL, m[last], 1) : __shfl_down_sync(FULL, m[last], 1);
    if (lane == edge_lane) in_px = cin;
    // A carry that does not raise a word's entry pixel raises nothing after it.
    const bool need = P::gt(P::mn(in_px, k[first]), m[first]);
    if (!__any_sync(FULL, need)) return;

    uint32_t A = m[last], B = k[0];
#pragma unroll
    for (int j = 1; j < N; ++j) B = P::mn(B, k[j]);
    if (lane == edge_lane) {
        A = P::mx(A, P::mn(cin, B));
        B = P::MINPX;  // the entry lane becomes a constant: nothing before it
    }
    if (DT == DT_I32) {
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) map_step_i32<FWD>(A, B, d);
    } else {
        uint32_t cur = A | (B << 16);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) cur = map_step_packed<FWD>(cur, d);
        A = cur & 0xffffu;
    }
    uint32_t c = FWD ? __shfl_up_sync(FULL, A, 1) : __shfl_down_sync(FULL, A, 1);
    if (lane == edge_lane) c = cin;
#pragma unroll
    for (int s = 0; s < N; ++s) {
        const int j = FWD ? s : N - 1 - s;
        c = P::mn(c, k[j]);
        m[j] = P::mx(m[j], c);
    }
}

// ------------------------------------------------------------- one sweep
// DOWN = raster order (rows top to bottom, each row left to right),
// otherwise anti-raster.  After a complete raster sweep every pixel satisfies
// its constraints towards N+ = {left, up-left, up, up-right}; after an
// anti-raster sweep towards N-.
//
// Rows are skipped when nothing they depend on can have changed since they
// last satisfied this sweep's constraints: a row is processed when the row
// before it (in sweep order) rose in this sweep, or when it or a vertical
// neighbour rose in the previous sweep (`dil`, already dilated by one row),
// or when its halo inputs are new (`force`, folded into `dil` by the caller).
// `chg` receives the rows that rose (bit r-1 for SMEM row r).
template <int DT, int CONN, int TH, bool DOWN>
__device__ __forceinline__ void sweep(TileSmem<TH>& sm, int lane, unsigned long long dil, unsigned long long& chg,
                                      bool& col_changed, uint32_t edge_mask, unsigned& row_steps) {
    using P = Px<DT>;
    constexpr int N = P::PPW;
    uint32_t prev[N];
    bool prev_valid = false, prev_changed = false;
    // the row words of step i are read during step i - 1 (only step i
    // writes its row), so their shared-memory latency overlaps a scan
    uint32_t next_m = sm.tm[(DOWN ? 1 : TH) * 32 + lane], next_k = sm.tk[(DOWN ? 1 : TH) * 32 + lane];
#pragma unroll 1
    for (int i = 0; i < TH; ++i) {
        const int r = DOWN ? 1 + i : TH - i;  // SMEM row
        const int rp = DOWN ? r - 1 : r + 1;  // SMEM row before it in sweep order
        const uint32_t old = next_m, kw = next_k;
        if (i + 1 < TH) {
            const int rn = DOWN ? r + 1 : r - 1;
            next_m = sm.tm[rn * 32 + lane];
            next_k = sm.tk[rn * 32 + lane];
        }
        if (!prev_changed && !((dil >> (r - 1)) & 1ull)) {
            prev_valid = false;
            continue;
        }
        if (!prev_valid) P::unpack(sm.tm[rp * 32 + lane], prev);
        ++row_steps;
        uint32_t m[N], k[N];
        P::unpack(old, m);
        P::unpack(kw, k);
        if (CONN == 8) {
            uint32_t left = __shfl_up_sync(FULL, prev[N - 1], 1);
            uint32_t right = __shfl_down_sync(FULL, prev[0], 1);
            if (lane == 0) left = sm.hLm[rp];
            if (lane == 31) right = sm.hRm[rp];
            if (N == 1) {
                m[0] = P::mx(m[0], P::mn(P::mx3(left, prev[0], right), k[0]));
            } else {
                // shared pairwise maxima of the previous row
                uint32_t pair[N > 1 ? N - 1 : 1];
#pragma unroll
                for (int j = 0; j + 1 < N; ++j) pair[j] = P::mx(prev[j], prev[j + 1]);
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    const uint32_t v = j == 0 ? P::mx(left, pair[0]) : j == N - 1 ? P::mx(pair[N - 2], right)
                                                                                   : P::mx(prev[j - 1], pair[j]);
                    m[j] = P::mx(m[j], P::mn(v, k[j]));
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < N; ++j) m[j] = P::mx(m[j], P::mn(prev[j], k[j]));
        }
        hscan<DT, DOWN>(m, k, DOWN ? sm.hLm[r] : sm.hRm[r], lane);
        const uint32_t nw = P::pack(m);
        prev_changed = __any_sync(FULL, nw != old);
        if (prev_changed) {
            sm.tm[r * 32 + lane] = nw;
            chg |= 1ull << (r - 1);
            col_changed |= ((nw ^ old) & edge_mask) != 0u;
        }
#pragma unroll
        for (int j = 0; j < N; ++j) prev[j] = m[j];
        prev_valid = true;
    }
    __syncwarp();
}

// ------------------------------------------------------- in-tile passes
// The tile converges through vertical and horizontal passes, the separable
// form of the reference's XForward / XBackward / YDownward / YUpward
// propagation (MR.cu:34-161), on blocks of eight rows in shared memory:
//   vertical (vblock): a lane walks its own word column over the block's
//     rows, down and up, entered by the rows beside the block
//     (8-connectivity: then a step that adds the diagonals);
//   horizontal (hblock): eight lanes hold a row, 16 bytes each, so most of a
//     row's closure is in-lane work and the clamp maps cross three lane steps
//     instead of five.
// What bounds both is a warp's own instruction rate: min, max and byte
// permutes issue every other cycle in one of the SM's four schedulers, so a
// block costs a warp its instructions twice over in cycles whatever else the
// SM does (measured alone and with 24 warps per SM: vertical 4-connected one
// direction 371 / 436 cycles per block, horizontal 682-932 / 870-1200).  A
// tile is therefore visited by as many warps as it has blocks (solve_tile),
// one on each scheduler, instead of by one warp block after block.
// The halo columns enter once, before the passes (halo_columns): they do not
// change during a visit, so no pass looks at them again.
// Rows are numbered as in shared memory (1..TH); block b has rows 8b+1..8b+8.

// What rose in a block (votes): its first row, the six between, its last row,
// a pixel of the tile's first or last column; RF_AGAIN: a diagonal raised
// something in the vertical pass, which a walk may carry on.
enum : unsigned { RF_FIRST = 1u, RF_INNER = 2u, RF_LAST = 4u, RF_COL = 8u, RF_AGAIN = 16u, RF_ROWS = 7u };

// OR of a per-lane 64-bit mask over the warp.
__device__ __forceinline__ unsigned long long warp_or64(unsigned long long v) {
    const unsigned lo = __reduce_or_sync(FULL, (unsigned)v);
    const unsigned hi = __reduce_or_sync(FULL, (unsigned)(v >> 32));
    return ((unsigned long long)hi << 32) | lo;
}

// A row's words in the form the vertical walk uses: uint8 the word's even and
// odd bytes, each byte doubled to 16 bits (which keeps the order and costs
// one byte permute); others the word itself.
template <int DT>
struct VRow {
    static constexpr int N = DT == DT_U8 ? 2 : 1;
    uint32_t v[N];
    __device__ __forceinline__ void set(uint32_t w) {
        if constexpr (DT == DT_U8) {
            v[0] = __byte_perm(w, 0u, 0x2200);
            v[1] = __byte_perm(w, 0u, 0x3311);
        } else {
            v[0] = w;
        }
    }
    __device__ __forceinline__ uint32_t word() const {
        if constexpr (DT == DT_U8)
            return __byte_perm(v[0], v[1], 0x6240);
        else
            return v[0];
    }
    __device__ __forceinline__ bool differs(const VRow& o) const {
        if constexpr (DT == DT_U8)
            return ((v[0] ^ o.v[0]) | (v[1] ^ o.v[1])) != 0u;
        else
            return v[0] != o.v[0];
    }
};

// Diagonals: byte selectors that put the word one pixel to the left / right
// of a row's together from the lane's word and its neighbour lane's (uint8:
// of the odd / even half).  In the first / last lane, where the tile ends,
// they pick a pixel that the lane has already.
struct EdgeSel {
    unsigned left, right;
    __device__ __forceinline__ explicit EdgeSel(int lane)
        : left(lane == 0 ? 0x5454u : 0x5432u), right(lane == 31 ? 0x3232u : 0x5432u) {}
};

template <int DT>
__device__ __forceinline__ uint32_t vmx(uint32_t a, uint32_t b) {
    return DT == DT_I32 ? (uint32_t)max((int)a, (int)b) : __vmaxu2(a, b);
}
template <int DT>
__device__ __forceinline__ uint32_t vmn(uint32_t a, uint32_t b) {
    return DT == DT_I32 ? (uint32_t)min((int)a, (int)b) : __vminu2(a, b);
}

// Each pixel the larger of its left and right neighbours in the row (a lane
// without a neighbour lane reads its own word).
template <int DT>
__device__ __forceinline__ VRow<DT> beside(const VRow<DT>& p, const EdgeSel& sel) {
    VRow<DT> h;
    if constexpr (DT == DT_U8) {
        // the even bytes' neighbours are the odd half and the odd half
        // shifted in from the left, the odd bytes' the even half and the even
        // half shifted in from the right
        const uint32_t left = __shfl_up_sync(FULL, p.v[1], 1), right = __shfl_down_sync(FULL, p.v[0], 1);
        h.v[0] = __vmaxu2(p.v[1], __byte_perm(left, p.v[1], sel.left));
        h.v[1] = __vmaxu2(p.v[0], __byte_perm(p.v[0], right, sel.right));
    } else {
        const uint32_t left = __shfl_up_sync(FULL, p.v[0], 1), right = __shfl_down_sync(FULL, p.v[0], 1);
        if (DT == DT_U16)
            h.v[0] = __vmaxu2(__byte_perm(left, p.v[0], sel.left), __byte_perm(p.v[0], right, sel.right));
        else
            h.v[0] = vmx<DT>(left, right);
    }
    return h;
}

// m = max(m, min(p, k)).
template <int DT>
__device__ __forceinline__ void vstep(VRow<DT>& m, const VRow<DT>& k, const VRow<DT>& p) {
#pragma unroll
    for (int j = 0; j < VRow<DT>::N; ++j) m.v[j] = vmx<DT>(m.v[j], vmn<DT>(p.v[j], k.v[j]));
}

// 8-connectivity, known to the kernel (CONN) or, with CONN 0, looked up.
template <int CONN>
__device__ __forceinline__ bool eight(bool conn8) {
    return CONN == 0 ? conn8 : CONN == 8;
}

// What a row offers the row above or below it.
template <int DT, int CONN>
__device__ __forceinline__ VRow<DT> offers(const VRow<DT>& p, const EdgeSel& sel, bool conn8 = false) {
    VRow<DT> q = p;
    if (eight<CONN>(conn8)) {
        const VRow<DT> h = beside<DT>(p, sel);
#pragma unroll
        for (int j = 0; j < VRow<DT>::N; ++j) q.v[j] = vmx<DT>(p.v[j], h.v[j]);
    }
    return q;
}

// Vertical pass over block b.  `due`: the walks that violated constraints in
// the block may call for (VD_DOWN, VD_UP), and the rows beside the block that
// rose (VD_ABOVE, VD_BELOW), which call for a walk only if they raise the
// block's first / last row: looked at first, since many do not.  Returns RF_*
// (warp-uniform).
// 8-connectivity: the rows beside the block enter with their diagonals, the
// walks go straight up and down, and one step over all rows at once then adds
// the diagonals between the block's rows; a path that a diagonal opens goes
// on in the next pass (RF_AGAIN).  Walks that take the diagonals along wait
// 24 cycles for a shuffle in every row (852 cycles a block alone), take a
// fifth more instructions, and must be repeated whenever they change
// anything, where this must only when a diagonal did.
enum : unsigned { VD_DOWN = 1u, VD_UP = 2u, VD_ABOVE = 4u, VD_BELOW = 8u };
template <int DT, int CONN>
__device__ __forceinline__ unsigned vblock(uint32_t* tm, const uint32_t* tk, int lane, int b, uint32_t edge_mask,
                                           const EdgeSel& sel, bool conn8, unsigned due) {
    constexpr int N = VRow<DT>::N;
    uint32_t* rows = tm + (8 * b + 1) * 32 + lane;
    const uint32_t* krows = tk + (8 * b + 1) * 32 + lane;
    VRow<DT> above, below;
    above.set(rows[-32]);
    below.set(rows[8 * 32]);
    VRow<DT> m[8], k[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        m[i].set(rows[i * 32]);
        k[i].set(krows[i * 32]);
    }
    if (due & (VD_DOWN | VD_ABOVE)) {
        const VRow<DT> was = m[0];
        vstep<DT>(m[0], k[0], offers<DT, CONN>(above, sel, conn8));
        if (!(due & VD_DOWN) && __any_sync(FULL, m[0].differs(was))) due |= VD_DOWN;
    }
    if (due & (VD_UP | VD_BELOW)) {
        const VRow<DT> was = m[7];
        vstep<DT>(m[7], k[7], offers<DT, CONN>(below, sel, conn8));
        if (!(due & VD_UP) && __any_sync(FULL, m[7].differs(was))) due |= VD_UP;
    }
    if (!(due & (VD_DOWN | VD_UP))) return 0u;
    // A pixel that rose from the pixel above it cannot raise that one again,
    // so a walk leaves the other direction clean.
    if (due & VD_DOWN) {
#pragma unroll
        for (int i = 1; i < 8; ++i) vstep<DT>(m[i], k[i], m[i - 1]);
    }
    if (due & VD_UP) {
#pragma unroll
        for (int i = 6; i >= 0; --i) vstep<DT>(m[i], k[i], m[i + 1]);
    }
    uint32_t diag = 0u;
    if (eight<CONN>(conn8)) {
        VRow<DT> before, here = beside<DT>(m[0], sel);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            VRow<DT> after, q;
            if (i < 7) after = beside<DT>(m[i + 1], sel);
#pragma unroll
            for (int j = 0; j < N; ++j)
                q.v[j] = i == 0 ? after.v[j] : i == 7 ? before.v[j] : vmx<DT>(before.v[j], after.v[j]);
            const VRow<DT> was = m[i];
            vstep<DT>(m[i], k[i], q);
#pragma unroll
            for (int j = 0; j < N; ++j) diag |= was.v[j] ^ m[i].v[j];
            before = here;
            here = after;
        }
    }
    // (the rows as they were are read again: registers are short here)
    uint32_t inner = 0u;
#pragma unroll
    for (int i = 1; i < 7; ++i) inner |= m[i].word() ^ rows[i * 32];
    const uint32_t first = m[0].word() ^ rows[0], last = m[7].word() ^ rows[7 * 32];
    const uint32_t all = first | inner | last;
    if (!__any_sync(FULL, all != 0u)) return 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) rows[i * 32] = m[i].word();
    unsigned f = __any_sync(FULL, first != 0u) ? RF_FIRST : 0u;
    if (__any_sync(FULL, inner != 0u)) f |= RF_INNER;
    if (__any_sync(FULL, last != 0u)) f |= RF_LAST;
    if (__any_sync(FULL, (all & edge_mask) != 0u)) f |= RF_COL;
    if (eight<CONN>(conn8) && __any_sync(FULL, diag != 0u)) f |= RF_AGAIN;
    return f;
}

// Q pairs of rows scanned together in one direction, uint8 / uint16: pixel
// j of a pair's two rows shares one word as u16x2 (first row low), so every
// min / max, and each step of the clamp-map scan (A and B in a word each),
// serves two rows at once.  The algebra is hscan's, element-wise.
template <bool FWD, int Q, int N>
__device__ __forceinline__ void hscan_pairs(uint32_t (&m)[Q][N], const uint32_t (&k)[Q][N], const uint32_t (&cin)[Q],
                                            int lane) {
    const int first = FWD ? 0 : N - 1, last = FWD ? N - 1 : 0;
    const int edge_lane = FWD ? 0 : 31;
    bool need = false;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
#pragma unroll
        for (int s = 1; s < N; ++s) {
            const int j = FWD ? s : N - 1 - s;
            const int jp = FWD ? j - 1 : j + 1;
            m[q][j] = __vmaxu2(m[q][j], __vminu2(m[q][jp], k[q][j]));
        }
        uint32_t in_px = FWD ? __shfl_up_sync(FULL, m[q][last], 1) : __shfl_down_sync(FULL, m[q][last], 1);
        if (lane == edge_lane) in_px = cin[q];
        need |= __vcmpgtu2(__vminu2(in_px, k[q][first]), m[q][first]) != 0u;
    }
    if (!__any_sync(FULL, need)) return;
    uint32_t A[Q], B[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        A[q] = m[q][last];
        B[q] = k[q][0];
#pragma unroll
        for (int j = 1; j < N; ++j) B[q] = __vminu2(B[q], k[q][j]);
        if (lane == edge_lane) {
            A[q] = __vmaxu2(A[q], __vminu2(cin[q], B[q]));
            B[q] = 0u;  // the entry lane becomes a constant: nothing before it
        }
    }
#pragma unroll
    for (int d = 1; d < 32; d <<= 1)
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const uint32_t Ap = FWD ? __shfl_up_sync(FULL, A[q], d) : __shfl_down_sync(FULL, A[q], d);
            const uint32_t Bp = FWD ? __shfl_up_sync(FULL, B[q], d) : __shfl_down_sync(FULL, B[q], d);
            A[q] = __vmaxu2(__vminu2(Ap, B[q]), A[q]);
            B[q] = __vminu2(Bp, B[q]);
        }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        uint32_t c = FWD ? __shfl_up_sync(FULL, A[q], 1) : __shfl_down_sync(FULL, A[q], 1);
        if (lane == edge_lane) c = cin[q];
#pragma unroll
        for (int s = 0; s < N; ++s) {
            const int j = FWD ? s : N - 1 - s;
            c = __vminu2(c, k[q][j]);
            m[q][j] = __vmaxu2(m[q][j], c);
        }
    }
}

// Two row words (a: first row, b: second) as the pair words of hscan_pairs
// and back.  uint8: pixel j of both rows from the words' even / odd bytes;
// uint16: the words' low / high halves.
template <int DT>
__device__ __forceinline__ void pair_pack(uint32_t a, uint32_t b, uint32_t (&p)[Px<DT>::PPW]) {
    if constexpr (DT == DT_U8) {
        constexpr uint32_t E = 0x00ff00ffu;
        const uint32_t la = a & E, ha = (a >> 8) & E, lb = b & E, hb = (b >> 8) & E;
        p[0] = __byte_perm(la, lb, 0x5410);
        p[1] = __byte_perm(ha, hb, 0x5410);
        p[2] = __byte_perm(la, lb, 0x7632);
        p[3] = __byte_perm(ha, hb, 0x7632);
    } else {
        p[0] = __byte_perm(a, b, 0x5410);
        p[1] = __byte_perm(a, b, 0x7632);
    }
}
template <int DT>
__device__ __forceinline__ void pair_unpack(const uint32_t (&p)[Px<DT>::PPW], uint32_t& a, uint32_t& b) {
    if constexpr (DT == DT_U8) {
        const uint32_t t = __byte_perm(p[0], p[1], 0x6240), u = __byte_perm(p[2], p[3], 0x6240);
        a = __byte_perm(t, u, 0x5410);
        b = __byte_perm(t, u, 0x7632);
    } else {
        a = __byte_perm(p[0], p[1], 0x5410);
        b = __byte_perm(p[0], p[1], 0x7632);
    }
}

// Horizontal pass over block b: each row to its one-dimensional fixed point.
// Lane L holds 16 bytes (part L % 8) of two rows (pair L / 8 of the block): a
// row's closure is a forward and a backward chain in the lane (side by side,
// each from the row as it was: what a pixel gets comes from one side, so
// their maximum is the closure), then, if some lane's outermost pixel can
// raise its neighbour lane's, the lanes' clamp maps in both directions at
// once (three steps of two shuffles each) and one pass applying what enters
// each lane from either side.  A row spread over the 32 lanes, a word each,
// needs five scan steps and shares every shuffle among fewer pixels (about
// twice the instructions).  uint8, cycles of a block alone / of the SM with
// it busy: 738 / 148; chains one after the other 801 / 141; sixteen lanes of
// eight pixels 782 / 162.
// uint8 / uint16 hold pixel j of the two rows in one word as u16x2 (uint8
// bytes doubled, as in VRow); int32 the two rows in words of their own.
template <int DT>
struct HLane {
    static constexpr int N = 4 * Px<DT>::PPW;       // pixels of a row that a lane holds
    static constexpr int S = DT == DT_I32 ? 2 : 1;  // words per pixel of the row pair
    static constexpr uint32_t MINV = DT == DT_I32 ? 0x80000000u : 0u;
    __device__ static __forceinline__ uint32_t mx(uint32_t a, uint32_t b) {
        return DT == DT_I32 ? (uint32_t)max((int)a, (int)b) : __vmaxu2(a, b);
    }
    __device__ static __forceinline__ uint32_t mn(uint32_t a, uint32_t b) {
        return DT == DT_I32 ? (uint32_t)min((int)a, (int)b) : __vminu2(a, b);
    }
    __device__ static __forceinline__ uint32_t mx3(uint32_t a, uint32_t b, uint32_t c) {
        return DT == DT_I32 ? (uint32_t)__vimax3_s32((int)a, (int)b, (int)c) : __vimax3_u16x2(a, b, c);
    }
    __device__ static __forceinline__ uint32_t mn3(uint32_t a, uint32_t b, uint32_t c) {
        return DT == DT_I32 ? (uint32_t)__vimin3_s32((int)a, (int)b, (int)c) : __vimin3_u16x2(a, b, c);
    }
    __device__ static __forceinline__ bool any_gt(uint32_t a, uint32_t b) {
        return DT == DT_I32 ? (int)a > (int)b : __vmaxu2(a, b) != b;
    }
    __device__ static __forceinline__ void split(const uint4& ra, const uint4& rb, uint32_t (&v)[S][N]) {
        const uint32_t a[4] = {ra.x, ra.y, ra.z, ra.w}, b[4] = {rb.x, rb.y, rb.z, rb.w};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            if constexpr (DT == DT_U8) {
                v[0][4 * w] = __byte_perm(a[w], b[w], 0x4400);
                v[0][4 * w + 1] = __byte_perm(a[w], b[w], 0x5511);
                v[0][4 * w + 2] = __byte_perm(a[w], b[w], 0x6622);
                v[0][4 * w + 3] = __byte_perm(a[w], b[w], 0x7733);
            } else if constexpr (DT == DT_U16) {
                v[0][2 * w] = __byte_perm(a[w], b[w], 0x5410);
                v[0][2 * w + 1] = __byte_perm(a[w], b[w], 0x7632);
            } else {
                v[0][w] = a[w];
                v[1][w] = b[w];
            }
        }
    }
    __device__ static __forceinline__ void join(const uint32_t (&v)[S][N], uint4& ra, uint4& rb) {
        uint32_t a[4], b[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            if constexpr (DT == DT_U8) {
                const uint32_t t = __byte_perm(v[0][4 * w], v[0][4 * w + 1], 0x6240);
                const uint32_t u = __byte_perm(v[0][4 * w + 2], v[0][4 * w + 3], 0x6240);
                a[w] = __byte_perm(t, u, 0x5410);
                b[w] = __byte_perm(t, u, 0x7632);
            } else if constexpr (DT == DT_U16) {
                a[w] = __byte_perm(v[0][2 * w], v[0][2 * w + 1], 0x5410);
                b[w] = __byte_perm(v[0][2 * w], v[0][2 * w + 1], 0x7632);
            } else {
                a[w] = v[0][w];
                b[w] = v[1][w];
            }
        }
        ra = make_uint4(a[0], a[1], a[2], a[3]);
        rb = make_uint4(b[0], b[1], b[2], b[3]);
    }
};

template <int DT>
__device__ __forceinline__ unsigned hblock(uint32_t* tm, const uint32_t* tk, int lane, int b) {
    using P = Px<DT>;
    using H = HLane<DT>;
    constexpr int N = H::N, S = H::S;
    const int part = lane & 7, pair = lane >> 3;
    const int at = (8 * b + 2 * pair + 1) * 32 + part * 4;
    const uint4 oa = *reinterpret_cast<const uint4*>(&tm[at]);
    const uint4 ob = *reinterpret_cast<const uint4*>(&tm[at + 32]);
    uint32_t m[S][N], k[S][N];
    H::split(oa, ob, m);
    H::split(*reinterpret_cast<const uint4*>(&tk[at]), *reinterpret_cast<const uint4*>(&tk[at + 32]), k);
    // the lane's own closure, then whether an outermost pixel can raise the
    // pixel beside it in the next lane
    bool need = false;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        uint32_t bw[N];
        bw[N - 1] = m[s][N - 1];
#pragma unroll
        for (int j = N - 2; j >= 0; --j) bw[j] = H::mx(m[s][j], H::mn(bw[j + 1], k[s][j]));
#pragma unroll
        for (int j = 1; j < N; ++j) m[s][j] = H::mx(m[s][j], H::mn(m[s][j - 1], k[s][j]));
#pragma unroll
        for (int j = 0; j + 1 < N; ++j) m[s][j] = H::mx(m[s][j], bw[j]);
        uint32_t l = __shfl_up_sync(FULL, m[s][N - 1], 1, 8), r = __shfl_down_sync(FULL, m[s][0], 1, 8);
        if (part == 0) l = H::MINV;
        if (part == 7) r = H::MINV;
        need |= H::any_gt(H::mn(l, k[s][0]), m[s][0]) || H::any_gt(H::mn(r, k[s][N - 1]), m[s][N - 1]);
    }
    if (__any_sync(FULL, need)) {
#pragma unroll
        for (int s = 0; s < S; ++s) {
            // clamp maps (A, B) of the lane in either direction (see
            // map_step_packed): the closure's exit pixel, the least mask
            uint32_t Bf = k[s][0];
#pragma unroll
            for (int j = 1; j + 1 < N; j += 2) Bf = H::mn3(Bf, k[s][j], k[s][j + 1]);
            Bf = H::mn(Bf, k[s][N - 1]);
            uint32_t Af = m[s][N - 1], Ab = m[s][0], Bb = Bf;
#pragma unroll
            for (int d = 1; d < 8; d <<= 1) {
                const uint32_t af = __shfl_up_sync(FULL, Af, d, 8), bf = __shfl_up_sync(FULL, Bf, d, 8);
                const uint32_t ab = __shfl_down_sync(FULL, Ab, d, 8), bb = __shfl_down_sync(FULL, Bb, d, 8);
                Af = H::mx(H::mn(af, Bf), Af);
                Bf = H::mn(bf, Bf);
                Ab = H::mx(H::mn(ab, Bb), Ab);
                Bb = H::mn(bb, Bb);
            }
            uint32_t cf = __shfl_up_sync(FULL, Af, 1, 8), cb = __shfl_down_sync(FULL, Ab, 1, 8);
            if (part == 0) cf = H::MINV;
            if (part == 7) cb = H::MINV;
            // what enters from the left reaches pixel j through the masks up
            // to j, what enters from the right through those from j on
            uint32_t f[N];
#pragma unroll
            for (int j = 0; j < N; ++j) f[j] = cf = H::mn(cf, k[s][j]);
#pragma unroll
            for (int j = N - 1; j >= 0; --j) {
                cb = H::mn(cb, k[s][j]);
                m[s][j] = H::mx3(m[s][j], f[j], cb);
            }
        }
    }
    uint4 na, nb;
    H::join(m, na, nb);
    const uint32_t xa = (na.x ^ oa.x) | (na.y ^ oa.y) | (na.z ^ oa.z) | (na.w ^ oa.w);
    const uint32_t xb = (nb.x ^ ob.x) | (nb.y ^ ob.y) | (nb.z ^ ob.z) | (nb.w ^ ob.w);
    if (!__any_sync(FULL, (xa | xb) != 0u)) return 0u;
    *reinterpret_cast<uint4*>(&tm[at]) = na;
    *reinterpret_cast<uint4*>(&tm[at + 32]) = nb;
    const uint32_t xc = part == 0   ? ((na.x ^ oa.x) | (nb.x ^ ob.x)) & P::FIRST_MASK
                        : part == 7 ? ((na.w ^ oa.w) | (nb.w ^ ob.w)) & P::LAST_MASK
                                    : 0u;
    const unsigned va = __ballot_sync(FULL, xa != 0u), vb = __ballot_sync(FULL, xb != 0u);
    unsigned f = (va & 0xffu) ? RF_FIRST : 0u;
    if ((va & 0xffffff00u) | (vb & 0x00ffffffu)) f |= RF_INNER;
    if (vb & 0xff000000u) f |= RF_LAST;
    if (__any_sync(FULL, xc != 0u)) f |= RF_COL;
    return f;
}

// Raises the first and last pixel column of block b from the halo columns
// (for 8-connectivity their three neighbours there, corners included); lanes
// 0-7 the rows of the first column, lanes 8-15 of the last.  Returns RF_*.
template <int DT, int CONN, int TH>
__device__ __forceinline__ unsigned halo_columns(TileSmem<TH>& sm, int lane, int b, bool conn8) {
    using P = Px<DT>;
    const int r = 8 * b + 1 + (lane & 7);
    const bool right = (lane & 8) != 0;
    const uint32_t* h = right ? sm.hRm : sm.hLm;
    uint32_t v = h[r];
    if (eight<CONN>(conn8)) v = P::mx3(v, h[r - 1], h[r + 1]);
    const int off = right ? 128 - P::BPP : 0;
    unsigned char* px = reinterpret_cast<unsigned char*>(&sm.tm[r * 32]) + off;
    v = P::mn(v, P::ld_px(reinterpret_cast<const unsigned char*>(&sm.tk[r * 32]) + off));
    const bool rose = lane < 16 && P::gt(v, P::ld_px(px));
    __syncwarp();
    if (rose) P::st_px(px, v);
    const unsigned bal = __ballot_sync(FULL, rose);
    const unsigned rows = (bal | (bal >> 8)) & 0xffu;
    if (rows == 0u) return 0u;
    return ((rows & 1u) ? RF_FIRST : 0u) | ((rows & 0x7eu) ? RF_INNER : 0u) | ((rows & 0x80u) ? RF_LAST : 0u) | RF_COL;
}

// --------------------------------------------------------------- tile visit
template <int DT>
__device__ __forceinline__ uint32_t load_word_plain(const unsigned char* row, int npx, bool coherent) {
    using P = Px<DT>;
    if (npx >= P::PPW)
        return coherent ? __ldcg(reinterpret_cast<const unsigned int*>(row))
                        : __ldg(reinterpret_cast<const unsigned int*>(row));
    uint32_t p[P::PPW];
#pragma unroll
    for (int i = 0; i < P::PPW; ++i)
        p[i] = i < npx ? (coherent ? P::ld_px_cg(row + i * P::BPP) : P::ld_px(row + i * P::BPP)) : P::MINPX;
    return P::pack(p);
}

// Stores block b's rows from shared memory to the tile's own pixels
// (MR.cu:335-364; here plain stores: the visiting CTA owns the tile).  Where
// the rows lie on 16-byte boundaries and the tile inside the image's width,
// eight lanes store a row, four rows per instruction.
template <int DT, int TH>
__device__ __forceinline__ void write_back_block(const ImgDesc& d, const TileSmem<TH>& sm, int lane, int b, int x0,
                                                 int y0) {
    using P = Px<DT>;
    const bool wide = x0 + 32 * P::PPW <= d.W && ((reinterpret_cast<size_t>(d.marker) | (size_t)d.pitch_m) & 15u) == 0u;
    if (wide) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = 8 * b + 4 * h + (lane >> 3);
            if (y0 + r < d.H)
                __stcg(reinterpret_cast<uint4*>(d.marker + (size_t)(y0 + r) * d.pitch_m + (size_t)x0 * P::BPP +
                                                (lane & 7) * 16),
                       *reinterpret_cast<const uint4*>(&sm.tm[(r + 1) * 32 + (lane & 7) * 4]));
        }
        return;
    }
    const int px0 = x0 + lane * P::PPW, npx = d.W - px0;
    if (npx <= 0) return;
#pragma unroll 1
    for (int r = 8 * b; r < 8 * b + 8 && y0 + r < d.H; ++r) {
        unsigned char* mrow = d.marker + (size_t)(y0 + r) * d.pitch_m + (size_t)px0 * P::BPP;
        const uint32_t w = sm.tm[(r + 1) * 32 + lane];
        if (npx >= P::PPW) {
            __stcg(reinterpret_cast<unsigned int*>(mrow), w);
        } else {
            uint32_t p[P::PPW];
            P::unpack(w, p);
#pragma unroll
            for (int i = 0; i < P::PPW; ++i)
                if (i < npx) P::st_px(mrow + i * P::BPP, p[i]);
        }
    }
}

// Neighbour detection (MR.cu:366-512, pull form) for block b: the NB_* bits
// of the neighbour tiles holding a pixel q next to a pixel p of this block
// with marker[q] < min(marker[p], mask[q]), looking only at the sides that
// rose (f, RF_*).  The halo values in shared memory are the neighbours'
// pixels as fetched; they can only have risen since, so a stale halo gives at
// most an extra notification, never a missed one.
template <int DT, int CONN, int TH>
__device__ __forceinline__ unsigned detect_neighbours(const TileSmem<TH>& sm, int lane, int b, unsigned f,
                                                      bool conn8) {
    const EdgeSel sel(lane);
    using P = Px<DT>;
    constexpr int NB = TH / 8;
    unsigned nb = 0u;
    const bool n = b == 0 && (f & RF_FIRST), s = b == NB - 1 && (f & RF_LAST);
    if (n || s) {
        // a step of the vertical walk over the halo row (one of the two: a
        // tile has at least two blocks)
        const int row = n ? 1 : TH, halo = n ? 0 : TH + 1;
        VRow<DT> p, m, k;
        p.set(sm.tm[row * 32 + lane]);
        const uint32_t w = sm.tm[halo * 32 + lane];
        m.set(w);
        k.set(sm.tk[halo * 32 + lane]);
        vstep<DT>(m, k, offers<DT, CONN>(p, sel, conn8));
        if (__any_sync(FULL, m.word() != w)) nb |= n ? NB_N : NB_S;
    }
    if (f & RF_COL) {
        // lanes 0-9 / 16-25: the rows from the one before the block to the
        // one after it in the left / right halo column
        const int i = lane & 15, r = 8 * b + i;
        const bool right = (lane & 16) != 0;
        bool up = false;
        if (eight<CONN>(conn8) ? i < 10 : i >= 1 && i < 9) {
            const unsigned char* col = reinterpret_cast<const unsigned char*>(sm.tm) + (right ? 128 - P::BPP : 0);
            uint32_t v = P::MINPX;
            if (eight<CONN>(conn8)) {
                if (r > 1) v = P::mx(v, P::ld_px(col + (r - 1) * 128));
                if (r < TH) v = P::mx(v, P::ld_px(col + (r + 1) * 128));
            }
            if (r >= 1 && r <= TH) v = P::mx(v, P::ld_px(col + r * 128));
            v = P::mn(v, right ? sm.hRk[r] : sm.hLk[r]);
            up = P::gt(v, right ? sm.hRm[r] : sm.hLm[r]);
        }
        const unsigned bal = __ballot_sync(FULL, up);
        unsigned l = bal & 0xffffu, e = bal >> 16;
        if (b == 0) {  // the corner rows
            if (l & 1u) nb |= NB_NW;
            if (e & 1u) nb |= NB_NE;
            l &= ~1u;
            e &= ~1u;
        }
        if (b == NB - 1) {
            if (l & 0x200u) nb |= NB_SW;
            if (e & 0x200u) nb |= NB_SE;
            l &= ~0x200u;
            e &= ~0x200u;
        }
        if (l) nb |= NB_W;
        if (e) nb |= NB_E;
    }
    return nb;
}

// ------------------------------------------------------- pixel queue
// Third in-tile solver, for revisits: a FIFO of tile pixels in shared memory
// instead of whole-tile passes.  Seeds: the pixels of the tile's boundary
// ring whose constraint towards any neighbour (halo included) is violated;
// each is raised to what its neighbours allow and queued.  A round pops up to
// 32 pixels, one per lane; each raises its in-tile neighbours q to
// min(value, mask[q]) when that is higher (a compare-and-swap on the packed
// word, lanes may share a word) and newly raised pixels are queued, placed
// by ballot and population count.  Every update is a valid monotone step of
// the propagation rule (MR.cu:43-44) and the queue empties only when no
// queued pixel can raise a neighbour, so the tile ends at its fixed point.
// Returns false (the caller finishes the tile with passes over every row)
// when the FIFO would overflow or a bound is reached; what was raised stands.
// `rows_chg` (per lane) collects the rows that rose (bit r - 1), `col_now`
// whether the tile's first / last pixel column rose.
template <int DT>
__device__ __forceinline__ uint32_t pq_get(const uint32_t* words, int r, int c) {
    using P = Px<DT>;
    const uint32_t w = *(const volatile uint32_t*)&words[r * 32 + c / P::PPW];
    constexpr int B = 8 * P::BPP;
    return B == 32 ? w : (w >> (B * (c % P::PPW))) & ((1u << B) - 1u);
}

// Raises pixel (r, c) of `words` to v when v is higher; true when this lane
// raised it.  *fail is set when the compare-and-swap loop gives up.
template <int DT>
__device__ __forceinline__ bool pq_raise(uint32_t* words, int r, int c, uint32_t v, bool* fail) {
    using P = Px<DT>;
    uint32_t* w = &words[r * 32 + c / P::PPW];
    if constexpr (DT == DT_I32) {
        return atomicMax(reinterpret_cast<int*>(w), (int)v) < (int)v;
    } else {
        constexpr int B = 8 * P::BPP;
        const int sh = B * (c % P::PPW);
        const uint32_t msk = ((1u << B) - 1u) << sh;
        uint32_t old = *(volatile uint32_t*)w;
        for (int it = 0; it < 64; ++it) {
            if (((old & msk) >> sh) >= v) return false;
            const uint32_t got = atomicCAS(w, old, (old & ~msk) | (v << sh));
            if (got == old) return true;
            old = got;
        }
        *fail = true;
        return false;
    }
}

template <int DT, int CONN, int TH>
__device__ bool pq_solve(TileSmemPq<TH>& sm, int lane, unsigned long long& rows_chg, bool& col_now, unsigned& rounds) {
    using P = Px<DT>;
    constexpr int TW = 32 * P::PPW;
    int head = 0, tail = 0;  // warp-uniform
    bool fail = false;
    // value of any pixel of rows 0..TH+1, columns -1..TW (halo columns)
    auto val = [&](int r, int c) -> uint32_t {
        if (c < 0) return sm.hLm[r];
        if (c >= TW) return sm.hRm[r];
        return pq_get<DT>(sm.tm, r, c);
    };
    // queue the pixels of the lanes with `want` (warp-uniform call)
    auto enqueue = [&](bool want, int r, int c) {
        const unsigned b = __ballot_sync(FULL, want);
        const int n = __popc(b);
        if (n == 0) return;
        if (tail - head + n > kPqCap) {
            fail = true;
            return;
        }
        if (want) {
            const int rank = __popc(b & ((1u << lane) - 1u));
            sm.pq[(tail + rank) % kPqCap] = (unsigned short)(r * TW + c);
        }
        tail += n;
    };
    auto raised = [&](int r, int c) {
        rows_chg |= 1ull << (r - 1);
        if (c == 0 || c == TW - 1) col_now = true;
    };
    // seeds: the boundary ring (top and bottom rows, first and last columns)
    constexpr int RING = 2 * TW + 2 * TH;
    for (int i0 = 0; i0 < RING; i0 += 32) {
        const int i = i0 + lane;
        int r = 0, c = 0;
        bool on = i < RING;
        if (i < TW) { r = 1; c = i; }
        else if (i < 2 * TW) { r = TH; c = i - TW; }
        else if (i < 2 * TW + TH) { r = i - 2 * TW + 1; c = 0; }
        else { r = i - 2 * TW - TH + 1; c = TW - 1; }
        bool up = false;
        if (on) {
            const uint32_t k = pq_get<DT>(sm.tk, r, c);
            uint32_t best = P::mx(val(r - 1, c), val(r + 1, c));
            best = P::mx(best, P::mx(val(r, c - 1), val(r, c + 1)));
            if (CONN == 8) {
                best = P::mx(best, P::mx(val(r - 1, c - 1), val(r - 1, c + 1)));
                best = P::mx(best, P::mx(val(r + 1, c - 1), val(r + 1, c + 1)));
            }
            const uint32_t cand = P::mn(best, k);
            if (P::gt(cand, pq_get<DT>(sm.tm, r, c)) && pq_raise<DT>(sm.tm, r, c, cand, &fail)) {
                up = true;
                raised(r, c);
            }
        }
        enqueue(up, r, c);
        if (__any_sync(FULL, fail)) return false;
    }
    // rounds
    constexpr int DR[8] = {-1, 1, 0, 0, -1, -1, 1, 1};
    constexpr int DC[8] = {0, 0, -1, 1, -1, 1, -1, 1};
    while (head != tail) {
        if (++rounds > 4096u) return false;
        const int k = min(tail - head, 32);
        int r = 0, c = 0;
        uint32_t v = 0u;
        const bool mine = lane < k;
        if (mine) {
            const int p = sm.pq[(head + lane) % kPqCap];
            r = p / TW;
            c = p - r * TW;
            v = pq_get<DT>(sm.tm, r, c);
        }
        __syncwarp();
        head += k;
#pragma unroll
        for (int dir = 0; dir < CONN; ++dir) {
            const int rq = r + DR[dir], cq = c + DC[dir];
            bool up = false;
            if (mine && rq >= 1 && rq <= TH && cq >= 0 && cq < TW) {
                const uint32_t cand = P::mn(v, pq_get<DT>(sm.tk, rq, cq));
                if (P::gt(cand, pq_get<DT>(sm.tm, rq, cq)) && pq_raise<DT>(sm.tm, rq, cq, cand, &fail)) {
                    up = true;
                    raised(rq, cq);
                }
            }
            enqueue(up, rq, cq);
            if (__any_sync(FULL, fail)) return false;
        }
    }
    return true;
}

template <int W>
__device__ __forceinline__ void cta_sync() {
    if (W == 1)
        __syncwarp();
    else
        __syncthreads();
}

// Fetches tile (tx, ty) of image d with its one-pixel halo (MR.cu:232-312);
// called by all W warps of the CTA.  Where the image has tensor maps, the
// first thread issues one box of TH+2 rows x 128 bytes per plane (rows /
// columns outside the image arrive as zeros), else the warps copy the words
// asynchronously (all in flight at once, no registers; through registers in
// batches of eight rows the fetch took four times as long).  The halo columns
// are single pixels, a load per lane and block.  Returns false when the
// bounded wait for the boxes ran out.
template <int DT, int TH, int W>
__device__ __forceinline__ bool fetch_tile(const ImgDesc& d, int tx, int ty, TileSmem<TH>& sm, int warp, int lane,
                                           unsigned& phase, long long timeout_ns) {
    using P = Px<DT>;
    constexpr int TW = 32 * P::PPW, BPW = TH / 8 / W;  // blocks per warp
    const int x0 = tx * TW, y0 = ty * TH;
    const int W_ = d.W, H = d.H;
    const int px0 = x0 + lane * P::PPW;  // first pixel of this lane's word
    const int npx = W_ - px0;            // >= PPW: full word, (0, PPW): partial, <= 0: outside
    const int r0 = warp == 0 ? 0 : 8 * BPW * warp + 1, r1 = warp == W - 1 ? TH + 1 : 8 * BPW * (warp + 1);
    const bool tma = d.tmaps != nullptr;
    if (tma) {
        if (warp == 0 && lane == 0) {
            fence_proxy_async_smem();  // earlier generic accesses of tm / tk before the async writes
            fence_proxy_async_global();
            mbar_arrive_expect_tx(&sm.mbar, 2u * 128u * (TH + 2));
            const unsigned char* maps = static_cast<const unsigned char*>(d.tmaps);
            tma_load_2d(sm.tm, maps, x0 * P::BPP, y0 - 1, &sm.mbar);
            tma_load_2d(sm.tk, maps + 128, x0 * P::BPP, y0 - 1, &sm.mbar);
        }
        __syncwarp();
    } else {
        const size_t off = (size_t)(npx > 0 ? px0 : 0) * P::BPP;
#pragma unroll 4
        for (int r = r0; r <= r1; ++r) {
            const int y = y0 - 1 + r;
            const bool in_y = y >= 0 && y < H;
            const unsigned char* mrow = d.marker + (size_t)y * d.pitch_m + off;
            const unsigned char* krow = d.mask + (size_t)y * d.pitch_k + off;
            if (in_y && npx >= P::PPW) {
                cp_async_4(&sm.tm[r * 32 + lane], mrow);
                cp_async_4(&sm.tk[r * 32 + lane], krow);
            } else {
                uint32_t mw = P::MINW, kw = P::MINW;
                if (in_y && npx > 0) {
                    mw = load_word_plain<DT>(mrow, npx, true);
                    kw = load_word_plain<DT>(krow, npx, false);
                }
                sm.tm[r * 32 + lane] = mw;
                sm.tk[r * 32 + lane] = kw;
            }
        }
    }
    {
        // halo columns, in flight together with the rows: lanes 0-7 the left
        // marker pixels of a block, then the left mask, right marker, right
        // mask; the corner rows with the first and the last block
        const int j = lane & 7, which = lane >> 3;
        uint32_t* h = which == 0 ? sm.hLm : which == 1 ? sm.hLk : which == 2 ? sm.hRm : sm.hRk;
        const int x = which < 2 ? x0 - 1 : x0 + TW;
        const bool in_x = x >= 0 && x < W_;
        const unsigned char* plane = (which & 1) ? d.mask : d.marker;
        const long long pitch = (which & 1) ? d.pitch_k : d.pitch_m;
        auto halo = [&](int r) -> uint32_t {
            const int y = y0 - 1 + r;
            if (!in_x || y < 0 || y >= H) return P::MINPX;
            return P::ld_px_cg(plane + (size_t)y * pitch + (size_t)x * P::BPP);
        };
        uint32_t v[BPW], vc = 0u;
#pragma unroll
        for (int i = 0; i < BPW; ++i) v[i] = halo(8 * (BPW * warp + i) + 1 + j);
        const int corner = warp == 0 && j == 0 ? 0 : warp == W - 1 && j == 7 ? TH + 1 : -1;
        if (corner >= 0) vc = halo(corner);
#pragma unroll
        for (int i = 0; i < BPW; ++i) h[8 * (BPW * warp + i) + 1 + j] = v[i];
        if (corner >= 0) h[corner] = vc;
    }
    if (tma) {
        // bounded wait for the box loads
        const long long t0 = globaltimer_ns();
        unsigned spins = 0;
        bool ok = true;
        while (!mbar_try_wait(&sm.mbar, phase)) {
            if ((++spins & 1023u) == 0u && globaltimer_ns() - t0 > timeout_ns) {
                ok = false;
                break;
            }
        }
        phase ^= 1u;
        if (!__all_sync(FULL, ok)) return false;
        if (DT == DT_I32) {
            // zero fill is not the int32 minimum: rewrite what lies outside
            for (int r = r0; r <= r1; ++r) {
                const int y = y0 - 1 + r;
                if (npx <= 0 || y < 0 || y >= H) sm.tm[r * 32 + lane] = sm.tk[r * 32 + lane] = P::MINW;
            }
        }
    } else {
        cp_async_wait_all();
    }
    return true;
}

// What rose in a warp's blocks: masks by block, and the tile's first / last
// row.
struct Rose {
    unsigned rows = 0u, col = 0u;
    bool top = false, bottom = false;
};

// Local convergence (MR.cu:320-325) by the W warps of a CTA, each with the
// blocks next to one another.  Every round a warp goes over its blocks
// (downward, then upward, in turn), runs the vertical pass where a constraint
// may be violated and, if that raised something (or the side columns did),
// the horizontal pass; a block that rose is looked at again, as is the block
// beside a first or last row that rose.  The warps read the rows beside their
// blocks while their owners may be raising them: pixels only rise, so an old
// value is a valid one, and the owner marks the reader's block after the row,
// for the next round.  Rounds end when nothing is left to look at, at the
// tile's fixed point; the result does not depend on the order of updates.
// `sides` (NB_* bits) names the halo sides whose pixels are new since the
// tile last converged (all sides on a first visit).  Returns false when the
// rounds do not end (a defect, reported instead of a hang).
template <int DT, int CONN, int TH, int W, class SM>
__device__ __forceinline__ bool solve_tile(SM& sm, int warp, int lane, unsigned& row_steps, Rose& rose) {
    using P = Px<DT>;
    constexpr int BPW = TH / 8 / W;
    constexpr unsigned LASTB = 1u << (BPW - 1);
    const uint32_t edge_mask = lane == 0 ? P::FIRST_MASK : lane == 31 ? P::LAST_MASK : 0u;
    const EdgeSel sel(lane);
    const int b0 = BPW * warp;
    // by block: due for the downward / upward walk, the row above / below
    // rose, due for the horizontal pass
    unsigned dd = 0u, du = 0u, da = 0u, db = 0u, dh = 0u;
    unsigned marks = 0u;  // 1 the warp above, 2 the warp below is to look again
    const unsigned sides = sm.sides;
    const bool conn8 = sm.d.conn == 8;
    // takes over what a pass raised (f, RF_*) in the warp's block i
    auto took = [&](unsigned f, int i) {
        if (!(f & RF_ROWS)) return;
        rose.rows |= 1u << i;
        if (f & RF_COL) rose.col |= 1u << i;
        if (f & RF_FIRST) {
            if (i > 0)
                db |= 1u << (i - 1);
            else if (warp > 0)
                marks |= 1u;
            else
                rose.top = true;
        }
        if (f & RF_LAST) {
            if (i < BPW - 1)
                da |= 2u << i;
            else if (warp < W - 1)
                marks |= 2u;
            else
                rose.bottom = true;
        }
    };
    if (sides == 0xffu) {
        dd = du = dh = 2u * LASTB - 1u;
    } else {
        if (warp == 0 && (sides & (NB_N | NB_NW | NB_NE))) da |= 1u;
        if (warp == W - 1 && (sides & (NB_S | NB_SW | NB_SE))) db |= LASTB;
    }
    if (sides & ~(NB_N | NB_S)) {
#pragma unroll 1
        for (int i = 0; i < BPW; ++i) {
            const unsigned f = halo_columns<DT, CONN, TH>(sm, lane, b0 + i, conn8);
            if (f & RF_ROWS) {
                dd |= 1u << i;
                du |= 1u << i;
                dh |= 1u << i;
                took(f, i);
            }
        }
        __syncwarp();
    }
    bool up = false;
#pragma unroll 1
    for (unsigned round = 0;; ++round, up = !up) {
        if constexpr (W > 1) {
            if (round != 0u) {
                volatile unsigned* mine = sm.mark[round & 1u][warp];
                const unsigned above = mine[0], below = mine[1];
                __syncwarp();
                if (above) da |= 1u;
                if (below) db |= LASTB;
                if (lane == 0 && above) mine[0] = 0u;
                if (lane == 0 && below) mine[1] = 0u;
            }
        }
#pragma unroll 1
        for (int n = 0; n < BPW; ++n) {
            const int i = up ? BPW - 1 - n : n;
            const unsigned bit = 1u << i;
            if ((dd | du | da | db) & bit) {
                const unsigned due = ((dd & bit) ? VD_DOWN : 0u) | ((du & bit) ? VD_UP : 0u) |
                                     ((da & bit) ? VD_ABOVE : 0u) | ((db & bit) ? VD_BELOW : 0u);
                dd &= ~bit;
                du &= ~bit;
                da &= ~bit;
                db &= ~bit;
                const unsigned f = vblock<DT, CONN>(sm.tm, sm.tk, lane, b0 + i, edge_mask, sel, conn8, due);
                __syncwarp();
                row_steps += 8u;
                took(f, i);
                if (f & RF_ROWS) dh |= bit;
                if (f & RF_AGAIN) {
                    dd |= bit;
                    du |= bit;
                }
            }
            if (dh & bit) {
                dh &= ~bit;
                const unsigned f = hblock<DT>(sm.tm, sm.tk, lane, b0 + i);
                __syncwarp();
                row_steps += 8u;
                took(f, i);
                if (f & RF_ROWS) {
                    dd |= bit;
                    du |= bit;
                }
            }
        }
        bool more = (dd | du | da | db) != 0u;
        if constexpr (W > 1) {
            if (lane == 0 && marks != 0u) {
                __threadfence_block();  // the rows before the marks
                if (marks & 1u) *(volatile unsigned*)&sm.mark[(round & 1u) ^ 1u][warp - 1][1] = 1u;
                if (marks & 2u) *(volatile unsigned*)&sm.mark[(round & 1u) ^ 1u][warp + 1][0] = 1u;
            }
            more = __syncthreads_or(more || marks != 0u) != 0;
            marks = 0u;
        }
        if (!more || round > (1u << 20)) {
            if (warp == 0 && lane == 0) sm.count.sweeps += round + 1u;
            return !more;
        }
    }
}

// One visit of tile (tx, ty) by a CTA of W warps: fetch, local convergence,
// store of the blocks that rose, and the neighbour tiles to notify in sm.nb.
// Called by all warps; after it the stores are the first warp's to publish,
// which may then go on to the next tile.  Returns false when a bounded wait
// ran out.
// CONN 0, for batches that mix connectivities: it is looked up.  Such a batch
// runs all the code there is at once, a copy per pixel type and connectivity of
// 40 KB each, and with four of them (64 mixed images, uint8 and uint16) an issue
// waited 8.7 cycles for instructions; with one per type the batch takes 2.84 ms
// instead of 3.59, where a single image would lose 2 % to the looking up.
template <int DT, int CONN, int TH, int W>
__device__ __forceinline__ bool visit_tile(TileSmemPasses<TH, W>& sm, int warp, int lane, unsigned& phase,
                                           long long timeout_ns, unsigned& row_steps) {
    constexpr int BPW = TH / 8 / W;
    const bool clerk = warp == 0 && lane == 0;  // keeps the visit's clock
    if (clerk) sm.count.cycles[1] -= clock64();
    bool ok = fetch_tile<DT, TH, W>(sm.d, sm.tx, sm.ty, sm, warp, lane, phase, timeout_ns);
    if (W > 1) {
        if (__syncthreads_or(!ok)) return false;
    } else {
        __syncwarp();
        if (!ok) return false;
    }
    if (clerk) {
        const long long t = clock64();
        sm.count.cycles[1] += t;
        sm.count.cycles[2] -= t;
    }
    Rose rose;
    ok = solve_tile<DT, CONN, TH, W>(sm, warp, lane, row_steps, rose);
    if (clerk) {
        const long long t = clock64();
        sm.count.cycles[2] += t;
        sm.count.cycles[3] -= t;
    }
    if (rose.rows != 0u) {
        unsigned nb = NB_STORED;
#pragma unroll 1
        for (int i = 0; i < BPW; ++i) {
            if (!((rose.rows >> i) & 1u)) continue;
            write_back_block<DT, TH>(sm.d, sm, lane, BPW * warp + i, sm.tx * 32 * Px<DT>::PPW, sm.ty * TH);
        }
#pragma unroll 1
        for (int i = 0; i < BPW; ++i) {
            unsigned f = (rose.col >> i) & 1u ? RF_COL : 0u;
            if (i == 0 && rose.top) f |= RF_FIRST;
            if (i == BPW - 1 && rose.bottom) f |= RF_LAST;
            if (f != 0u) nb |= detect_neighbours<DT, CONN, TH>(sm, lane, BPW * warp + i, f, sm.d.conn == 8);
        }
        if (lane == 0) atomicOr(&sm.nb, nb);
    }
    fence_proxy_async_smem();
    cta_sync<W>();
    if (clerk) sm.count.cycles[3] += clock64();
    return ok;
}

// The visits with the alternative solvers, for callers that ask for them
// (iwpp_config.solver 1 and 3), by one warp.  All solvers are sequences of valid
// monotone updates that stop at the tile's fixed point, so they give the same
// bytes.

// What rose in a visit by one warp, or since it last published: rows (bit r - 1
// for SMEM row r), and a side column (per lane).
struct RoseAlt {
    unsigned long long rows = 0ull;
    bool col = false;
    bool published = false;  // some of it was published before
};

// Stores what rose and returns the NB_* bits of the neighbours that it raises.
// (A pixel is next to halo pixels that its own block's detection looks at.)
template <int DT, int CONN, int TH>
__device__ __forceinline__ unsigned publish_alt(const TileSmem<TH>& sm, int lane, const RoseAlt& rose) {
    const unsigned f_col = __any_sync(FULL, rose.col) ? RF_COL : 0u;
    unsigned nb = 0u;
#pragma unroll 1
    for (int b = 0; b < TH / 8; ++b) {
        const unsigned rb = (unsigned)(rose.rows >> (8 * b)) & 0xffu;
        if (rb == 0u) continue;
        write_back_block<DT, TH>(sm.d, sm, lane, b, sm.tx * 32 * Px<DT>::PPW, sm.ty * TH);
        nb |= detect_neighbours<DT, CONN, TH>(sm, lane, b,
                                              ((rb & 1u) ? RF_FIRST : 0u) | ((rb & 0x80u) ? RF_LAST : 0u) | f_col,
                                              CONN == 8);
    }
    return nb;
}

// Row sweeps, raster and anti-raster, until one after the first two changes
// nothing.  `early` can publish intermediate results: after a sweep that raised
// a boundary row or column, if early.want() says so (the async queue, while many
// warps wait for work), the rows risen so far are stored and the neighbours that
// they raise handed to early.flush() while the sweeps go on, which one warp
// takes long over; `rose` then holds what rose after the last flush.
template <int DT, int CONN, int TH, class Early>
__device__ __forceinline__ void solve_sweeps(TileSmem<TH>& sm, int lane, unsigned& row_steps, RoseAlt& rose,
                                             Early& early) {
    using P = Px<DT>;
    constexpr unsigned long long ALL = TH == 64 ? ~0ull : ((1ull << TH) - 1ull);
    constexpr unsigned long long TOP = 1ull, BOT = 1ull << (TH - 1);
    const uint32_t edge_mask = lane == 0 ? P::FIRST_MASK : lane == 31 ? P::LAST_MASK : 0u;
    const unsigned sides = sm.sides;
    // Rows whose halo inputs are new are processed by the first two sweeps:
    // the top row by the raster sweep (N, NW, NE), the bottom row by the
    // anti-raster sweep (S, SW, SE), every row when a side column that feeds
    // the sweep changed (W, and E through the up-right / down-right diagonals
    // for 8-connectivity; the reverse for the anti-raster sweep).  Other rows
    // are skipped while nothing they depend on has changed.
    const unsigned side_down = CONN == 8 ? (NB_W | NB_E) : NB_W;
    const unsigned side_up = CONN == 8 ? (NB_W | NB_E) : NB_E;
    const unsigned long long force_down = (sides & side_down) ? ALL : (sides & (NB_N | NB_NW | NB_NE)) ? TOP : 0ull;
    const unsigned long long force_up = (sides & side_up) ? ALL : (sides & (NB_S | NB_SW | NB_SE)) ? BOT : 0ull;
    unsigned long long chg_prev = 0ull;
    unsigned n = 0u;
    for (;; ++n) {
        unsigned long long dil = chg_prev | (chg_prev << 1) | (chg_prev >> 1);
        if (n == 0) dil |= force_down;
        if (n == 1) dil |= force_up;
        dil &= ALL;
        unsigned long long chg = 0ull;
        bool col_now = false;
        if (dil != 0ull) {
            if ((n & 1u) == 0u)
                sweep<DT, CONN, TH, true>(sm, lane, dil, chg, col_now, edge_mask, row_steps);
            else
                sweep<DT, CONN, TH, false>(sm, lane, dil, chg, col_now, edge_mask, row_steps);
        }
        rose.rows |= chg;
        rose.col |= col_now;
        chg_prev = chg;
        if (chg == 0ull && n >= 1u) break;
        if constexpr (Early::kEnabled) {
            if (((chg & (TOP | BOT)) != 0ull || __any_sync(FULL, col_now)) && early.want(lane)) {
                early.flush(publish_alt<DT, CONN, TH>(sm, lane, rose), lane);
                rose.rows = 0ull;
                rose.col = false;
                rose.published = true;
            }
        }
    }
    if (lane == 0) sm.count.sweeps += n + 1u;
}

// A revisit by the pixel queue; a first visit, or one that the queue cannot
// finish, by the passes.
template <int DT, int CONN, int TH>
__device__ __forceinline__ bool solve_pq(TileSmemPq<TH>& sm, int lane, unsigned& row_steps, RoseAlt& rose) {
    constexpr unsigned long long TOP = 1ull, BOT = 1ull << (TH - 1);
    if (sm.sides != 0xffu) {
        unsigned rounds = 0u;
        unsigned long long mine = 0ull;
        const bool solved = pq_solve<DT, CONN, TH>(sm, lane, mine, rose.col, rounds);
        __syncwarp();
        rose.rows = warp_or64(mine);
        row_steps += rounds;
        if (lane == 0) sm.count.sweeps += 1u;
        if (solved) return true;
        if (lane == 0) sm.sides = 0xffu;
        __syncwarp();
    }
    Rose r;
    const bool ok = solve_tile<DT, CONN, TH, 1>(sm, 0, lane, row_steps, r);
    for (int b = 0; b < TH / 8; ++b)
        if ((r.rows >> b) & 1u) rose.rows |= 0x7eull << (8 * b);  // (which of a block's inner rows does not matter)
    if (r.top) rose.rows |= TOP;
    if (r.bottom) rose.rows |= BOT;
    rose.col |= r.col != 0u;
    return ok;
}

// PQ: by the pixel queue, else by row sweeps.
template <int DT, int CONN, int TH, bool PQ, class SM, class Early>
__device__ __forceinline__ bool visit_tile_alt(SM& sm, int lane, unsigned& phase, long long timeout_ns,
                                               unsigned& row_steps, Early& early) {
    if (lane == 0) sm.count.cycles[1] -= clock64();
    bool ok = fetch_tile<DT, TH, 1>(sm.d, sm.tx, sm.ty, sm, 0, lane, phase, timeout_ns);
    __syncwarp();
    if (!ok) return false;
    if (lane == 0) {
        const long long t = clock64();
        sm.count.cycles[1] += t;
        sm.count.cycles[2] -= t;
    }
    RoseAlt rose;
    if constexpr (PQ)
        ok = solve_pq<DT, CONN, TH>(sm, lane, row_steps, rose);
    else
        solve_sweeps<DT, CONN, TH>(sm, lane, row_steps, rose, early);
    if (lane == 0) {
        const long long t = clock64();
        sm.count.cycles[2] += t;
        sm.count.cycles[3] -= t;
    }
    const unsigned nb = publish_alt<DT, CONN, TH>(sm, lane, rose);
    if (lane == 0) sm.nb = nb | (rose.rows != 0ull || rose.published ? (unsigned)NB_STORED : 0u);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) sm.count.cycles[3] += clock64();
    return ok;
}

}  // namespace iwpp
