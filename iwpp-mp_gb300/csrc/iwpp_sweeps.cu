// iwpp_sweeps.cu -- elementwise precondition clip and whole-image directional
// sweeps.
//
// clip:   the reference's clipImage (IWPP MP/src/MorphologicalReconstruction.cu:827-836),
//         marker = min(marker, mask), one 32-bit word per thread.
// sweeps: the reference's *PropagationEntireImage kernels (MR.cu:547-753)
//         and the iRec1D* alternatives (IWPP MP DQ/src/MorphologicalReconstruction.cu:817-1074),
//         rule m = max(m, min(prev, mask)) along one axis.
//   +X / -X: one warp per row, the whole row as one max-min scan (128-byte
//            chunks, carry from chunk to chunk), exact and coalesced.
//   +Y / -Y: 4-connected, one warp per column strip (or segment of one),
//            rows streamed through shared memory with cp.async far ahead;
//            8-connectivity also takes the two diagonal pixels of the
//            previous row inside a 128-byte strip, segments of rows first on
//            their own, then their entries.  The result is the walk's, row
//            by row, whatever the order.
#include <algorithm>

#include "iwpp_engine.cuh"

namespace iwpp {

template <int DT>
__device__ __forceinline__ void load_pair(const unsigned char* mrow, const unsigned char* krow, int npx,
                                          uint32_t& mw, uint32_t& kw) {
    mw = load_word_plain<DT>(mrow, npx, true);
    kw = load_word_plain<DT>(krow, npx, false);
}

template <int DT>
__device__ __forceinline__ void store_word_plain(unsigned char* mrow, int npx, uint32_t w) {
    using P = Px<DT>;
    if (npx >= P::PPW) {
        *reinterpret_cast<unsigned int*>(mrow) = w;
    } else {
        uint32_t p[P::PPW];
        P::unpack(w, p);
#pragma unroll
        for (int i = 0; i < P::PPW; ++i)
            if (i < npx) P::st_px(mrow + i * P::BPP, p[i]);
    }
}

// ------------------------------------------------------------------- clip
template <int DT>
__global__ void clip_kernel(ImgDesc d) {
    using P = Px<DT>;
    const int words = (d.W + P::PPW - 1) / P::PPW;
    const long long total = (long long)words * d.H;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int y = (int)(i / words), wi = (int)(i - (long long)y * words);
        const int px0 = wi * P::PPW, npx = d.W - px0;
        unsigned char* mrow = d.marker + (size_t)y * d.pitch_m + (size_t)px0 * P::BPP;
        const unsigned char* krow = d.mask + (size_t)y * d.pitch_k + (size_t)px0 * P::BPP;
        uint32_t mw, kw;
        load_pair<DT>(mrow, krow, npx, mw, kw);
        uint32_t m[P::PPW], k[P::PPW];
        P::unpack(mw, m);
        P::unpack(kw, k);
#pragma unroll
        for (int j = 0; j < P::PPW; ++j) m[j] = P::mn(m[j], k[j]);
        const uint32_t c = P::pack(m);
        if (c != mw) store_word_plain<DT>(mrow, npx, c);
    }
}

// ---------------------------------------------------------------- staging
// Copies the rows of up to 64 images at once (grid.y), a warp per piece of a
// row in turn.  The row is written as the aligned words inside it, each put
// together from the two aligned source words around it, and single bytes at
// the ends (at most three each), so that a row of any alignment costs what an
// aligned one does.  Bound by DRAM / L2 / link traffic: read and write each byte
// once.  Pieces, since a warp per row left a short wide image to a few warps,
// each with a few hundred bytes in flight (a clip of one row of 20
// million bytes 81 ms, 0.35 so).
struct StageList {
    StageCopy c[64];
};
constexpr int kStageWords = 256;  // words of a piece

// Pieces of a row of `bytes` bytes, whatever its alignment.
__host__ __device__ static long long stage_pieces(long long bytes) {
    return bytes <= 4ll * kStageWords ? 1 : (bytes / 4 + kStageWords - 1) / kStageWords;
}

// PIECES: rows of more than one.
template <bool PIECES>
__device__ __forceinline__ void stage_copy(const StageCopy& c, int lane, long long pieces) {
    const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long u = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5); u < c.rows * pieces;
         u += nwarps) {
        const long long y = PIECES ? u / pieces : u, piece = PIECES ? u - y * pieces : 0;
        const unsigned char* src = static_cast<const unsigned char*>(c.src) + y * c.src_pitch;
        unsigned char* dst = static_cast<unsigned char*>(c.dst) + y * c.dst_pitch;
        const long long n = c.row_bytes;
        const long long lead = min((long long)((0u - (unsigned)reinterpret_cast<size_t>(dst)) & 3u), n);
        const long long words = (n - lead) >> 2, tail = lead + 4 * words;
        const long long end = PIECES ? min(words, (piece + 1) * kStageWords) : words;
        const unsigned char* from = src + lead;  // source of the first aligned word of dst
        const unsigned sh = (unsigned)reinterpret_cast<size_t>(from) & 3u;
        const unsigned* ws = reinterpret_cast<const unsigned*>(from - sh);
        unsigned* wd = reinterpret_cast<unsigned*>(dst + lead);
        if (sh == 0u) {
#pragma unroll 4
            for (long long i = piece * kStageWords + lane; i < end; i += 32) wd[i] = ws[i];
        } else {
            // the source words around the row's first and last bytes hold
            // bytes of other rows or of nothing: those words byte by byte
#pragma unroll 4
            for (long long i = piece * kStageWords + lane; i < end; i += 32) {
                unsigned w;
                if (i > 0 && i + 1 < words) {
                    w = __funnelshift_r(ws[i], ws[i + 1], 8 * sh);
                } else {
                    const unsigned char* b = from + 4 * i;
                    w = (unsigned)b[0] | (unsigned)b[1] << 8 | (unsigned)b[2] << 16 | (unsigned)b[3] << 24;
                }
                wd[i] = w;
            }
        }
        if (PIECES && piece != 0) continue;
        if (lane < 3 && lane < lead) dst[lane] = src[lane];
        if (lane >= 4 && tail + lane - 4 < n) dst[tail + lane - 4] = src[tail + lane - 4];
    }
}

__global__ void __launch_bounds__(256) stage_copy_kernel(const __grid_constant__ StageList list) {
    const StageCopy& c = list.c[blockIdx.y];
    const int lane = threadIdx.x & 31;
    const long long pieces = stage_pieces(c.row_bytes);
    if (pieces == 1)
        stage_copy<false>(c, lane, 1);
    else
        stage_copy<true>(c, lane, pieces);
}

cudaError_t launch_stage_copies(const std::vector<StageCopy>& copies, cudaStream_t s, int* launches) {
    for (size_t i = 0; i < copies.size(); i += 64) {
        StageList list{};
        const size_t n = copies.size() - i < 64 ? copies.size() - i : 64;
        long long units = 1;
        for (size_t j = 0; j < n; ++j) {
            list.c[j] = copies[i + j];
            units = std::max(units, copies[i + j].rows * stage_pieces(copies[i + j].row_bytes));
        }
        // eight pieces per block; at most four waves of blocks, which share the
        // largest image
        const long long want = (units + 7) / 8, most = kSms * 32 / (long long)n + 1;
        stage_copy_kernel<<<dim3((unsigned)(want < most ? want : most), (unsigned)n), 256, 0, s>>>(list);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        if (launches) ++*launches;
    }
    return cudaSuccess;
}

// ------------------------------------------------------ fixed-point check
// Counts the pixels c that a neighbour p could still raise:
// min(m[p], mask[c]) > m[c].  Zero on every reconstruction (it is a fixed
// point of the propagation rule, MR.cu:43-44); a size-independent check for
// images too large for a CPU comparison.
template <int DT>
__global__ void fixed_point_kernel(ImgDesc d, unsigned long long* count) {
    using P = Px<DT>;
    const long long total = (long long)d.W * d.H;
    unsigned long long mine = 0ull;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int y = (int)(i / d.W), x = (int)(i - (long long)y * d.W);
        const unsigned char* mrow = d.marker + (size_t)y * d.pitch_m;
        const uint32_t m = P::ld_px(mrow + (size_t)x * P::BPP);
        const uint32_t k = P::ld_px(d.mask + (size_t)y * d.pitch_k + (size_t)x * P::BPP);
        if (!P::gt(k, m)) continue;  // m == mask[c] (or above it): nothing can raise it
        uint32_t best = P::MINPX;
        for (int dy = -1; dy <= 1; ++dy) {
            const int yy = y + dy;
            if (yy < 0 || yy >= d.H) continue;
            const unsigned char* row = d.marker + (size_t)yy * d.pitch_m;
            for (int dx = -1; dx <= 1; ++dx) {
                const int xx = x + dx;
                if ((dx == 0 && dy == 0) || xx < 0 || xx >= d.W) continue;
                if (d.conn == 4 && dx != 0 && dy != 0) continue;
                best = P::mx(best, P::ld_px(row + (size_t)xx * P::BPP));
            }
        }
        if (P::gt(P::mn(best, k), m)) ++mine;
    }
    const unsigned long long warp_sum = __reduce_add_sync(0xffffffffu, (unsigned)mine);
    if ((threadIdx.x & 31) == 0 && warp_sum) atomicAdd(count, warp_sum);
}

// --------------------------------------------------------------- X sweeps
// Chunks a warp keeps in flight ahead of the one it scans: the row's loads
// do not depend on the carry, so they are issued kXAhead chunks early into a
// register ring (the walk is otherwise one global-memory latency per chunk).
// A chunk is loaded before any store of this warp to it, and no other warp
// touches the row, so no load reads a value this sweep has replaced.
// Measured on 16384^2 rows: 2 ahead takes 14-24 % off a uint8 / uint16
// sweep and 5 % off int32; 4 or 8 ahead gain less (int32: lose).
constexpr int kXAhead = 2;

template <int DT, bool FWD>
__global__ void sweep_x_kernel(ImgDesc d) {
    if (gated_off(d)) return;
    using P = Px<DT>;
    constexpr int TW = 32 * P::PPW;
    const int lane = threadIdx.x & 31;
    const int row = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (row >= d.H) return;
    const int chunks = (d.W + TW - 1) / TW;
    unsigned char* mbase = d.marker + (size_t)row * d.pitch_m;
    const unsigned char* kbase = d.mask + (size_t)row * d.pitch_k;
    // chunk cc in walk order: its first pixel for this lane and how many of
    // the lane's pixels lie inside the row
    auto px0_of = [&](int cc) { return (FWD ? cc : chunks - 1 - cc) * TW + lane * P::PPW; };
    auto fetch = [&](int cc, uint32_t& mw, uint32_t& kw) {
        mw = P::MINW;
        kw = P::MINW;
        if (cc >= chunks) return;
        const int px0 = px0_of(cc), npx = d.W - px0;
        if (npx > 0) load_pair<DT>(mbase + (size_t)px0 * P::BPP, kbase + (size_t)px0 * P::BPP, npx, mw, kw);
    };
    uint32_t mq[kXAhead], kq[kXAhead];
#pragma unroll
    for (int q = 0; q < kXAhead; ++q) fetch(q, mq[q], kq[q]);
    uint32_t carry = P::MINPX;
    for (int c0 = 0; c0 < chunks; c0 += kXAhead) {
#pragma unroll
        for (int q = 0; q < kXAhead; ++q) {
            const int cc = c0 + q;
            if (cc >= chunks) break;  // warp-uniform
            const uint32_t mw = mq[q], kw = kq[q];
            fetch(cc + kXAhead, mq[q], kq[q]);
            uint32_t m[P::PPW], k[P::PPW];
            P::unpack(mw, m);
            P::unpack(kw, k);
            hscan<DT, FWD>(m, k, carry, lane);
            const uint32_t nw = P::pack(m);
            const int px0 = px0_of(cc), npx = d.W - px0;
            if (npx > 0 && nw != mw) store_word_plain<DT>(mbase + (size_t)px0 * P::BPP, npx, nw);
            carry = FWD ? __shfl_sync(FULL, m[P::PPW - 1], 31) : __shfl_sync(FULL, m[0], 0);
        }
    }
}

// The same sweep with 16-byte lanes (a warp chunk is 512 bytes): the lane's
// four words are scanned in registers and the warp's clamp-map composition
// runs once per 16 bytes instead of once per 4, which is what the 4-byte form
// spends its issue slots on.  Rows must start on 16-byte boundaries (base
// and pitch of both planes); the row's last partial lane is loaded and
// stored word by word.
template <int DT, bool FWD>
__global__ void sweep_x16_kernel(ImgDesc d) {
    if (gated_off(d)) return;
    using P = Px<DT>;
    constexpr int WPL = 4;             // words per lane
    constexpr int N = WPL * P::PPW;    // pixels per lane
    constexpr int CW = 32 * N;         // pixels per chunk
    const int lane = threadIdx.x & 31;
    const int row = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (row >= d.H) return;
    const int chunks = (d.W + CW - 1) / CW;
    unsigned char* mbase = d.marker + (size_t)row * d.pitch_m;
    const unsigned char* kbase = d.mask + (size_t)row * d.pitch_k;
    auto px0_of = [&](int cc) { return (FWD ? cc : chunks - 1 - cc) * CW + lane * N; };
    auto fetch = [&](int cc, uint4& mv, uint4& kv) {
        mv = make_uint4(P::MINW, P::MINW, P::MINW, P::MINW);
        kv = mv;
        if (cc >= chunks) return;
        const int px0 = px0_of(cc), npx = d.W - px0;
        if (npx >= N) {
            mv = __ldcg(reinterpret_cast<const uint4*>(mbase + (size_t)px0 * P::BPP));
            kv = __ldg(reinterpret_cast<const uint4*>(kbase + (size_t)px0 * P::BPP));
        } else if (npx > 0) {
            uint32_t mw[WPL], kw[WPL];
#pragma unroll
            for (int w = 0; w < WPL; ++w) {
                const int n = npx - w * P::PPW;
                mw[w] = P::MINW;
                kw[w] = P::MINW;
                if (n > 0)
                    load_pair<DT>(mbase + (size_t)(px0 + w * P::PPW) * P::BPP,
                                  kbase + (size_t)(px0 + w * P::PPW) * P::BPP, n, mw[w], kw[w]);
            }
            mv = make_uint4(mw[0], mw[1], mw[2], mw[3]);
            kv = make_uint4(kw[0], kw[1], kw[2], kw[3]);
        }
    };
    uint4 mq[kXAhead], kq[kXAhead];
#pragma unroll
    for (int q = 0; q < kXAhead; ++q) fetch(q, mq[q], kq[q]);
    uint32_t carry = P::MINPX;
    for (int c0 = 0; c0 < chunks; c0 += kXAhead) {
#pragma unroll
        for (int q = 0; q < kXAhead; ++q) {
            const int cc = c0 + q;
            if (cc >= chunks) break;  // warp-uniform
            const uint4 mv = mq[q], kv = kq[q];
            fetch(cc + kXAhead, mq[q], kq[q]);
            const uint32_t mw[WPL] = {mv.x, mv.y, mv.z, mv.w}, kw[WPL] = {kv.x, kv.y, kv.z, kv.w};
            uint32_t m[N], k[N];
#pragma unroll
            for (int w = 0; w < WPL; ++w) {
                uint32_t a[P::PPW], b[P::PPW];
                P::unpack(mw[w], a);
                P::unpack(kw[w], b);
#pragma unroll
                for (int j = 0; j < P::PPW; ++j) {
                    m[w * P::PPW + j] = a[j];
                    k[w * P::PPW + j] = b[j];
                }
            }
            hscan<DT, FWD, N>(m, k, carry, lane);
            uint32_t nw[WPL];
            bool chg = false;
#pragma unroll
            for (int w = 0; w < WPL; ++w) {
                uint32_t a[P::PPW];
#pragma unroll
                for (int j = 0; j < P::PPW; ++j) a[j] = m[w * P::PPW + j];
                nw[w] = P::pack(a);
                chg |= nw[w] != mw[w];
            }
            const int px0 = px0_of(cc), npx = d.W - px0;
            if (chg && npx > 0) {
                unsigned char* dst = mbase + (size_t)px0 * P::BPP;
                if (npx >= N) {
                    *reinterpret_cast<uint4*>(dst) = make_uint4(nw[0], nw[1], nw[2], nw[3]);
                } else {
#pragma unroll
                    for (int w = 0; w < WPL; ++w)
                        if (npx - w * P::PPW > 0) store_word_plain<DT>(dst + w * 4, npx - w * P::PPW, nw[w]);
                }
            }
            carry = FWD ? __shfl_sync(FULL, m[N - 1], 31) : __shfl_sync(FULL, m[0], 0);
        }
    }
}

// The same sweep over two rows per warp (uint8; the pairing also holds for
// uint16).  Pixel j of a lane's 16 bytes in both rows shares one word as
// u16x2 (first row low), so the in-lane scan, the carry vote and the
// clamp-map scan (hscan_pairs) run once for the two rows: about half the
// issue slots of two sweep_x16_kernel rows.  An odd image's last warp has no
// second row: it reads as the minimum and is not stored.
template <int DT, bool FWD>
__global__ void sweep_x16p_kernel(ImgDesc d) {
    if (gated_off(d)) return;
    using P = Px<DT>;
    static_assert(DT != DT_I32, "int32 rows are not paired");
    constexpr int WPL = 4;             // words per lane
    constexpr int N = WPL * P::PPW;    // pixels per lane (and pair words)
    constexpr int CW = 32 * N;         // pixels per chunk
    const int lane = threadIdx.x & 31;
    const int ra = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 2, rb = ra + 1;
    if (ra >= d.H) return;
    const bool has_b = rb < d.H;
    const int chunks = (d.W + CW - 1) / CW;
    unsigned char* ma = d.marker + (size_t)ra * d.pitch_m;
    const unsigned char* ka = d.mask + (size_t)ra * d.pitch_k;
    unsigned char* mb = has_b ? ma + d.pitch_m : ma;
    const unsigned char* kb = has_b ? ka + d.pitch_k : ka;
    auto px0_of = [&](int cc) { return (FWD ? cc : chunks - 1 - cc) * CW + lane * N; };
    auto fetch_row = [&](const unsigned char* mrow, const unsigned char* krow, bool live, int cc, uint4& mv,
                         uint4& kv) {
        mv = make_uint4(P::MINW, P::MINW, P::MINW, P::MINW);
        kv = mv;
        if (cc >= chunks || !live) return;
        const int px0 = px0_of(cc), npx = d.W - px0;
        if (npx >= N) {
            mv = __ldcg(reinterpret_cast<const uint4*>(mrow + (size_t)px0 * P::BPP));
            kv = __ldg(reinterpret_cast<const uint4*>(krow + (size_t)px0 * P::BPP));
        } else if (npx > 0) {
            uint32_t mw[WPL], kw[WPL];
#pragma unroll
            for (int w = 0; w < WPL; ++w) {
                const int n = npx - w * P::PPW;
                mw[w] = P::MINW;
                kw[w] = P::MINW;
                if (n > 0)
                    load_pair<DT>(mrow + (size_t)(px0 + w * P::PPW) * P::BPP,
                                  krow + (size_t)(px0 + w * P::PPW) * P::BPP, n, mw[w], kw[w]);
            }
            mv = make_uint4(mw[0], mw[1], mw[2], mw[3]);
            kv = make_uint4(kw[0], kw[1], kw[2], kw[3]);
        }
    };
    auto store_row = [&](unsigned char* mrow, int cc, const uint32_t (&nw)[WPL]) {
        const int px0 = px0_of(cc), npx = d.W - px0;
        if (npx <= 0) return;
        unsigned char* dst = mrow + (size_t)px0 * P::BPP;
        if (npx >= N) {
            *reinterpret_cast<uint4*>(dst) = make_uint4(nw[0], nw[1], nw[2], nw[3]);
        } else {
#pragma unroll
            for (int w = 0; w < WPL; ++w)
                if (npx - w * P::PPW > 0) store_word_plain<DT>(dst + w * 4, npx - w * P::PPW, nw[w]);
        }
    };
    uint4 maq[kXAhead], kaq[kXAhead], mbq[kXAhead], kbq[kXAhead];
#pragma unroll
    for (int q = 0; q < kXAhead; ++q) {
        fetch_row(ma, ka, true, q, maq[q], kaq[q]);
        fetch_row(mb, kb, has_b, q, mbq[q], kbq[q]);
    }
    uint32_t carry[1] = {0u};  // both rows' entry pixel: the minimum
    for (int c0 = 0; c0 < chunks; c0 += kXAhead) {
#pragma unroll
        for (int q = 0; q < kXAhead; ++q) {
            const int cc = c0 + q;
            if (cc >= chunks) break;  // warp-uniform
            const uint4 mav = maq[q], kav = kaq[q], mbv = mbq[q], kbv = kbq[q];
            fetch_row(ma, ka, true, cc + kXAhead, maq[q], kaq[q]);
            fetch_row(mb, kb, has_b, cc + kXAhead, mbq[q], kbq[q]);
            const uint32_t wa[WPL] = {mav.x, mav.y, mav.z, mav.w}, wb[WPL] = {mbv.x, mbv.y, mbv.z, mbv.w};
            const uint32_t va[WPL] = {kav.x, kav.y, kav.z, kav.w}, vb[WPL] = {kbv.x, kbv.y, kbv.z, kbv.w};
            uint32_t m[1][N], k[1][N];
#pragma unroll
            for (int w = 0; w < WPL; ++w) {
                uint32_t pm[P::PPW], pk[P::PPW];
                pair_pack<DT>(wa[w], wb[w], pm);
                pair_pack<DT>(va[w], vb[w], pk);
#pragma unroll
                for (int j = 0; j < P::PPW; ++j) {
                    m[0][w * P::PPW + j] = pm[j];
                    k[0][w * P::PPW + j] = pk[j];
                }
            }
            hscan_pairs<FWD, 1, N>(m, k, carry, lane);
            uint32_t na[WPL], nb[WPL];
            bool chg_a = false, chg_b = false;
#pragma unroll
            for (int w = 0; w < WPL; ++w) {
                uint32_t pm[P::PPW];
#pragma unroll
                for (int j = 0; j < P::PPW; ++j) pm[j] = m[0][w * P::PPW + j];
                pair_unpack<DT>(pm, na[w], nb[w]);
                chg_a |= na[w] != wa[w];
                chg_b |= nb[w] != wb[w];
            }
            if (chg_a) store_row(ma, cc, na);
            if (chg_b && has_b) store_row(mb, cc, nb);
            carry[0] = FWD ? __shfl_sync(FULL, m[0][N - 1], 31) : __shfl_sync(FULL, m[0][0], 0);
        }
    }
}

// --------------------------------------------------------------- Y sweeps
// 16-byte asynchronous global -> shared copy (cp.async, LDGSTS) and its group
// bookkeeping.
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The 4-connected sweeps stream rows through a ring in shared memory, kRing
// rows of a plane ahead, in cp.async groups of kGroup rows.
constexpr int kRing = 64, kGroup = 8;

// Vertical sweeps by strips (8-connected ones, and 4-connected ones of rows
// that the ring kernels below do not stream).  A 128-byte column strip is
// closed: its rows take the three pixels (4-connected: one) of the row before
// them inside the strip (a lane holds a word).  Row by row that is a chain of
// 50 cycles a row and more, and with the diagonals a run of rows is no
// per-column map that could be composed; one warp walking a strip's whole
// height took 500 us for 4096 rows whatever the width.  But the sweep is the
// least solution of "each row at least what the row before it offers", so the
// rows can be taken in any order that ends with no row left to raise:
//   sweep_strip_local_kernel: segments of kStripRows rows, a warp each, as if
//     nothing entered them;
//   sweep_strip_enter_kernel, kStripEnter times: a warp per segment, what the
//     row before the segment offers, on from there while the rows rise; the
//     row before it may itself be rising meanwhile;
//   sweep_strip_settle_kernel: a warp per strip, the segments in order, any entry
//     that still raises something, on from there while the rows rise.
// Same bytes as the walk.  Measured on 4096^2 uint8 h-domes (+Y / -Y, us): the
// walk 496 / 516; segments of 64 rows with 1 / 2 / 4 / 8 enter steps 144 / 81 /
// 70 / 87, of 128 rows 70 / 60 / 66 / 83, of 32 rows 304 / 203 / 111 / 105.
// Bound by the chain, about 70 cycles a row of one warp, where a front runs down
// many segments (the settle step's walk: rows far ahead in shared memory, the
// last strip's partial words masked and not loaded pixel by pixel).  With a
// group of rows ahead in registers and the last strip's pixels one by one, and
// now, us: 16384^2 uint8 spiral 8-connected 1931 / 838, 8191 x 8190 uint16
// spiral 4-connected (staged) 4734 / 1392, 8190 x 8192 int32 spiral 8-connected
// 1008 / 428, 1028 x 8192 uint8, one front down the whole height, 1346 / 567.
constexpr int kStripRows = 128;
constexpr int kStripEnter = 2;
// images up to this height: one walk, whose launch is all it costs (1024 x 182
// uint16 12 us; in segments 29 and three more launches)
constexpr int kStripWhole = 384;
constexpr int kStripThreads = 128;

// A lane's word column of a strip, rows by their index in sweep order.
template <int DT, int CONN, bool DOWN>
struct Strip {
    using P = Px<DT>;
    unsigned char* m;
    const unsigned char* k;
    long long pitch_m, pitch_k;
    int npx, H;
    uint32_t keep;  // the bits of the lane's word that are the image's
    __device__ __forceinline__ Strip(const ImgDesc& d, int strip, int lane) : H(d.H) {
        const int px0 = strip * 32 * P::PPW + lane * P::PPW;
        npx = d.W - px0;
        keep = npx >= P::PPW ? FULL : npx > 0 ? (1u << (8 * P::BPP * npx)) - 1u : 0u;
        const size_t off = (size_t)(npx > 0 ? px0 : 0) * P::BPP;
        const int first = DOWN ? 0 : d.H - 1;
        pitch_m = DOWN ? d.pitch_m : -d.pitch_m;
        pitch_k = DOWN ? d.pitch_k : -d.pitch_k;
        m = d.marker + (size_t)first * d.pitch_m + off;
        k = d.mask + (size_t)first * d.pitch_k + off;
    }
    __device__ __forceinline__ uint32_t marker(int i) const {
        return i < H && npx > 0 ? load_word_plain<DT>(m + i * pitch_m, npx, true) : P::MINW;
    }
    __device__ __forceinline__ uint32_t mask(int i) const {
        return i < H && npx > 0 ? load_word_plain<DT>(k + i * pitch_k, npx, false) : P::MINW;
    }
    __device__ __forceinline__ void store(int i, uint32_t w) const {
        if (npx > 0) store_word_plain<DT>(m + i * pitch_m, npx, w);
    }
    // The word of a row, in every row but the image's last where the strip is
    // not inside the image's width (INSIDE): there a lane has a word, a part of
    // one or nothing, and loads a whole word all the same (with what lies
    // between the row's end and the next row, or its row's first word).
    __device__ __forceinline__ uint32_t word_at(const unsigned char* row) const {
        return __ldcg(reinterpret_cast<const unsigned int*>(row));
    }
    // What of it is the image's.
    template <bool INSIDE>
    __device__ __forceinline__ uint32_t own(uint32_t w) const {
        if (INSIDE) return w;
        return DT == DT_I32 ? (npx > 0 ? w : P::MINW) : w & keep;
    }
    // Row i below row i - 1 (in `prev`); true when it rises.
    __device__ __forceinline__ bool step(VRow<DT>& prev, int i, const EdgeSel& sel) const {
        const uint32_t was = marker(i);
        VRow<DT> v, kv;
        v.set(was);
        kv.set(mask(i));
        vstep<DT>(v, kv, offers<DT, CONN>(prev, sel));
        const uint32_t w = v.word();
        if (w != was) store(i, w);
        prev = v;
        return __any_sync(FULL, w != was);
    }
    // Eight rows from row i (marker words `old`, at `at`, mask words `kw`);
    // whether the lane's word of the last one rises.  Stores after the chain: a
    // branch for them in every row of the last strip cost as much as the row.
    template <bool INSIDE>
    __device__ __forceinline__ bool group(VRow<DT>& prev, const uint32_t (&old)[8], const uint32_t (&kw)[8], int i,
                                          unsigned char* at, const EdgeSel& sel) const {
        uint32_t out[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            VRow<DT> v, kv;
            v.set(own<INSIDE>(old[q]));
            kv.set(own<INSIDE>(kw[q]));
            vstep<DT>(v, kv, offers<DT, CONN>(prev, sel));
            out[q] = v.word();
            prev = v;
        }
        uint32_t rose = 0u;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const bool r = out[q] != own<INSIDE>(old[q]);
            rose |= r ? 1u << q : 0u;
            if ((INSIDE || npx >= P::PPW) && r) *reinterpret_cast<unsigned int*>(at + q * pitch_m) = out[q];
        }
        if (!INSIDE && DT != DT_I32 && npx < P::PPW && rose != 0u) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if ((rose >> q) & 1u) store(i + q, out[q]);
        }
        return (rose & 128u) != 0u;
    }
    // The first row of a walk's groups of eight and the end of them: the image's
    // last row is stepped by itself in the last strip.  False: the walk is over.
    template <bool STOP, bool INSIDE>
    __device__ __forceinline__ bool groups(VRow<DT>& prev, int& i, int end, int& groups_end, const EdgeSel& sel) const {
        groups_end = end;
        if (!INSIDE) {
            if (DOWN)
                groups_end = min(end, H - 1);
            else if (i == 0)
                return step(prev, i++, sel) || !STOP;
        }
        return true;
    }
    // Walks rows from `i` below row i - 1 (in `prev`); with STOP until a group
    // of eight ends with a row that does not rise, else to row `end`.  Strips
    // inside the image's width (all but the last) run on bare words.
    //   walk: the next group's words in registers.
    //   walk_ahead: kRing rows ahead in shared memory, for one warp's long way
    //     down: 70 cycles a row, where a group ahead waits for memory (150).
    template <bool STOP>
    __device__ __forceinline__ void walk(const VRow<DT>& prev, int i, int end, const EdgeSel& sel) const {
        if (__all_sync(FULL, npx >= P::PPW))
            walk_rows<STOP, true>(prev, i, end, sel);
        else
            walk_rows<STOP, false>(prev, i, end, sel);
    }
    template <bool STOP, bool INSIDE>
    __device__ __forceinline__ void walk_rows(VRow<DT> prev, int i, int end, const EdgeSel& sel) const {
        int groups_end;
        if (!groups<STOP, INSIDE>(prev, i, end, groups_end, sel)) return;
        uint32_t gm[2][8], gk[2][8];
        const unsigned char *pm = m + i * pitch_m, *pk = k + i * pitch_k;  // the next group to load
        unsigned char* at = m + i * pitch_m;                               // the group in hand
        int next = i;
        auto refill = [&](int g) {
            if (next + 8 <= groups_end) {
#pragma unroll
                for (int q = 0; q < 8; ++q) gm[g][q] = word_at(pm + q * pitch_m);
#pragma unroll
                for (int q = 0; q < 8; ++q) gk[g][q] = word_at(pk + q * pitch_k);
            }
            next += 8;
            pm += 8 * pitch_m;
            pk += 8 * pitch_k;
        };
        refill(0);
        refill(1);
#pragma unroll 1
        while (i + 8 <= groups_end) {
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                if (i + 8 <= groups_end) {
                    const bool x = group<INSIDE>(prev, gm[g], gk[g], i, at, sel);
                    if (STOP && !__any_sync(FULL, x)) return;
                    refill(g);
                    i += 8;
                    at += 8 * pitch_m;
                }
            }
        }
#pragma unroll 1
        for (; i < end; ++i)
            if (!step(prev, i, sel) && STOP) return;
    }
    using Ring = uint32_t[kRing][32];
    // Returns the row that it stopped at.
    __device__ __forceinline__ int walk_ahead(const VRow<DT>& prev, int i, int end, const EdgeSel& sel, Ring& rm,
                                              Ring& rk, int lane) const {
        return __all_sync(FULL, npx >= P::PPW) ? walk_ring<true>(prev, i, end, sel, rm, rk, lane)
                                               : walk_ring<false>(prev, i, end, sel, rm, rk, lane);
    }
    template <bool INSIDE>
    __device__ __forceinline__ int walk_ring(VRow<DT> prev, int i, int end, const EdgeSel& sel, Ring& rm, Ring& rk,
                                             int lane) const {
        int groups_end;
        if (!groups<true, INSIDE>(prev, i, end, groups_end, sel)) return i;
        const unsigned char *pm = m + i * pitch_m, *pk = k + i * pitch_k;
        unsigned char* at = m + i * pitch_m;
        int next = i, slot = 0;
        auto refill = [&](int s) {  // a lane reads only words that it copied
            if (next + 8 <= groups_end) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    cp_async_4(&rm[s + q][lane], pm + q * pitch_m);
                    cp_async_4(&rk[s + q][lane], pk + q * pitch_k);
                }
            }
            cp_async_commit();
            next += 8;
            pm += 8 * pitch_m;
            pk += 8 * pitch_k;
        };
        for (int s = 0; s < kRing; s += 8) refill(s);
        bool rises = true;
#pragma unroll 1
        while (rises && i + 8 <= groups_end) {
            cp_async_wait<kRing / 8 - 1>();
            uint32_t old[8], kw[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                old[q] = rm[slot + q][lane];
                kw[q] = rk[slot + q][lane];
            }
            rises = __any_sync(FULL, group<INSIDE>(prev, old, kw, i, at, sel));
            refill(slot);
            slot = (slot + 8) % kRing;
            i += 8;
            at += 8 * pitch_m;
        }
        cp_async_wait<0>();
#pragma unroll 1
        while (rises && i < end) rises = step(prev, i++, sel);
        return i;
    }
};

template <int DT, int CONN, bool DOWN>
__global__ void __launch_bounds__(kStripThreads) sweep_strip_local_kernel(ImgDesc d, int strips, int segs,
                                                                    int seg_rows) {
    if (gated_off(d)) return;
    const int lane = threadIdx.x & 31;
    const long long wid = (long long)blockIdx.x * (kStripThreads / 32) + (threadIdx.x >> 5);
    if (wid >= (long long)strips * segs) return;
    const int seg = (int)(wid / strips), strip = (int)(wid - (long long)seg * strips);
    const Strip<DT, CONN, DOWN> st(d, strip, lane);
    const EdgeSel sel(lane);
    const int i0 = seg * seg_rows, end = min(i0 + seg_rows, d.H);
    VRow<DT> prev;
    prev.set(Px<DT>::MINW);
    st.template walk<false>(prev, i0, end, sel);
}

template <int DT, int CONN, bool DOWN>
__global__ void __launch_bounds__(kStripThreads) sweep_strip_enter_kernel(ImgDesc d, int strips, int segs) {
    if (gated_off(d)) return;
    const int lane = threadIdx.x & 31;
    const long long wid = (long long)blockIdx.x * (kStripThreads / 32) + (threadIdx.x >> 5);
    if (wid >= (long long)strips * (segs - 1)) return;
    const int seg = 1 + (int)(wid / strips), strip = (int)(wid % strips);
    const Strip<DT, CONN, DOWN> st(d, strip, lane);
    const int i0 = seg * kStripRows;
    VRow<DT> prev;
    prev.set(st.marker(i0 - 1));
    st.template walk<true>(prev, i0, min(i0 + kStripRows, d.H), EdgeSel(lane));
}

// One warp goes over all of a strip's entries: what it takes on images of very
// many rows (4 x 4000000 uint8, 31250 entries, one 4-connected
// sweep 6430 us with the rows of eight in flight, 1670 with 16, 1420 with 32).
constexpr int kEntries = 32;

template <int DT, int CONN, bool DOWN>
__global__ void __launch_bounds__(32) sweep_strip_settle_kernel(ImgDesc d, int segs) {
    if (gated_off(d)) return;
    __shared__ uint32_t ring_m[kRing][32], ring_k[kRing][32];
    const int lane = threadIdx.x;
    const Strip<DT, CONN, DOWN> st(d, (int)blockIdx.x, lane);
    const EdgeSel sel(lane);
    int reached = 0;
    // the rows that are loaded word by word (the image's last one is not)
    const int groups_end = DOWN ? d.H - 1 : d.H;
#pragma unroll 1
    for (int s0 = 1; s0 < segs; s0 += kEntries) {
        // many entries' rows in flight together; a walk that goes past an
        // entry below has satisfied it, and one that does not reach it leaves
        // the row above it as read.  So no row is copied to shared memory
        // after this thread wrote it.
        uint32_t above[kEntries], first[kEntries], kw[kEntries];
        if ((s0 + kEntries - 1) * kStripRows < groups_end) {
            const unsigned char* pm = st.m + (s0 * kStripRows - 1) * st.pitch_m;
            const unsigned char* pk = st.k + s0 * kStripRows * st.pitch_k;
#pragma unroll
            for (int q = 0; q < kEntries; ++q) {
                above[q] = st.word_at(pm + q * kStripRows * st.pitch_m);
                first[q] = st.word_at(pm + (q * kStripRows + 1) * st.pitch_m);
                kw[q] = st.word_at(pk + q * kStripRows * st.pitch_k);
            }
        } else {
#pragma unroll
            for (int q = 0; q < kEntries; ++q) {
                const int i = (s0 + q) * kStripRows;
                above[q] = first[q] = kw[q] = Px<DT>::MINW;
                if (i < groups_end) {
                    above[q] = st.word_at(st.m + (i - 1) * st.pitch_m);
                    first[q] = st.word_at(st.m + i * st.pitch_m);
                    kw[q] = st.word_at(st.k + i * st.pitch_k);
                } else if (i < d.H) {  // the image's last row
                    above[q] = st.marker(i - 1);
                    first[q] = st.marker(i);
                    kw[q] = st.mask(i);
                }
            }
        }
        unsigned due = 0u;
#pragma unroll
        for (int q = 0; q < kEntries; ++q) {
            VRow<DT> p, v, kv;
            p.set(st.template own<false>(above[q]));
            v.set(st.template own<false>(first[q]));
            kv.set(st.template own<false>(kw[q]));
            const VRow<DT> was = v;
            vstep<DT>(v, kv, offers<DT, CONN>(p, sel));
            if (__any_sync(FULL, v.differs(was))) due |= 1u << q;
        }
        while (due != 0u) {
            const int i = (s0 + __ffs((int)due) - 1) * kStripRows;
            due &= due - 1u;
            if (i < reached) continue;
            VRow<DT> prev;
            prev.set(st.marker(i - 1));
            reached = st.walk_ahead(prev, i, d.H, sel, ring_m, ring_k, lane);
        }
    }
}

constexpr int kRingN = 64;  // rows in flight per plane in the narrow variant

// Vertical sweeps for 4-connectivity (the whole-image init passes use them for
// either connectivity: the pixel above / below alone is a valid update), rows
// of whole strips on 16-byte boundaries (by_strips takes the others).
//
// uint8 / uint16: a warp covers a 64-byte strip, two bytes per lane (uint8: two
// pixels as one u16x2 register; uint16: one pixel), so the chain per row is one min and one max, and twice as many
// warps share the image.
//
// Tall images are cut into segments of kSegRows rows so that more warps
// share each column: the update of one column over a run of rows is
// x -> max(min(x, B), A) for the value x entering the run (A = the run's
// last value when nothing enters, B = the minimum of the mask over the run),
// and such maps compose.  MODE 1 computes (A, B) per segment and column
// without storing; sweep_y_carry_kernel chains them into the value entering
// each segment; MODE 2 sweeps every segment from that value and stores.
// MODE 0 is one warp over the whole column.
constexpr int kSegRows = 1024;

template <int DT, bool DOWN, int MODE>
__global__ void __launch_bounds__(32) sweep_y4n_kernel(ImgDesc d, uint32_t* seg_a, uint32_t* seg_b,
                                                       const uint32_t* seg_in) {
    if (gated_off(d)) return;
    static_assert(DT == DT_U8 || DT == DT_U16, "two-byte lanes");
    constexpr int NR = kRingN, NG = kRingN / kGroup;
    __shared__ __align__(16) uint16_t ring_m[kRingN][32];
    __shared__ __align__(16) uint16_t ring_k[kRingN][32];
    const int lane = threadIdx.x & 31;
    const int strip = (int)blockIdx.x;
    const long long b0 = (long long)strip * 64 + lane * 2;  // this lane's bytes in a row
    // rows (in sweep order) of this block's segment
    const int i0 = MODE == 0 ? 0 : (int)blockIdx.y * kSegRows;
    const int H = MODE == 0 ? d.H : min(kSegRows, d.H - i0);
    const size_t seg_idx = ((size_t)blockIdx.y * gridDim.x + strip) * 32 + lane;
    const long long step_m = DOWN ? d.pitch_m : -d.pitch_m, step_k = DOWN ? d.pitch_k : -d.pitch_k;
    const unsigned char* m0 = d.marker + (size_t)(DOWN ? 0 : d.H - 1) * d.pitch_m + (long long)i0 * step_m;
    const unsigned char* k0 = d.mask + (size_t)(DOWN ? 0 : d.H - 1) * d.pitch_k + (long long)i0 * step_k;
    // 4 pieces of 16 bytes per row and plane, 8 rows per instruction
    auto issue_group = [&](int g0) {
        const int piece = lane & 3, i = g0 + (lane >> 2);
        if (i < H) {
            const int slot = i % NR;
            const long long o = (long long)strip * 64 + piece * 16;
            cp_async16(&ring_m[slot][piece * 8], m0 + (long long)i * step_m + o);
            cp_async16(&ring_k[slot][piece * 8], k0 + (long long)i * step_k + o);
        }
    };
    for (int g = 0; g < NG; ++g) {
        issue_group(g * kGroup);
        cp_async_commit();
    }
    uint32_t prev = MODE == 2 ? seg_in[seg_idx] : 0u;
    uint32_t kmin = DT == DT_U8 ? 0x00ff00ffu : 0xffffu;
    unsigned char* mo = const_cast<unsigned char*>(m0) + b0;
    for (int base = 0; base < H; base += kGroup) {
        cp_async_wait<NG - 1>();
        __syncwarp();
        const int sb = base % NR;
        uint32_t out[kGroup], orig[kGroup];
#pragma unroll
        for (int q = 0; q < kGroup; ++q) {
            uint32_t m = ring_m[sb + q][lane], k = ring_k[sb + q][lane];
            orig[q] = m;
            const bool live = base + q < H;  // rows past the segment: stale slots
            if (DT == DT_U8) {
                m = __byte_perm(m, 0u, 0x4140);
                k = __byte_perm(k, 0u, 0x4140);
                const uint32_t v = __vmaxu2(m, __vminu2(prev, k));
                if (MODE == 1) {
                    if (live) {
                        prev = v;
                        kmin = __vminu2(kmin, k);
                    }
                } else {
                    prev = v;
                }
                out[q] = __byte_perm(v, 0u, 0x0020);
            } else {
                const uint32_t v = max(m, min(prev, k));
                if (MODE == 1) {
                    if (live) {
                        prev = v;
                        kmin = min(kmin, k);
                    }
                } else {
                    prev = v;
                }
                out[q] = v;
            }
        }
        if (MODE != 1) {
            // only the elements that rose are stored: an unchanged store
            // would still dirty its L2 sector and cost a DRAM write-back
#pragma unroll
            for (int q = 0; q < kGroup; ++q)
                if (base + q < H && out[q] != orig[q])
                    *reinterpret_cast<uint16_t*>(mo + (long long)(base + q) * step_m) = (uint16_t)out[q];
        }
        __syncwarp();
        issue_group(base + NR);
        cp_async_commit();
    }
    cp_async_wait<0>();
    if (MODE == 1) {
        seg_a[seg_idx] = prev;
        seg_b[seg_idx] = kmin;
    }
}

// int32: one pixel per lane, 128-byte strips, a warp each over the whole
// height.  Not in segments: at four bytes a pixel the two extra plane reads cost
// more than the parallelism gains (its strips already give 512 warps on a
// 16384-wide image).
template <bool DOWN>
__global__ void __launch_bounds__(32) sweep_y4i_kernel(ImgDesc d) {
    if (gated_off(d)) return;
    constexpr int NG = kRing / kGroup;
    __shared__ __align__(16) uint32_t ring_m[kRing][32];
    __shared__ __align__(16) uint32_t ring_k[kRing][32];
    const int lane = threadIdx.x & 31;
    const long long sbase = (long long)blockIdx.x * 128;
    const int H = d.H;
    const long long step_m = DOWN ? d.pitch_m : -d.pitch_m, step_k = DOWN ? d.pitch_k : -d.pitch_k;
    unsigned char* m0 = d.marker + (size_t)(DOWN ? 0 : H - 1) * d.pitch_m + sbase;
    const unsigned char* k0 = d.mask + (size_t)(DOWN ? 0 : H - 1) * d.pitch_k + sbase;
    // 8 pieces of 16 bytes per row and plane, 4 rows per instruction
    auto issue_group = [&](int g0) {
        const int piece = lane & 7;
#pragma unroll
        for (int rr = 0; rr < kGroup; rr += 4) {
            const int i = g0 + rr + (lane >> 3);
            if (i < H) {
                const int slot = i % kRing;
                cp_async16(&ring_m[slot][piece * 4], m0 + (long long)i * step_m + piece * 16);
                cp_async16(&ring_k[slot][piece * 4], k0 + (long long)i * step_k + piece * 16);
            }
        }
    };
    for (int g = 0; g < NG; ++g) {
        issue_group(g * kGroup);
        cp_async_commit();
    }
    int prev = INT_MIN;
    unsigned char* mo = m0 + lane * 4;
    for (int base = 0; base < H; base += kGroup) {
        cp_async_wait<NG - 1>();
        __syncwarp();  // pieces copied by other lanes are visible to this one
        const int sb = base % kRing;
        int out[kGroup];
#pragma unroll
        for (int q = 0; q < kGroup; ++q) {
            const int m = (int)ring_m[sb + q][lane], k = (int)ring_k[sb + q][lane];
            out[q] = prev = max(m, min(prev, k));
        }
#pragma unroll
        for (int q = 0; q < kGroup; ++q)
            if (base + q < H) *reinterpret_cast<int*>(mo + (long long)(base + q) * step_m) = out[q];
        __syncwarp();  // the slots just read are refilled next
        issue_group(base + kRing);
        cp_async_commit();
    }
    cp_async_wait<0>();
}

// The value entering every segment of every column: x_0 = nothing (0),
// x_{j+1} = max(min(x_j, B_j), A_j).  One thread per lane slot of a strip.
template <int DT>
__global__ void sweep_y_carry_kernel(int nseg, int slots, const uint32_t* seg_a, const uint32_t* seg_b,
                                     uint32_t* seg_in) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t >= slots) return;
    uint32_t x = 0u;
    for (int j = 0; j < nseg; ++j) {
        const size_t idx = (size_t)j * slots + t;
        seg_in[idx] = x;
        if (DT == DT_U8)
            x = __vmaxu2(__vminu2(x, seg_b[idx]), seg_a[idx]);
        else
            x = max(min(x, seg_b[idx]), seg_a[idx]);
    }
}

static bool aligned16(const ImgDesc& d) {
    return ((reinterpret_cast<uintptr_t>(d.marker) | reinterpret_cast<uintptr_t>(d.mask)) & 15u) == 0u &&
           ((d.pitch_m | d.pitch_k) & 15) == 0;
}

// Vertical sweeps by 128-byte strips in place: 8-connected ones, and
// 4-connected ones of rows off the 16-byte boundary or not a whole number of
// the ring kernels' strips wide, which those would have to load element by
// element (2000 x 768 uint8 240 us, by strips 42; 1416 x 5514 uint8 574 and
// 54, uint16 487 and 54; 708 x 5514 int32 1640 and 33).  The others stay with
// the ring kernels: their segments' maps compose, so a long vertical path costs
// nothing (whole calls: 16384^2 spiral 409 us, by strips 594; 128 x 100000 sparse
// seeds 263 and 2730).
static bool by_strips(const ImgDesc& d) {
    const long long row = (long long)d.W * (d.dtype == DT_U8 ? 1 : d.dtype == DT_U16 ? 2 : 4);
    return d.conn == 8 || !aligned16(d) || row % (d.dtype == DT_I32 ? 128 : 64) != 0;
}

size_t sweep_scratch_bytes(const ImgDesc& d) {
    if (by_strips(d) || d.dtype == DT_I32 || d.H <= 2 * kSegRows) return 0;
    const long long strips = (long long)d.W * (d.dtype == DT_U8 ? 1 : 2) / 64;
    const long long nseg = (d.H + kSegRows - 1) / kSegRows;
    return (size_t)(3 * nseg * strips * 32 * 4);
}

// ------------------------------------------------------------ host side
static unsigned blocks_for(long long threads, int block) {
    long long b = (threads + block - 1) / block;
    if (b < 1) b = 1;
    if (b > (1ll << 30)) b = 1ll << 30;
    return (unsigned)b;
}

cudaError_t launch_fixed_point_check(const ImgDesc& d, unsigned long long* count, cudaStream_t s) {
    if (d.W == 0 || d.H == 0) return cudaSuccess;
    unsigned blocks = blocks_for((long long)d.W * d.H, 256);
    if (blocks > kSms * 16u) blocks = kSms * 16u;
    if (d.dtype == DT_U8)
        fixed_point_kernel<DT_U8><<<blocks, 256, 0, s>>>(d, count);
    else if (d.dtype == DT_U16)
        fixed_point_kernel<DT_U16><<<blocks, 256, 0, s>>>(d, count);
    else
        fixed_point_kernel<DT_I32><<<blocks, 256, 0, s>>>(d, count);
    return cudaGetLastError();
}

cudaError_t launch_clip(const ImgDesc& d, cudaStream_t s) {
    if (d.W == 0 || d.H == 0) return cudaSuccess;
    const int ppw = d.dtype == DT_U8 ? 4 : d.dtype == DT_U16 ? 2 : 1;
    const long long words = (long long)((d.W + ppw - 1) / ppw) * d.H;
    unsigned blocks = blocks_for(words, 256);
    if (blocks > kSms * 16u) blocks = kSms * 16u;
    if (d.dtype == DT_U8)
        clip_kernel<DT_U8><<<blocks, 256, 0, s>>>(d);
    else if (d.dtype == DT_U16)
        clip_kernel<DT_U16><<<blocks, 256, 0, s>>>(d);
    else
        clip_kernel<DT_I32><<<blocks, 256, 0, s>>>(d);
    return cudaGetLastError();
}

// A vertical sweep by 128-byte strips; returns the launches.
template <int DT, int CONN, bool DOWN>
static int launch_strips(const ImgDesc& d, int strips, cudaStream_t s) {
    const bool whole = d.H <= kStripWhole;
    const int seg_rows = whole ? d.H : kStripRows, segs = whole ? 1 : (d.H + kStripRows - 1) / kStripRows;
    auto grid = [&](long long n) { return (unsigned)((n * strips + kStripThreads / 32 - 1) / (kStripThreads / 32)); };
    sweep_strip_local_kernel<DT, CONN, DOWN><<<grid(segs), kStripThreads, 0, s>>>(d, strips, segs, seg_rows);
    if (whole) return 1;
    for (int r = 0; r < kStripEnter; ++r)
        sweep_strip_enter_kernel<DT, CONN, DOWN><<<grid(segs - 1), kStripThreads, 0, s>>>(d, strips, segs);
    sweep_strip_settle_kernel<DT, CONN, DOWN><<<(unsigned)strips, 32, 0, s>>>(d, segs);
    return 2 + kStripEnter;
}

template <int DT>
static int launch_sweep_t(const ImgDesc& d, int direction, cudaStream_t s, void* scratch) {
    using P = Px<DT>;
    constexpr int TW = 32 * P::PPW;
    if (direction == 0 || direction == 2) {
        const unsigned blocks = blocks_for((long long)d.H * 32, 128);
        if (aligned16(d) && DT == DT_U8) {
            // two rows per warp (uint16 measured no faster: its lanes hold
            // half as many pixels, so the scan is a smaller share)
            const unsigned pblocks = blocks_for((long long)((d.H + 1) / 2) * 32, 128);
            if (direction == 0)
                sweep_x16p_kernel<DT_U8, true><<<pblocks, 128, 0, s>>>(d);
            else
                sweep_x16p_kernel<DT_U8, false><<<pblocks, 128, 0, s>>>(d);
        } else if (aligned16(d)) {
            if (direction == 0)
                sweep_x16_kernel<DT, true><<<blocks, 128, 0, s>>>(d);
            else
                sweep_x16_kernel<DT, false><<<blocks, 128, 0, s>>>(d);
        } else if (direction == 0) {
            sweep_x_kernel<DT, true><<<blocks, 128, 0, s>>>(d);
        } else {
            sweep_x_kernel<DT, false><<<blocks, 128, 0, s>>>(d);
        }
        return 1;
    } else {
        const int strips = (d.W + TW - 1) / TW;
        const bool down = direction == 1;
        if (d.conn == 8)
            return down ? launch_strips<DT, 8, true>(d, strips, s) : launch_strips<DT, 8, false>(d, strips, s);
        if (by_strips(d))
            return down ? launch_strips<DT, 4, true>(d, strips, s) : launch_strips<DT, 4, false>(d, strips, s);
        if constexpr (DT == DT_I32) {
            if (down)
                sweep_y4i_kernel<true><<<(unsigned)strips, 32, 0, s>>>(d);
            else
                sweep_y4i_kernel<false><<<(unsigned)strips, 32, 0, s>>>(d);
        } else {
            const unsigned nblocks = (unsigned)((long long)d.W * P::BPP / 64);
            if (scratch && sweep_scratch_bytes(d) > 0) {
                // segments: aggregate, chain, sweep
                const int nseg = (d.H + kSegRows - 1) / kSegRows;
                const int slots = (int)nblocks * 32;
                uint32_t* a = static_cast<uint32_t*>(scratch);
                uint32_t* b = a + (size_t)nseg * slots;
                uint32_t* in = b + (size_t)nseg * slots;
                const dim3 grid(nblocks, (unsigned)nseg);
                if (down)
                    sweep_y4n_kernel<DT, true, 1><<<grid, 32, 0, s>>>(d, a, b, nullptr);
                else
                    sweep_y4n_kernel<DT, false, 1><<<grid, 32, 0, s>>>(d, a, b, nullptr);
                sweep_y_carry_kernel<DT><<<(unsigned)((slots + 127) / 128), 128, 0, s>>>(nseg, slots, a, b, in);
                if (down)
                    sweep_y4n_kernel<DT, true, 2><<<grid, 32, 0, s>>>(d, nullptr, nullptr, in);
                else
                    sweep_y4n_kernel<DT, false, 2><<<grid, 32, 0, s>>>(d, nullptr, nullptr, in);
                return 3;
            } else if (down) {
                sweep_y4n_kernel<DT, true, 0><<<nblocks, 32, 0, s>>>(d, nullptr, nullptr, nullptr);
            } else {
                sweep_y4n_kernel<DT, false, 0><<<nblocks, 32, 0, s>>>(d, nullptr, nullptr, nullptr);
            }
        }
        return 1;
    }
}

cudaError_t launch_sweep(const ImgDesc& d, int direction, cudaStream_t s, void* scratch, int* launches) {
    if (d.W == 0 || d.H == 0) return cudaSuccess;
    int n;
    if (d.dtype == DT_U8)
        n = launch_sweep_t<DT_U8>(d, direction, s, scratch);
    else if (d.dtype == DT_U16)
        n = launch_sweep_t<DT_U16>(d, direction, s, scratch);
    else
        n = launch_sweep_t<DT_I32>(d, direction, s, scratch);
    if (launches) *launches += n;
    return cudaGetLastError();
}

}  // namespace iwpp
