// iwpp_engine_kernel.cuh -- the persistent kernel of the tile engine and its
// queues (see iwpp_engine.cuh for the design and the reference citations),
// instantiated queue by queue in
// iwpp_engine_{mutex,double,unique,async}.cu.
#pragma once

#include "iwpp_engine.cuh"

namespace iwpp {

__device__ __forceinline__ unsigned ld_volatile(const unsigned* p) { return *(const volatile unsigned*)p; }
__device__ __forceinline__ int ld_volatile(const int* p) { return *(const volatile int*)p; }

__device__ __forceinline__ void set_error(Ctrl* c, unsigned code) { atomicCAS(&c->error, 0u, code); }

// Async ring: positions below this are the job's initial entries (every
// tile, or the seed list after the front stage), the rest map to ring slots.
__device__ __forceinline__ unsigned ring_base(const EngineArgs& a) {
    return a.init_list ? ld_volatile(&a.ctrl->ninit) : a.G;
}

// Image of global tile g: the last image whose tile_base <= g.
__device__ __forceinline__ int find_image(const EngineArgs& a, unsigned g) {
    int lo = 0, hi = a.nimg - 1;
#pragma unroll 1
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((unsigned)__ldg(&a.imgs[mid].tile_base) <= g)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// A tile's shared memory in a kernel (SOLVE_*), and its visit for the image's
// pixel type.
template <int TH, int W, int SOLVE>
struct SmemOf {
    using T = TileSmemPasses<TH, W>;
};
template <int TH, int W>
struct SmemOf<TH, W, SOLVE_SWEEPS> {
    using T = TileSmem<TH>;
};
template <int TH, int W>
struct SmemOf<TH, W, SOLVE_PQ> {
    using T = TileSmemPq<TH>;
};

template <int DT, int CONN, int TH, int W, int SOLVE, class SM, class Early>
__device__ __forceinline__ bool visit_as(const EngineArgs& a, SM& sm, int warp, int lane, unsigned& phase,
                                         unsigned& row_steps, Early& early) {
    if constexpr (SOLVE == SOLVE_PASSES)
        return visit_tile<DT, CONN, TH, W>(sm, warp, lane, phase, a.timeout_ns, row_steps);
    else if (sm.d.conn == 8)
        return visit_tile_alt<DT, 8, TH, SOLVE == SOLVE_PQ>(sm, lane, phase, a.timeout_ns, row_steps, early);
    else
        return visit_tile_alt<DT, 4, TH, SOLVE == SOLVE_PQ>(sm, lane, phase, a.timeout_ns, row_steps, early);
}

template <int CONN, int TH, int W, int SOLVE, class SM, class Early>
__device__ __forceinline__ bool dispatch_visit(const EngineArgs& a, SM& sm, int warp, int lane, unsigned& phase,
                                               unsigned& row_steps, Early& early) {
    switch (sm.d.dtype) {
        case DT_U8: return visit_as<DT_U8, CONN, TH, W, SOLVE>(a, sm, warp, lane, phase, row_steps, early);
        case DT_U16: return visit_as<DT_U16, CONN, TH, W, SOLVE>(a, sm, warp, lane, phase, row_steps, early);
        default: return visit_as<DT_I32, CONN, TH, W, SOLVE>(a, sm, warp, lane, phase, row_steps, early);
    }
}

// The side of a neighbour tile that faces direction `dir` of this tile.
__device__ __constant__ static const int kNbOpposite[8] = {1, 0, 3, 2, 7, 6, 5, 4};

// ---------------------------------------------------------------- mutex

// The global mutex (IWPP MP/src/globalQueue.cu:35, :114, a CAS spin without
// a bound) as a ticket lock: one atomic per acquisition instead of a CAS
// storm from every waiting warp, hand-over in arrival order, acquire /
// release ordering instead of full fences; waiters poll the ticket being
// served with a back-off proportional to their place in line, and a
// wall-clock bound ends in DEV_ERR_TIMEOUT.  A waiter that gives up leaves
// the error flag set, which ends every other waiter too.
__device__ __forceinline__ unsigned long long ld_acquire64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// The mutex stack's entry count and the ticket being served, read without
// the lock (hints: look-ahead, quiescence).
__device__ __forceinline__ int stack_top(const Ctrl* c) {
    return (int)(unsigned)(*(const volatile unsigned long long*)&c->lock_word >> 32);
}
__device__ __forceinline__ unsigned lock_serving(const Ctrl* c) {
    return (unsigned)*(const volatile unsigned long long*)&c->lock_word;
}

// Acquires the lock; *top is the stack's entry count at the hand-over.
__device__ inline bool mutex_lock(const EngineArgs& a, unsigned* ticket, int* top) {
    const unsigned t = atomicAdd(&a.ctrl->lock_next, 1u);
    *ticket = t;
    const long long t0 = globaltimer_ns();
    unsigned spins = 0;
    for (;;) {
        const unsigned long long w = ld_acquire64(&a.ctrl->lock_word);
        const unsigned s = (unsigned)w;
        if (s == t) {
            *top = (int)(unsigned)(w >> 32);
            return true;
        }
        const unsigned place = t - s;
        __nanosleep(32u * (place < 32u ? place : 32u));
        if ((++spins & 15u) == 0u) {
            if (ld_volatile(&a.ctrl->error) != 0u) return false;
            if (globaltimer_ns() - t0 > a.timeout_ns) {
                set_error(a.ctrl, DEV_ERR_TIMEOUT);
                return false;
            }
        }
    }
}

// Releases the lock, publishing the stack's new entry count with it.
__device__ __forceinline__ void mutex_unlock(const EngineArgs& a, unsigned ticket, int top) {
    st_release64(&a.ctrl->lock_word, ((unsigned long long)(unsigned)top << 32) | (unsigned long long)(ticket + 1u));
}

// ------------------------------------------------------------------ push
// Inserts the entries of the lanes with `want` set into the queue: the mutex
// stack under one lock acquisition (IWPP MP/src/globalQueue.cu:25-81), or the
// write queue with one atomicAdd reservation per warp
// (IWPP MP DQ/src/globalQueue.cu:14-47).  A short insertion sets the
// overflow flag (the reference's memLeak, MR.cu:524-526); the tiles stay
// DIRTY and are recovered by the restart.  push_entries returns their number.
// The mutex stack's insertion: one lock acquisition for the warp's entries.
// `counted`: `pending` already holds them (entries moving from a CTA
// buffer); else they are added to it before the release can publish them.
__device__ inline void mutex_push_global(const EngineArgs& a, bool want, unsigned gn, int lane, bool counted) {
    const unsigned ballot = __ballot_sync(FULL, want);
    if (ballot == 0u) return;
    const int n = __popc(ballot);
    const int rank = __popc(ballot & ((1u << lane) - 1u));
    int base = -1;
    unsigned ticket = 0u;
    if (lane == 0) {
        int top = 0;
        if (mutex_lock(a, &ticket, &top)) {
            if ((unsigned)top + (unsigned)n <= a.cap) {
                base = top;
                if (!counted) atomicAdd(&a.ctrl->pending, n);  // before the entries can be taken
            } else {
                atomicExch(&a.ctrl->overflow, 1u);
                if (counted) atomicSub(&a.ctrl->pending, n);  // lost: the restart recovers the tiles
                mutex_unlock(a, ticket, top);
            }
        }
    }
    base = __shfl_sync(FULL, base, 0);
    if (base < 0) return;
    if (want) {
        a.q0[base + rank] = gn;
        __threadfence();  // the entry before the release that publishes it
    }
    __syncwarp();
    if (lane == 0) mutex_unlock(a, ticket, base + n);
}

template <int VAR>
__device__ int push_entries(const EngineArgs& a, bool want, unsigned gn, int lane, unsigned* wq) {
    const unsigned ballot = __ballot_sync(FULL, want);
    if (ballot == 0u) return 0;
    const int n = __popc(ballot);
    const int rank = __popc(ballot & ((1u << lane) - 1u));
    if (VAR == VAR_MUTEX) {
        mutex_push_global(a, want, gn, lane, false);
    } else if (VAR == VAR_ASYNC) {
        // positions [base, base + n) of the ring; `pending` first, so the job
        // cannot look finished while these entries exist
        unsigned base = 0u;
        if (lane == 0) {
            atomicAdd(&a.ctrl->pending, n);
            base = atomicAdd(&a.ctrl->atail, (unsigned)n);
        }
        base = __shfl_sync(FULL, base, 0);
        if (want) {
            const unsigned slot = (base + (unsigned)rank - ring_base(a)) % a.cap;
            const long long t0 = globaltimer_ns();
            unsigned spins = 0;
            // the slot's previous occupant has normally been taken long ago
            while (atomicCAS(&a.q0[slot], 0u, gn + 1u) != 0u) {
                __nanosleep(64);
                if ((++spins & 255u) == 0u && globaltimer_ns() - t0 > a.timeout_ns) {
                    set_error(a.ctrl, DEV_ERR_TIMEOUT);
                    break;
                }
            }
        }
    } else {
        unsigned base = 0u;
        if (lane == 0) base = atomicAdd(&a.ctrl->wn, (unsigned)n);
        base = __shfl_sync(FULL, base, 0);
        if (want) {
            const unsigned pos = base + (unsigned)rank;
            if (pos < a.cap)
                wq[pos] = gn;
            else
                atomicExch(&a.ctrl->overflow, 1u);
        }
    }
    return n;
}

// ------------------------------------------------- mutex: CTA buffers
// The MP discipline keeps one LIFO stack under one lock, and what
// serialises it is one acquisition per insertion and per take.  Each CTA
// therefore keeps the entries it inserts in a shared-memory buffer and takes
// from it first; the global stack sees a batch take when the buffer runs dry,
// a spill when it fills, and a share when the global stack is empty while
// CTAs elsewhere wait.  Buffered entries count in `pending`, so the
// termination rule (nothing pending, nothing stacked) is unchanged.  Where the
// CTA's first warp alone works the queue the buffer needs no lock; where its
// warps each work it (SHARED, the solvers of one warp per tile) they take
// turns at it, and one of them at a time goes to the global stack for all.
constexpr int kCtaBuf = 64;    // entries a CTA buffers
constexpr int kCtaSpill = 48;  // above this a push spills the buffer down to kCtaKeep
constexpr int kCtaKeep = 16;

struct MutexCtaBuf {
    int n;
    unsigned e[kCtaBuf];
    int lock;
    int taker;    // 1 while one of this CTA's warps works the global stack
    int waiting;  // this CTA's warps waiting for work
};
__shared__ MutexCtaBuf s_cq;

__device__ __forceinline__ int cq_count() { return *(volatile int*)&s_cq.n; }

// The buffer's lock, held by one of this CTA's warps (lane 0) for a few
// shared-memory accesses at a time; the bound is never reached in a working job.
template <bool SHARED>
__device__ __forceinline__ bool cq_lock(const EngineArgs& a) {
    if (SHARED) {
        unsigned spins = 0;
        while (atomicCAS(&s_cq.lock, 0, 1) != 0) {
            __nanosleep(32);
            if (++spins > (1u << 22)) {
                set_error(a.ctrl, DEV_ERR_TIMEOUT);
                return false;
            }
        }
        __threadfence_block();
    }
    return true;
}
template <bool SHARED>
__device__ __forceinline__ void cq_unlock() {
    if (SHARED) {
        __threadfence_block();
        atomicExch(&s_cq.lock, 0);
    }
}

// Moves up to 32 of the buffer's newest entries beyond `keep` to the global
// stack (one acquisition).
template <bool SHARED>
__device__ inline void cta_spill(const EngineArgs& a, int lane, int keep) {
    int m = 0, base = 0;
    if (lane == 0 && cq_lock<SHARED>(a)) {
        const int n = cq_count();
        m = min(max(n - keep, 0), 32);
        base = n - m;
        *(volatile int*)&s_cq.n = base;
        if (m == 0) cq_unlock<SHARED>();
    }
    m = __shfl_sync(FULL, m, 0);
    base = __shfl_sync(FULL, base, 0);
    if (m == 0) return;
    const unsigned mine = lane < m ? *(volatile unsigned*)&s_cq.e[base + lane] : 0u;
    __syncwarp();
    if (lane == 0) cq_unlock<SHARED>();
    mutex_push_global(a, lane < m, mine, lane, true);
}

// Inserts the entries of the lanes with `want` set into this CTA's buffer
// (what does not fit goes to the global stack), spilling a full buffer.
// `counted`: `pending` already holds them.  Returns their number.
template <bool SHARED>
__device__ inline int cta_push(const EngineArgs& a, bool want, unsigned gn, int lane, bool counted = false) {
    const unsigned ballot = __ballot_sync(FULL, want);
    if (ballot == 0u) return 0;
    const int n = __popc(ballot);
    const int rank = __popc(ballot & ((1u << lane) - 1u));
    int base = 0, k = 0;
    bool mine = false;  // lane 0: the lock is held
    if (lane == 0) {
        if (!counted) atomicAdd(&a.ctrl->pending, n);  // before any of them can be taken
        mine = cq_lock<SHARED>(a);
        if (mine) {
            base = cq_count();
            k = min(n, kCtaBuf - base);
        }
    }
    base = __shfl_sync(FULL, base, 0);
    k = __shfl_sync(FULL, k, 0);
    if (want && rank < k) *(volatile unsigned*)&s_cq.e[base + rank] = gn;
    __syncwarp();
    if (mine) {
        *(volatile int*)&s_cq.n = base + k;
        cq_unlock<SHARED>();
    }
    __syncwarp();
    if (n > k) mutex_push_global(a, want && rank >= k, gn, lane, true);
    if (__shfl_sync(FULL, cq_count(), 0) > kCtaSpill) cta_spill<SHARED>(a, lane, kCtaKeep);
    return n;
}

// The buffer's newest entry, or ~0u.
template <bool SHARED>
__device__ inline unsigned cta_take(const EngineArgs& a, int lane) {
    unsigned g = ~0u;
    if (lane == 0 && cq_count() > 0 && cq_lock<SHARED>(a)) {
        const int n = cq_count();
        if (n > 0) {
            g = *(volatile unsigned*)&s_cq.e[n - 1];
            *(volatile int*)&s_cq.n = n - 1;
        }
        cq_unlock<SHARED>();
    }
    return __shfl_sync(FULL, g, 0);
}

// ------------------------------------------------------------ one entry
// Takes tile g.  False: another CTA owns it (that owner sees DIRTY when it
// releases).  *sides: the halo sides to look at, 0 for a tile that is not
// DIRTY.  One exchange sets ACTIVE and takes DIRTY and the sides over; where
// the tile was ACTIVE already (a duplicate entry), what the exchange took
// goes back to the owner, and an owner that released the tile in between
// leaves it to this CTA.
__device__ __forceinline__ bool take_tile(const EngineArgs& a, unsigned g, int lane, unsigned* sides) {
    unsigned old = 0u;
    if (lane == 0) {
        for (;;) {
            old = atomicExch(&a.state[g], ST_ACTIVE);
            const unsigned rest = old & (ST_DIRTY | ST_SIDES);
            if (!(old & ST_ACTIVE) || rest == 0u) break;
            if (atomicOr(&a.state[g], rest) & (ST_ACTIVE | ST_DIRTY)) break;
        }
        fence_gpu();  // acquire: neighbours' stores before their DIRTY
    }
    old = __shfl_sync(FULL, old, 0);
    if (old & ST_ACTIVE) return false;
    *sides = (old & ST_DIRTY) == 0u ? 0u : (old & ST_SIDES) != 0u ? (old & ST_SIDES) >> ST_SIDE_SHIFT : 0xffu;
    return true;
}

// Lane < 8: marks the neighbour tile in direction `lane` DIRTY if it is in
// `nb`; true where it is to be inserted (*gn).  *fresh: it was neither DIRTY nor
// being visited.
template <int VAR>
__device__ __forceinline__ bool mark_neighbour(const EngineArgs& a, const ImgDesc& d, int tx, int ty, unsigned nb,
                                               int lane, unsigned* gn, bool* fresh) {
    if (!((nb >> lane) & 1u)) return false;
    const int nx = tx + kNbDx[lane], ny = ty + kNbDy[lane];
    if (nx < 0 || nx >= d.tiles_x || ny < 0 || ny >= d.tiles_y) return false;
    *gn = (unsigned)d.tile_base + (unsigned)(ny * d.tiles_x + nx);
    const unsigned old = atomicOr(&a.state[*gn], ST_DIRTY | (1u << (ST_SIDE_SHIFT + (unsigned)kNbOpposite[lane])));
    *fresh = (old & (ST_DIRTY | ST_ACTIVE)) == 0u;
    return VAR == VAR_UNIQUE || VAR == VAR_ASYNC ? *fresh : true;
}

// Publication before a tile has converged, for the solvers of one warp per
// tile with the async queue: while more than half of the warps wait for work (a
// quarter or an eighth switches too early on h-dome images, three quarters too
// late on long corridors) a visit that raised a boundary of its tile stores
// what it has and inserts those neighbours at once, so that they can start.
// Several warps per tile are done too soon for it to pay (every workload
// slower).  Row sweeps, us with / without it: sparse seeds 4096^2 u8 710 / 822,
// h-domes 2048 x 1500 u16 338 / 378, 300 x 200 u8 211 / 225, 4096^2 u8 446 / 434.
template <int VAR>
struct EarlyFlush {
    static constexpr bool kEnabled = VAR == VAR_ASYNC;
    const EngineArgs& a;
    const ImgDesc& d;
    const int &tx, &ty;
    unsigned& pushes;
    int half;  // of the warps that take entries
    __device__ __forceinline__ bool want(int lane) const {
        unsigned v = 0u;
        if (lane == 0) {
            const unsigned head = ld_volatile(&a.ctrl->ahead), tail = ld_volatile(&a.ctrl->atail);
            v = (int)(head - tail) > half ? 1u : 0u;
        }
        return __shfl_sync(FULL, v, 0) != 0u;
    }
    __device__ __forceinline__ void flush(unsigned nb, int lane) const {
        __syncwarp();
        fence_gpu();  // release: the rows just stored before the neighbours' DIRTY
        bool fresh = false;
        unsigned gn = 0u;
        const bool want = lane < 8 && mark_neighbour<VAR>(a, d, tx, ty, nb, lane, &gn, &fresh);
        const int pushed = push_entries<VAR>(a, want, gn, lane, nullptr);
        if (lane == 0) pushes += (unsigned)pushed;
    }
};

// After a visit of tile (tx, ty) = g: marks the neighbour tiles in `nb`
// DIRTY and inserts them (VAR_UNIQUE / VAR_ASYNC: only those that were
// neither pending nor being visited), and releases g, inserting it again if
// it was marked DIRTY meanwhile (next round for the double / unique queues;
// not revisited at once with half-updated neighbours).  The atomics of all of
// them are in flight together.  With the async queue and the mutex stack one
// of the newly dirty neighbours is not inserted but returned: the CTA visits
// it next itself, following the propagation front without a trip through the
// queue.  Returns ~0u when there is none.
template <int VAR, bool SHARED>
__device__ __forceinline__ unsigned leave_tile(const EngineArgs& a, const ImgDesc& d, int tx, int ty, unsigned g,
                                               unsigned nb, int lane, unsigned* wq, int* pushed) {
    bool fresh = false, want = false;
    unsigned gn = 0u;
    if (lane < 8) {
        want = mark_neighbour<VAR>(a, d, tx, ty, nb, lane, &gn, &fresh);
    } else if (lane == 8) {
        gn = g;
        want = (atomicAnd(&a.state[g], ~ST_ACTIVE) & ST_DIRTY) != 0u;
    }
    unsigned cont = ~0u;
    if (VAR == VAR_ASYNC || VAR == VAR_MUTEX) {
        const unsigned ballot = __ballot_sync(FULL, want && fresh);
        if (ballot != 0u) {
            const int leader = __ffs(ballot) - 1;
            cont = __shfl_sync(FULL, gn, leader);
            if (lane == leader) want = false;
        }
    }
    *pushed = VAR == VAR_MUTEX ? cta_push<SHARED>(a, want, gn, lane) : push_entries<VAR>(a, want, gn, lane, wq);
    return cont;
}

// ------------------------------------------------------- mutex worker
// The global stack's side of a take, for the one warp of its CTA that works
// it: up to kMutexBatch entries under the lock (enough for this CTA's
// waiting warps, or the stack divided among the CTAs while it is long; the
// reference takes one, IWPP MP/src/MorphologicalReconstruction.cu:221), the
// first returned in *g, the rest buffered for the CTA.  Returns 0 with an
// entry, 1 when the job is over for this warp (finished or an error), 2 when
// there is nothing to take now.  On overflow the quiescent stack is refilled
// with every tile (MR.cu:785-806).
template <bool SHARED>
__device__ inline int mutex_global_take(const EngineArgs& a, int lane, unsigned* g) {
    // Look before queueing for the lock: a ticket only while the stack holds
    // more entries than there are warps in line (a ticket lock serves in
    // arrival order, so warps queued for an empty stack would delay every
    // warp that inserts), or when the job looks finished but an overflow
    // needs the refill.  A finished job (nothing stacked or pending, no
    // overflow) is left without the lock.
    int look = 0;  // 0 back off, 1 take a ticket, 2 finished
    if (lane == 0) {
        const int top = stack_top(a.ctrl);
        const int pend = ld_volatile(&a.ctrl->pending);
        const unsigned line = ld_volatile(&a.ctrl->lock_next) - lock_serving(a.ctrl);
        if (pend == 0 && top == 0 && ld_volatile(&a.ctrl->overflow) == 0u)
            look = 2;
        else if (top > (int)line || pend == 0)
            look = 1;
    }
    look = __shfl_sync(FULL, look, 0);
    if (look == 2) return 1;
    if (look == 0) return 2;
    int n = 0, base = 0, outcome = 0;  // outcome: 0 entries / nothing, 1 exit, 2 refill
    unsigned ticket = 0u;
    int top = 0;
    if (lane == 0) {
        if (!mutex_lock(a, &ticket, &top)) {
            outcome = 1;
        } else {
            if (top > 0) {
                n = max(top / (int)gridDim.x, 1 + (SHARED ? *(volatile int*)&s_cq.waiting : 0));
                n = n > kMutexBatch ? kMutexBatch : n;
                n = n > top ? top : n;
                base = top - n;
            } else if (ld_volatile(&a.ctrl->pending) == 0) {
                if (ld_volatile(&a.ctrl->overflow) != 0u) {
                    if ((int)ld_volatile(&a.ctrl->restarts) >= a.max_restarts) {
                        set_error(a.ctrl, DEV_ERR_OVERFLOW);
                        outcome = 1;
                    } else {
                        outcome = 2;
                    }
                } else {
                    outcome = 1;
                }
            }
            if (n == 0 && outcome != 2) mutex_unlock(a, ticket, top);
        }
    }
    n = __shfl_sync(FULL, n, 0);
    base = __shfl_sync(FULL, base, 0);
    outcome = __shfl_sync(FULL, outcome, 0);
    if (outcome == 1) return 1;
    if (outcome == 2) {
        // quiescent with lost insertions: refill with every tile (lock held)
        for (unsigned i = (unsigned)lane; i < a.G && i < a.cap; i += 32u) a.q0[i] = a.G - 1u - i;
        __threadfence();
        __syncwarp();
        if (lane == 0) {
            const int cnt_all = (int)(a.G < a.cap ? a.G : a.cap);
            atomicAdd(&a.ctrl->pending, cnt_all);
            atomicExch(&a.ctrl->overflow, 0u);
            atomicAdd(&a.ctrl->restarts, 1u);
            mutex_unlock(a, ticket, cnt_all);
        }
        __syncwarp();
        return 2;
    }
    if (n == 0) return 2;
    // copy the taken entries out before the lock is released
    unsigned mine = 0u;
    if (lane < n) mine = __ldcg(&a.q0[base + lane]);  // from L2: the slot may have been cached before
    // (the vote needs every lane's value: the loads are done before the release)
    __ballot_sync(FULL, mine == ~0u);
    if (lane == 0) mutex_unlock(a, ticket, base);
    *g = __shfl_sync(FULL, mine, 0);
    cta_push<SHARED>(a, lane >= 1 && lane < n, mine, lane, true);
    return 0;
}

// A queue entry that names no tile ends the job with an error.
__device__ __forceinline__ bool names_a_tile(const EngineArgs& a, int lane, unsigned g) {
    if (g < a.G) return true;
    if (lane == 0) set_error(a.ctrl, DEV_ERR_INTERNAL);
    return false;
}

// The queues, as a CTA's first warp works them, or each of the WORKERS warps of
// one where a warp visits a tile alone: get() finds the next entry (false when
// the job is over or failed), done() counts it finished after its visit and
// those of the neighbours that the worker went on to.

// One persistent launch.  The next entry comes from the CTA's buffer; when
// that is empty, a batch is taken from the global LIFO stack
// (mutex_global_take).  Termination: nothing is stacked and no inserted entry
// is unfinished (`pending` == 0, buffered entries included), which replaces
// activeBlocksCount (IWPP MP/src/globalQueue.cu:134-145).
template <int WORKERS>
struct MutexQueue {
    static constexpr int VAR = VAR_MUTEX;
    static constexpr bool SHARED = WORKERS > 1;
    unsigned* wq = nullptr;
    unsigned ns = 64;

    // this CTA's slice of the initial stack, without the lock (it lies above
    // the stack's top, and `pending` counts it already); the lowest position
    // ends on the buffer's top, so it is taken first, as from the stack
    __device__ void start(const EngineArgs& a, int lane) {
        if (!SHARED || threadIdx.x < 32) {
            const unsigned pf = ld_volatile(&a.ctrl->prefill);
            const unsigned base = ld_volatile(&a.ctrl->prefill_base) + blockIdx.x * pf;
            for (unsigned j = (unsigned)lane; j < pf; j += 32u) s_cq.e[j] = __ldcg(&a.q0[base + pf - 1u - j]);
            if (lane == 0) {
                s_cq.n = (int)pf;
                s_cq.lock = s_cq.taker = s_cq.waiting = 0;
            }
        }
        if (SHARED)
            __syncthreads();
        else
            __syncwarp();
    }
    __device__ bool get(const EngineArgs& a, int lane, unsigned* out) {
        long long idle_since = 0;
        unsigned idle_progress = 0u;
        bool idle = false, got = false;  // idle: counted in ctrl->idle
        ns = 64;
        for (;;) {
            if (ld_volatile(&a.ctrl->error) != 0u) break;
            unsigned g = cta_take<SHARED>(a, lane);
            int outcome = 0;
            if (g == ~0u) {
                int taker = 1;
                if (SHARED) taker = __shfl_sync(FULL, lane == 0 ? atomicCAS(&s_cq.taker, 0, 1) == 0 : 0, 0);
                if (taker) {
                    outcome = mutex_global_take<SHARED>(a, lane, &g);
                    __syncwarp();
                    if (SHARED && lane == 0) atomicExch(&s_cq.taker, 0);
                } else {
                    // another warp of this CTA is at the global stack: wait for
                    // its batch, leaving when the job is over
                    const bool over = ld_volatile(&a.ctrl->pending) == 0 && stack_top(a.ctrl) == 0 &&
                                      ld_volatile(&a.ctrl->overflow) == 0u;
                    outcome = __shfl_sync(FULL, over ? 1 : 2, 0);
                }
            }
            if (outcome == 1) break;
            if (outcome == 0) {
                got = names_a_tile(a, lane, g);
                *out = g;
                break;
            }
            // nothing to take but work in flight: back off, bounded by progress
            if (!idle && lane == 0) {
                atomicAdd(&a.ctrl->idle, 1u);
                if (SHARED) atomicAdd(&s_cq.waiting, 1);
            }
            idle = true;
            const unsigned prog = ld_volatile(&a.ctrl->progress);
            const long long now = globaltimer_ns();
            if (idle_since == 0 || prog != idle_progress) {
                idle_since = now;
                idle_progress = prog;
            } else if (now - idle_since > a.timeout_ns) {
                if (lane == 0) set_error(a.ctrl, DEV_ERR_TIMEOUT);
                break;
            }
            __nanosleep(ns);
            if (ns < 2048) ns <<= 1;
        }
        if (idle && lane == 0) {
            atomicSub(&a.ctrl->idle, 1u);
            if (SHARED) atomicSub(&s_cq.waiting, 1);
        }
        return __shfl_sync(FULL, got ? 1 : 0, 0) != 0;
    }
    __device__ void done(const EngineArgs& a, int lane) {
        if (lane == 0) {
            atomicAdd(&a.ctrl->progress, 1u);
            atomicSub(&a.ctrl->pending, 1);  // after this entry's insertions
        }
        // share: the global stack is empty while CTAs elsewhere wait
        int share = 0;
        if (lane == 0 && cq_count() >= 2 && stack_top(a.ctrl) == 0 &&
            ld_volatile(&a.ctrl->idle) > (SHARED ? (unsigned)*(volatile int*)&s_cq.waiting : 0u))
            share = 1;
        if (__shfl_sync(FULL, share, 0)) cta_spill<SHARED>(a, lane, __shfl_sync(FULL, cq_count(), 0) / 2);
    }
};

// Ring positions 0..n0-1 are the initial tiles (no storage: every tile in
// id order, or the seed list after the front stage); position p >= n0 lives in
// slot (p - n0) % cap.  A CTA claims the next position with one atomicAdd and
// waits for a producer to fill it.  Every filled position is claimed by
// exactly one CTA, and when `pending` (filled, unfinished entries) reaches
// zero no producer is left: the CTA that finishes the last entry sets `done`
// and fills the slots that CTAs wait at with kRingEnd, so a waiting CTA
// watches its own slot and hardly ever the job's counters.
constexpr unsigned kRingEnd = 0xffffffffu;

struct AsyncQueue {
    static constexpr int VAR = VAR_ASYNC;
    unsigned* wq = nullptr;
    unsigned n0 = 0;

    __device__ void start(const EngineArgs& a, int) { n0 = ring_base(a); }
    __device__ bool get(const EngineArgs& a, int lane, unsigned* out) {
        unsigned p = 0u;
        if (lane == 0) p = atomicAdd(&a.ctrl->ahead, 1u);
        p = __shfl_sync(FULL, p, 0);
        if (p < n0) {
            *out = a.init_list ? __ldcg(&a.init_list[p]) : p;
            return names_a_tile(a, lane, *out);
        }
        unsigned v = 0u;
        if (lane == 0) {
            const unsigned slot = (p - n0) % a.cap;
            long long idle_since = globaltimer_ns();
            unsigned idle_progress = 0u;
            unsigned ns = 32, spins = 0;
            for (;;) {
                // The slot is this CTA's alone: watch it with plain loads (a
                // waiting CTA issues no atomics) and take it once set.
                if (ld_volatile(&a.q0[slot]) != 0u) {
                    v = atomicExch(&a.q0[slot], 0u);
                    break;
                }
                // the end of the job at the first look and now and then,
                // progress (for the bound on the wait) rarely
                if ((spins & 15u) == 0u && (ld_volatile(&a.ctrl->done) != 0u || ld_volatile(&a.ctrl->error) != 0u)) {
                    v = kRingEnd;
                    break;
                }
                if ((++spins & 63u) == 0u) {
                    const unsigned prog = ld_volatile(&a.ctrl->progress);
                    const long long now = globaltimer_ns();
                    if (prog != idle_progress) {
                        idle_progress = prog;
                        idle_since = now;
                    } else if (now - idle_since > a.timeout_ns) {
                        set_error(a.ctrl, DEV_ERR_TIMEOUT);
                        v = kRingEnd;
                        break;
                    }
                }
                __nanosleep(ns);
                if (ns < 256) ns <<= 1;
            }
        }
        v = __shfl_sync(FULL, v, 0);
        *out = v - 1u;
        return v != kRingEnd && names_a_tile(a, lane, *out);
    }
    __device__ void done(const EngineArgs& a, int lane) {
        unsigned last = 0u, from = 0u, to = 0u;
        if (lane == 0) {
            atomicAdd(&a.ctrl->progress, 1u);
            // after this entry's insertions, which counted themselves first
            last = atomicSub(&a.ctrl->pending, 1) == 1 ? 1u : 0u;
            if (last) {
                // `done` first: a CTA that claims a position after `ahead` is
                // read here sees it at its first look
                atomicExch(&a.ctrl->done, 1u);
                __threadfence();
                from = ld_volatile(&a.ctrl->atail);
                to = ld_volatile(&a.ctrl->ahead);
            }
        }
        if (!__shfl_sync(FULL, last, 0)) return;
        from = __shfl_sync(FULL, from, 0);
        to = __shfl_sync(FULL, to, 0);
        // at most one claimed position per worker of the grid, fewer than `cap`
        for (unsigned p = from + (unsigned)lane; (int)(to - p) > 0; p += 32u)
            *(volatile unsigned*)&a.q0[(p - n0) % a.cap] = kRingEnd;
    }
};

// --------------------------------------------------------- grid barrier
// All workers of the (cooperative) launch.  The last one to arrive performs the
// round transition.  Waits are bounded; returns false when the job failed.
template <int WORKERS>
__device__ inline bool grid_barrier_round(const EngineArgs& a) {
    int ok = 1;
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
        Ctrl* c = a.ctrl;
        const unsigned gen = ld_volatile(&c->bar_gen);
        __threadfence();
        const unsigned arrived = atomicAdd(&c->bar_count, 1u);
        // (with the phantom-work test hook the barrier waits for one worker
        // more than the grid has, so every waiter runs out of time)
        if (arrived == gridDim.x * WORKERS - 1u + (a.phantom ? 1u : 0u)) {
            // Round transition (IWPP MP DQ/src/globalQueue.cu:139-157 swapQueues,
            // UQ/src/globalQueue.cu:159-168 resetReadQueue, and the overflow
            // restart of DQ/MR.cu:1242-1323, all on the device).
            __threadfence();
            const unsigned wn = ld_volatile(&c->wn);
            unsigned rn;
            if (ld_volatile(&c->overflow) != 0u) {
                if ((int)c->restarts >= a.max_restarts) {
                    set_error(c, DEV_ERR_OVERFLOW);
                    rn = 0u;
                } else {
                    c->restarts += 1u;
                    c->vfull = 1u;
                    rn = a.G;
                }
                c->overflow = 0u;
            } else {
                c->vfull = 0u;
                rn = wn < a.cap ? wn : a.cap;
            }
            c->qsel ^= 1u;
            c->rn = rn;
            c->wn = 0u;
            c->rcur = 0u;
            c->rounds += 1u;
            if (rn == 0u || ld_volatile(&c->error) != 0u) c->done = 1u;
            c->bar_count = 0u;
            __threadfence();
            atomicAdd(&c->bar_gen, 1u);
        } else {
            const long long t0 = globaltimer_ns();
            unsigned ns = 64;
            while (ld_volatile(&c->bar_gen) == gen) {
                __nanosleep(ns);
                if (ns < 2048) ns <<= 1;
                if (ld_volatile(&c->error) != 0u) {
                    ok = 0;
                    break;
                }
                if (globaltimer_ns() - t0 > a.timeout_ns) {
                    set_error(c, DEV_ERR_TIMEOUT);
                    ok = 0;
                    break;
                }
            }
            __threadfence();
        }
    }
    return __shfl_sync(FULL, ok, 0) != 0;
}

// ------------------------------------------------------- round queues
template <int V, int WORKERS>
struct RoundQueue {
    static constexpr int VAR = V;
    unsigned* wq = nullptr;
    unsigned rn = 0, vfull = 0;

    __device__ void start(const EngineArgs& a, int) {
        rn = ld_volatile(&a.ctrl->rn);
        vfull = ld_volatile(&a.ctrl->vfull);
        wq = ld_volatile(&a.ctrl->qsel) ? a.q0 : a.q1;
    }
    __device__ bool get(const EngineArgs& a, int lane, unsigned* out) {
        for (;;) {
            unsigned idx = 0u;
            if (lane == 0) idx = atomicAdd(&a.ctrl->rcur, 1u);
            idx = __shfl_sync(FULL, idx, 0);
            if (idx < rn) {
                *out = vfull ? idx : __ldcg(&(wq == a.q0 ? a.q1 : a.q0)[idx]);
                return names_a_tile(a, lane, *out);
            }
            if (!grid_barrier_round<WORKERS>(a)) return false;
            if (ld_volatile(&a.ctrl->done) != 0u) return false;
            start(a, lane);
        }
    }
    __device__ void done(const EngineArgs&, int) {}
};

template <int VAR, int WORKERS>
struct QueueOf {
    using T = RoundQueue<VAR, WORKERS>;
};
template <int WORKERS>
struct QueueOf<VAR_MUTEX, WORKERS> {
    using T = MutexQueue<WORKERS>;
};
template <int WORKERS>
struct QueueOf<VAR_ASYNC, WORKERS> {
    using T = AsyncQueue;
};

// --------------------------------------------------------------- kernels
// A CTA of W warps works on one tile at a time.  Its first warp runs the
// queue and hands the tile to the CTA's warps through shared memory.  The
// kernels with the alternative in-tile solvers, apart so that their registers
// and code cost the passes nothing, have WORKERS warps that each work on a
// tile of their own (W 1).  Registers: 24 warps per SM (80 registers) with four
// and eight warps per tile, 20 (96) with two, whose loop over a warp's blocks
// needs them; 16 and 32 warps measured the same or slower (32: a fifth slower,
// spills); 12 (168) with one.
constexpr int kAltWorkers = 4;

template <int VAR, int TH, int W, int SOLVE, int CONN>
__global__ void __launch_bounds__(SOLVE == SOLVE_PASSES ? 32 * W : 32 * kAltWorkers,
                                  SOLVE != SOLVE_PASSES ? 12 / kAltWorkers : W == 2 ? 10 : 24 / W)
    engine_kernel(const __grid_constant__ EngineArgs a) {
    constexpr int WORKERS = SOLVE == SOLVE_PASSES ? 1 : kAltWorkers;
    static_assert(WORKERS == 1 || W == 1, "several workers: a warp each");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int worker = WORKERS > 1 ? threadIdx.x >> 5 : 0, warp = WORKERS > 1 ? 0 : threadIdx.x >> 5;
    // 128-byte align the tiles (the launch adds 128 bytes of slack)
    const uint32_t base = smem_u32(smem_raw);
    using Smem = typename SmemOf<TH, W, SOLVE>::T;
    Smem& sm = reinterpret_cast<Smem*>(smem_raw + ((128u - (base & 127u)) & 127u))[worker];
    if (warp == 0 && lane == 0) {
        mbar_init(&sm.mbar, 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        sm.nb = 0u;
        sm.count = VisitCount{};
        if (a.nimg == 1) {
            sm.d = a.one;
            sm.d.tmaps = a.one_tma ? a.one_maps : nullptr;
        } else {
            sm.d = a.imgs[0];
        }
    }
    if constexpr (SOLVE == SOLVE_PASSES) {
        if (lane == 0) sm.mark[0][warp][0] = sm.mark[0][warp][1] = sm.mark[1][warp][0] = sm.mark[1][warp][1] = 0u;
    }
    cta_sync<W>();
    unsigned phase = 0u, row_steps = 0u;
    typename QueueOf<VAR, WORKERS>::T queue;
    if (warp == 0) queue.start(a, lane);
    bool visited = false;  // first warp: tile g was visited
    unsigned g = 0u;
    for (;;) {
        if (warp == 0) {
            bool have = false, found = false;  // an entry in hand (g); a tile to visit (g)
            unsigned sides = 0u;
            if (visited) {
                const long long q0 = clock64();
                const unsigned nb = sm.nb;
                __syncwarp();
                if (lane == 0) sm.nb = 0u;
                // Release: all warps' stores before the neighbours' DIRTY and
                // before the tile's ACTIVE bit clears (its next owner reads
                // them).  By the lanes whose atomics follow, after the barrier
                // that ended the visit.
                if (nb & NB_STORED) fence_gpu();
                int pushed = 0;
                const unsigned cont =
                    leave_tile<VAR, (WORKERS > 1)>(a, sm.d, sm.tx, sm.ty, g, nb, lane, queue.wq, &pushed);
                if (lane == 0) {
                    sm.count.cycles[4] += clock64() - q0;
                    sm.count.visits += 1u;
                    sm.count.pushes += (unsigned)pushed;
                }
                if (cont != ~0u) {
                    g = cont;
                    have = true;
                } else {
                    queue.done(a, lane);
                }
            }
            const long long q0 = clock64();
            while (have || queue.get(a, lane, &g)) {
                have = false;
                if (take_tile(a, g, lane, &sides)) {
                    if (sides != 0u) {
                        found = true;
                        break;
                    }
                    // not DIRTY: released at once, unless it became so
                    bool again = false;
                    if (lane == 0) again = (atomicAnd(&a.state[g], ~ST_ACTIVE) & ST_DIRTY) != 0u;
                    const int pushed =
                        VAR == VAR_MUTEX ? cta_push<(WORKERS > 1)>(a, again, g, lane)
                                         : push_entries<VAR>(a, again, g, lane, queue.wq);
                    if (lane == 0) sm.count.pushes += (unsigned)pushed;
                }
                queue.done(a, lane);
            }
            if (found && a.nimg != 1 &&
                !(g - (unsigned)sm.d.tile_base < (unsigned)(sm.d.tiles_x * sm.d.tiles_y))) {
                // another image of the batch
                const int ii = find_image(a, g);
                __syncwarp();
                const unsigned* src = reinterpret_cast<const unsigned*>(&a.imgs[ii]);
                if (lane < (int)(sizeof(ImgDesc) / 4)) reinterpret_cast<unsigned*>(&sm.d)[lane] = __ldg(&src[lane]);
                __syncwarp();
            }
            if (found) {
                const int t = (int)(g - (unsigned)sm.d.tile_base), ty = t / sm.d.tiles_x;
                if (lane == 0) {
                    sm.ty = ty;
                    sm.tx = t - ty * sm.d.tiles_x;
                    sm.sides = sides;
                }
            }
            if (lane == 0) {
                sm.go = found ? 1u : 0u;
                sm.count.cycles[0] += clock64() - q0;
            }
            visited = found;
        }
        cta_sync<W>();
        if (sm.go == 0u) break;
        EarlyFlush<VAR> early{a, sm.d, sm.tx, sm.ty, sm.count.pushes, (int)(gridDim.x * WORKERS / 2u)};
        if (!dispatch_visit<CONN, TH, W, SOLVE>(a, sm, warp, lane, phase, row_steps, early)) {
            if (warp == 0 && lane == 0) set_error(a.ctrl, DEV_ERR_TIMEOUT);
            break;
        }
    }
    if (lane == 0) {
        if (row_steps) atomicAdd(&a.ctrl->row_steps, (unsigned long long)row_steps);
        if (warp == 0) {
            const VisitCount& c = sm.count;
            if (c.visits) atomicAdd(&a.ctrl->visits, (unsigned long long)c.visits);
            if (c.sweeps) atomicAdd(&a.ctrl->sweeps, (unsigned long long)c.sweeps);
            if (c.pushes) atomicAdd(&a.ctrl->pushes, (unsigned long long)c.pushes);
            for (int i = 0; i < 5; ++i)
                if (c.cycles[i] > 0) atomicAdd(&a.ctrl->phase[i], (unsigned long long)c.cycles[i]);
        }
    }
}

template <int VAR, int CONN>
void* kernel_for(int tile_rows, int warps) {
    if (tile_rows == 32) return reinterpret_cast<void*>(&engine_kernel<VAR, 32, 4, SOLVE_PASSES, CONN>);
    if (warps == 8) return reinterpret_cast<void*>(&engine_kernel<VAR, 64, 8, SOLVE_PASSES, CONN>);
    if (warps == 4) return reinterpret_cast<void*>(&engine_kernel<VAR, 64, 4, SOLVE_PASSES, CONN>);
    return reinterpret_cast<void*>(&engine_kernel<VAR, 64, 2, SOLVE_PASSES, CONN>);
}

template <int VAR, int SOLVE>
void* kernel_for(int tile_rows) {
    return tile_rows == 32 ? reinterpret_cast<void*>(&engine_kernel<VAR, 32, 1, SOLVE, 0>)
                           : reinterpret_cast<void*>(&engine_kernel<VAR, 64, 1, SOLVE, 0>);
}

// The kernel of a queue and an in-tile solver (SOLVE_*) for tiles of a shape and
// images of one connectivity (4, 8) or of both (0).
template <int VAR>
void* kernel_for(int tile_rows, int warps, int solve, int conn) {
    return solve == SOLVE_SWEEPS ? kernel_for<VAR, SOLVE_SWEEPS>(tile_rows)
           : solve == SOLVE_PQ   ? kernel_for<VAR, SOLVE_PQ>(tile_rows)
           : conn == 4           ? kernel_for<VAR, 4>(tile_rows, warps)
           : conn == 8           ? kernel_for<VAR, 8>(tile_rows, warps)
                                 : kernel_for<VAR, 0>(tile_rows, warps);
}

// Each queue's kernels are a translation unit of their own
// (iwpp_engine_{mutex,double,unique,async}.cu): they take long to compile.
extern template void* kernel_for<VAR_MUTEX>(int, int, int, int);
extern template void* kernel_for<VAR_DOUBLE>(int, int, int, int);
extern template void* kernel_for<VAR_UNIQUE>(int, int, int, int);
extern template void* kernel_for<VAR_ASYNC>(int, int, int, int);

}  // namespace iwpp
