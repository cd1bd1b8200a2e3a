// song_search.cuh -- sm_100a kernels of the SONG graph search (device code
// and instance selection; the song_search*.cu files hold the instances).
//
// One warp owns one query at a time; several warps share a CTA and a
// persistent grid pulls queries from a device work counter, so every SM
// keeps many independent traversals (and their neighbour gathers) in flight.
// The reference runs one query per single-warp block with lane 0 doing all
// queue and Bloom work serially (kernalGraph.h:184-299).
//
// Results are bit-exact with the reference, including tie order and the
// QueryTrace counters, because the per-query state is the reference's own
// state and every step keeps its order:
//  * Candidates / Results (gpuHeap.h:8-108) stay unsorted slot arrays in
//    shared memory with exactly the reference's slot moves.  The O(cap)
//    scans become a two-level tournament: slots are grouped 32 at a time
//    (one slot per lane), each group's (max, first slot) and (min, first
//    slot) summary lives in a register of lane g, and "first maximal slot"
//    or "first minimal slot" is two redux.sync over those summaries.  A slot
//    write refreshes only its group (one shared load per lane + redux).
//    Ties break on the lowest slot -- the reference's first-index rule.
//  * A row of up to 32 neighbours is handled at once, lane j = slot j, but
//    the Bloom test of neighbour j sees the bits of neighbours < j exactly as
//    bf_test/bf_set in j order do (bloomFilter.h:34-48): see bloom_test.
//  * Distances follow warp_l2 (kernalGraph.h:157-170): 32 partial sums of
//    (q_i - b_i)^2 over i = l (mod 32) with FMA, then the reference's
//    shfl_down tree.  Only the rows that passed the Bloom test are read, 8
//    lanes per row with 16-byte loads, each lane holding four of the partial
//    sums (l2_rows).  Integer vectors in [0, 255] (the SIFT-shaped case) are
//    read as bytes instead: every order of exact integer sums gives the same
//    FP32 value (l2_u8).
//  * Pushes are applied in lane (= j) order; a push into a full queue only
//    evicts when strictly closer than the current first maximum, and the
//    maximum never grows while a queue is full, so lanes that lose against
//    the running maximum drop out with one ballot.
//  * The final trim (pop_worst) and drain (drain_best) are replayed exactly;
//    when the k+1 smallest results have distinct distances their outcome is
//    simply those k in ascending order, which is taken directly.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <type_traits>

#include "song_kernels.cuh"

namespace song {

extern std::atomic<int64_t> g_launches;

using KernelFn = void (*)(const SearchArgs);

// A chosen kernel instance and its launch shape.
struct KernelSel {
    KernelFn fn = nullptr;      // candidate ids in shared memory
    KernelFn fn_tmc = nullptr;  // tm only: the candidate ids in TMEM too
    KernelFn fn_tmd = nullptr;  // tm only, not all: result distances in TMEM too
    KernelFn fn_nt = nullptr;   // the three without the trace, where they exist
    KernelFn fn_tmc_nt = nullptr;
    KernelFn fn_tmd_nt = nullptr;
    int tm = 0;                 // result ids in TMEM (the CTA allocates tensor memory)
    int qr = 0;                 // queues in registers: up to 32 * qr slots
    int threads = 256;
    bool query_smem = true;
};

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr unsigned NONE = 0xffffffffu;  // "no slot" / empty group

// The mixing constants of bloomFilter.h:14-19: two per hash function.
__constant__ uint64_t kBloomMix[8] = {
    0x4bcb391f924ed183ULL, 0xa0ab69ccd854fc0aULL, 0x91086b9cecf5e3b7ULL, 0xc68e01641bead407ULL,
    0x3a7b976128a30449ULL, 0x6d122efabfc4d99fULL, 0xe6700ef8715030e2ULL, 0x80dd0c3bffcfb45bULL,
};

__device__ __forceinline__ unsigned fbits(float x) { return __float_as_uint(x); }

inline int round_up(int x, int m) { return (x + m - 1) / m * m; }

// Read-only loads of base rows (the read-only data path; an L1 no-allocate
// variant measured slightly slower).
__device__ __forceinline__ float4 ld_row(const float4* p) { return __ldg(p); }
__device__ __forceinline__ uint4 ld_row(const uint4* p) { return __ldg(p); }
__device__ __forceinline__ unsigned lanemask_lt(int lane) { return (1u << lane) - 1u; }

// Tensor memory (TMEM) access of one warp: 32 lanes x 32-bit columns.  The
// wait is part of the same asm statement, so the loaded value is never used
// before the load has completed, and a store has completed before the next
// access of the same column.
__device__ __forceinline__ unsigned tm_ld(uint32_t taddr) {
    unsigned r;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r)
        : "r"(taddr)
        : "memory");
    return r;
}
// Two columns with one wait.
__device__ __forceinline__ void tm_ld2(uint32_t a0, uint32_t a1, unsigned& r0, unsigned& r1) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%2];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x1.b32 {%1}, [%3];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r0), "=r"(r1)
        : "r"(a0), "r"(a1)
        : "memory");
}
__device__ __forceinline__ void tm_st(uint32_t taddr, unsigned v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};\n\t"
        "tcgen05.wait::st.sync.aligned;"
        :
        : "r"(taddr), "r"(v)
        : "memory");
}
// Two columns with one wait.
__device__ __forceinline__ void tm_st2(uint32_t a0, uint32_t a1, unsigned v0, unsigned v1) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%2};\n\t"
        "tcgen05.st.sync.aligned.32x32b.x1.b32 [%1], {%3};\n\t"
        "tcgen05.wait::st.sync.aligned;"
        :
        : "r"(a0), "r"(a1), "r"(v0), "r"(v1)
        : "memory");
}

// Slot queue of capacity <= 1024 * GPL.  Distances live in shared memory;
// ids live in shared memory (TM = 0) or in the warp's 32 TMEM lanes, one
// column per group of 32 slots, slot 32g + l at lane l of column tid + g
// (TM = 1).  TD = 1 (with TM = 1): the distances too, in the columns from
// tdd on, laid out like the ids.  The summary of group g (slots 32g ..
// 32g+31) is held by lane g % 32 in entry g / 32.  Distances are
// non-negative, so their bit patterns order like the floats.  All scalar
// fields are warp-uniform.
template <int GPL, int TM = 0, int TD = 0>
struct Queue {
    float* d;      // TD = 0
    int* id;       // TM = 0
    uint32_t tid;  // TM = 1: TMEM address of group 0's id column
    uint32_t tdd;  // TD = 1: TMEM address of group 0's distance column
    int sz;
    int cap;
    unsigned xb[GPL], xi[GPL];  // group maximum bits, first slot holding it (NONE = empty)
    unsigned nb[GPL], ni[GPL];  // group minimum bits, first slot holding it
    // The queue's maximum and its first slot while cx holds (results queue
    // only: its maximum is read at every early-stop check and push): kept
    // through appends and evictions instead of recomputed from the group
    // summaries each time.
    unsigned cxb, cxi;
    bool cx;
};

// Id of slot s (warp-uniform s; every lane gets it).
template <int GPL, int TM, int TD>
__device__ __forceinline__ int q_id(const Queue<GPL, TM, TD>& q, int s) {
    if constexpr (TM) {
        const unsigned r = tm_ld(q.tid + (uint32_t)(s >> 5));
        return (int)__shfl_sync(FULL, r, s & 31);
    } else {
        return q.id[s];
    }
}

// Id of slot s := v (warp-uniform s and v; called by every lane).
template <int GPL, int TM, int TD>
__device__ __forceinline__ void q_set_id(Queue<GPL, TM, TD>& q, int s, int v, int lane) {
    if constexpr (TM) {
        const uint32_t a = q.tid + (uint32_t)(s >> 5);
        unsigned r = tm_ld(a);
        if (lane == (s & 31)) r = (unsigned)v;
        tm_st(a, r);
    } else {
        if (lane == 0) q.id[s] = v;
    }
}

// Distance bits of slot s (warp-uniform s; every lane gets them).
template <int GPL, int TM, int TD>
__device__ __forceinline__ unsigned q_dbits(const Queue<GPL, TM, TD>& q, int s) {
    if constexpr (TD) {
        const unsigned r = tm_ld(q.tdd + (uint32_t)(s >> 5));
        return __shfl_sync(FULL, r, s & 31);
    } else {
        return fbits(q.d[s]);
    }
}

// Slot s := (distance bits b, id v) (warp-uniform s, b, v; called by every
// lane).  TD: both columns read with one wait.
template <int GPL, int TM, int TD>
__device__ __forceinline__ void q_set_slot(Queue<GPL, TM, TD>& q, int s, unsigned b, int v, int lane) {
    if constexpr (TD) {
        const uint32_t ai = q.tid + (uint32_t)(s >> 5), ad = q.tdd + (uint32_t)(s >> 5);
        unsigned ri, rd;
        tm_ld2(ai, ad, ri, rd);
        if (lane == (s & 31)) {
            ri = (unsigned)v;
            rd = b;
        }
        tm_st2(ai, ad, ri, rd);
    } else {
        if (lane == 0) reinterpret_cast<unsigned*>(q.d)[s] = b;
        q_set_id(q, s, v, lane);
    }
}

// Distance bits of slot s := b (warp-uniform s and b; called by every lane).
template <int GPL, int TM, int TD>
__device__ __forceinline__ void q_set_dbits(Queue<GPL, TM, TD>& q, int s, unsigned b, int lane) {
    if constexpr (TD) {
        const uint32_t ad = q.tdd + (uint32_t)(s >> 5);
        unsigned r = tm_ld(ad);
        if (lane == (s & 31)) r = b;
        tm_st(ad, r);
    } else {
        if (lane == 0) reinterpret_cast<unsigned*>(q.d)[s] = b;
    }
}

template <int GPL, int TM, int TD>
__device__ __forceinline__ void q_init(Queue<GPL, TM, TD>& q, float* d, int* id, uint32_t tid,
                                       uint32_t tdd, int cap) {
    q.d = d;
    q.id = id;
    q.tid = tid;
    q.tdd = tdd;
    q.sz = 0;
    q.cap = cap;
    q.cx = false;
#pragma unroll
    for (int r = 0; r < GPL; ++r) {
        q.xb[r] = 0u;
        q.xi[r] = NONE;
        q.nb[r] = 0xffffffffu;
        q.ni[r] = NONE;
    }
}

// Refresh the summary of group g from the slot array.  MIN: also the minimum.
// `b`: this lane's slot's distance bits (0 if the slot is empty).
template <bool MIN, int GPL, int TM, int TD>
__device__ __forceinline__ void group_update_b(Queue<GPL, TM, TD>& q, int g, int lane, unsigned b) {
    const int s = (g << 5) + lane;
    const bool occ = s < q.sz;
    const unsigned mx = __reduce_max_sync(FULL, b);
    const unsigned mxi = __reduce_min_sync(FULL, (occ && b == mx) ? (unsigned)s : NONE);
    unsigned mn = 0xffffffffu, mni = NONE;
    if constexpr (MIN) {
        mn = __reduce_min_sync(FULL, occ ? b : 0xffffffffu);
        mni = __reduce_min_sync(FULL, (occ && b == mn) ? (unsigned)s : NONE);
    }
    if ((g & 31) == lane) {
        const int r = g >> 5;
#pragma unroll
        for (int t = 0; t < GPL; ++t) {
            if (t == r) {
                q.xb[t] = mx;
                q.xi[t] = mxi;
                if constexpr (MIN) {
                    q.nb[t] = mn;
                    q.ni[t] = mni;
                }
            }
        }
    }
}

template <bool MIN, int GPL, int TM, int TD>
__device__ __forceinline__ void group_update(Queue<GPL, TM, TD>& q, int g, int lane) {
    const bool occ = (g << 5) + lane < q.sz;
    unsigned b;
    if constexpr (TD) {
        const unsigned c = tm_ld(q.tdd + (uint32_t)g);
        b = occ ? c : 0u;
    } else {
        b = occ ? fbits(q.d[(g << 5) + lane]) : 0u;
    }
    group_update_b<MIN>(q, g, lane, b);
}

// First slot holding the maximum over [0, sz) (gpuHeap.h:29, :73, :83, :93).
template <int GPL, int TM, int TD>
__device__ __forceinline__ void root_max(const Queue<GPL, TM, TD>& q, unsigned& mb, unsigned& mi) {
    unsigned b = 0u, i = NONE;
#pragma unroll
    for (int r = 0; r < GPL; ++r)
        if (q.xi[r] != NONE && (i == NONE || q.xb[r] > b)) {
            b = q.xb[r];
            i = q.xi[r];
        }
    mb = __reduce_max_sync(FULL, i != NONE ? b : 0u);
    mi = __reduce_min_sync(FULL, (i != NONE && b == mb) ? i : NONE);
}

// First slot holding the minimum over [0, sz) (gpuHeap.h:42, :263).
template <int GPL, int TM, int TD>
__device__ __forceinline__ void root_min(const Queue<GPL, TM, TD>& q, unsigned& mb, unsigned& mi) {
    unsigned b = 0xffffffffu, i = NONE;
#pragma unroll
    for (int r = 0; r < GPL; ++r)
        if (q.ni[r] != NONE && (i == NONE || q.nb[r] < b)) {
            b = q.nb[r];
            i = q.ni[r];
        }
    mb = __reduce_min_sync(FULL, i != NONE ? b : 0xffffffffu);
    mi = __reduce_min_sync(FULL, (i != NONE && b == mb) ? i : NONE);
}

// Move the last slot into slot `hole` and shrink (the removal of
// Candidates::pop_min, Results::pop_worst and drain_best).
template <bool MIN, int GPL, int TM, int TD>
__device__ __forceinline__ void q_remove(Queue<GPL, TM, TD>& q, int hole, int lane) {
    const int last = q.sz - 1;
    __syncwarp();
    if (hole != last) {
        if constexpr (TD) {
            q_set_slot(q, hole, q_dbits(q, last), q_id(q, last), lane);
        } else if constexpr (TM) {
            if (lane == 0) q.d[hole] = q.d[last];
            q_set_id(q, hole, q_id(q, last), lane);
        } else {
            if (lane == 0) q.d[hole] = q.d[last];
            if (lane == 0) q.id[hole] = q.id[last];
        }
    }
    __syncwarp();
    q.sz = last;
    q.cx = false;
    group_update<MIN>(q, hole >> 5, lane);
    if ((last >> 5) != (hole >> 5)) group_update<MIN>(q, last >> 5, lane);
}

// Maximum and its first slot (gpuHeap.h:29, :73), from the cache when it holds.
template <int GPL, int TM, int TD>
__device__ __forceinline__ void root_max_c(Queue<GPL, TM, TD>& q, unsigned& mb, unsigned& mi) {
    if (!q.cx) {
        root_max(q, q.cxb, q.cxi);
        q.cx = true;
    }
    mb = q.cxb;
    mi = q.cxi;
}

// Id of slot `hole`, then q_remove(hole): the same queue afterwards, with the
// TMEM columns of `hole` and of the last slot read once (one wait) instead
// of once per id access.
template <bool MIN, int GPL, int TM, int TD>
__device__ __forceinline__ int q_pop(Queue<GPL, TM, TD>& q, int hole, int lane) {
    static_assert(!TD, "pops serve the candidate queue, whose distances are in shared memory");
    if constexpr (!TM) {
        const int id = q.id[hole];
        q_remove<MIN>(q, hole, lane);
        return id;
    } else {
        const int last = q.sz - 1;
        const uint32_t ch = q.tid + (uint32_t)(hole >> 5), cl = q.tid + (uint32_t)(last >> 5);
        unsigned rh, rl;
        if (ch == cl) {
            rh = tm_ld(ch);
            rl = rh;
        } else {
            tm_ld2(ch, cl, rh, rl);
        }
        const int id = (int)__shfl_sync(FULL, rh, hole & 31);
        const unsigned idl = __shfl_sync(FULL, rl, last & 31);
        __syncwarp();
        if (hole != last) {
            if (lane == 0) q.d[hole] = q.d[last];
            if (lane == (hole & 31)) rh = idl;
            tm_st(ch, rh);
        }
        __syncwarp();
        q.sz = last;
        q.cx = false;
        group_update<MIN>(q, hole >> 5, lane);
        if ((last >> 5) != (hole >> 5)) group_update<MIN>(q, last >> 5, lane);
        return id;
    }
}

// Push (d, nb) of every lane in N, in lane order, with the semantics of
// Candidates::push / Results::try_push (gpuHeap.h:23-36, :68-77).
// Returns how many pushes were accepted.  `stage` (32 ints, TM = 1 only)
// receives the ids in rank order for the column writes of an append.
// RC: keep the queue's cached maximum (cxb, cxi) current.
template <bool MIN, bool RC = false, int GPL, int TM, int TD>
__device__ __forceinline__ int q_push(Queue<GPL, TM, TD>& q, unsigned N, float d, int nb, int lane,
                                      int* stage) {
    if (N == 0u) return 0;
    const bool mine = (N >> lane) & 1u;
    const int rank = __popc(N & lanemask_lt(lane));
    const int nm = __popc(N);
    const int room = q.cap - q.sz;
    int acc = 0;
    if (room > 0) {
        const int a = nm < room ? nm : room;
        if (mine && rank < a) {
            if constexpr (TD) stage[32 + rank] = (int)fbits(d);
            else q.d[q.sz + rank] = d;
            if constexpr (TM) stage[rank] = nb;
            else q.id[q.sz + rank] = nb;
        }
        __syncwarp();
        const int g0 = q.sz >> 5, g1 = (q.sz + a - 1) >> 5;
        if constexpr (TD) {  // ids and distances, column by column; each group's summary from its column
            const int sz0 = q.sz;
            q.sz += a;
            for (int g = g0; g <= g1; ++g) {
                const uint32_t ci = q.tid + (uint32_t)g, cd = q.tdd + (uint32_t)g;
                unsigned ri, rd;
                tm_ld2(ci, cd, ri, rd);
                const int rr = (g << 5) + lane - sz0;
                if (rr >= 0 && rr < a) {
                    ri = (unsigned)stage[rr];
                    rd = (unsigned)stage[32 + rr];
                }
                tm_st2(ci, cd, ri, rd);
                group_update_b<MIN>(q, g, lane, (g << 5) + lane < q.sz ? rd : 0u);
            }
            q.sz = sz0;
            __syncwarp();
        } else if constexpr (TM) {  // slots sz .. sz+a-1 take the staged ids, column by column
            for (int g = g0; g <= g1; ++g) {
                const uint32_t col = q.tid + (uint32_t)g;
                unsigned r = tm_ld(col);
                const int rr = (g << 5) + lane - q.sz;
                if (rr >= 0 && rr < a) r = (unsigned)stage[rr];
                tm_st(col, r);
            }
            __syncwarp();
        }
        if (RC && q.cx) {  // the appended entries sit after every slot: only a larger one moves the maximum
            const bool app = mine && rank < a;
            const unsigned am = __reduce_max_sync(FULL, app ? fbits(d) : 0u);
            if (am > q.cxb) {
                const int fl = __ffs(__ballot_sync(FULL, app && fbits(d) == am)) - 1;
                q.cxb = am;
                q.cxi = (unsigned)(q.sz + __popc(N & lanemask_lt(fl)));
            }
        }
        q.sz += a;
        if constexpr (!TD)
            for (int g = g0; g <= g1; ++g) group_update<MIN>(q, g, lane);
        acc = a;
    }
    if (nm > room) {
        unsigned M, fi;
        if constexpr (RC) root_max_c(q, M, fi);
        else root_max(q, M, fi);
        unsigned rest = __ballot_sync(FULL, mine && rank >= room && fbits(d) < M);
        while (rest) {
            const int j = __ffs(rest) - 1;
            const float dj = __shfl_sync(FULL, d, j);
            const int nj = __shfl_sync(FULL, nb, j);
            if constexpr (TD) {  // the slot's two columns, then the group's summary from the distance column
                const int g = (int)(fi >> 5);
                const uint32_t ci = q.tid + (uint32_t)g, cd = q.tdd + (uint32_t)g;
                unsigned ri, rd;
                tm_ld2(ci, cd, ri, rd);
                if (lane == (int)(fi & 31)) {
                    ri = (unsigned)nj;
                    rd = fbits(dj);
                }
                tm_st2(ci, cd, ri, rd);
                group_update_b<MIN>(q, g, lane, (g << 5) + lane < q.sz ? rd : 0u);
            } else {
                if (lane == 0) q.d[fi] = dj;
                q_set_id(q, (int)fi, nj, lane);
                __syncwarp();
                group_update<MIN>(q, (int)(fi >> 5), lane);
            }
            ++acc;
            root_max(q, M, fi);
            rest &= ~(1u << j);
            rest &= __ballot_sync(FULL, fbits(d) < M);
        }
        if constexpr (RC) {
            q.cxb = M;
            q.cxi = fi;
            q.cx = true;
        }
    }
    return acc;
}

// The same slot queue for up to 32 * R slots with its distances in registers:
// slot 32 r + l is d[r] of lane l (kEmpty past sz: the largest value unsigned,
// the smallest signed), ids in shared memory.  Maximum, minimum and every
// slot write are a few instructions on registers and two redux.sync, where
// the queue above goes through shared memory and the group summaries: a push
// into a full queue is a chain of about 200 cycles instead of 330 (measured,
// one warp alone), and it needs neither TMEM nor shared memory for distances.
// The work per operation grows with R and passes the summaries' at R = 8
// (launch_search has the figures).
constexpr unsigned kEmpty = 0xffffffffu;
template <int R>
struct RQueue {
    unsigned d[R];
    int* id;
    int sz;
    int cap;
    // maximum and its first slot while cx; minimum and its first slot while nx
    unsigned cxb, cxi, nxb, nxi;
    bool cx, nx;
};

// x := r == key ? v : x.  As one asm statement, or the compiler turns a chain
// of these over r into an indexed access and moves the queue to local memory.
__device__ __forceinline__ void pick_if(unsigned& x, int r, int key, unsigned v) {
    asm("{\n\t.reg .pred p;\n\t"
        "setp.eq.s32 p, %1, %2;\n\t"
        "selp.b32 %0, %3, %0, p;\n\t}"
        : "+r"(x) : "r"(r), "r"(key), "r"(v));
}

template <int R>
__device__ __forceinline__ void q_init(RQueue<R>& q, int* id, int cap) {
#pragma unroll
    for (int r = 0; r < R; ++r) q.d[r] = kEmpty;
    q.id = id;
    q.sz = 0;
    q.cap = cap;
    q.cx = q.nx = false;
}

// Slot whose distance bits are `b`, the lowest of them (some slot holds b).
// (Ballots over the registers instead of the redux measured twice as slow.)
template <int R>
__device__ __forceinline__ unsigned first_slot(const RQueue<R>& q, unsigned b, int lane) {
    unsigned f = NONE;
#pragma unroll
    for (int r = R - 1; r >= 0; --r)
        if (q.d[r] == b) f = (unsigned)(32 * r + lane);
    return __reduce_min_sync(FULL, f);
}

template <int R>
__device__ __forceinline__ void root_max(const RQueue<R>& q, unsigned& mb, unsigned& mi, int lane) {
    int m = (int)q.d[0];
#pragma unroll
    for (int r = 1; r < R; ++r) m = max(m, (int)q.d[r]);
    mb = (unsigned)__reduce_max_sync(FULL, m);
    mi = first_slot(q, mb, lane);
}

template <int R>
__device__ __forceinline__ void root_min(const RQueue<R>& q, unsigned& mb, unsigned& mi, int lane) {
    unsigned m = q.d[0];
#pragma unroll
    for (int r = 1; r < R; ++r) m = min(m, q.d[r]);
    mb = __reduce_min_sync(FULL, m);
    mi = first_slot(q, mb, lane);
}

template <int R>
__device__ __forceinline__ void root_max_c(RQueue<R>& q, unsigned& mb, unsigned& mi, int lane) {
    if (!q.cx) {
        root_max(q, q.cxb, q.cxi, lane);
        q.cx = true;
    }
    mb = q.cxb;
    mi = q.cxi;
}

template <int R>
__device__ __forceinline__ void root_min_c(RQueue<R>& q, unsigned& mb, unsigned& mi, int lane) {
    if (!q.nx) {
        root_min(q, q.nxb, q.nxi, lane);
        q.nx = true;
    }
    mb = q.nxb;
    mi = q.nxi;
}

// Distance bits of slot s := b (warp-uniform s and b).
template <int R>
__device__ __forceinline__ void q_set_dbits(RQueue<R>& q, int s, unsigned b, int lane) {
    const int key = lane == (s & 31) ? s >> 5 : -1;
#pragma unroll
    for (int r = 0; r < R; ++r) pick_if(q.d[r], r, key, b);
}

// Move the last slot into slot `hole` and shrink.
template <int R>
__device__ __forceinline__ void q_remove(RQueue<R>& q, int hole, int lane) {
    const int last = q.sz - 1;
    unsigned x = q.d[0];
#pragma unroll
    for (int r = 1; r < R; ++r) pick_if(x, r, last >> 5, q.d[r]);
    x = __shfl_sync(FULL, x, last & 31);
    __syncwarp();
    if (lane == 0) q.id[hole] = q.id[last];
    __syncwarp();
    q_set_dbits(q, hole, x, lane);
    q_set_dbits(q, last, kEmpty, lane);
    q.sz = last;
    q.cx = q.nx = false;
}

template <int R>
__device__ __forceinline__ int q_pop(RQueue<R>& q, int hole, int lane) {
    const int id = q.id[hole];
    q_remove(q, hole, lane);
    return id;
}

// Push (d, nb) of lanes 0 .. popc(N) - 1 (N is a run of low bits), in lane
// order.  MIN: keep the cached minimum only while no pushed distance reaches
// it.
template <bool MIN, int R>
__device__ __forceinline__ int q_push(RQueue<R>& q, unsigned N, float d, int nb, int lane) {
    if (N == 0u) return 0;
    const int nm = __popc(N);
    const bool mine = lane < nm;
    const unsigned db = fbits(d);
    const int room = q.cap - q.sz;
    int acc = 0;
    if (MIN && q.nx && __ballot_sync(FULL, mine && db <= q.nxb)) q.nx = false;
    if (room > 0) {
        const int a = nm < room ? nm : room;
        const int rk = (lane - q.sz) & 31;  // the push whose slot is one of this lane's
        const unsigned x = __shfl_sync(FULL, db, rk);
        if (mine && lane < a) q.id[q.sz + lane] = nb;
        __syncwarp();
        const int key = rk < a ? (q.sz + rk) >> 5 : -1;
#pragma unroll
        for (int r = 0; r < R; ++r) pick_if(q.d[r], r, key, x);
        q.sz += a;
        q.cx = false;
        acc = a;
    }
    if (nm > room) {
        unsigned M, fi;
        root_max_c(q, M, fi, lane);
        unsigned rest = __ballot_sync(FULL, mine && lane >= room && db < M);
        while (rest) {
            const int j = __ffs(rest) - 1;
            const unsigned dj = __shfl_sync(FULL, db, j);
            // one slot may be evicted again and again, by other lanes: redux and
            // shuffles do not order their writes
            if (lane == j) q.id[fi] = nb;
            __syncwarp();
            q_set_dbits(q, (int)fi, dj, lane);
            if (MIN && fi == q.nxi) q.nx = false;
            ++acc;
            root_max(q, M, fi, lane);
            rest &= ~(1u << j);
            rest &= __ballot_sync(FULL, db < M);
        }
        q.cxb = M;
        q.cxi = fi;
    }
    __syncwarp();
    return acc;
}

struct BloomCfg {
    uint64_t nbits;  // BF_WORDS * 64
    uint32_t words;  // BF_WORDS
    uint32_t wmask;  // BF_WORDS - 1 when a power of two
    int shift;       // log2(BF_WORDS), or -1
    int nhash;       // BF_NHASH
};

// bf_hash (bloomFilter.h:23-30) for a node id x >= 0.  The first x ^= x>>33
// of the reference is the identity for x < 2^33 and is left out.
__device__ __forceinline__ uint64_t bf_mix(int h, uint32_t x) {
    uint64_t y = (uint64_t)x * kBloomMix[2 * h];
    y ^= y >> 33;
    y *= kBloomMix[2 * h + 1];
    return y ^ (y >> 33);
}

// Bloom test-and-set of one chunk of up to 32 ids (lane j = j-th id of the
// row, nb < 0 = empty slot), equivalent to the reference's
//   for j: if (!bf_test(nb_j)) { bf_set(nb_j); new_j = true; }
// in two steps: bloom_test returns the lanes that hold an unset position and
// sets their positions, bloom_new drops from them the lanes that an earlier
// id of the same row covers.
//
// Reference order matters only through bits set by earlier ids of the same
// row: id j is skipped iff each of its positions is in B0 (the filter before
// the row) or is a position of an earlier valid id (an id that was itself
// skipped adds nothing new, so it may be counted too).  Lanes with all
// positions in B0 are skipped.  The others set their missing bits with an
// atomic or; if none ever finds its bit already set, no missing position is
// shared by two lanes and the B0 test alone is exact.  Otherwise (rare with a
// large filter) every lane checks its missing positions against those of the
// lanes before it.  The final filter is B0 plus all positions of the new ids
// either way, as in the reference.
//
// The chain of this test is what an expansion waits for most: the hashes of a
// power-of-two filter are branch-free code (a branch per hash and per
// division took 900 cycles where these take 300), and the rows of the lanes
// that bloom_test returns are read before bloom_new waits for the atomics.
struct BloomRow {
    uint32_t pos[4];  // positions (0xffffffff: unused)
    unsigned unc;     // hashes whose position was unset
    bool event;       // one of them was set by an atomic before this one
};

__device__ __forceinline__ unsigned bloom_test(uint64_t* bloom, int nb, const BloomCfg& bc, BloomRow& br) {
    const uint32_t* words = reinterpret_cast<const uint32_t*>(bloom);
    // the same bit as a 32-bit word: the low half of 64-bit word w is word 2w
    uint32_t wd[4], bt[4];
    if (bc.shift >= 0) {
        const uint32_t mask = (uint32_t)bc.nbits - 1u;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const uint32_t p = (uint32_t)bf_mix(h, (uint32_t)nb) & mask;
            const uint32_t b64 = p >> bc.shift;
            br.pos[h] = p;
            wd[h] = 2u * (p & bc.wmask) + (b64 >> 5);
            bt[h] = 1u << (b64 & 31u);
        }
    } else {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const uint32_t p = (uint32_t)(bf_mix(h, (uint32_t)nb) % bc.nbits);
            const uint32_t b64 = p / bc.words;
            br.pos[h] = p;
            wd[h] = 2u * (p % bc.words) + (b64 >> 5);
            bt[h] = 1u << (b64 & 31u);
        }
    }
    unsigned unc = 0;
#pragma unroll
    for (int h = 0; h < 4; ++h)
        if (!(words[wd[h]] & bt[h])) unc |= 1u << h;
    unc = nb >= 0 ? unc & ((1u << bc.nhash) - 1u) : 0u;
    br.unc = unc;
    __syncwarp();
    // predicated, so that the four are in flight together
    unsigned old[4];
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(bloom);
#pragma unroll
    for (int h = 0; h < 4; ++h)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.u32 p, %3, 0;\n\t"
            "mov.u32 %0, 0;\n\t"
            "@p atom.shared.or.b32 %0, [%1], %2;\n\t}"
            : "=&r"(old[h])
            : "r"(base + 4u * wd[h]), "r"(bt[h]), "r"((unc >> h) & 1u)
            : "memory");
    br.event = ((old[0] & bt[0]) | (old[1] & bt[1]) | (old[2] & bt[2]) | (old[3] & bt[3])) != 0u;
    return __ballot_sync(FULL, unc != 0u);
}

__device__ __forceinline__ unsigned bloom_new(const BloomRow& br, unsigned fresh, const BloomCfg& bc, int lane) {
    if (__ballot_sync(FULL, br.event) == 0u) {
        __syncwarp();
        return fresh;
    }
    unsigned cov = 0;
    unsigned src = fresh;
    while (src) {
        const int i = __ffs(src) - 1;
        src &= src - 1u;
        uint32_t p[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) p[h] = __shfl_sync(FULL, br.pos[h], i);
        if (lane > i && br.unc) {
#pragma unroll
            for (int h = 0; h < 4; ++h)
#pragma unroll
                for (int g = 0; g < 4; ++g)  // a position of a hash that is not used sets nothing
                    if (((br.unc >> h) & 1u) && g < bc.nhash && br.pos[h] == p[g]) cov |= 1u << h;
        }
    }
    __syncwarp();
    return __ballot_sync(FULL, (br.unc & ~cov) != 0u);
}

// Four floats of the query from element i on: 16 aligned bytes of shared
// memory (QG = 0, zero padded to a multiple of 4), or the caller's own row in
// global memory (any alignment, zero past dim): QG = 1 through the read-only
// path, QG = 2 with plain loads, for the serving kernel, whose request slots
// are rewritten while it runs.  (For QG = 1 too, plain loads took 8 % longer at
// 200 dimensions and queue 200, through their registers, and loads from L2 up
// to 37 %.)
template <int QG>
__device__ __forceinline__ float4 query4(const float* q, int i, int dim) {
    if constexpr (QG == 0) {
        return *reinterpret_cast<const float4*>(q + i);
    } else {
        auto at = [&](int j) { return QG == 1 ? __ldg(q + j) : *(q + j); };
        return make_float4(at(i), i + 1 < dim ? at(i + 1) : 0.0f, i + 2 < dim ? at(i + 2) : 0.0f,
                           i + 3 < dim ? at(i + 3) : 0.0f);
    }
}

// Elements of a row's float4 number c at or past dim := 0.
__device__ __forceinline__ void drop_past(float4& x, int c, int dim) {
    const int r = dim - 4 * c;
    if (r < 4) x.w = 0.0f;
    if (r < 3) x.z = 0.0f;
    if (r < 2) x.y = 0.0f;
}

__device__ __forceinline__ void sq_diff4(const float4 q, const float4 x, float (&s)[4]) {
    float t;
    t = q.x - x.x; s[0] = fmaf(t, t, s[0]);
    t = q.y - x.y; s[1] = fmaf(t, t, s[1]);
    t = q.z - x.z; s[2] = fmaf(t, t, s[2]);
    t = q.w - x.w; s[3] = fmaf(t, t, s[3]);
}

// Squared L2 in the reference's exact order (warp_l2, kernalGraph.h:157-170:
// lane l sums i = l (mod 32) in increasing i with FMA, then a shfl_down tree
// of 16, 8, 4, 2, 1) for the m rows of the list; a lane gets row `want`'s.
// They are read 4 at a time, 8 lanes per row: lane t of a group holds the
// partial sums of the reference's lanes 4t .. 4t + 3, since those
// elements of every 32 are one 16-byte load, and the tree becomes shuffles
// of 4, 2 and 1 between the lanes of a group (offsets 16, 8, 4) and of the
// four sums among themselves (offsets 2, 1); a + b = b + a, so which side
// keeps the sum does not matter.  The query is zero padded to 4 elements and
// what a row holds past dim is dropped (a caller's rows may hold anything
// there): a zero difference leaves every sum as it is.
//
// What bounds it is the wait for the rows, so the loads of up to 4 rows are
// issued 8 per lane ahead of the sums (one round trip for dim <= 256), those
// of up to 8 rows 4 + 4; 4 and 2 + 2 at 80 registers and 6 CTAs per SM
// measured 10 % slower at 200 dimensions and 33 % at 960.  Reading each row
// with 32 lanes of 4 bytes and reducing all 32 slots of the adjacency row in
// unrolled code, as before, took 2-4 times the instructions and more code
// than the instruction cache holds: 10,000 queries x 200 dimensions at ef 512
// 36.3 -> 8.6 ms (200,000 nodes, 0.47 -> 2.0 TB/s of gathered rows), 1,000 x
// 960 at ef 256 7.0 -> 2.5 ms, 10,000 x 24 at ef 128 4.4 -> 2.7 ms.
template <int QG>
__device__ __forceinline__ float l2_rows(const float* __restrict__ base, int ld, int dim,
                                         const float* q, int m, int want, const int* rows, int lane) {
    const int grp = lane >> 3, t = lane & 7;
    const int nch = (dim + 3) >> 2;  // float4 per row
    const bool ragged = dim & 3;
    // loads in flight per lane and rows per pass; as few as can be where this is
    // the rare path (QG), whose registers the byte rows' path would pay for
    constexpr int U = QG ? 1 : 8, P = QG ? 4 : 8;
    float out = 0.0f;
    for (int p0 = 0; p0 < m; p0 += P) {
        const int ra = p0 + grp, rb = ra + 4;
        const bool va = ra < m, vb = rb < m;
        const float4* pa = reinterpret_cast<const float4*>(base + (size_t)(va ? rows[ra] : 0) * ld);
        float sa[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        float r;
        if (P == 8 && m - p0 > 4) {
            const float4* pb = reinterpret_cast<const float4*>(base + (size_t)(vb ? rows[rb] : 0) * ld);
            float sb[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            for (int c0 = t; c0 < nch; c0 += 4 * U) {
                float4 xa[(U + 1) / 2], xb[(U + 1) / 2];
#pragma unroll
                for (int e = 0; e < U / 2; ++e) {
                    const int c = c0 + 8 * e;
                    const bool in = c < nch;
                    xa[e] = (in && va) ? ld_row(pa + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                    xb[e] = (in && vb) ? ld_row(pb + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                if (ragged) {
#pragma unroll
                    for (int e = 0; e < U / 2; ++e) {
                        drop_past(xa[e], c0 + 8 * e, dim);
                        drop_past(xb[e], c0 + 8 * e, dim);
                    }
                }
#pragma unroll
                for (int e = 0; e < U / 2; ++e) {
                    const int c = c0 + 8 * e;
                    if (c < nch) {
                        const float4 qc = query4<QG>(q, 4 * c, dim);
                        sq_diff4(qc, xa[e], sa);
                        sq_diff4(qc, xb[e], sb);
                    }
                }
            }
            __syncwarp();
            // offset 16 (lanes t, t ^ 4): lanes t < 4 keep row a, the others row b
            const bool up = t & 4;
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float o = __shfl_xor_sync(FULL, up ? sa[i] : sb[i], 4);
                v[i] = (up ? sb[i] : sa[i]) + o;
            }
            // offset 8 (t ^ 2) keeps sums {0, 1} or {2, 3}, offset 4 (t ^ 1) one of them
            const bool u2 = t & 2, u1 = t & 1;
            const float w0 = (u2 ? v[2] : v[0]) + __shfl_xor_sync(FULL, u2 ? v[0] : v[2], 2);
            const float w1 = (u2 ? v[3] : v[1]) + __shfl_xor_sync(FULL, u2 ? v[1] : v[3], 2);
            r = (u1 ? w1 : w0) + __shfl_xor_sync(FULL, u1 ? w0 : w1, 1);
            r += __shfl_xor_sync(FULL, r, 2);  // offset 2: sums i and i ^ 2
            r += __shfl_xor_sync(FULL, r, 1);  // offset 1: sums i and i ^ 1
        } else {
            for (int c0 = t; c0 < nch; c0 += 8 * U) {
                float4 xa[U];
#pragma unroll
                for (int e = 0; e < U; ++e) {
                    const int c = c0 + 8 * e;
                    xa[e] = (c < nch && va) ? ld_row(pa + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                if (ragged) {
#pragma unroll
                    for (int e = 0; e < U; ++e) drop_past(xa[e], c0 + 8 * e, dim);
                }
#pragma unroll
                for (int e = 0; e < U; ++e) {
                    const int c = c0 + 8 * e;
                    if (c < nch) sq_diff4(query4<QG>(q, 4 * c, dim), xa[e], sa);
                }
            }
            __syncwarp();
            // offset 16 keeps sums {0, 1} or {2, 3}, offset 8 one of them; offset 4
            // adds the two halves of that sum; then offsets 2 and 1 as above
            const bool u4 = t & 4, u2 = t & 2;
            const float v0 = (u4 ? sa[2] : sa[0]) + __shfl_xor_sync(FULL, u4 ? sa[0] : sa[2], 4);
            const float v1 = (u4 ? sa[3] : sa[1]) + __shfl_xor_sync(FULL, u4 ? sa[1] : sa[3], 4);
            r = (u2 ? v1 : v0) + __shfl_xor_sync(FULL, u2 ? v0 : v1, 2);
            r += __shfl_xor_sync(FULL, r, 1);  // offset 4
            r += __shfl_xor_sync(FULL, r, 4);  // offset 2
            r += __shfl_xor_sync(FULL, r, 2);  // offset 1
        }
        // the row of rank r sits in group r % 4, the second rows in lanes 4 .. 7
        const float g = __shfl_sync(FULL, r, ((want & 3) << 3) | (P == 8 ? want & 4 : 0));
        if (want / P == p0 / P) out = g;
    }
    __syncwarp();
    return out;
}

// Squared L2 of integer vectors in [0, 255] from their byte rows:
// sum (q - b)^2 = sum q^2 + sum b^2 - 2 sum q*b, each term an exact unsigned
// byte dot product (dp4a), so the result is the exact integer distance --
// the same FP32 value the reference's float arithmetic produces, since all
// of its partial sums are integers below 2^24 (dim <= 256).  Rows are read
// in 16-byte chunks, 8 lanes per row, NC chunks per lane, 4 rows per pass
// and two passes in flight; `qb` holds this lane's query chunks and `qq`
// the query's sum of squares.  The m rows are the list's, and a lane gets row
// `want`'s distance.  FOUR: more than 8 rows take 16 per pass, four passes'
// loads in flight (short queues, whose expansions find many new rows: 1 query
// at ef 50 140 -> 133 us, 10,000 at ef 50 1.01 -> 0.98 ms).
template <int NC, int FOUR = 0>
__device__ __forceinline__ float l2_u8(const uint8_t* __restrict__ base, int ld, int nch,
                                       const uint4 (&qb)[NC], int qq, int m, int want,
                                       const int* rows, int lane) {
    const int grp = lane >> 3, t = lane & 7;
    float out = 0.0f;
    if (FOUR && NC == 1 && m > 8) {
        for (int p0 = 0; p0 < m; p0 += 16) {
            uint4 x[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int ri = p0 + 4 * r + grp;
                x[r] = (ri < m && t < nch) ? ld_row(reinterpret_cast<const uint4*>(base + (size_t)rows[ri] * ld) + t) : make_uint4(0u, 0u, 0u, 0u);
            }
            int sm[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                unsigned qa = 0u, ba = 0u;
                qa = __dp4a(qb[0].x, x[r].x, qa);
                qa = __dp4a(qb[0].y, x[r].y, qa);
                qa = __dp4a(qb[0].z, x[r].z, qa);
                qa = __dp4a(qb[0].w, x[r].w, qa);
                ba = __dp4a(x[r].x, x[r].x, ba);
                ba = __dp4a(x[r].y, x[r].y, ba);
                ba = __dp4a(x[r].z, x[r].z, ba);
                ba = __dp4a(x[r].w, x[r].w, ba);
                sm[r] = (int)ba - 2 * (int)qa;
            }
#pragma unroll
            for (int w = 4; w >= 1; w >>= 1)
#pragma unroll
                for (int r = 0; r < 4; ++r) sm[r] += __shfl_xor_sync(FULL, sm[r], w);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int g = __shfl_sync(FULL, sm[r], (want & 3) << 3);
                if ((want >> 2) == (p0 >> 2) + r) out = (float)(qq + g);
            }
        }
        __syncwarp();
        return out;
    }
    for (int p0 = 0; p0 < m; p0 += 8) {
        const int ra = p0 + grp, rb = p0 + 4 + grp;
        const bool va = ra < m, vb = rb < m;
        const uint4* pa = reinterpret_cast<const uint4*>(base + (size_t)(va ? rows[ra] : 0) * ld);
        const uint4* pb = reinterpret_cast<const uint4*>(base + (size_t)(vb ? rows[rb] : 0) * ld);
        uint4 xa[NC], xb[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int ch = t + 8 * c;
            xa[c] = (va && ch < nch) ? ld_row(pa + ch) : make_uint4(0u, 0u, 0u, 0u);
            xb[c] = (vb && ch < nch) ? ld_row(pb + ch) : make_uint4(0u, 0u, 0u, 0u);
        }
        unsigned qa = 0u, ba = 0u, qbb = 0u, bbb = 0u;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            qa = __dp4a(qb[c].x, xa[c].x, qa);
            qa = __dp4a(qb[c].y, xa[c].y, qa);
            qa = __dp4a(qb[c].z, xa[c].z, qa);
            qa = __dp4a(qb[c].w, xa[c].w, qa);
            ba = __dp4a(xa[c].x, xa[c].x, ba);
            ba = __dp4a(xa[c].y, xa[c].y, ba);
            ba = __dp4a(xa[c].z, xa[c].z, ba);
            ba = __dp4a(xa[c].w, xa[c].w, ba);
            qbb = __dp4a(qb[c].x, xb[c].x, qbb);
            qbb = __dp4a(qb[c].y, xb[c].y, qbb);
            qbb = __dp4a(qb[c].z, xb[c].z, qbb);
            qbb = __dp4a(qb[c].w, xb[c].w, qbb);
            bbb = __dp4a(xb[c].x, xb[c].x, bbb);
            bbb = __dp4a(xb[c].y, xb[c].y, bbb);
            bbb = __dp4a(xb[c].z, xb[c].z, bbb);
            bbb = __dp4a(xb[c].w, xb[c].w, bbb);
        }
        int sa = (int)ba - 2 * (int)qa, sb = (int)bbb - 2 * (int)qbb;
#pragma unroll
        for (int w = 4; w >= 1; w >>= 1) {
            sa += __shfl_xor_sync(FULL, sa, w);
            sb += __shfl_xor_sync(FULL, sb, w);
        }
        // row of rank r sits in group r % 4 of pass r / 4
        const int ga = __shfl_sync(FULL, sa, (want & 3) << 3);
        const int gb = __shfl_sync(FULL, sb, (want & 3) << 3);
        if ((want >> 2) == (p0 >> 2)) out = (float)(qq + ga);
        if ((want >> 2) == (p0 >> 2) + 1) out = (float)(qq + gb);
    }
    __syncwarp();
    return out;
}

// Hamming distances: popcount(q ^ b) over the dim code words (warp_hamming,
// hashKernelGraph.h:215-224; integer, so order-free) of the m rows of the
// list; a lane gets row `want`'s.  A row is W4 uint4 wide and W4 lanes read
// it, one each (`qc`: this lane's uint4 of the query), 32 / W4 rows per pass;
// words at or past dim are padding and never count, whatever they hold.  A
// lane per row instead had only the new rows' lanes loading, W4 dependent
// lines each.
template <int W4>
__device__ __forceinline__ float ham_rows(const uint32_t* __restrict__ base, int ld, int dim,
                                          const uint4 qc, int m, int want, const int* rows, int lane) {
    constexpr int P = 32 / W4;
    const int t = lane & (W4 - 1), grp = lane / W4;
    const int r = dim - 4 * t;  // words of this lane's uint4 that count
    float out = 0.0f;
    for (int p0 = 0; p0 < m; p0 += P) {
        int s = 0;
        if (p0 + grp < m && r > 0) {
            uint4 x = ld_row(reinterpret_cast<const uint4*>(base + (size_t)rows[p0 + grp] * ld) + t);
            if (r < 2) x.y = qc.y;
            if (r < 3) x.z = qc.z;
            if (r < 4) x.w = qc.w;
            s = __popc(x.x ^ qc.x) + __popc(x.y ^ qc.y) + __popc(x.z ^ qc.z) + __popc(x.w ^ qc.w);
        }
#pragma unroll
        for (int w = W4 / 2; w >= 1; w >>= 1) s += __shfl_xor_sync(FULL, s, w);
        const int g = __shfl_sync(FULL, s, (want % P) * W4);
        if (want / P == p0 / P) out = (float)g;
    }
    __syncwarp();
    return out;
}

// Writes the k results (kernalGraph.h:292-296): `while (sz > k) pop_worst()`
// then `drain_best(out, k)`, -1 padding.  The k+1 smallest results are
// extracted first (into the free candidate arrays); if their distances are
// strictly increasing the replay's outcome is exactly those k in order.
// Otherwise the extraction is undone and the trims and drains are replayed.
// `scratch` (TM = 1: at least cap ints of shared memory) holds the slots of
// the extracted results; with TM = 0 the free candidate id array does.
template <int GPL, int TM, int TD, int TMC>
__device__ __forceinline__ int finish(Queue<GPL, TM, TD>& res, Queue<GPL, TMC>& cand, int k,
                                      int32_t* out, float* outd, int lane, int* scratch) {
    const int ng = (res.sz + 31) >> 5;
    for (int g = 0; g < ng; ++g) group_update<true>(res, g, lane);
    const int cnt = res.sz < k ? res.sz : k;
    const int take = res.sz < k + 1 ? res.sz : k + 1;
    unsigned* xv = reinterpret_cast<unsigned*>(cand.d);  // extracted distance bits
    int* xs = TMC ? scratch : cand.id;                   // their slots
    for (int i = 0; i < take; ++i) {
        unsigned mb, mi;
        root_min(res, mb, mi);
        if (lane == 0) {
            xv[i] = mb;
            xs[i] = (int)mi;
        }
        q_set_dbits(res, (int)mi, 0xffffffffu, lane);  // out of every minimum
        __syncwarp();
        group_update<true>(res, (int)(mi >> 5), lane);
    }
    bool distinct = true;
    for (int i = lane; i + 1 < take; i += 32) distinct &= xv[i] < xv[i + 1];
    distinct = __all_sync(FULL, distinct);
    if (distinct) {
        if constexpr (TM) {
            for (int i = 0; i < cnt; ++i) {
                const int id = q_id(res, xs[i]);
                if (lane == (i & 31)) out[i] = id;
            }
            for (int i = lane; i < cnt; i += 32)
                if (outd) outd[i] = __uint_as_float(xv[i]);
        } else {
            for (int i = lane; i < cnt; i += 32) {
                out[i] = res.id[xs[i]];
                if (outd) outd[i] = __uint_as_float(xv[i]);
            }
        }
    } else {
        if constexpr (TD) {
            for (int i = 0; i < take; ++i) q_set_dbits(res, xs[i], xv[i], lane);
        } else {
            for (int i = lane; i < take; i += 32) reinterpret_cast<unsigned*>(res.d)[xs[i]] = xv[i];
        }
        __syncwarp();
        for (int g = 0; g < ng; ++g) group_update<true>(res, g, lane);
        while (res.sz > k) {  // Results::pop_worst
            unsigned mb, mi;
            root_max(res, mb, mi);
            q_remove<true>(res, (int)mi, lane);
        }
        for (int i = 0; i < cnt; ++i) {  // Results::drain_best
            unsigned mb, mi;
            root_min(res, mb, mi);
            const int id = q_id(res, (int)mi);
            if (lane == 0) {
                out[i] = id;
                if (outd) outd[i] = __uint_as_float(mb);
            }
            q_remove<true>(res, (int)mi, lane);
        }
    }
    for (int i = cnt + lane; i < k; i += 32) {
        out[i] = -1;
        if (outd) outd[i] = INFINITY;
    }
    return cnt;
}

// The same for queues in registers (`scratch`: 2 * cap ints).
template <int R>
__device__ __forceinline__ int finish(RQueue<R>& res, int k, int32_t* out, float* outd, int lane, int* scratch) {
    const int cnt = res.sz < k ? res.sz : k;
    const int take = res.sz < k + 1 ? res.sz : k + 1;
    unsigned* xv = reinterpret_cast<unsigned*>(scratch);  // extracted distance bits
    int* xs = scratch + res.cap;                          // their slots
    for (int i = 0; i < take; ++i) {
        unsigned mb, mi;
        root_min(res, mb, mi, lane);
        if (lane == 0) {
            xv[i] = mb;
            xs[i] = (int)mi;
        }
        q_set_dbits(res, (int)mi, kEmpty, lane);
    }
    __syncwarp();
    bool distinct = true;
    for (int i = lane; i + 1 < take; i += 32) distinct &= xv[i] < xv[i + 1];
    distinct = __all_sync(FULL, distinct);
    if (distinct) {
        for (int i = lane; i < cnt; i += 32) {
            out[i] = res.id[xs[i]];
            if (outd) outd[i] = __uint_as_float(xv[i]);
        }
    } else {
        for (int i = 0; i < take; ++i) q_set_dbits(res, xs[i], xv[i], lane);
        while (res.sz > k) {  // Results::pop_worst
            unsigned mb, mi;
            root_max(res, mb, mi, lane);
            q_remove(res, (int)mi, lane);
        }
        for (int i = 0; i < cnt; ++i) {  // Results::drain_best
            unsigned mb, mi;
            root_min(res, mb, mi, lane);
            const int id = res.id[mi];
            if (lane == 0) {
                out[i] = id;
                if (outd) outd[i] = __uint_as_float(mb);
            }
            q_remove(res, (int)mi, lane);
        }
    }
    for (int i = cnt + lane; i < k; i += 32) {
        out[i] = -1;
        if (outd) outd[i] = INFINITY;
    }
    return cnt;
}

// Place in shared memory of query element i for the compressed rows: lane t of
// 8 reads the elements of row chunk t + 8 b (EPC of them) four at a time, so
// the four's 8 places are side by side.  In element order the 8 lanes' reads
// were 32 or 64 bytes apart, 2 and 4 bank conflicts each (4,000 queries x 960
// dimensions, FP8, ef 384: 6.14 -> 5.91 ms).
template <int DT>
__device__ __forceinline__ int lowp_place(int i) {
    constexpr int EPC = DT == SONG_PREC_BF16 ? 8 : 16;  // elements per 16-byte chunk
    const int c = i / EPC, piece = (i % EPC) >> 2;
    return ((c >> 3) * (EPC / 4) + piece) * 32 + (c & 7) * 4 + (i & 3);
}

// Accumulate (q - b)^2 over one 16-byte chunk of a compressed row: 8 BF16 or
// 16 FP8 e4m3 values (times the row's scale), FP32 arithmetic.  qc: the
// chunk's first four query elements, the next ones 32 floats on.
template <int DT>
__device__ __forceinline__ void chunk_l2(const uint4 x, const float* qc, float scale, float& acc) {
    const unsigned w[4] = {x.x, x.y, x.z, x.w};
    if constexpr (DT == SONG_PREC_BF16) {
        const float4 q0 = *reinterpret_cast<const float4*>(qc);
        const float4 q1 = *reinterpret_cast<const float4*>(qc + 32);
        const float q[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float lo = __uint_as_float(w[i] << 16);
            const float hi = __uint_as_float(w[i] & 0xffff0000u);
            float t = q[2 * i] - lo;
            acc = fmaf(t, t, acc);
            t = q[2 * i + 1] - hi;
            acc = fmaf(t, t, acc);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 q = *reinterpret_cast<const float4*>(qc + 32 * i);
            const __half2_raw h01 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[i] & 0xffffu), __NV_E4M3);
            const __half2_raw h23 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[i] >> 16), __NV_E4M3);
            const float2 b01 = __half22float2(__half2(h01));
            const float2 b23 = __half22float2(__half2(h23));
            float t = fmaf(-scale, b01.x, q.x);
            acc = fmaf(t, t, acc);
            t = fmaf(-scale, b01.y, q.y);
            acc = fmaf(t, t, acc);
            t = fmaf(-scale, b23.x, q.z);
            acc = fmaf(t, t, acc);
            t = fmaf(-scale, b23.y, q.w);
            acc = fmaf(t, t, acc);
        }
    }
}

// Precision-form distances of the m rows of the list (a lane gets row
// `want`'s): 4 rows per pass, 8 lanes per row, 16-byte loads of the
// compressed rows, query from shared memory, two passes in flight.
template <int DT>
__device__ __forceinline__ float l2_lowp(const SearchArgs& a, const float* sq, int m, int want,
                                         const int* rows, int lane) {
    constexpr int EPC = DT == SONG_PREC_BF16 ? 8 : 16;  // elements per 16-byte chunk
    const int grp = lane >> 3, t = lane & 7;
    const int nchunk = a.lowp_ld >> 4;
    const float* qt = sq + 4 * t;  // chunk t + 8 b of the query: 8 EPC b floats on
    const unsigned char* lp = reinterpret_cast<const unsigned char*>(a.lowp);
    float out = 0.0f;
    for (int p0 = 0; p0 < m; p0 += 8) {
        const int ra = p0 + grp, rb = p0 + 4 + grp;
        const bool va = ra < m, vb = rb < m;
        const int ia = va ? rows[ra] : 0, ib = vb ? rows[rb] : 0;
        const uint4* pa = reinterpret_cast<const uint4*>(lp + (size_t)ia * a.lowp_ld);
        const uint4* pb = reinterpret_cast<const uint4*>(lp + (size_t)ib * a.lowp_ld);
        float sca = 1.0f, scb = 1.0f;
        if constexpr (DT == SONG_PREC_FP8) {
            sca = va ? __ldg(a.scales + ia) : 0.0f;
            scb = vb ? __ldg(a.scales + ib) : 0.0f;
        }
        // rows are whole multiples of 8 chunks; loads in flight per lane: 4 of one
        // row, or 2 of each of two rows
        float sa = 0.0f, sb = 0.0f;
        if (m - p0 > 4) {
            for (int c0 = t; c0 < nchunk; c0 += 16) {
                uint4 xa[2], xb[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const bool in = c0 + 8 * e < nchunk;
                    xa[e] = (in && va) ? ld_row(pa + c0 + 8 * e) : make_uint4(0u, 0u, 0u, 0u);
                    xb[e] = (in && vb) ? ld_row(pb + c0 + 8 * e) : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (c0 + 8 * e < nchunk) {
                        chunk_l2<DT>(xa[e], qt + (c0 - t + 8 * e) * EPC, sca, sa);
                        chunk_l2<DT>(xb[e], qt + (c0 - t + 8 * e) * EPC, scb, sb);
                    }
                }
            }
        } else {
            for (int c0 = t; c0 < nchunk; c0 += 32) {
                uint4 xa[4];
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    xa[e] = (c0 + 8 * e < nchunk && va) ? ld_row(pa + c0 + 8 * e) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (c0 + 8 * e < nchunk) chunk_l2<DT>(xa[e], qt + (c0 - t + 8 * e) * EPC, sca, sa);
            }
        }
#pragma unroll
        for (int w = 4; w >= 1; w >>= 1) {
            sa += __shfl_xor_sync(FULL, sa, w);
            sb += __shfl_xor_sync(FULL, sb, w);
        }
        const float ga = __shfl_sync(FULL, sa, (want & 3) << 3);
        const float gb = __shfl_sync(FULL, sb, (want & 3) << 3);
        if ((want >> 2) == (p0 >> 2)) out = ga;
        if ((want >> 2) == (p0 >> 2) + 1) out = gb;
    }
    __syncwarp();
    return out;
}

// Squared FP32 distance of the row `row` (nullptr: none) for each group of 8
// lanes, summed per lane over every 8th float4 and then over the lanes: 8
// loads in flight per lane, or the final re-rank (every entry of a queue) is
// a chain of one load after the other (with the one-row pass of l2_lowp,
// 4,000 queries x 960 dimensions at ef 384: FP8 7.48 -> 6.14 ms, BF16 9.38 ->
// 6.94 ms).
__device__ __forceinline__ float rerank_row(const float4* row, int nch, const float* sq, int lane) {
    constexpr int U = 8;
    const int t = lane & 7;
    float acc = 0.0f;
    for (int c0 = t; c0 < nch; c0 += 8 * U) {
        float4 x[U];
#pragma unroll
        for (int e = 0; e < U; ++e)
            x[e] = (row != nullptr && c0 + 8 * e < nch) ? ld_row(row + c0 + 8 * e) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int e = 0; e < U; ++e) {
            if (c0 + 8 * e < nch) {
                const float4 q = *reinterpret_cast<const float4*>(sq + 4 * (c0 + 8 * e));
                float u = q.x - x[e].x;
                acc = fmaf(u, u, acc);
                u = q.y - x[e].y;
                acc = fmaf(u, u, acc);
                u = q.z - x[e].z;
                acc = fmaf(u, u, acc);
                u = q.w - x[e].w;
                acc = fmaf(u, u, acc);
            }
        }
    }
#pragma unroll
    for (int w = 4; w >= 1; w >>= 1) acc += __shfl_xor_sync(FULL, acc, w);
    return acc;
}

// Precision form, final step: exact FP32 distances of every entry of the
// results queue (FP32 rows, 8 lanes per row), then the k smallest by
// (distance, id) in ascending order, -1 padded.
template <int GPL, int TM, int TD, int TMC>
__device__ __forceinline__ int rerank_finish(const SearchArgs& a, Queue<GPL, TM, TD>& res,
                                             Queue<GPL, TMC>& cand, const float* sq, int32_t* out,
                                             float* outd, int lane) {
    const int m = res.sz;
    float* rd = cand.d;
    int* rid = cand.id;  // TM = 0 only; with TM = 1 the ids stay in res's TMEM columns
    const float* base = reinterpret_cast<const float*>(a.base);
    const int nch = a.ld >> 2;  // float4 per FP32 row
    const int grp = lane >> 3, t = lane & 7;
    unsigned gid = 0;  // TM = 1: ids of the current group, lane l = slot 32g + l
    for (int p0 = 0; p0 < m; p0 += 4) {
        const int r = p0 + grp;
        const bool v = r < m;
        int id;
        if constexpr (TM) {
            if ((p0 & 31) == 0) gid = tm_ld(res.tid + (uint32_t)(p0 >> 5));
            id = (int)__shfl_sync(FULL, gid, r & 31);
            if (!v) id = 0;
        } else {
            id = v ? res.id[r] : 0;
        }
        const float acc = rerank_row(v ? reinterpret_cast<const float4*>(base + (size_t)id * a.ld) : nullptr, nch, sq, lane);
        if (t == 0 && v) {
            rd[r] = acc;
            if constexpr (!TM) rid[r] = id;
        }
    }
    __syncwarp();
    const int cnt = m < a.k ? m : a.k;
    for (int i = 0; i < cnt; ++i) {
        unsigned bb = 0xffffffffu, bi = 0xffffffffu;
        for (int s0 = 0; s0 < m; s0 += 32) {  // warp-uniform trip count (TMEM loads are collective)
            const int s2 = s0 + lane;
            unsigned id;
            if constexpr (TM) id = tm_ld(res.tid + (uint32_t)(s0 >> 5));
            else id = s2 < m ? (unsigned)rid[s2] : 0u;
            if (s2 < m) {
                const unsigned b = fbits(rd[s2]);
                if (b < bb || (b == bb && id < bi)) {
                    bb = b;
                    bi = id;
                }
            }
        }
        const unsigned mb = __reduce_min_sync(FULL, bb);
        const unsigned mi = __reduce_min_sync(FULL, bb == mb ? bi : 0xffffffffu);
        if (lane == 0) {
            out[i] = (int)mi;
            if (outd) outd[i] = __uint_as_float(mb);
        }
        for (int s0 = 0; s0 < m; s0 += 32) {  // taken: out of every later minimum
            const int s2 = s0 + lane;
            unsigned id;
            if constexpr (TM) id = tm_ld(res.tid + (uint32_t)(s0 >> 5));
            else id = s2 < m ? (unsigned)rid[s2] : 0u;
            if (s2 < m && id == mi) rd[s2] = __uint_as_float(0xffffffffu);
        }
        __syncwarp();
    }
    for (int i = cnt + lane; i < a.k; i += 32) {
        out[i] = -1;
        if (outd) outd[i] = INFINITY;
    }
    return cnt;
}


// The same for queues in registers: ids in res.id, distances in `rd` (cap
// floats of shared memory).
template <int R>
__device__ __forceinline__ int rerank_finish(const SearchArgs& a, RQueue<R>& res, const float* sq, int32_t* out,
                                             float* outd, int lane, float* rd) {
    const int m = res.sz;
    const float* base = reinterpret_cast<const float*>(a.base);
    const int nch = a.ld >> 2;  // float4 per FP32 row
    const int grp = lane >> 3, t = lane & 7;
    for (int p0 = 0; p0 < m; p0 += 4) {
        const bool v = p0 + grp < m;
        const float4* row = v ? reinterpret_cast<const float4*>(base + (size_t)res.id[p0 + grp] * a.ld) : nullptr;
        const float acc = rerank_row(row, nch, sq, lane);
        if (t == 0 && v) rd[p0 + grp] = acc;
    }
    __syncwarp();
    // the k smallest by (distance, id): the queue's registers hold the new distances
    RQueue<R>& q = res;
#pragma unroll
    for (int r = 0; r < R; ++r) q.d[r] = 32 * r + lane < m ? fbits(rd[32 * r + lane]) : kEmpty;
    const int cnt = m < a.k ? m : a.k;
    for (int i = 0; i < cnt; ++i) {
        unsigned lm = q.d[0];
#pragma unroll
        for (int r = 1; r < R; ++r) lm = min(lm, q.d[r]);
        const unsigned mb = __reduce_min_sync(FULL, lm);
        unsigned bi = 0xffffffffu;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (q.d[r] == mb && 32 * r + lane < m) bi = min(bi, (unsigned)q.id[32 * r + lane]);
        const unsigned mi = __reduce_min_sync(FULL, bi);
        if (lane == 0) {
            out[i] = (int)mi;
            if (outd) outd[i] = __uint_as_float(mb);
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (q.d[r] == mb && 32 * r + lane < m && (unsigned)q.id[32 * r + lane] == mi) q.d[r] = kEmpty;
    }
    for (int i = cnt + lane; i < a.k; i += 32) {
        out[i] = -1;
        if (outd) outd[i] = INFINITY;
    }
    return cnt;
}

// ------------------------------------------------------------ learned model

// Warp-resident MLP over warp-uniform inputs f[kFeat] with FP16 weights and
// FP32 accumulation: relu(W1 f + b1) -> relu(W2 h + b2) -> W3 h + b3.
// Lane l evaluates hidden units l and l + 32.  For n_out == 1 every lane
// returns the output; otherwise lane o < n_out (<= 32) returns output o.
__device__ __forceinline__ float mlp_warp(const __half* __restrict__ w, const float (&f)[kFeat],
                                          int n_out, int lane) {
    const __half* W1 = w;
    const __half* b1 = W1 + kHid * kFeat;
    const __half* W2 = b1 + kHid;
    const __half* b2 = W2 + kHid * kHid;
    const __half* W3 = b2 + kHid;
    const __half* b3 = W3 + n_out * kHid;
    float h0 = __half2float(b1[lane]), h1 = __half2float(b1[lane + 32]);
    const __half2* r0 = reinterpret_cast<const __half2*>(W1 + lane * kFeat);
    const __half2* r1 = reinterpret_cast<const __half2*>(W1 + (lane + 32) * kFeat);
#pragma unroll
    for (int i = 0; i < kFeat / 2; ++i) {
        const float2 a = __half22float2(r0[i]);
        const float2 b = __half22float2(r1[i]);
        h0 = fmaf(a.x, f[2 * i], h0);
        h0 = fmaf(a.y, f[2 * i + 1], h0);
        h1 = fmaf(b.x, f[2 * i], h1);
        h1 = fmaf(b.y, f[2 * i + 1], h1);
    }
    h0 = fmaxf(h0, 0.0f);
    h1 = fmaxf(h1, 0.0f);
    float g0 = __half2float(b2[lane]), g1 = __half2float(b2[lane + 32]);
    const __half2* s0 = reinterpret_cast<const __half2*>(W2 + lane * kHid);
    const __half2* s1 = reinterpret_cast<const __half2*>(W2 + (lane + 32) * kHid);
#pragma unroll 4
    for (int j = 0; j < 32; j += 2) {
        const float x0 = __shfl_sync(FULL, h0, j), x1 = __shfl_sync(FULL, h0, j + 1);
        const float y0 = __shfl_sync(FULL, h1, j), y1 = __shfl_sync(FULL, h1, j + 1);
        const float2 a = __half22float2(s0[j >> 1]), c = __half22float2(s0[(j + 32) >> 1]);
        const float2 b = __half22float2(s1[j >> 1]), e = __half22float2(s1[(j + 32) >> 1]);
        g0 = fmaf(a.x, x0, fmaf(a.y, x1, fmaf(c.x, y0, fmaf(c.y, y1, g0))));
        g1 = fmaf(b.x, x0, fmaf(b.y, x1, fmaf(e.x, y0, fmaf(e.y, y1, g1))));
    }
    g0 = fmaxf(g0, 0.0f);
    g1 = fmaxf(g1, 0.0f);
    if (n_out == 1) {
        float z = fmaf(__half2float(W3[lane]), g0, __half2float(W3[lane + 32]) * g1);
#pragma unroll
        for (int w2 = 16; w2 >= 1; w2 >>= 1) z += __shfl_xor_sync(FULL, z, w2);
        return z + __half2float(b3[0]);
    }
    const int o = lane < n_out ? lane : 0;
    const __half2* t3 = reinterpret_cast<const __half2*>(W3 + o * kHid);
    float z = __half2float(b3[o]);
#pragma unroll 4
    for (int j = 0; j < 32; j += 2) {
        const float x0 = __shfl_sync(FULL, g0, j), x1 = __shfl_sync(FULL, g0, j + 1);
        const float y0 = __shfl_sync(FULL, g1, j), y1 = __shfl_sync(FULL, g1, j + 1);
        const float2 a = __half22float2(t3[j >> 1]), c = __half22float2(t3[(j + 32) >> 1]);
        z = fmaf(a.x, x0, fmaf(a.y, x1, fmaf(c.x, y0, fmaf(c.y, y1, z))));
    }
    return z;
}

// Running statistics of a search for the learned stop.  kd: lane i < K holds
// the i-th smallest distance computed so far (+inf if fewer), which is the
// i-th entry of the results' top-K, since results only lose their maximum.
struct StopState {
    float kd, kth, best, kth_prev, entry_d;
    int K, hops_kth, hops_best, n_new, n_res, n_front, nck;
};

__device__ __forceinline__ void stop_init(StopState& s, int k) {
    s.kd = s.kth = s.best = s.kth_prev = s.entry_d = INFINITY;
    s.K = k < 1 ? 1 : (k > 32 ? 32 : k);
    s.hops_kth = s.hops_best = s.n_new = s.n_res = s.n_front = s.nck = 0;
}

// Insert the distances of the lanes in N into the sorted top-K (lane order).
__device__ __forceinline__ void topk_insert(StopState& s, unsigned N, float d, int lane) {
    const bool mine = (N >> lane) & 1u;
    unsigned ins = __ballot_sync(FULL, mine && d < s.kth);
    while (ins) {
        const int j = __ffs(ins) - 1;
        const float v = __shfl_sync(FULL, d, j);
        const int p = __popc(__ballot_sync(FULL, lane < s.K && s.kd <= v));
        const float up = __shfl_up_sync(FULL, s.kd, 1);
        if (lane < s.K && lane > p) s.kd = up;
        if (lane == p) s.kd = v;
        if (v < s.best) s.hops_best = 0;
        const float nk = __shfl_sync(FULL, s.kd, s.K - 1);
        if (nk != s.kth) s.hops_kth = 0;
        s.kth = nk;
        s.best = __shfl_sync(FULL, s.kd, 0);
        ins &= ~(1u << j);
        ins &= __ballot_sync(FULL, mine && d < s.kth);
    }
}

// The kFeat stop features (warp-uniform), all finite and roughly in [0, 1].
// cnt1/cnt11/cnt125: frontier candidates closer than 1x / 1.1x / 1.25x the
// k-th best distance (the ones that can still improve the top-k).
__device__ __forceinline__ void stop_features(float (&f)[kFeat], const StopState& s, int t,
                                              float cmin, float worst, bool res_full,
                                              float cand_fill, float res_fill, int cnt1,
                                              int cnt11, int cnt125, int window) {
    const bool kf = s.kth < INFINITY;
    const float kth = kf ? fmaxf(s.kth, 1e-30f) : 1.0f;
    const float best = s.best < INFINITY ? s.best : 0.0f;
    const float wnd = 1.0f / (float)window;
    f[0] = log1pf((float)t) * 0.125f;
    f[1] = kf ? fminf(cmin / kth, 4.0f) * 0.25f : 1.0f;
    f[2] = kf ? fminf(best / kth, 1.0f) : 0.0f;
    f[3] = (kf && s.kth_prev < INFINITY) ? fminf(s.kth / fmaxf(s.kth_prev, 1e-30f), 1.0f) : 1.0f;
    f[4] = fminf((float)s.hops_kth, 256.0f) * (1.0f / 64.0f);
    f[5] = fminf((float)s.hops_best, 256.0f) * (1.0f / 64.0f);
    f[6] = (res_full && kf) ? fminf(worst / kth, 8.0f) * 0.125f : 1.0f;
    f[7] = (float)s.n_res * wnd;
    f[8] = (float)s.n_new * wnd;
    f[9] = cand_fill;
    f[10] = res_fill;
    f[11] = kf ? fminf(logf(kth / fmaxf(best, 1e-30f)), 8.0f) * 0.125f : 1.0f;
    f[12] = log1pf((float)s.hops_kth) * (1.0f / 6.0f);
    f[13] = log1pf((float)s.hops_best) * (1.0f / 6.0f);
    f[14] = res_full ? fminf(cmin / fmaxf(worst, 1e-30f), 2.0f) * 0.5f : 0.0f;
    f[15] = fminf((float)cnt1, 16.0f) * (1.0f / 16.0f);
    f[16] = kf ? 1.0f : 0.0f;
    f[17] = log1pf(kf ? s.kth : 0.0f) * (1.0f / 16.0f);
    f[18] = fminf((float)cnt125, 64.0f) * (1.0f / 64.0f);
    f[19] = log1pf(cmin < INFINITY ? cmin : 0.0f) * (1.0f / 16.0f);
    f[20] = (float)s.n_front * wnd;
    f[21] = fminf((float)cnt11, 32.0f) * (1.0f / 32.0f);
    f[22] = (kf && s.entry_d < INFINITY) ? fminf(s.entry_d / kth, 64.0f) * (1.0f / 64.0f) : 1.0f;
    f[23] = 1.0f;
}

// Order-preserving unsigned key of a float (for redux over signed values).
__device__ __forceinline__ unsigned fkey(float x) {
    const unsigned b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// KIND 0 = L2 (NE = 0: query in shared memory; NE < 0: byte rows of up to
// -NE chunks of 16 bytes per lane); KIND 1 = Hamming with NE uint4 of code
// per row.  GPL: queue groups per lane.
// DT: SONG_PREC_FP32 (the plain, bit-exact search) or the precision form on
// BF16 / FP8 rows (KIND 0, query in shared memory, FP32 re-rank at the end).
// LM: 0 plain; 1 learning traces; 2 learned entry and stop; 3 learned entry
// only (the instance for a stop model that cannot fire).
// TM = 1: the result ids live in this warp's TMEM lanes from column `tbase`
// (G = ceil(cap / 32) columns); TMC = 1: so do the candidate ids, in the G
// columns before them.  The per-warp shared-memory layout then has no id
// array for that queue.
// TR = 0: the per-query trace is not written (a.trace must be null), so its
// counters are dead code and free their registers.  TD = 1 (TM = TMC = 1):
// the results queue's distances in TMEM too.  SV = 1: called by the serving
// kernel, whose queries lie in memory that is written while it runs.
template <int KIND, int NE, int GPL, int DT, int LM, int TM = 0, int TMC = TM, int TR = 1, int TD = 0, int QR = 0,
          int SV = 0>
__device__ __forceinline__ void search_query(const SearchArgs& a, int qid, unsigned char* ws,
                                             int lane, uint32_t tbase = 0) {
    static_assert(!TD || (TM && TMC), "distances in TMEM go with the ids in TMEM");
    static_assert(!QR || (!TM && GPL == 1), "queues in registers use no TMEM");
    std::conditional_t<(QR > 0), RQueue<QR ? QR : 1>, Queue<GPL, TMC>> cand;
    std::conditional_t<(QR > 0), RQueue<QR ? QR : 1>, Queue<GPL, TM, TD>> res;
    // this warp's TMEM columns: [candidate ids (TMC)] [result ids (TM)] [result distances (TD)]
    const uint32_t ngrp = (uint32_t)((a.cap + 31) >> 5);
    const uint32_t tres = tbase + (TMC ? ngrp : 0u);
    if constexpr (QR) {
        q_init(cand, reinterpret_cast<int*>(ws + a.ci_off), a.cap);
        q_init(res, reinterpret_cast<int*>(ws + a.ri_off), a.cap);
    } else {
        q_init(cand, reinterpret_cast<float*>(ws + a.cd_off), reinterpret_cast<int*>(ws + a.ci_off),
               tbase, 0u, a.cap);
        q_init(res, reinterpret_cast<float*>(ws + a.rd_off), reinterpret_cast<int*>(ws + a.ri_off),
               tres, tres + ngrp, a.cap);
    }
    uint64_t* bloom = reinterpret_cast<uint64_t*>(ws + a.bl_off);
    float* sq = reinterpret_cast<float*>(ws + a.q_off);
    int* rows = reinterpret_cast<int*>(ws + a.rows_off);

    BloomCfg bc;
    bc.words = (uint32_t)a.bf_words;
    bc.nbits = (uint64_t)a.bf_words * 64ull;
    bc.shift = (a.bf_words & (a.bf_words - 1)) == 0 ? __ffs(a.bf_words) - 1 : -1;
    bc.wmask = (uint32_t)a.bf_words - 1u;
    bc.nhash = a.bf_nhash;

    // The query: KIND 0 keeps it in shared memory (zero padded to qdim), but for
    // NE < 0 (byte-row instances, an index with byte rows, dim <= 32 * 4 * -NE):
    // only the query's bytes, in registers; a query that is not integral in
    // [0, 255] takes the exact float path reading its floats from global
    // memory.  Fewer live registers let more queries reside per SM.
    constexpr bool kU8 = KIND == 0 && NE < 0;
    constexpr int kNC = kU8 ? -NE : 1;  // 16-byte query chunks per lane on the byte-row path
    uint4 qb[kU8 ? kNC : 1];
    const float* sqg = nullptr;  // byte-row instances: the query in global memory
    uint4 qcode;  // Hamming: this lane's uint4 of the query
    bool u8_mode = false;
    int qq = 0;
    if constexpr (KIND == 0) {
        const float* qg = reinterpret_cast<const float*>(a.queries) + (int64_t)qid * a.qld;
        if constexpr (kU8) {
            sqg = qg;
            float lo = INFINITY, hi = -INFINITY;
            bool integral = true;
            int s2 = 0;
            for (int i = lane; i < a.dim; i += 32) {
                const float v = __ldcg(qg + i);
                lo = fminf(lo, v);
                hi = fmaxf(hi, v);
                integral &= v == rintf(v);
                if (v >= 0.0f && v <= 255.0f) s2 += (int)v * (int)v;
            }
            integral = __all_sync(FULL, integral);
#pragma unroll
            for (int w = 16; w >= 1; w >>= 1) {
                lo = fminf(lo, __shfl_xor_sync(FULL, lo, w));
                hi = fmaxf(hi, __shfl_xor_sync(FULL, hi, w));
            }
            // byte rows hold a base in [0, 255]; a query there too makes every
            // partial sum an integer below 2^24 (dim <= 256): exact dp4a distances
            u8_mode = a.u8 != nullptr && integral && lo >= 0.0f && hi <= 255.0f;
            // the request before this one in its slot was read through L1: no lane may be
            // served its floats (plain loads are ordered by a fence after the claim)
            if (SV && !u8_mode) __threadfence();
            if (u8_mode) {
                qq = (int)__reduce_add_sync(FULL, (unsigned)s2);
#pragma unroll
                for (int c = 0; c < kNC; ++c) {  // lane t of 8: bytes 16(t + 8c) .. +15
                    const int e0 = 16 * ((lane & 7) + 8 * c);
                    unsigned w4[4];
#pragma unroll
                    for (int wd = 0; wd < 4; ++wd) {
                        unsigned wv = 0u;
#pragma unroll
                        for (int bt = 0; bt < 4; ++bt) {
                            const int e = e0 + 4 * wd + bt;
                            const unsigned bv = e < a.dim ? (unsigned)__ldcg(qg + e) : 0u;
                            wv |= bv << (8 * bt);
                        }
                        w4[wd] = wv;
                    }
                    qb[c] = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                }
            }
        } else {
            for (int i = lane; i < a.qdim; i += 32) {
                const float v = i < a.dim ? __ldcg(qg + i) : 0.0f;
                if constexpr (DT != SONG_PREC_FP32) sq[lowp_place<DT>(i)] = v;
                else sq[i] = v;
            }
        }
    } else {
        const uint32_t* qg = reinterpret_cast<const uint32_t*>(a.queries) + (int64_t)qid * a.qld;
        const int t4 = 4 * (lane & (NE - 1));
        uint32_t w[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) w[t] = (t4 + t) < a.dim ? __ldcg(qg + t4 + t) : 0u;
        qcode = make_uint4(w[0], w[1], w[2], w[3]);
    }
    for (int w = lane; w < a.bf_words; w += 32) bloom[w] = 0ull;
    __syncwarp();

    // Distances of the ids `nb` of the lanes in N, through the 32-entry list of
    // them in lane order: lane l gets its own, or with queues in registers the
    // l-th of the list (then N becomes the run of low bits that has one, and nb
    // the list).
    auto distances = [&](int& nb, unsigned& N) -> float {
        const int rank = __popc(N & lanemask_lt(lane));
        const int m = __popc(N);
        const bool mine = (N >> lane) & 1u;
        if (mine) rows[rank] = nb;
        __syncwarp();
        int want = mine ? rank : m + 32;  // m + 32: none
        if constexpr (QR) {
            want = lane < m ? lane : m + 32;
            nb = lane < m ? rows[lane] : -1;
            N = m == 32 ? FULL : (1u << m) - 1u;
        }
        float d;
        if constexpr (DT != SONG_PREC_FP32) {
            d = l2_lowp<DT>(a, sq, m, want, rows, lane);
        } else if constexpr (KIND == 0) {
            const float* base = reinterpret_cast<const float*>(a.base);
            if constexpr (kU8) {
                if (u8_mode) d = l2_u8<kNC, (QR > 0)>(a.u8, a.u8_ld, a.u8_ld >> 4, qb, qq, m, want, rows, lane);
                else d = l2_rows<1 + SV>(base, a.ld, a.dim, sqg, m, want, rows, lane);
            } else {
                d = l2_rows<0>(base, a.ld, a.dim, sq, m, want, rows, lane);
            }
        } else {
            d = ham_rows<NE>(reinterpret_cast<const uint32_t*>(a.base), a.ld, a.dim, qcode, m, want, rows, lane);
        }
        return d;
    };

    // Learned entry: distances to the hub nodes are the entry features; the
    // entry model's top hubs replace the p*n/N_MULTIPROBE seeds.
    StopState ss;
    stop_init(ss, a.k);
    int seed_id = -1, n_seeds = a.n_multiprobe;
    const bool given_seeds = a.qseeds != nullptr;  // caller-chosen entry points per query
    if (given_seeds) {
        n_seeds = a.n_qseeds;
        seed_id = lane < n_seeds ? __ldg(a.qseeds + (int64_t)qid * a.n_qseeds + lane) : -1;
        if (seed_id >= a.n) {  // never read out of range
            atomicExch(a.err, 1);
            seed_id = -1;
        }
    }
    if constexpr (LM > 0) {
        if (a.ecand != nullptr && !given_seeds) {
            // entry stage: this query's kEntryK nearest hubs (nearest first) from the
            // tensor-core kernel; the entry model re-scores them, or without a model
            // the nearest N_MULTIPROBE become the entry points
            const int64_t eo = (int64_t)qid * kEntryK;
            const int hub = lane < kEntryK ? __ldg(a.ecand + eo + lane) : -1;
            const float hd = hub >= 0 ? __ldg(a.edist + eo + lane) : INFINITY;
            float dmin = hd;
#pragma unroll
            for (int w = 16; w >= 1; w >>= 1) dmin = fminf(dmin, __shfl_xor_sync(FULL, dmin, w));
            const float rel = hub >= 0 ? hd / fmaxf(dmin, 1e-30f) : 0.0f;
            const int valid = __popc(__ballot_sync(FULL, hub >= 0));
            n_seeds = a.n_multiprobe < valid ? a.n_multiprobe : valid;
            if (n_seeds > 32) n_seeds = 32;
            if (LM == 1 && a.tr_entry_feat != nullptr && lane < kFeat)
                a.tr_entry_feat[(int64_t)qid * kFeat + lane] = hub >= 0 ? fminf(rel, 64.0f) * (1.0f / 64.0f) : 1.0f;
            if (a.entry_w != nullptr) {
                float f[kFeat];
#pragma unroll
                for (int i = 0; i < kFeat; ++i) {
                    const float ri = __shfl_sync(FULL, rel, i);
                    const int hi = __shfl_sync(FULL, hub, i);
                    f[i] = hi >= 0 ? fminf(ri, 64.0f) * (1.0f / 64.0f) : 1.0f;
                }
                const float z = mlp_warp(a.entry_w, f, kEntryK, lane);
                bool used = false;
                for (int s2 = 0; s2 < n_seeds; ++s2) {  // candidates by decreasing score
                    const unsigned key = (hub >= 0 && !used) ? fkey(z) : 0u;
                    const unsigned mk = __reduce_max_sync(FULL, key);
                    const int win = __ffs(__ballot_sync(FULL, hub >= 0 && !used && key == mk)) - 1;
                    const int h = __shfl_sync(FULL, hub, win);
                    if (lane == s2) seed_id = h;
                    if (lane == win) used = true;
                }
            } else {
                seed_id = lane < n_seeds ? hub : -1;
            }
            if (n_seeds < 1) {  // no hub at all: the reference's entry points
                n_seeds = a.n_multiprobe;
                seed_id = -1;
            }
        } else if (a.n_hubs > 0 && !given_seeds) {
            int hub = lane < a.n_hubs ? __ldg(a.hubs + lane) : -1;
            unsigned HN = __ballot_sync(FULL, hub >= 0);  // hubs are node ids: the lanes below n_hubs
            const float hd = distances(hub, HN);
            float dmin = hub >= 0 ? hd : INFINITY;
#pragma unroll
            for (int w = 16; w >= 1; w >>= 1) dmin = fminf(dmin, __shfl_xor_sync(FULL, dmin, w));
            const float rel = hub >= 0 ? hd / fmaxf(dmin, 1e-30f) : 0.0f;
            float f[kFeat];
#pragma unroll
            for (int i = 0; i < kFeat; ++i) f[i] = fminf(__shfl_sync(FULL, rel, i), 64.0f) * (1.0f / 64.0f);
            if (LM == 1 && a.tr_entry_feat != nullptr && lane < kFeat)
                a.tr_entry_feat[(int64_t)qid * kFeat + lane] = lane < a.n_hubs ? fminf(rel, 64.0f) * (1.0f / 64.0f) : 0.0f;
            if (a.entry_w != nullptr) {
                const float z = mlp_warp(a.entry_w, f, a.n_hubs, lane);
                n_seeds = a.n_multiprobe < a.n_hubs ? a.n_multiprobe : a.n_hubs;
                if (n_seeds > 32) n_seeds = 32;
                bool used = false;
                for (int s2 = 0; s2 < n_seeds; ++s2) {  // hubs by decreasing score
                    const unsigned key = (hub >= 0 && !used) ? fkey(z) : 0u;
                    const unsigned mk = __reduce_max_sync(FULL, key);
                    const int win = __ffs(__ballot_sync(FULL, hub >= 0 && !used && key == mk)) - 1;
                    const int h = __shfl_sync(FULL, hub, win);
                    if (lane == s2) seed_id = h;
                    if (lane == win) used = true;
                }
            }
        }
    }

    song_query_trace tr = {};
    bool seeding = true;  // the first pass inserts the N_MULTIPROBE entry points
    for (;;) {
        int limit;
        const int32_t* arow = nullptr;
        // first chunk of each adjacency row; learned searches with beam > 1 expand up
        // to 3 more rows this step (BLOCK_SIZE <= 32: one chunk per row)
        int first = -1, first2 = -1, first3 = -1, first4 = -1;
        int nrows = 1;
        if (seeding) {
            limit = n_seeds;  // seeds p*n/N_MULTIPROBE (kernalGraph.h:214-231)
        } else {              // expansion (kernalGraph.h:233-289)
            if (cand.sz == 0) break;
            unsigned mb, mi;
            int cn;
            if constexpr (QR) {
                root_min_c(cand, mb, mi, lane);
                cn = q_pop(cand, (int)mi, lane);
            } else {
                root_min(cand, mb, mi);
                cn = q_pop<true>(cand, (int)mi, lane);
            }
            const float cmin = __uint_as_float(mb);
            limit = a.block_size;
            arow = a.adj + (int64_t)cn * a.block_size;
            if (lane < limit) first = __ldg(arow + lane);
            tr.expanded_nodes += 1;
            unsigned wb = 0xffffffffu, wi;
            if (res.sz == res.cap) {  // early stop: full and strictly worse than the worst
                if constexpr (QR) root_max_c(res, wb, wi, lane);
                else if constexpr (LM == 0) root_max_c(res, wb, wi);  // cached: plain searches only
                else root_max(res, wb, wi);
                if (fbits(cmin) > wb) {
                    tr.early_stopped = 1;
                    break;
                }
            }
            if constexpr (LM > 0) {
                // Beam (learned searches only; not the reference's order): the next
                // best candidates are expanded in the same step while they would not
                // end the search, so their adjacency rows are fetched in one round trip.
                if (a.beam > 1 && a.block_size <= 32) {
                    for (int bb = 1; bb < a.beam && cand.sz > 0; ++bb) {
                        unsigned mb2, mi2;
                        if constexpr (QR) root_min_c(cand, mb2, mi2, lane);
                        else root_min(cand, mb2, mi2);
                        if (res.sz == res.cap && mb2 > wb) break;
                        int cn2;
                        if constexpr (QR) cn2 = q_pop(cand, (int)mi2, lane);
                        else cn2 = q_pop<true>(cand, (int)mi2, lane);
                        const int f = lane < limit ? __ldg(a.adj + (int64_t)cn2 * a.block_size + lane) : -1;
                        if (bb == 1) first2 = f;
                        else if (bb == 2) first3 = f;
                        else first4 = f;
                        tr.expanded_nodes += 1;
                        nrows = bb + 1;
                    }
                }
            }
            if constexpr (LM == 1 || LM == 2) {  // learned-stop checkpoint
                ss.hops_kth += nrows;
                ss.hops_best += nrows;
                const int t = tr.expanded_nodes;
                // A checkpoint right after the k-th distance improved (hops_kth == 0 after the
                // increment below is impossible; 1 means "improved by the last expansion")
                // cannot be the converged state the model looks for: no evaluation then.
                const bool want = LM == 1 || (a.stop_w != nullptr && a.stop_thr < INFINITY &&
                                              t >= a.min_expansions && ss.kth < INFINITY &&
                                              ss.hops_kth > 1);
                if (t % a.ckpt_every < nrows) {  // a multiple of ckpt_every was reached
                    if (want) {
                        int c1 = 0, c11 = 0, c125 = 0;
                        const float k1 = ss.kth, k11 = ss.kth * 1.1f, k125 = ss.kth * 1.25f;
                        auto count = [&](float v) {
                            c1 += v < k1;
                            c11 += v < k11;
                            c125 += v < k125;
                        };
                        if constexpr (QR) {
#pragma unroll
                            for (int r = 0; r < QR; ++r)
                                if (cand.d[r] != kEmpty) count(__uint_as_float(cand.d[r]));
                        } else {
                            for (int s2 = lane; s2 < cand.sz; s2 += 32) count(cand.d[s2]);
                        }
                        c1 = __reduce_add_sync(FULL, (unsigned)c1);
                        c11 = __reduce_add_sync(FULL, (unsigned)c11);
                        c125 = __reduce_add_sync(FULL, (unsigned)c125);
                        float f[kFeat];
                        stop_features(f, ss, t, cmin, __uint_as_float(wb), res.sz == res.cap,
                                      (float)cand.sz / (float)cand.cap, (float)res.sz / (float)res.cap,
                                      c1, c11, c125, a.ckpt_every * a.block_size);
                        if (LM == 1 && a.tr_feat != nullptr && ss.nck < a.max_ckpt) {
                            const int64_t row = (int64_t)qid * a.max_ckpt + ss.nck;
                            if (lane == 0) {
#pragma unroll
                                for (int i = 0; i < kFeat; ++i) a.tr_feat[row * kFeat + i] = f[i];
                                a.tr_kth[row] = ss.kth;
                            }
                            ss.nck += 1;
                        }
                        if (LM == 2) {
                            const float z = mlp_warp(a.stop_w, f, 1, lane);
                            if (z >= a.stop_thr) {
                                tr.early_stopped = 2;  // learned stop
                                break;
                            }
                        }
                    }
                    ss.kth_prev = ss.kth;
                    ss.n_new = ss.n_res = ss.n_front = 0;
                }
            }
            // The next pop is most often today's runner-up: warm its row in L2.  Learned
            // searches (short queues, rows mostly L2-resident) measured faster without it.
            if (LM == 0 && cand.sz > 0) {
                unsigned nb2, ni2;
                int nid;
                if constexpr (QR) {
                    root_min_c(cand, nb2, ni2, lane);  // kept for the next pop unless a push gets below it
                    nid = cand.id[ni2];
                } else {
                    root_min(cand, nb2, ni2);
                    nid = q_id(cand, (int)ni2);
                }
                if (lane == 0) {
                    const int32_t* nrow = a.adj + (int64_t)nid * a.block_size;
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(nrow));
                }
            }
        }
        for (int rr = 0; rr < nrows; ++rr)
        for (int c0 = 0; c0 < limit; c0 += 32) {
            const int j = c0 + lane;
            int nb = -1;
            if (j < limit) {
                if (seeding) {
                    nb = (given_seeds || (LM > 0 && seed_id >= 0)) ? seed_id
                                                  : (int)((unsigned long long)j * (unsigned long long)a.n /
                                                          (unsigned long long)a.n_multiprobe);
                } else if (rr == 0) {
                    nb = c0 == 0 ? first : __ldg(arow + j);
                } else {  // beam rows: one chunk each
                    nb = rr == 1 ? first2 : (rr == 2 ? first3 : first4);
                }
            }
            if (nb >= a.n) {  // impossible for a validated graph; never read out of range
                atomicExch(a.err, 1);
                nb = -1;
            }
            BloomRow br;
            const unsigned fresh = bloom_test(bloom, nb, bc, br);
            unsigned N = fresh;
            float d = distances(nb, N);
            const unsigned isnew = bloom_new(br, fresh, bc, lane);
            if (isnew != fresh) {  // covered by an earlier id of the row: not new, no push
                if constexpr (QR) {  // the list without them
                    const int m = __popc(isnew);
                    const int src = lane < m ? __popc(fresh & lanemask_lt((int)__fns(isnew, 0, lane + 1))) : 0;
                    d = __shfl_sync(FULL, d, src);
                    nb = __shfl_sync(FULL, nb, src);
                    if (lane >= m) nb = -1;
                    N = m == 32 ? FULL : (1u << m) - 1u;
                } else {
                    N = isnew;
                }
            }
            const int c = __popc(N);
            if (seeding) {
                tr.seed_count += c;
            } else {
                tr.neighbor_slots_scanned += min(32, limit - c0);
                tr.candidate_nodes += c;
            }
            tr.visited_nodes += c;
            tr.distance_evals += c;
            int pf, pr;
            if constexpr (QR) {
                pf = q_push<true>(cand, N, d, nb, lane);
                pr = q_push<false>(res, N, d, nb, lane);
            } else {
                pf = q_push<true>(cand, N, d, nb, lane, rows);
                pr = q_push<false, LM == 0>(res, N, d, nb, lane, rows);
            }
            tr.frontier_pushes += pf;
            tr.result_updates += pr;
            if constexpr (LM == 1 || LM == 2) {
                topk_insert(ss, N, d, lane);
                ss.n_new += c;
                ss.n_res += pr;
                ss.n_front += pf;
                if (seeding) {
                    float m = ((N >> lane) & 1u) ? d : INFINITY;
#pragma unroll
                    for (int w = 16; w >= 1; w >>= 1) m = fminf(m, __shfl_xor_sync(FULL, m, w));
                    ss.entry_d = fminf(ss.entry_d, m);
                }
            }
            if (N) {
                tr.peak_frontier = max(tr.peak_frontier, cand.sz);
                tr.peak_results = max(tr.peak_results, res.sz);
            }
        }
        seeding = false;
    }

    if constexpr (LM == 1) {
        if (lane == 0 && a.tr_count != nullptr) {
            a.tr_count[qid] = ss.nck;
            a.tr_final_kth[qid] = ss.kth;
        }
    }
    // a launch that may have started before the previous one on its stream
    // finished writes nothing until that launch is complete
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float* outd = a.out_dist ? a.out_dist + (int64_t)qid * a.k : nullptr;
    if constexpr (DT != SONG_PREC_FP32) {
        if (a.rerank) {  // the FP32 rows' distances read the query in element order
            const float* qg = reinterpret_cast<const float*>(a.queries) + (int64_t)qid * a.qld;
            __syncwarp();
            for (int i = lane; i < a.qdim; i += 32) sq[i] = i < a.dim ? __ldcg(qg + i) : 0.0f;
            __syncwarp();
        }
    }
    if constexpr (QR) {
        if (DT != SONG_PREC_FP32 && a.rerank)
            tr.result_count = rerank_finish(a, res, sq, a.out + (int64_t)qid * a.k, outd, lane,
                                            reinterpret_cast<float*>(bloom));
        else
            tr.result_count = finish(res, a.k, a.out + (int64_t)qid * a.k, outd, lane, reinterpret_cast<int*>(bloom));
    } else {
        if (DT != SONG_PREC_FP32 && a.rerank)
            tr.result_count = rerank_finish(a, res, cand, sq, a.out + (int64_t)qid * a.k, outd, lane);
        else
            tr.result_count = finish(res, cand, a.k, a.out + (int64_t)qid * a.k, outd, lane,
                                     reinterpret_cast<int*>(bloom));
    }
    if (TR && a.trace != nullptr && lane == 0) a.trace[qid] = tr;
}

// Launch shape of a search_kernel instance.  Queues of up to 1024 slots run
// in CTAs of 4 warps with at most 96 registers per thread, so that 5 CTAs
// (20 warps) fit an SM.  The search is latency-bound and gains from every
// resident query, but not at the price of spills: capped at 80 registers (6
// CTAs) the plain and entry-only instances spilled 100-190 bytes and ran
// 16 % (plain) and 13 % (learned) slower.  The plain and precision searches
// (LM = 0, queues of hundreds of slots) keep their result ids in TMEM (TM),
// one warp per TMEM lane quarter, and their candidate ids (the hotter queue:
// every expansion pops it) in shared memory: at ef 512 with a 512-word Bloom
// filter that still fits 5 CTAs per SM, where both id arrays in shared
// memory would not (measured 4-5 % faster than both in TMEM, 11 % faster
// than both in shared memory).  Both placements are compiled; the launcher
// takes the candidate ids into TMEM too when shared memory would otherwise
// cost resident CTAs (large queues and Bloom filters).  Learned searches run short queues, whose ids fit
// shared memory without costing warps, and there an id access is one
// shared-memory load instead of a TMEM round trip (measured 11 % faster).
// The trace and learned-stop instances (LM = 1, 2: checkpoint features, a
// running top-k) still spilled at 96 registers; they get 128 (4 CTAs, 16
// warps), measured 13-16 % faster.  Larger queues keep the ids in shared
// memory, up to 8 warps per CTA.
template <int KIND, int NE, int GPL, int DT, int LM, int QR = 0>
struct KernelShape {
    static constexpr int kTM = (GPL == 1 && LM == 0 && QR == 0) ? 1 : 0;   // result ids in TMEM
    static constexpr int kThreads = GPL == 1 ? 128 : 256;
    // byte-row instances (NE < 0) hold fewer query registers: 80 per thread and 6 CTAs
    // (plain, learned entry without the stop model: 72 and 7 CTAs spilled and took
    // 8 % longer at ef 256), 96 and 5 CTAs (learned entry and stop)
    static constexpr int kMinBlocks =
        GPL == 1 ? (LM == 1 ? 4
                            : (LM == 2 ? (NE < 0 ? 5 : 4) : (NE < 0 ? 6 : 5)))
                 : 1;
    // without the trace counters (TR = 0): one more CTA
    static constexpr int kMinBlocksNT = GPL == 1 && (NE < 0 || KIND == 1) ? kMinBlocks + 1 : kMinBlocks;
    // register queues: 96 registers (5 CTAs), without the trace counters 80 (6); float
    // rows keep 8 loads in flight and spilled at 96: 128 (4 CTAs), 15 % faster at 500
    // queries and 960 dimensions, the same at 10,000
    static constexpr int kMinBlocksQ = LM == 2 || (KIND == 0 && NE == 0 && DT == SONG_PREC_FP32) ? 4 : 5;
    static constexpr int kMinBlocksQNT = LM == 2 ? 5 : 6;
    static constexpr bool kQuerySmem = KIND == 0 && NE == 0;  // query kept in shared memory
};

// TMC = 1 (TM instances only): the candidate ids in TMEM as well.  TR = 0:
// no per-query trace.  TD = 1 (with TMC = 1): the result distances in TMEM.
template <int KIND, int NE, int GPL, int DT, int LM = 0, int TMC = 0, int TR = 1, int TD = 0, int QR = 0>
__global__ void __launch_bounds__((KernelShape<KIND, NE, GPL, DT, LM, QR>::kThreads),
                                  (QR ? (TR ? KernelShape<KIND, NE, GPL, DT, LM, QR>::kMinBlocksQ
                                            : KernelShape<KIND, NE, GPL, DT, LM, QR>::kMinBlocksQNT)
                                      : (TR ? KernelShape<KIND, NE, GPL, DT, LM, QR>::kMinBlocks
                                            : KernelShape<KIND, NE, GPL, DT, LM, QR>::kMinBlocksNT)))
    search_kernel(const SearchArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int TM = KernelShape<KIND, NE, GPL, DT, LM, QR>::kTM;
    static_assert(TM || !TMC, "candidate ids in TMEM need a TMEM allocation");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char* ws = smem + (size_t)warp * a.warp_smem;
    uint32_t tbase = 0;
    __shared__ uint32_t tm_slot;
    if constexpr (TM) {  // one TMEM allocation per CTA, warp w uses lanes 32(w%4) .. +31
        if (warp == 0) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                         :: "r"((uint32_t)__cvta_generic_to_shared(&tm_slot)), "r"(a.tm_cols)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tbase = tm_slot + ((uint32_t)(32 * (warp & 3)) << 16) +
                (uint32_t)((warp >> 2) * a.tm_warp_cols);
    }
    for (;;) {
        int qid = 0;
        if (lane == 0) qid = (int)atomicAdd(a.counter, 1u);
        qid = __shfl_sync(FULL, qid, 0);
        if (qid >= a.nq) break;
        search_query<KIND, NE, GPL, DT, LM, TM, TMC, TR, TD, QR>(a, qid, ws, lane, tbase);
    }
    // Every query of this launch has been claimed: a search launched after
    // this one on the stream with programmatic serialization may start on
    // the resources this launch's tail leaves idle (it reads only the index
    // and its own queries, and waits for this launch before it writes).
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if constexpr (TM) {  // every warp is done with TMEM before it is freed
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (warp == 0)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                         :: "r"(tm_slot), "r"(a.tm_cols) : "memory");
    }
    if (a.done != nullptr) {
        // The last CTA past its loop returns the work counter to zero for the
        // launch that takes this ring slot next, so no memset has to sit
        // between two launches on the stream.
        if constexpr (!TM) __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(a.done, 1u) == gridDim.x - 1) {
                atomicExch(a.counter, 0u);
                atomicExch(a.done, 0u);
            }
        }
    }
}

template <int KIND, int NE, int GPL, int DT, int LM = 0>
KernelSel ksel() {
    using S = KernelShape<KIND, NE, GPL, DT, LM>;
    KernelSel k;
    k.fn = search_kernel<KIND, NE, GPL, DT, LM, 0>;
    if constexpr (S::kTM) k.fn_tmc = search_kernel<KIND, NE, GPL, DT, LM, 1>;
    if constexpr ((NE < 0 || KIND == 1) && LM != 1) {  // trace-free copies where they fit one more CTA
        k.fn_nt = search_kernel<KIND, NE, GPL, DT, LM, 0, 0>;
        if constexpr (S::kTM) {
            k.fn_tmc_nt = search_kernel<KIND, NE, GPL, DT, LM, 1, 0>;
            k.fn_tmd_nt = search_kernel<KIND, NE, GPL, DT, LM, 1, 0, 1>;
        }
    }
    if constexpr (S::kTM && (NE < 0 || KIND == 1 || DT != SONG_PREC_FP32))
        k.fn_tmd = search_kernel<KIND, NE, GPL, DT, LM, 1, 1, 1>;
    k.tm = S::kTM;
    k.threads = S::kThreads;
    k.query_smem = S::kQuerySmem;
    return k;
}

template <int KIND, int NE, int DT, int LM, int QR>
KernelSel ksel_reg() {
    using S = KernelShape<KIND, NE, 1, DT, LM, QR>;
    KernelSel k;
    k.fn = search_kernel<KIND, NE, 1, DT, LM, 0, 1, 0, QR>;
    if constexpr (NE < 0 || KIND == 1) k.fn_nt = search_kernel<KIND, NE, 1, DT, LM, 0, 0, 0, QR>;
    k.qr = QR;
    k.threads = S::kThreads;
    k.query_smem = S::kQuerySmem;
    return k;
}

// The register-queue instance for a.cap slots; none above 256.
template <int KIND, int NE, int DT, int LM>
KernelSel reg_queues(const SearchArgs& a) {
    if (a.cap <= 64) return ksel_reg<KIND, NE, DT, LM, 2>();
    if (a.cap <= 128) return ksel_reg<KIND, NE, DT, LM, 4>();
    if (a.cap <= 160) return ksel_reg<KIND, NE, DT, LM, 5>();
    if (a.cap <= 256) return ksel_reg<KIND, NE, DT, LM, 8>();
    return KernelSel();
}

// The plain instance for a.cap slots.
template <int KIND, int NE, int DT>
KernelSel by_cap(const SearchArgs& a, bool reg) {
    if (reg) return reg_queues<KIND, NE, DT, 0>(a);
    if (a.cap <= 1024) return ksel<KIND, NE, 1, DT>();
    if (a.cap <= 2048) return ksel<KIND, NE, 2, DT>();
    if (a.cap <= 4096) return ksel<KIND, NE, 4, DT>();
    return KernelSel();
}

}  // namespace

// Instances by file (song_search_*.cu).  reg: queues in registers; an empty
// selection means none for these arguments.
// query_global: an instance that can read the query from global memory.
KernelSel pick_l2(const SearchArgs& a, bool reg, bool query_global = false);
KernelSel pick_lowp(const SearchArgs& a, bool reg);
KernelSel pick_hamming(const SearchArgs& a, bool reg);
KernelSel pick_learned(const SearchArgs& a, bool reg);

}  // namespace song
