// pg_kernels.cuh -- CUDA kernels of the perft engine (sm_103a).
//
// Breadth-first expansion of the reference's GPU path (perft_bb.h:1027-1138:
// per level count -> exclusive scan -> parent expansion -> generate + make,
// count-only leaf) re-planned for one GB300:
//   k_count_level   children per node of a level (countMoves)
//   k_scan          single-pass exclusive scan, decoupled look-back with a
//                   bounded spin (replaces moderngpu ScanD, scan.cuh:330)
//   k_plan          greedy split of a level into chunks whose children fit
//                   the next level's buffer (HBM budget)
//   k_count_plan    the three in one launch for a small level; k_step: with
//                   the expansion as well, for a few nodes
//   k_expand        generate + make into the next level; the CTA stages its
//                   nodes in shared memory, emits (parent, move) entries into
//                   a shared queue and writes children coalesced in 16-byte
//                   vectors (replaces IntervalExpand + generate_moves +
//                   makemove_and_count, perft_bb.h:601,983; intervalmove.cuh:405)
//   k_leaf          the last two plies inside one CTA: each thread sums one
//                   node's replies to its plain moves in sets (pg_reply.cuh)
//                   and queues the other moves as (parent, move) entries, then
//                   every thread makes + counts entries, so the per-thread
//                   work is even whatever the branching
//                   (replaces makeMove_and_perft_single_level_indices,
//                   perft_bb.h:412)
#pragma once
#include "pg_level.cuh"
#include "pg_movegen.cuh"
#include "pg_reply.cuh"

namespace pg {

// per-thread running sum for one group id; flushed with one atomic per
// group change and one per warp at the end when the warp shares the group
struct GroupAcc {
    static constexpr u32 NONE = 0xFFFFFFFFu;
    u32 g = NONE;
    u64 s = 0;
    __device__ __forceinline__ void add(u64* acc, u32 grp, u64 v)
    {
        if (grp != g) {
            if (s) atomicAdd(&acc[g], s);
            g = grp;
            s = 0;
        }
        s += v;
    }
    __device__ __forceinline__ void flush_warp(u64* acc)
    {
        const unsigned full = 0xFFFFFFFFu;
        const u32 g0 = __shfl_sync(full, g, 0);
        const bool same = __all_sync(full, g == g0 || s == 0);
        if (same) {
            u64 t = s;
            for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(full, t, o);
            if ((threadIdx.x & 31) == 0 && t && g0 != NONE) atomicAdd(&acc[g0], t);
        } else if (s) {
            atomicAdd(&acc[g], s);
        }
        s = 0;
        g = NONE;
    }
};

// exclusive scan of one u32 per thread over a CTA of T threads
template <int T>
__device__ __forceinline__ u32 block_excl_scan(u32 v, u32& total, u32* s_warp)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u32 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        u32 w = lane < T / 32 ? s_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 y = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < T / 32) s_warp[lane] = w;
    }
    __syncthreads();
    total = s_warp[T / 32 - 1];
    return (warp ? s_warp[warp - 1] : 0u) + x - v;
}

// writes the moves of one node whose queue positions fall in [lo, hi)
struct QEmit {
    u32* q;
    u32 pos, lo, hi, tag;
    // bits 25-28 carry the moving piece (PC_*) and PC_EP_FLAG for make_child
    __device__ __forceinline__ void operator()(u16 m, u32 piece)
    {
        if (pos >= lo && pos < hi) q[pos - lo] = tag | m | (piece << 25);
        ++pos;
    }
};

// reply_sum's emitters for the leaf

// the queued moves of one thread, in a column of CAP words of its own in shared
// memory (interleaved over the threads, STRIDE = threads) or local memory: the
// moves to make from its start, the king recounts from its end.  Moves that do
// not fit are only counted.
template <int STRIDE, int CAP> struct QColumn {
    u32* col;
    u32 tag, made, kings, eps;  // made counts the en-passant children (eps) too
    __device__ __forceinline__ void put(u32 ent)
    {
        if (made < (u32)CAP) col[made * STRIDE] = tag + ent;
        made++;
    }
    __device__ __forceinline__ void put_ep(u32 ent)
    {
        put(ent);
        eps++;
    }
    __device__ __forceinline__ void sets(u64 rest, u64 by_king, u32 first, u32 mul)
    {
        auto half = [&](u32 r, u32 k, u32 f) {
            for (u32 x = r | k; x; x &= x - 1) {
                const int t = __ffs(x) - 1;
                const u32 king = (k >> t) & 1u;
                const u32 at = king ? (u32)CAP - 1u - kings : made;
                kings += king;
                made += 1u - king;
                if (at < (u32)CAP) col[at * STRIDE] = f + (u32)t * mul;
            }
        };
        half((u32)rest, (u32)by_king, tag + first);
        half((u32)(rest >> 32), (u32)(by_king >> 32), tag + first + 32u * mul);
    }
};

// the same moves written at fixed positions by a second pass: those in
// [lo, hi), all kinds in one sequence
struct QWindow {
    u32* q;
    u32 pos, lo, hi, tag, kings;
    __device__ __forceinline__ void put(u32 ent)
    {
        if (pos >= lo && pos < hi) q[pos - lo] = tag + ent;
        pos++;
    }
    __device__ __forceinline__ void put_ep(u32 ent) { put(ent); }
    __device__ __forceinline__ void sets(u64 rest, u64 by_king, u32 first, u32 mul)
    {
        each_square(rest, [&](int t) { put(first + (u32)t * mul); });
        each_square(by_king, [&](int t) { put((first + (u32)t * mul) | Q_KING); });
        kings += popc(by_king);
    }
};
// One node's sum of replies and its queued moves, out of line: the call fixes
// which registers are live across the node phase, and the compiler spills a
// quarter as much as with the sum inlined into the queue's loops (260 -> 80 bytes
// a thread at 128 registers).  Board and results go in registers.  The batch
// workload's leaf 30.5 -> 29.9 ms, one position at depth 7 30.7 -> 29.4 ms, the
// persistent launch 32.7 -> 31.8 ms; the queued moves' count and king recount as
// calls of their own are slower (30.9 and 30.7 ms: their results are few and their
// boards live already).
struct Replies {
    u64 sum;
    u32 made, kings, eps;
};
template <int S, int STRIDE, int CAP>
__device__ __noinline__ Replies node_replies(u64 w, u64 p, u64 n, u64 bq, u64 rq, u64 k, u32* column, u32 tag)
{
    const Pos b{w, p, n, bq, rq, k};
    QColumn<STRIDE, CAP> e{column, tag, 0u, 0u, 0u};
    const u64 sum = reply_sum<S>(b, e);
    return Replies{sum, e.made, e.kings, e.eps};
}
// one node's part of a queue window (rare: a CTA with more children than its
// queue holds), out of line so that the leaf keeps one copy of reply_sum
template <int S> __device__ __noinline__ void queue_window(const Pos& b, u32* q, u32 off, u32 lo, u32 hi, u32 tag)
{
    QWindow e{q, off, lo, hi, tag, 0u};
    reply_sum<S>(b, e);
}

struct ArrEmit {
    u16* out;
    u32 n;
    __device__ __forceinline__ void operator()(u16 m)
    {
        if (n < 256) out[n] = m;
        ++n;
    }
};

struct BoardEmit {
    Pos* out;
    u32 n;
    __device__ __forceinline__ void operator()(const Pos& p)
    {
        if (n < 256) out[n] = p;
        ++n;
    }
};

template <class SL> __device__ __forceinline__ u32 count_any(const Pos& b)
{
    return st_side(b) ? count_moves<1, SL>(b) : count_moves<0, SL>(b);
}

// ---------------------------------------------------------------------------
// operator-surface kernels (mixed sides, one thread per position)
// ---------------------------------------------------------------------------

template <class SL>
__global__ void k_count_batch(const Pos* __restrict__ in, u32 n, u32* __restrict__ out)
{
    stage_tables<SL>();
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = count_any<SL>(in[i]);
}

template <class SL>
__global__ void k_gen_moves_batch(const Pos* __restrict__ in, u32 n, u16* __restrict__ out, u32* __restrict__ nout)
{
    stage_tables<SL>();
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        ArrEmit e{out + (u64)i * 256, 0};
        const Pos b = in[i];
        if (st_side(b)) gen_moves<1, SL>(b, e); else gen_moves<0, SL>(b, e);
        nout[i] = e.n;
    }
}

template <class SL>
__global__ void k_gen_boards_batch(const Pos* __restrict__ in, u32 n, Pos* __restrict__ out, u32* __restrict__ nout)
{
    stage_tables<SL>();
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        BoardEmit e{out + (u64)i * 256, 0};
        const Pos b = in[i];
        if (st_side(b)) gen_boards<1, SL>(b, e); else gen_boards<0, SL>(b, e);
        nout[i] = e.n;
    }
}

static __global__ void k_make_batch(Pos* __restrict__ pos, const u16* __restrict__ mv, u32 n)
{
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        Pos b = pos[i];
        if (st_side(b)) make_move<1>(b, mv[i]); else make_move<0>(b, mv[i]);
        pos[i] = b;
    }
}

// the children of one position by its *n moves (at most 256)
static __global__ void k_make_children(const Pos* __restrict__ root, const u16* __restrict__ mv, const u32* __restrict__ n,
                                       Pos* __restrict__ out)
{
    const u32 i = threadIdx.x;
    if (i >= min(*n, 256u)) return;
    Pos b = *root;
    if (st_side(b)) make_move<1>(b, mv[i]); else make_move<0>(b, mv[i]);
    out[i] = b;
}

__device__ __forceinline__ u64 splitmix_next(u64& s)
{
    u64 z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// seeded random legal playouts (procedure documented at pg_random_playouts)
template <class SL>
__global__ void k_playouts(Pos start, u64 seed, u32 n, int min_plies, int max_plies, int min_moves, int depth_lo,
                           int depth_hi, Pos* __restrict__ out, unsigned char* __restrict__ depths, u32* err)
{
    stage_tables<SL>();
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        u16 mv[256];
        bool done = false;
        for (u64 a = 0; a < 100000 && !done; a++) {
            u64 s = seed ^ ((u64)i << 32) ^ (a * 0xA24BAED4963EE407ull);
            const int plies = min_plies + (int)(splitmix_next(s) % (u64)(max_plies - min_plies + 1));
            Pos p = start;
            bool ok = true;
            for (int k = 0; k < plies; k++) {
                ArrEmit e{mv, 0};
                if (st_side(p)) gen_moves<1, SL>(p, e); else gen_moves<0, SL>(p, e);
                if (!e.n) {
                    ok = false;
                    break;
                }
                const u16 m = mv[splitmix_next(s) % min(e.n, 256u)];
                if (st_side(p)) make_move<1>(p, m); else make_move<0>(p, m);
            }
            if (ok && (int)count_any<SL>(p) >= min_moves) {
                out[i] = p;
                done = true;
            }
        }
        if (!done) atomicOr(err, ERR_PLAYOUT_ATTEMPTS);
        if (depths) {
            u64 s = seed ^ ((u64)i << 32) ^ 0x5851F42D4C957F2Dull;
            depths[i] = (unsigned char)(depth_lo + (int)(splitmix_next(s) % (u64)(depth_hi - depth_lo + 1)));
        }
    }
}

// ---------------------------------------------------------------------------
// engine kernels
// ---------------------------------------------------------------------------

// The bodies of the level kernels are device functions so that the
// persistent driver (pg_persist.cuh) runs the same code as the per-level
// launches; the kernels below are thin wrappers.  The bodies take no
// __restrict__ on data another phase of a persistent launch writes.

template <int S, class SL>
__device__ __forceinline__ void count_level_body(const LevelView& lv, u32 start, u32 n, u32* cnt, u32 min_rem)
{
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const u32 rem = lv.rem[start + i];
        cnt[i] = (rem >= min_rem && rem < REM_DEAD) ? count_moves<S, SL>(load_board(lv, start + i)) : 0u;
    }
}

template <int S, class SL>
__global__ void k_count_level(LevelView lv, u32 start, u32 n, u32* __restrict__ cnt, u32 min_rem)
{
    stage_tables<SL>();
    count_level_body<S, SL>(lv, start, n, cnt, min_rem);
}

// The scan of a small level's children counts and its chunk plan, by one CTA of
// 256; returns the number of children.  The plan goes straight to pinned host
// memory (nchunks 0: the children do not fit one chunk of `cap`, k_plan has to
// split them; pad: the error bits).  children (or null): their number for a launch
// sequence that does not return to the host between levels; 0 there when they do
// not fit, so that the launches behind do nothing.
__device__ __forceinline__ u64 plan_level(u32 n, const u32* cnt, u64* offs, u64 cap, PlanOut* plan, const u32* err, u32* children)
{
    constexpr int T = 256;
    __shared__ u64 s_warp[T / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u32 per = (n + T - 1) / T, c0 = min(n, tid * per), c1 = min(n, c0 + per);
    u64 sum = 0;
    for (u32 i = c0; i < c1; i++) sum += __ldcg(cnt + i);
    u64 x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    u64 run = x - sum, total = 0;
    for (int w = 0; w < T / 32; w++) {
        if (w < warp) run += s_warp[w];
        total += s_warp[w];
    }
    for (u32 i = c0; i < c1; i++) {
        offs[i] = run;
        run += __ldcg(cnt + i);
    }
    if (tid == 0) {
        offs[n] = total;
        plan->nchunks = total <= cap ? 1u : 0u;
        if (children) *children = total <= cap ? (u32)total : 0u;
        plan->pad = *err;
        plan->total = total;
        plan->bnd[0] = 0;
        plan->bnd[1] = n;
        plan->coff[0] = 0;
        plan->coff[1] = total;
    }
    return total;
}

// Children counts, their scan and the chunk plan of a small level (n up to
// PLAN_FUSED_MAX) in one launch: the last CTA to finish its counts scans them
// all.  ahead: the level's size (null: n) and where its children's number goes.
template <int S, class SL>
__global__ void __launch_bounds__(256) k_count_plan(LevelView lv, u32 start, u32 n, u32* cnt, u32 min_rem, u64* offs, u64 cap,
                                                    PlanOut* plan, u32* done, const u32* err, Ahead ahead)
{
    stage_tables<SL>();
    if (ahead.nodes) n = *ahead.nodes;
    count_level_body<S, SL>(lv, start, n, cnt, min_rem);
    __shared__ u32 s_done;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_done = atomicAdd(done, 1u);
    __syncthreads();
    if (s_done != gridDim.x - 1) return;
    __threadfence();
    plan_level(n, cnt, offs, cap, plan, err, ahead.children);
}

constexpr int LEAF_GATHER = 4;  // nodes a thread looks at when the CTA collects the live ones of a sparse level
constexpr int LEAF_COLUMN = 48;  // queued moves a thread holds before they are gathered

// Nodes per CTA and chunk of a launch over n nodes: the launch's CTAs share a
// small level, fewer nodes than threads each (whole warps of them once there
// are that many).  The node phase then runs on some of a CTA's warps and the
// children, ten (leaf) or thirty (expansion) a node, on all of them, where a full
// chunk would leave SMs idle and give every thread its nodes' children one after
// the other.
struct Share {
    u32 cta, ctas;  // which of the CTAs that work on these nodes this one is
};
__device__ __forceinline__ Share whole_grid() { return Share{blockIdx.x, gridDim.x}; }
__device__ __forceinline__ u32 node_chunk(u32 n, u32 threads, const Share& sh)
{
    const u32 even = (n + sh.ctas - 1) / sh.ctas;
    return min(threads, even <= 32u ? even : (even + 31u) & ~31u);
}

template <class SL, int T, int QCAP> struct BlockSmem {
    static constexpr int tables = table_smem_bytes<SL>();
    static constexpr int boards = T * (int)sizeof(Pos);
    static constexpr int queue = QCAP * 4;
    static constexpr int bytes = tables + boards + queue + T * 4 + T;
};

// the leaf's: no remaining depths, but the threads' columns (in local memory
// where the byte-lookup policy's tables leave no room)
template <class SL, int T, int QCAP> struct LeafSmem {
    static constexpr int tables = table_smem_bytes<SL>();
    static constexpr int boards = T * (int)sizeof(Pos);
    static constexpr int queue = QCAP * 4;
    static constexpr bool column_shared = SL::kId != 2;
    static constexpr int column_at = tables + boards + queue + T * 8;
    static constexpr int bytes = column_at + (column_shared ? T * LEAF_COLUMN * 4 : 0);
};

// register cap: at least PG_LEAF_MIN_WARPS resident warps per SM
#ifndef PG_LEAF_MIN_WARPS
#define PG_LEAF_MIN_WARPS 16
#endif
template <int T> constexpr int min_blocks() { return (PG_LEAF_MIN_WARPS * 32 + T - 1) / T; }

// the last plies of every node with remaining depth <= 2, inside one CTA
// (pg_leaf_body.inc).  The kernel includes the statements in its own body,
// not through this function: with the arguments left in the parameter space
// the compiler keeps more registers for the count (measured 0.5-0.9% faster
// than calling the inlined function).  LV is LevelView or any type with the
// same grp[] / rem[] subscripts and a load_board overload.
template <int S, class SL, int T, int QCAP, bool SPARSE, class LV>
__device__ __forceinline__ void leaf_body(LV lv, u32 start, u32 n, u64* __restrict__ acc, u32* ticket, u32 max_rem,
                                          const u32* n_dev, const Share share)
{
    extern __shared__ __align__(16) unsigned char pg_dyn_smem[];
#include "pg_leaf_body.inc"
}

template <int S, class SL, int T, int QCAP, bool SPARSE>
__global__ void __launch_bounds__(T, min_blocks<T>()) k_leaf(LevelView lv, u32 start, u32 n, u64* __restrict__ acc, u32* ticket,
                                                            u32 max_rem, const u32* __restrict__ n_dev)
{
    extern __shared__ __align__(16) unsigned char pg_dyn_smem[];
    stage_tables<SL>();
    const Share share = whole_grid();
#include "pg_leaf_body.inc"
}

// children of the nodes [a, b) of a level into the next level; offs is the
// exclusive scan of the children counts, child slots start at offs[a]
// parent_out (transposition-table mode): each child's group becomes its own
// slot and its parent's slot is written to parent_out
template <int S, class SL, int T, int QCAP>
__device__ __forceinline__ void expand_body(const LevelView& in, u32 start, u32 a, u32 b, const u64* offs,
                                            const LevelView& out, u32* ticket, u32* parent_out, const Share share)
{
    extern __shared__ __align__(16) unsigned char pg_dyn_smem[];
    using L = BlockSmem<SL, T, QCAP>;
    Pos* sb = reinterpret_cast<Pos*>(pg_dyn_smem + L::tables);
    u32* q = reinterpret_cast<u32*>(pg_dyn_smem + L::tables + L::boards);
    u32* sg = q + QCAP;
    unsigned char* sr = reinterpret_cast<unsigned char*>(sg + T);
    __shared__ u32 s_chunk;
    const int tid = threadIdx.x;
    const u64 out_base = offs[a];
    const u32 per = node_chunk(b - a, T, share);
    for (;;) {
        if (tid == 0) s_chunk = atomicAdd(ticket, 1u);
        __syncthreads();
        const u64 c0 = (u64)a + (u64)s_chunk * per;
        if (c0 >= b) break;
        const u64 c1 = min(c0 + per, (u64)b);
        const u64 i = c0 + tid;
        const u64 chunk_off = offs[c0];
        const u32 total = (u32)(offs[c1] - chunk_off);
        const u64 chunk_out = chunk_off - out_base;
        Pos bd{0, 0, 0, 0, 0, 0};
        u32 c = 0, off = 0, grp = 0;
        unsigned char rem = 0;
        if (i < c1) {
            const u64 o0 = offs[i];
            c = (u32)(offs[i + 1] - o0);
            off = (u32)(o0 - chunk_off);
            bd = load_board(in, start + i);
            grp = in.grp[start + i];
            rem = in.rem[start + i];
        }
        sb[tid] = bd;
        sg[tid] = grp;  // every slot holds a group in range, whatever a queue entry names
        sr[tid] = rem;
        for (u32 lo = 0; lo < total; lo += QCAP) {
            const u32 hi = min(lo + (u32)QCAP, total);
            if (c && off < hi && off + c > lo) {
                QEmit e{q, off, lo, hi, (u32)tid << 16};
                gen_leaf<S>(bd, e);
            }
            __syncthreads();
            const u32 m = hi - lo;
            for (u32 e = tid; e < m; e += T) {
                const u32 ent = q[e];
                const u32 p = (ent >> 16) & (T - 1);  // in bounds even if a queue slot was left unwritten
                Pos ch = sb[p];
                make_move<S>(ch, (u16)(ent & 0xFFFFu));
                const u64 o = chunk_out + lo + e;
                store_board(out, o, ch);
                if (parent_out) {
                    out.grp[o] = (u32)o;
                    parent_out[o] = (u32)(start + c0 + p);
                } else {
                    out.grp[o] = sg[p];
                }
                out.rem[o] = (unsigned char)(sr[p] - 1);
            }
            __syncthreads();
        }
        __syncthreads();
    }
}

template <int S, class SL, int T, int QCAP>
__global__ void __launch_bounds__(T, min_blocks<T>()) k_expand(LevelView in, u32 start, u32 a, u32 b, const u64* __restrict__ offs,
                                              LevelView out, u32* ticket, u32* __restrict__ parent_out = nullptr,
                                              Ahead ahead = Ahead{})
{
    stage_tables<SL>();
    if (ahead.children) {
        if (*ahead.children == 0) return;  // none, or more than `out` holds
        if (ahead.nodes) b = *ahead.nodes;
    }
    expand_body<S, SL, T, QCAP>(in, start, a, b, offs, out, ticket, parent_out, whole_grid());
}

// Counts, plan and expansion of a level of a few nodes (STEP_MAX) by one CTA of
// 256 threads.  Such a call is a chain of launches, each as long as a thread takes
// through its code: one less a level.  One position at depth 3 / 4 / 5: 61 / 82 /
// 121 -> 56 / 73 / 111 us (means of three).
template <int S, class SL, int QCAP>
__global__ void __launch_bounds__(256, min_blocks<256>()) k_step(LevelView in, u32 start, u32 n, u32* cnt, u32 min_rem, u64* offs,
                                                                u64 cap, PlanOut* plan, const u32* err, Ahead ahead, LevelView out,
                                                                u32* ticket)
{
    stage_tables<SL>();
    if (ahead.nodes) n = *ahead.nodes;
    count_level_body<S, SL>(in, start, n, cnt, min_rem);
    __syncthreads();
    const u64 total = plan_level(n, cnt, offs, cap, plan, err, ahead.children);
    __syncthreads();
    if (total == 0 || total > cap) return;
    expand_body<S, SL, 256, QCAP>(in, start, 0, n, offs, out, ticket, nullptr, Share{0u, 1u});
}

}  // namespace pg
