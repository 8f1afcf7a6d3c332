// pg_ops_impl.cuh -- launch wrappers instantiated once per slider policy.
// Included by exactly one translation unit per policy (pg_sl_*.cu).
#pragma once
#include <algorithm>

#include "pg_kernels.cuh"
#include "pg_ops.cuh"

namespace pg {
namespace {

// shared-memory queue entries per CTA.  The leaf queues the moves that are not
// counted in sets, about 10 a node: 16 per thread hold them in one window on
// most CTAs, and a CTA with more gathers another window from its columns.
// (Every 16th position of the batched workload: 30.7 ms with 16, 30.8 with 20
// to 32, 31.0 with 12: what the queue takes is missing in the L1.)
// The expansion queues every move: 64 per thread hold the children of nodes
// with ~50 moves.  The byte-lookup policy gives 158 KB of the CTA's shared
// memory to its tables and keeps 8.
template <class SL, int T> struct QcapFor {
    static constexpr int leaf = SL::kId == 2 ? T * 8 : T * 16;
    static constexpr int expand = SL::kId == 2 ? T * 8 : T * 64;
};

inline int full_grid(int per_sm, int T, u64 items, int num_sms)
{
    const u64 want = std::max<u64>(1, (items + T - 1) / T);
    return (int)std::min<u64>(want, (u64)per_sm * (u64)num_sms);
}

template <class SL>
cudaError_t upload_tables(const HostTables& t)
{
    return upload_static_tables(t);
}

template <int S, class SL, int T, bool SPARSE>
cudaError_t leaf_t(const LevelView& lv, u32 start, u32 n, u64* acc, u32* ticket, u32 max_rem, const u32* n_dev,
                   cudaStream_t st, int sms)
{
    constexpr int Q = QcapFor<SL, T>::leaf;
    using L = LeafSmem<SL, T, Q>;
    auto fn = k_leaf<S, SL, T, Q, SPARSE>;
    static KernelSetup setup;
    if (const cudaError_t e = setup.once((const void*)fn, T, L::bytes)) return e;
    // a CTA for every node until the chip is full (node_chunk)
    const int grid = full_grid(setup.per_sm, T, SPARSE ? n : (u64)n * T, sms);
    fn<<<grid, T, L::bytes, st>>>(lv, start, n, acc, ticket, max_rem, n_dev);
    return cudaGetLastError();
}

template <int S, class SL, int T>
cudaError_t expand_t(const LevelView& in, u32 start, u32 a, u32 b, const u64* offs, const LevelView& out, u32* ticket,
                     Ahead ahead, cudaStream_t st, int sms)
{
    constexpr int Q = QcapFor<SL, T>::expand;
    using L = BlockSmem<SL, T, Q>;
    auto fn = k_expand<S, SL, T, Q>;
    static KernelSetup setup;
    if (const cudaError_t e = setup.once((const void*)fn, T, L::bytes)) return e;
    const int grid = full_grid(setup.per_sm, T, (u64)(b - a) * T, sms);
    fn<<<grid, T, L::bytes, st>>>(in, start, a, b, offs, out, ticket, nullptr, ahead);
    return cudaGetLastError();
}

// The CTA size is the caller's, on a sparse level too; the duplicate pass takes 256
// where it is left open (64 positions at depth 6, the whole call: 17.1 ms with
// 256 threads, 17.4 with 512, 21.4 with 128).
template <int S, class SL, bool SPARSE>
cudaError_t leaf_size(int T, const LevelView& lv, u32 start, u32 n, u64* acc, u32* ticket, u32 max_rem, const u32* n_dev,
                      cudaStream_t st, int sms)
{
    return T == 128   ? leaf_t<S, SL, 128, SPARSE>(lv, start, n, acc, ticket, max_rem, n_dev, st, sms)
           : T == 512 ? leaf_t<S, SL, 512, SPARSE>(lv, start, n, acc, ticket, max_rem, n_dev, st, sms)
                      : leaf_t<S, SL, 256, SPARSE>(lv, start, n, acc, ticket, max_rem, n_dev, st, sms);
}

template <class SL>
cudaError_t leaf_any(int side, int T, const LevelView& lv, u32 start, u32 n, u64* acc, u32* ticket, u32 max_rem,
                     bool sparse, const u32* n_dev, cudaStream_t st, int sms)
{
    if (sparse)
        return side ? leaf_size<1, SL, true>(T, lv, start, n, acc, ticket, max_rem, n_dev, st, sms)
                    : leaf_size<0, SL, true>(T, lv, start, n, acc, ticket, max_rem, n_dev, st, sms);
    return side ? leaf_size<1, SL, false>(T, lv, start, n, acc, ticket, max_rem, n_dev, st, sms)
                : leaf_size<0, SL, false>(T, lv, start, n, acc, ticket, max_rem, n_dev, st, sms);
}

template <class SL>
cudaError_t expand_any(int side, int T, const LevelView& in, u32 start, u32 a, u32 b, const u64* offs,
                       const LevelView& out, u32* ticket, Ahead ahead, cudaStream_t st, int sms)
{
    if (T == 128) return side ? expand_t<1, SL, 128>(in, start, a, b, offs, out, ticket, ahead, st, sms) : expand_t<0, SL, 128>(in, start, a, b, offs, out, ticket, ahead, st, sms);
    if (T == 512) return side ? expand_t<1, SL, 512>(in, start, a, b, offs, out, ticket, ahead, st, sms) : expand_t<0, SL, 512>(in, start, a, b, offs, out, ticket, ahead, st, sms);
    return side ? expand_t<1, SL, 256>(in, start, a, b, offs, out, ticket, ahead, st, sms) : expand_t<0, SL, 256>(in, start, a, b, offs, out, ticket, ahead, st, sms);
}

template <int S, class SL>
cudaError_t count_level_t(const LevelView& lv, u32 start, u32 n, u32* cnt, u32 min_rem, cudaStream_t st, int sms)
{
    auto fn = k_count_level<S, SL>;
    constexpr int smem = table_smem_bytes<SL>();
    static KernelSetup setup;
    if (const cudaError_t e = setup.once((const void*)fn, 256, smem)) return e;
    const int grid = full_grid(setup.per_sm, 256, n, sms);
    fn<<<grid, 256, smem, st>>>(lv, start, n, cnt, min_rem);
    return cudaGetLastError();
}

template <class SL>
cudaError_t count_level_any(int side, const LevelView& lv, u32 start, u32 n, u32* cnt, u32 min_rem, cudaStream_t st,
                            int sms)
{
    return side ? count_level_t<1, SL>(lv, start, n, cnt, min_rem, st, sms)
                : count_level_t<0, SL>(lv, start, n, cnt, min_rem, st, sms);
}

template <int S, class SL>
cudaError_t count_plan_t(const LevelView& lv, u32 start, u32 n, u32* cnt, u32 min_rem, u64* offs, u64 cap, PlanOut* plan,
                         u32* done, const u32* err, Ahead ahead, cudaStream_t st)
{
    auto fn = k_count_plan<S, SL>;
    constexpr int smem = table_smem_bytes<SL>();
    static KernelSetup setup;
    if (const cudaError_t e = setup.once((const void*)fn, 256, smem)) return e;
    fn<<<(n + 255) / 256, 256, smem, st>>>(lv, start, n, cnt, min_rem, offs, cap, plan, done, err, ahead);
    return cudaGetLastError();
}

template <class SL>
cudaError_t count_plan_any(int side, const LevelView& lv, u32 start, u32 n, u32* cnt, u32 min_rem, u64* offs, u64 cap,
                           PlanOut* plan, u32* done, const u32* err, Ahead ahead, cudaStream_t st)
{
    return side ? count_plan_t<1, SL>(lv, start, n, cnt, min_rem, offs, cap, plan, done, err, ahead, st)
                : count_plan_t<0, SL>(lv, start, n, cnt, min_rem, offs, cap, plan, done, err, ahead, st);
}

template <int S, class SL>
cudaError_t step_t(const LevelView& lv, u32 start, u32 n, u32* cnt, u32 min_rem, u64* offs, u64 cap, PlanOut* plan, const u32* err,
                   Ahead ahead, const LevelView& out, u32* ticket, cudaStream_t st)
{
    constexpr int Q = QcapFor<SL, 256>::expand;
    using L = BlockSmem<SL, 256, Q>;
    auto fn = k_step<S, SL, Q>;
    static KernelSetup setup;
    if (const cudaError_t e = setup.once((const void*)fn, 256, L::bytes)) return e;
    fn<<<1, 256, L::bytes, st>>>(lv, start, n, cnt, min_rem, offs, cap, plan, err, ahead, out, ticket);
    return cudaGetLastError();
}

template <class SL>
cudaError_t step_any(int side, const LevelView& lv, u32 start, u32 n, u32* cnt, u32 min_rem, u64* offs, u64 cap, PlanOut* plan,
                     const u32* err, Ahead ahead, const LevelView& out, u32* ticket, cudaStream_t st)
{
    return side ? step_t<1, SL>(lv, start, n, cnt, min_rem, offs, cap, plan, err, ahead, out, ticket, st)
                : step_t<0, SL>(lv, start, n, cnt, min_rem, offs, cap, plan, err, ahead, out, ticket, st);
}

inline int small_grid(u32 n, int T) { return (int)std::max<u32>(1, std::min<u32>((n + T - 1) / T, 8192)); }

template <class SL>
cudaError_t count_batch(const Pos* in, u32 n, u32* out, cudaStream_t st)
{
    constexpr int smem = table_smem_bytes<SL>();
    static KernelSetup setup;
    if (const cudaError_t e = setup.once((const void*)k_count_batch<SL>, 128, smem)) return e;
    k_count_batch<SL><<<small_grid(n, 128), 128, smem, st>>>(in, n, out);
    return cudaGetLastError();
}

template <class SL>
cudaError_t gen_moves_batch(const Pos* in, u32 n, u16* out, u32* nout, cudaStream_t st)
{
    constexpr int smem = table_smem_bytes<SL>();
    static KernelSetup setup;
    if (const cudaError_t e = setup.once((const void*)k_gen_moves_batch<SL>, 128, smem)) return e;
    k_gen_moves_batch<SL><<<small_grid(n, 128), 128, smem, st>>>(in, n, out, nout);
    return cudaGetLastError();
}

template <class SL>
cudaError_t gen_boards_batch(const Pos* in, u32 n, Pos* out, u32* nout, cudaStream_t st)
{
    constexpr int smem = table_smem_bytes<SL>();
    static KernelSetup setup;
    if (const cudaError_t e = setup.once((const void*)k_gen_boards_batch<SL>, 128, smem)) return e;
    k_gen_boards_batch<SL><<<small_grid(n, 128), 128, smem, st>>>(in, n, out, nout);
    return cudaGetLastError();
}

inline cudaError_t make_batch(Pos* pos, const u16* mv, u32 n, cudaStream_t st)
{
    k_make_batch<<<small_grid(n, 128), 128, 0, st>>>(pos, mv, n);
    return cudaGetLastError();
}

inline cudaError_t make_children(const Pos* root, const u16* mv, const u32* n, Pos* out, cudaStream_t st)
{
    k_make_children<<<1, 256, 0, st>>>(root, mv, n, out);
    return cudaGetLastError();
}

template <class SL>
cudaError_t playouts(const Pos& start, u64 seed, u32 n, int min_plies, int max_plies, int min_moves, int depth_lo,
                     int depth_hi, Pos* out, unsigned char* depths, u32* err, cudaStream_t st)
{
    constexpr int smem = table_smem_bytes<SL>();
    static KernelSetup setup;
    if (const cudaError_t e = setup.once((const void*)k_playouts<SL>, 64, smem)) return e;
    k_playouts<SL><<<small_grid(n, 64), 64, smem, st>>>(start, seed, n, min_plies, max_plies, min_moves, depth_lo,
                                                          depth_hi, out, depths, err);
    return cudaGetLastError();
}

}  // namespace

#define PG_DEFINE_OPS(SLT, NAME, ENUM)                                                                   \
    const SliderOps g_ops_##NAME = {#NAME,          ENUM,                    upload_tables<SLT>,           \
                                    leaf_any<SLT>,  expand_any<SLT>,         count_level_any<SLT>,         \
                                    count_plan_any<SLT>, step_any<SLT>,                                           \
                                    count_batch<SLT>, gen_moves_batch<SLT>,  gen_boards_batch<SLT>,        \
                                    make_batch,     make_children,           playouts<SLT>};

}  // namespace pg
