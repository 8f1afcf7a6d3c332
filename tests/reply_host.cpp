// Host build of the move generator's headers for test_reply_sum.py: the CUDA
// qualifiers and intrinsics they use, spelled in plain C++, and one entry
// that counts the last two plies of boards both ways.
#include <algorithm>
#include <cstdint>
#include <cstring>

#define __device__
#define __host__
#define __constant__
#define __shared__
#define __noinline__
#define __forceinline__ inline
#define __align__(n) __attribute__((aligned(n)))

struct uint4 { unsigned x, y, z, w; };
struct Dim { int x; };
static Dim threadIdx{0}, blockDim{1};
typedef int cudaError_t;
using std::max;
using std::min;
template <class T> static T __ldg(const T* p) { return *p; }
static int __popc(unsigned x) { return __builtin_popcount(x); }
static int __popcll(unsigned long long x) { return __builtin_popcountll(x); }
static int __ffs(unsigned x) { return __builtin_ffs((int)x); }
static int __ffsll(long long x) { return __builtin_ffsll(x); }
static int __clzll(long long x) { return x ? __builtin_clzll((unsigned long long)x) : 64; }
static unsigned long long __brevll(unsigned long long x)
{
    unsigned long long r = 0;
    for (int i = 0; i < 64; i++) r |= ((x >> i) & 1ull) << (63 - i);
    return r;
}
static unsigned __activemask() { return 1u; }
static int __any_sync(unsigned, int p) { return p; }
static void __syncthreads() {}
template <class D> static int cudaMemcpyToSymbol(D& d, const void* s, size_t n) { memcpy((void*)&d, s, n); return 0; }
static int cudaStreamSynchronize(int) { return 0; }

#include "pg_reply.cuh"

namespace pg {
unsigned char pg_dyn_smem[16];

struct Moves {  // the emitter of both generators
    u16 mv[4096];
    u32 pc[4096];
    u32 n = 0, kings = 0;
    u32 king_entry[4096];
    void operator()(u16 m, u32 piece) { put((u32)m | (piece << Q_PIECE_SHIFT)); }
    void put(u32 ent)
    {
        mv[n] = (u16)ent;
        pc[n++] = (ent >> Q_PIECE_SHIFT) & 15u;
    }
    void put_ep(u32 ent) { put(ent); }
    void sets(u64 rest, u64 by_king, u32 first, u32 mul)
    {
        each_square(rest, [&](int t) { put(first + (u32)t * mul); });
        each_square(by_king, [&](int t) { king_entry[kings++] = first + (u32)t * mul; });
    }
};

template <int S> static u64 replies(const Pos& b, const Moves& e)
{
    u64 sum = 0;
    for (u32 i = 0; i < e.n; i++) {
        Pos c = b;
        make_child<S>(c, e.mv[i], e.pc[i]);
        sum += count_moves_ks1<1 - S>(c);
    }
    for (u32 i = 0; i < e.kings; i++)
        sum += king_replies<S>(b, (u16)e.king_entry[i], (e.king_entry[i] >> Q_PIECE_SHIFT) & 15u);
    return sum;
}

template <int S> static void both_ways(const Pos& b, u64* split, u64* made, u32* moves, u32* queued)
{
    Moves all, rest;
    gen_from_facts<S>(b, ks_facts<S>(b), all);
    *made = replies<S>(b, all);
    *split = reply_sum<S>(b, rest);
    *split += replies<S>(b, rest);
    *moves = all.n;
    *queued = rest.n + rest.kings;
}
}  // namespace pg

extern "C" int reply_both_ways(const pg::Pos* b, u32 n, u64* split, u64* made, u32* moves, u32* queued)
{
    const pg::HostTables* t = pg::host_tables();
    if (!t) return 1;
    pg::upload_static_tables(*t);
    for (u32 i = 0; i < n; i++) {
        if (pg::st_side(b[i])) pg::both_ways<1>(b[i], split + i, made + i, moves + i, queued + i);
        else pg::both_ways<0>(b[i], split + i, made + i, moves + i, queued + i);
    }
    return 0;
}
