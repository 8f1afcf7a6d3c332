// pg_noalloc.cu -- batched perft for callers that must not allocate device
// memory.
//
// Some callers cannot call cudaMalloc: a serving process that reserved all of
// the GPU's memory up front for its own pool, a framework whose allocator
// owns the device and forbids side allocations, or code that runs where
// allocation is not allowed (a host callback, a timed region that must not
// call into the allocator).  pg_perft_batch_noalloc serves them: every byte
// of working memory it needs lives in one file-scope device array of a fixed
// size (NA_SCRATCH_BYTES, 60 MiB), which every GPU that loads the library
// holds until the process exits.  The caller passes device pointers for the
// inputs and the output; nothing is allocated by the call (no cudaMalloc,
// cudaFree or allocating library routine).  The call synchronises its stream
// (it reads the partition and the children totals back to the host) and
// returns when d_out is written.
//
// The kernels run the engine's own code (leaf, count, scan, expand) on the
// scratch array instead of engine-owned buffers, one launch a step for both
// sides, for depths 0..3: a depth-3 root is expanded once into the scratch level and
// both levels finish in the two-ply leaf kernel.  Every size check (positions,
// depths, the children of the depth-3 positions of both sides together) is
// made before the first leaf kernel, so a call that returns PG_ERR_CAPACITY
// has only zeroed d_out.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "pg_kernels.cuh"

namespace pg {
namespace {

constexpr u32 NA_MAX_ROOTS = 1u << 16;      // positions per call
constexpr u32 NA_MAX_CHILDREN = 1u << 20;   // depth-2 nodes made from depth-3 roots per call (both sides)
constexpr int NA_MAX_DEPTH = 3;
constexpr int NA_T = 256;

constexpr u64 align256(u64 x) { return (x + 255) & ~255ull; }
// scratch layout
constexpr u64 NA_L0_PL = 0;                                               // 3 planes x 64 Ki x 16 B
constexpr u64 NA_L0_GRP = align256(NA_L0_PL + 3ull * NA_MAX_ROOTS * 16);
constexpr u64 NA_L0_REM = align256(NA_L0_GRP + 4ull * NA_MAX_ROOTS);
constexpr u64 NA_L0_CNT = align256(NA_L0_REM + 1ull * NA_MAX_ROOTS);
constexpr u64 NA_L0_OFFS = align256(NA_L0_CNT + 4ull * NA_MAX_ROOTS);
// the exclusive scan of the children with its total: n + 1 words
constexpr u64 NA_L1_PL = align256(NA_L0_OFFS + 8ull * (NA_MAX_ROOTS + 2));
constexpr u64 NA_L1_GRP = align256(NA_L1_PL + 3ull * NA_MAX_CHILDREN * 16);
constexpr u64 NA_L1_REM = align256(NA_L1_GRP + 4ull * NA_MAX_CHILDREN);
constexpr u64 NA_STATUS = align256(NA_L1_REM + 1ull * NA_MAX_CHILDREN);
constexpr u64 NA_STATUS_WORDS = NA_MAX_ROOTS / SCAN_TILE + 2;
constexpr u64 NA_CTRL = align256(NA_STATUS + 8 * NA_STATUS_WORDS);
// control words: [0..3] partition counters, [4..15] tickets (7 used), [16] flags, [17] scan errors
constexpr u64 NA_CTRL_WORDS = 32;
constexpr u64 NA_SCRATCH_BYTES = align256(NA_CTRL + 4 * NA_CTRL_WORDS);
static_assert(NA_SCRATCH_BYTES <= 60ull << 20, "scratch over its stated 60 MiB");

enum : u32 { NA_BAD_POSITION = 1, NA_BAD_DEPTH = 2, NA_NOT_SET_UP = 4 };
constexpr u32 NA_MAGIC = 0x9A11A10Cu;

}  // namespace

// In host code this name is only a stand-in for the device array; the device
// address comes from cudaGetSymbolAddress, on every call.
static __device__ __align__(256) unsigned char g_noalloc_scratch[NA_SCRATCH_BYTES];
// NA_MAGIC once this device's move tables were uploaded.  A device reset
// reloads the module: the marker reads 0 again and the next call uploads
// the tables again instead of counting with empty ones.
static __device__ u32 g_na_ready;

namespace {

// roots into level 0 (as k_partition_roots), the counts cleared, and the checks:
// boards that board_ok takes, depths within 0..3, this device's set-up marker
__global__ void k_na_roots(const Pos* __restrict__ pos, const unsigned char* __restrict__ depths, u32 n, LevelView lv,
                           u32* counters /* [0] white, [1] black, [3] largest depth */, u32* flags, u64* __restrict__ out)
{
    u32 bad = blockIdx.x == 0 && threadIdx.x == 0 && g_na_ready != NA_MAGIC ? (u32)NA_NOT_SET_UP : 0u;
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const Pos b = pos[i];
        const u32 d = depths[i];
        if (!board_ok(b.w, b.p, b.n, b.bq, b.rq, b.k)) bad |= NA_BAD_POSITION;
        if (d > (u32)NA_MAX_DEPTH) bad |= NA_BAD_DEPTH;
        const u32 slot = st_side(b) ? n - 1 - atomicAdd(&counters[1], 1u) : atomicAdd(&counters[0], 1u);
        store_board(lv, slot, b);
        lv.grp[slot] = i;
        lv.rem[slot] = (unsigned char)d;
        atomicMax(&counters[3], d);
        out[i] = 0;
    }
    if (bad) atomicOr(flags, bad);
}

struct NaDevice {
    bool ready = false;
    unsigned char* scratch = nullptr;
    int sms = 0;
    int leaf_per_sm = 0, expand_per_sm = 0;  // resident CTAs
};
NaDevice g_na_dev[64];
std::mutex g_na_mu;

struct NaViews {
    LevelView l0, l1;
    u32* cnt0;
    u64* offs0;
    u64* status;
    u32* ctrl;
};

NaViews views(unsigned char* s)
{
    NaViews v;
    v.l0.pl0 = (ulonglong2*)(s + NA_L0_PL);
    v.l0.pl1 = v.l0.pl0 + NA_MAX_ROOTS;
    v.l0.pl2 = v.l0.pl1 + NA_MAX_ROOTS;
    v.l0.grp = (u32*)(s + NA_L0_GRP);
    v.l0.rem = s + NA_L0_REM;
    v.l1.pl0 = (ulonglong2*)(s + NA_L1_PL);
    v.l1.pl1 = v.l1.pl0 + NA_MAX_CHILDREN;
    v.l1.pl2 = v.l1.pl1 + NA_MAX_CHILDREN;
    v.l1.grp = (u32*)(s + NA_L1_GRP);
    v.l1.rem = s + NA_L1_REM;
    v.cnt0 = (u32*)(s + NA_L0_CNT);
    v.offs0 = (u64*)(s + NA_L0_OFFS);
    v.status = (u64*)(s + NA_STATUS);
    v.ctrl = (u32*)(s + NA_CTRL);
    return v;
}

// the view of lv from node k on
__device__ __forceinline__ LevelView from_node(const LevelView& lv, u64 k)
{
    LevelView r = lv;
    r.pl0 += k;
    r.pl1 += k;
    r.pl2 += k;
    r.grp += k;
    r.rem += k;
    return r;
}

// Both sides in one launch.  For calls of some thousands of positions one side's
// launch is mostly the latency of a few rounds, and the other's can run beside it
// (at the limits, 65,536 positions and 1,048,576 children, each side has many
// rounds).  The sides share the SMs by their nodes, whole SMs each, since the two
// sides' code together is more than an SM's instruction caches hold.  20,001
// positions at depths 0 to 3: 313 us with launches of one side each, 199 us so.
__device__ __forceinline__ Share side_share(u32 nw, u32 nb, u32 sms, bool& black)
{
    const u32 slots = min(sms, gridDim.x), layers = gridDim.x / slots;  // the grid is a multiple of slots
    u32 ws = (u32)(((u64)slots * nw + (nw + nb) / 2) / max(nw + nb, 1u));
    if (nw && nb) ws = min(max(ws, 1u), slots - 1);  // both have nodes: two CTAs at least
    const u32 slot = blockIdx.x % slots, layer = blockIdx.x / slots;
    black = slot >= ws;
    return black ? Share{layer * (slots - ws) + slot - ws, layers * (slots - ws)} : Share{layer * ws + slot, layers * ws};
}

constexpr int NA_LEAF_Q = NA_T * 16, NA_EXPAND_Q = NA_T * 32;
static_assert(BlockSmem<SlKS, NA_T, NA_EXPAND_Q>::bytes <= 48 * 1024, "dynamic shared memory above the default limit");
constexpr int NA_LEAF_SMEM = LeafSmem<SlKS, NA_T, NA_LEAF_Q>::bytes;
constexpr int NA_EXPAND_SMEM = BlockSmem<SlKS, NA_T, NA_EXPAND_Q>::bytes;

// the nodes [0, k) of a level, of side `first`, and [k, n), of the other one;
// k = *split, or split_at[*split] (the children of the first *split nodes)
__device__ __forceinline__ u32 split_of(const u32* split, const u64* split_at)
{
    return split_at ? (u32)split_at[*split] : *split;
}
__global__ void __launch_bounds__(NA_T, min_blocks<NA_T>())
k_na_leaf(LevelView lv, u32 n, int first, const u32* split, const u64* split_at, u64* out, u32* tickets, u32 sms)
{
    const u32 k = split_of(split, split_at);
    const u32 nw = first ? n - k : k, nb = n - nw;
    bool black;
    const Share share = side_share(nw, nb, sms, black);
    if (black) leaf_body<1, SlKS, NA_T, NA_LEAF_Q, false>(lv, first ? 0u : k, nb, out, tickets, 2u, nullptr, share);
    else leaf_body<0, SlKS, NA_T, NA_LEAF_Q, false>(lv, first ? k : 0u, nw, out, tickets + 1, 2u, nullptr, share);
}

// the children of [0, nw) (white to move) and of [nw, n), in that order
__global__ void __launch_bounds__(NA_T, min_blocks<NA_T>())
k_na_expand(LevelView in, u32 n, const u32* split, const u64* offs, LevelView out, u32* tickets, u32 sms)
{
    const u32 nw = *split;
    bool black;
    const Share share = side_share(nw, n - nw, sms, black);
    if (black) expand_body<1, SlKS, NA_T, NA_EXPAND_Q>(in, 0, nw, n, offs, from_node(out, offs[nw]), tickets, nullptr, share);
    else expand_body<0, SlKS, NA_T, NA_EXPAND_Q>(in, 0, 0, nw, offs, out, tickets + 1, nullptr, share);
}

// children of the depth-3 positions, once all positions are known to be valid
__global__ void __launch_bounds__(256) k_na_count(LevelView lv, u32 n, u32* __restrict__ cnt, const u32* flags)
{
    if (*flags) return;
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        cnt[i] = lv.rem[i] == 3 ? count_any<SlKS>(load_board(lv, i)) : 0u;
}

// CTAs for a launch over n nodes of both sides: one a node until the SMs are
// full, then whole rounds of SMs
int pair_grid(int per_sm, u32 n, int sms)
{
    const u32 want = (u32)std::min<u64>(n, (u64)per_sm * sms);
    return (int)std::max<u32>(1, want <= (u32)sms ? want : want / sms * sms);
}

// per-device set-up, with that device current: the scratch array's device
// address (looked up on every call, so a device reset that moves the module
// is followed) and, the first time and whenever the address changed or a
// kernel found the set-up marker cleared, this translation unit's copy of the
// move tables (knight and king moves, and the magic tables the count reads the
// king's rays from) and the marker
int na_setup(int dev, bool force, NaDevice*& out)
{
    std::lock_guard<std::mutex> lk(g_na_mu);
    if (dev < 0 || dev >= 64) {
        set_error("pg_perft_batch_noalloc: device %d out of range", dev);
        return PG_ERR_INVALID_ARGUMENT;
    }
    NaDevice& d = g_na_dev[dev];
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
        set_error("cudaGetSymbolAddress(g_noalloc_scratch) failed: %s", cudaGetErrorString(e));
        return PG_ERR_CUDA;
    }
    if (!d.ready || force || p != (void*)d.scratch) {
        d.ready = false;
        const HostTables* t = host_tables();
        if (!t) {
            set_error("move table construction failed");
            return PG_ERR_CUDA;
        }
        e = upload_static_tables(*t);
        if (e != cudaSuccess) {
            set_error("move table upload failed: %s", cudaGetErrorString(e));
            return PG_ERR_CUDA;
        }
        e = cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) {
            set_error("device query failed: %s", cudaGetErrorString(e));
            return PG_ERR_CUDA;
        }
        e = cudaFuncSetAttribute(k_na_leaf, cudaFuncAttributeMaxDynamicSharedMemorySize, NA_LEAF_SMEM);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.leaf_per_sm, k_na_leaf, NA_T, NA_LEAF_SMEM);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.expand_per_sm, k_na_expand, NA_T, NA_EXPAND_SMEM);
        if (e != cudaSuccess || d.leaf_per_sm < 1 || d.expand_per_sm < 1) {
            set_error("kernel set-up failed: %s", cudaGetErrorString(e));
            return PG_ERR_CUDA;
        }
        const u32 magic = NA_MAGIC;
        e = cudaMemcpyToSymbol(g_na_ready, &magic, sizeof(magic));
        if (e != cudaSuccess) {
            set_error("set-up marker upload failed: %s", cudaGetErrorString(e));
            return PG_ERR_CUDA;
        }
        d.scratch = (unsigned char*)p;
        d.ready = true;
    }
    out = &d;
    return PG_OK;
}

}  // namespace
}  // namespace pg

using namespace pg;

#define NA_CUDA(call)                                                                   \
    do {                                                                                \
        cudaError_t e_ = (call);                                                        \
        if (e_ != cudaSuccess) {                                                        \
            set_error("%s failed: %s", #call, cudaGetErrorString(e_));                  \
            return PG_ERR_CUDA;                                                         \
        }                                                                               \
    } while (0)

extern "C" int pg_perft_batch_noalloc(const pg_board* d_pos, const uint8_t* d_depths, uint32_t n,
                                      uint64_t* d_out, void* stream)
{
    if (n == 0) return PG_OK;
    if (!d_pos || !d_depths || !d_out) {
        set_error("null argument");
        return PG_ERR_INVALID_ARGUMENT;
    }
    if (n > NA_MAX_ROOTS) {
        set_error("pg_perft_batch_noalloc: %u positions exceed the maximum of %u per call", n, NA_MAX_ROOTS);
        return PG_ERR_CAPACITY;
    }
    int dev = 0;
    NA_CUDA(cudaGetDevice(&dev));
    cudaStream_t st = (cudaStream_t)stream;
    const Pos* pos = (const Pos*)d_pos;
    u64* out = (u64*)d_out;
    NaDevice* d = nullptr;
    struct {
        u32 words[18];
        u64 total;
    } head;
    NaViews v;
    for (int attempt = 0;; attempt++) {
        int r = na_setup(dev, attempt > 0, d);
        if (r != PG_OK) return r;
        v = views(d->scratch);
        u32* ctrl = v.ctrl;
        // the counters and the scan status words start at zero (the array keeps
        // the previous call's contents); k_na_roots clears the output
        NA_CUDA(cudaMemsetAsync(v.status, 0, NA_SCRATCH_BYTES - NA_STATUS, st));
        const int g = (int)std::min<u32>((n + 255) / 256, 1024);
        k_na_roots<<<g, 256, 0, st>>>(pos, d_depths, n, v.l0, ctrl, ctrl + 16, out);
        // the depth-3 positions' children, counted and scanned before the host
        // looks, so that every limit is checked before any leaf kernel runs
        k_na_count<<<g, 256, 0, st>>>(v.l0, n, v.cnt0, ctrl + 16);
        k_scan<<<(n + SCAN_TILE - 1) / SCAN_TILE, SCAN_T, 0, st>>>(v.cnt0, n, v.offs0, v.status, ctrl + 4, ctrl + 17);
        NA_CUDA(cudaGetLastError());
        NA_CUDA(cudaMemcpyAsync(head.words, ctrl, sizeof(head.words), cudaMemcpyDeviceToHost, st));
        NA_CUDA(cudaMemcpyAsync(&head.total, v.offs0 + n, sizeof(u64), cudaMemcpyDeviceToHost, st));
        NA_CUDA(cudaStreamSynchronize(st));
        if (!(head.words[16] & NA_NOT_SET_UP)) break;
        if (attempt > 0) {
            set_error("pg_perft_batch_noalloc: device set-up did not take effect");
            return PG_ERR_CUDA;
        }
    }
    if (head.words[16] & NA_BAD_POSITION) {
        set_error("pg_perft_batch_noalloc: a position is not a valid board");
        return PG_ERR_INVALID_POSITION;
    }
    if (head.words[16] & NA_BAD_DEPTH) {
        set_error("pg_perft_batch_noalloc: depths are limited to 0..%d", NA_MAX_DEPTH);
        return PG_ERR_CAPACITY;
    }
    if (head.words[17]) {
        set_error("pg_perft_batch_noalloc: device error flags 0x%x", head.words[17]);
        return PG_ERR_DEVICE_TIMEOUT;
    }
    const u32 maxd = head.words[3];
    const u64 total = maxd == 3 ? head.total : 0;
    if (total > NA_MAX_CHILDREN) {
        set_error("pg_perft_batch_noalloc: the depth-3 positions have %llu children, over the maximum of %u "
                  "per call",
                  (unsigned long long)total, NA_MAX_CHILDREN);
        return PG_ERR_CAPACITY;
    }
    // level 0: nodes with remaining depth <= 2 finish in the leaf kernel
    u32* white = v.ctrl;
    u32* tickets = v.ctrl + 6;
    const u32 sms = (u32)d->sms;
    k_na_leaf<<<pair_grid(d->leaf_per_sm, n, d->sms), NA_T, NA_LEAF_SMEM, st>>>(v.l0, n, 0, white, nullptr, out, tickets, sms);
    if (total) {
        // black-to-move children of the white-to-move positions first
        k_na_expand<<<pair_grid(d->expand_per_sm, n, d->sms), NA_T, NA_EXPAND_SMEM, st>>>(v.l0, n, white, v.offs0, v.l1,
                                                                                         tickets + 2, sms);
        k_na_leaf<<<pair_grid(d->leaf_per_sm, (u32)total, d->sms), NA_T, NA_LEAF_SMEM, st>>>(
            v.l1, (u32)total, 1, white, v.offs0, out, tickets + 4, sms);
    }
    NA_CUDA(cudaGetLastError());
    NA_CUDA(cudaStreamSynchronize(st));
    return PG_OK;
}
