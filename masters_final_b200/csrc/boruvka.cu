// Boruvka minimum spanning forest, connected components and the EAC final
// clustering (lifetime cut) on B200.
//
// Reference: MyML/MyML/graph/mst.py:417-809 (boruvka_minho_gpu and kernels),
// MyML/MyML/graph/connected_components.py:176-345, MyML/MyML/EAC/eac.py:199-391.
//
// Design (not the reference's):
//  * Every undirected edge is ONE 64-bit word: weight-order bits | min(u,v) |
//    max(u,v) | the entry's offset in the row of min(u,v) (graph MST; the
//    spare bits) | direction, with u, v the ORIGINAL endpoints, offered to the selection
//    slots of both its ends.  A round never rewrites edges; it only drops the
//    ones that became internal.  The current endpoints are the roots of u
//    and v in a union-find forest over the original vertices.
//  * Min-edge selection is an atomicMin of a 64-bit selection key per
//    supervertex: (weight, min, max) for the MST -- a strict total order, so
//    the forest is unique -- or (weight, other end's supervertex) for the
//    reference's connected-components numbering.  Lanes of a warp holding
//    edges of the same supervertex are pre-reduced with a segmented shuffle
//    scan, so one atomic is issued per run, not per edge.
//  * All Boruvka rounds of a phase run in ONE persistent kernel (k_rounds):
//    a cooperative grid whose blocks meet at bounded grid barriers, or a
//    single block for small graphs.  Contraction is fused with the NEXT
//    round's min-edge selection: each edge is read once and written at most
//    once per round.
//  * Mutual picks are broken towards the larger id like the reference; roots
//    are found by a bounded pointer chase with path halving; supervertices are
//    renumbered in root order, which is the reference's numbering.
//  * The MST grows by weight phases (Kruskal's prefix property), so heavy
//    edges that lighter ones made internal are dropped by one filtering read.
#include "eacb_common.cuh"
#include "scan_impl.cuh"

#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

namespace eacb {

enum { SEL_MST = 0, SEL_CC = 1 };

struct Pack {
    int vbits;
    int obits;       // row-offset bits (0: none)
    int wshift;      // 2*vbits + obits + 1
    uint64_t vmask;
    uint64_t omask;  // (1 << obits) - 1: also the "offset not recorded" value
    __host__ __device__ uint32_t a(uint64_t k) const { return (uint32_t)((k >> (vbits + obits + 1)) & vmask); }
    __host__ __device__ uint32_t b(uint64_t k) const { return (uint32_t)((k >> (obits + 1)) & vmask); }
    __host__ __device__ uint32_t w(uint64_t k) const { return (uint32_t)(k >> wshift); }
    __host__ __device__ uint32_t src(uint64_t k) const { return (k & 1) ? b(k) : a(k); }
    __host__ __device__ uint32_t dst(uint64_t k) const { return (k & 1) ? a(k) : b(k); }
    // off: where the entry min -> max sits in the row of min (omask: not
    // recorded); it is the lowest field of the selection key, so among
    // parallel entries of one row the first one wins
    __host__ __device__ uint64_t make(uint32_t w, uint32_t u, uint32_t v, uint64_t off) const
    {
        uint32_t lo = u < v ? u : v, hi = u < v ? v : u;
        return ((uint64_t)w << wshift) | ((uint64_t)lo << (vbits + obits + 1)) |
               ((uint64_t)hi << (obits + 1)) | ((off & omask) << 1) | (uint64_t)(u > v);
    }
    __host__ __device__ uint64_t make(uint32_t w, uint32_t u, uint32_t v) const
    {
        return make(w, u, v, omask);
    }
    // MST selection key (weight, min, max, offset) and its decoding
    __host__ __device__ uint64_t mst_sel(uint64_t k) const { return k >> 1; }
    __host__ __device__ uint32_t sel_a(uint64_t s) const { return (uint32_t)((s >> (vbits + obits)) & vmask); }
    __host__ __device__ uint32_t sel_b(uint64_t s) const { return (uint32_t)((s >> obits) & vmask); }
    __host__ __device__ uint32_t sel_w(uint64_t s) const { return (uint32_t)(s >> (2 * vbits + obits)); }
    __host__ __device__ uint64_t sel_off(uint64_t s) const { return s & omask; }
};

// with_offsets: the bits left over in the word hold the entry's row offset
// (a graph MST returns entry ids: k_key2eid reads them instead of searching
// the row).
static int make_pack(int32_t n_vertices, int wbits, Pack &pk, bool with_offsets = false)
{
    int vbits = 1;
    while (vbits < 31 && ((int64_t)1 << vbits) < (int64_t)n_vertices) vbits++;
    if (wbits + 2 * vbits + 1 > 64) return EACB_ERR_UNSUPPORTED;
    const int spare = 64 - (wbits + 2 * vbits + 1);
    pk.vbits = vbits;
    pk.obits = with_offsets ? (spare < 24 ? spare : 24) : 0;
    pk.wshift = 2 * vbits + pk.obits + 1;
    pk.vmask = ((uint64_t)1 << vbits) - 1;
    pk.omask = ((uint64_t)1 << pk.obits) - 1;
    return EACB_OK;
}

static int dtype_bits(int dt)
{
    switch (dt) {
    case EACB_U8: return 8;
    case EACB_U16: return 16;
    case EACB_I32: case EACB_U32: case EACB_F32: return 32;
    default: return -1;
    }
}

// Order-preserving unsigned image of a weight.
__device__ __forceinline__ uint32_t wword(uint8_t x) { return x; }
__device__ __forceinline__ uint32_t wword(uint16_t x) { return x; }
__device__ __forceinline__ uint32_t wword(uint32_t x) { return x; }
__device__ __forceinline__ uint32_t wword(int32_t x) { return (uint32_t)x ^ 0x80000000u; }
__device__ __forceinline__ uint32_t wword(float x)
{
    uint32_t u = __float_as_uint(x == 0.0f ? 0.0f : x);   // -0 == +0
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

constexpr uint64_t kNone = ~0ull;

// atomicMin that is skipped when the candidate cannot lower the slot.  Within
// a kernel the slots only decrease, so a (possibly older) L2 value that the
// candidate does not beat means the atomic would change nothing; late
// rounds, whose few supervertices receive most edges, then issue few atomics.
__device__ __forceinline__ void min_if_lower(unsigned long long *slot, uint64_t v)
{
    if (v < __ldcg(slot)) atomicMin(slot, (unsigned long long)v);
}

// An offer that never waits: a reduction with no return value.  For kernels
// whose slots each receive few offers (a graph's first phase: a vertex is
// offered its incident edges only), where the check load of min_if_lower
// would put an L2 round trip between consecutive offers of a thread.
__device__ __forceinline__ void offer_min(unsigned long long *slot, uint64_t v, bool check)
{
    if (check) min_if_lower(slot, v);
    else atomicMin(slot, (unsigned long long)v);
}

// One atomicMin per run of equal `su` among consecutive lanes.
__device__ __forceinline__ void seg_min_atomic(bool valid, int32_t su, uint64_t sel,
                                               unsigned long long *best)
{
    const int lane = threadIdx.x & 31;
    int32_t key = valid ? su : -1 - lane;
    int32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
    bool head = (lane == 0) || (prev != key);
    unsigned heads = __ballot_sync(0xffffffffu, head);
    int start = 31 - __clz(heads & ((2u << lane) - 1u));
    uint64_t m = valid ? sel : kNone;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        uint64_t o = __shfl_up_sync(0xffffffffu, m, d);
        if (lane - d >= start) m = (o < m) ? o : m;
    }
    int32_t next = __shfl_down_sync(0xffffffffu, key, 1);
    bool tail = (lane == 31) || (next != key);
    if (valid && tail) min_if_lower(&best[su], m);
}

constexpr int kET = 256;   // edge-tile threads
constexpr int kEI = 8;     // edges per thread (striped): 2048 edges per tile
constexpr int64_t kETile = (int64_t)kET * kEI;

// Edge sources for the tile kernel ------------------------------------------
// Each source splits an edge into fetch() (independent global loads, issued
// for all items of a thread before any is used) and resolve() (the dependent
// work), so a thread keeps all its loads in flight at once.
// Undirected keys (MST selection keys) below a weight cap, one word each
struct SrcForest {
    typedef uint64_t Raw;
    const uint64_t *keys;   // selection keys (w, a, b)
    int64_t n_keys;
    int64_t wmax;           // keep weights <= wmax (-1 keeps none)
    Pack pk;
    __device__ __forceinline__ void fetch(int64_t i, Raw &r) const
    {
        r = keys[i < n_keys ? i : i - n_keys];
    }
    // resolve() needs the item index for the direction: passed through k
    __device__ __forceinline__ bool resolve_dir(const Raw &s, bool reverse, uint64_t &k,
                                                int32_t &su, int32_t &sv, uint32_t &w) const
    {
        w = pk.sel_w(s);
        if ((int64_t)w > wmax) return false;
        const uint32_t a = pk.sel_a(s), b = pk.sel_b(s);
        k = (s << 1) | (uint64_t)reverse;
        su = (int32_t)(reverse ? b : a);
        sv = (int32_t)(reverse ? a : b);
        return true;
    }
};

template <typename Src>
__device__ __forceinline__ bool resolve_item(const Src &src, const typename Src::Raw &r,
                                             int64_t i, uint64_t &k, int32_t &su, int32_t &sv,
                                             uint32_t &w)
{
    return src.resolve(r, k, su, sv, w);
}

template <>
__device__ __forceinline__ bool resolve_item<SrcForest>(const SrcForest &src, const uint64_t &r,
                                                        int64_t i, uint64_t &k, int32_t &su,
                                                        int32_t &sv, uint32_t &w)
{
    return src.resolve_dir(r, false, k, su, sv, w);
}

// Tile kernel: keep-filter + order-preserving compaction + fused min-edge
// selection for the next round.  eout may equal the source array (in-place
// contraction): a tile writes only after its prefix is known, i.e. after
// every earlier tile has read its input, and never past its own input end.
template <int MODE, typename Src>
__global__ void __launch_bounds__(kET)
k_edge_tile(Src src, int64_t n_in, uint64_t *eout, unsigned long long *best,
            uint64_t *status, int *counter, int64_t *d_count, int *err,
            const int64_t *d_n = nullptr)
{
    __shared__ int s_tile;
    __shared__ int s_off[kEI][kET / 32];
    __shared__ int64_t s_prefix;
    // with d_n the edge count is read on the device and the blocks loop over
    // tiles (persistent grid); tile ids are taken in increasing order, so
    // every tile a block waits on is held by a running block
    if (d_n) n_in = *d_n;
    const int64_t n_tiles = (n_in + kETile - 1) / kETile;
    for (;;) {
    if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1);
    __syncthreads();
    const int64_t tile = s_tile;
    __syncthreads();
    if (tile >= n_tiles) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = tile * kETile;
    typename Src::Raw raw[kEI];
#pragma unroll
    for (int it = 0; it < kEI; ++it) {
        const int64_t i = base + (int64_t)it * kET + threadIdx.x;
        if (i < n_in) src.fetch(i, raw[it]);
    }
    uint64_t k[kEI];
    int32_t su[kEI], sv[kEI];
    uint32_t w[kEI];
    bool keep[kEI];
#pragma unroll
    for (int it = 0; it < kEI; ++it) {
        const int64_t i = base + (int64_t)it * kET + threadIdx.x;
        su[it] = sv[it] = 0;
        w[it] = 0;
        k[it] = 0;
        keep[it] = (i < n_in) && resolve_item(src, raw[it], i, k[it], su[it], sv[it], w[it]);
    }
    unsigned bal[kEI];
#pragma unroll
    for (int it = 0; it < kEI; ++it) {
        bal[it] = __ballot_sync(0xffffffffu, keep[it]);
        if (lane == 0) s_off[it][warp] = __popc(bal[it]);
        const uint64_t sel =
            MODE == SEL_MST ? (k[it] >> 1) : (((uint64_t)w[it] << 32) | (uint32_t)sv[it]);
        seg_min_atomic(keep[it], su[it], sel, best);
        // the word stands for both directions: the other end's offer
        if (keep[it])
            min_if_lower(&best[sv[it]],
                         MODE == SEL_MST ? (k[it] >> 1)
                                         : (((uint64_t)w[it] << 32) | (uint32_t)su[it]));
    }
    __syncthreads();
    if (warp == 0) {
        // exclusive scan of the kEI x 8 per-warp counts in (item, warp) order
        constexpr int N = kEI * (kET / 32);
        constexpr int PER = N / 32;
        int c[PER];
        int sum = 0;
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            int idx = lane * PER + q;
            c[q] = s_off[idx / (kET / 32)][idx % (kET / 32)];
            sum += c[q];
        }
        int incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += o;
        }
        int run = incl - sum;
        int tot = __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            int idx = lane * PER + q;
            s_off[idx / (kET / 32)][idx % (kET / 32)] = run;
            run += c[q];
        }
        int64_t pre = lookback(status, tile, tot, 0, err);
        if (lane == 0) {
            s_prefix = pre;
            const int64_t ntiles = (n_in + kETile - 1) / kETile;
            if (tile == ntiles - 1) *d_count = pre + tot;
        }
    }
    __syncthreads();
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int it = 0; it < kEI; ++it) {
        if (bal[it] & (1u << lane)) {
            int64_t pos = s_prefix + s_off[it][warp] + __popc(bal[it] & lt);
            eout[pos] = k[it];
        }
    }
    if (!d_n) return;            // one tile per block
    __syncthreads();             // shared state is reused by the next tile
    }
}

// ---------------------------------------------------------------------------
// Weight phases (MST mode).  For a strict total order of the edges, the
// minimum spanning forest of the edges up to a key is exactly the MST
// restricted to those edges (Kruskal's prefix property).  So the forest is
// grown phase by phase over weight ranges: a phase contracts the edges of its
// range whose endpoints are still in different components, then the next
// phase starts from those components.  Heavy edges that the light ones made
// internal are dropped by one filtering read instead of being carried through
// every round.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t wbucket(uint32_t w, int wbits)
{
    return wbits <= 8 ? w : (w >> (wbits - 8));
}

// 256-bin histograms.  Weights are heavily skewed (most co-association
// dissimilarities sit in a few top bins), so a shared atomic per element
// would serialise on those bins: lanes of a warp holding the same bin combine
// first (match_any), and every warp owns a private copy of the bins.
constexpr int kHistThreads = 256;

__device__ __forceinline__ void hist_add(unsigned *h, uint32_t b, bool valid)
{
    const unsigned act = __ballot_sync(0xffffffffu, valid);
    if (!valid) return;
    const unsigned peers = __match_any_sync(act, b);
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&h[b], (unsigned)__popc(peers));
}

__device__ __forceinline__ void hist_flush(unsigned (*h)[256], unsigned long long *hist)
{
    __syncthreads();
    for (int b = threadIdx.x; b < 256; b += blockDim.x) {
        unsigned long long t = 0;
        for (int w = 0; w < kHistThreads / 32; ++w) t += h[w][b];
        if (t) atomicAdd(&hist[b], t);
    }
}

template <typename WT>
__global__ void __launch_bounds__(kHistThreads)
k_whist_csr(const WT *weight, int64_t E, int wbits, unsigned long long *hist)
{
    __shared__ unsigned h[kHistThreads / 32][256];
    for (int i = threadIdx.x; i < (kHistThreads / 32) * 256; i += blockDim.x) (&h[0][0])[i] = 0;
    __syncthreads();
    unsigned *mine = h[threadIdx.x >> 5];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // the loop bound is warp-uniform (match_any needs the whole warp)
    for (int64_t e0 = (int64_t)blockIdx.x * blockDim.x; e0 < E; e0 += stride) {
        const int64_t e = e0 + threadIdx.x;
        const bool ok = e < E;
        hist_add(mine, ok ? wbucket(wword(weight[e]), wbits) & 255 : 0, ok);
    }
    hist_flush(h, hist);
}

// uint8 weights, 16 per thread per step (128-bit loads).  Every lane owns a
// private column of 256 counters (bank = lane, so no conflicts and no
// atomics): counts[warp][bin][lane], 32 KB per warp, two warps per block.
constexpr int kHist8Threads = 64;
constexpr size_t kHist8Smem = (size_t)(kHist8Threads / 32) * 256 * 32 * sizeof(uint32_t);
__global__ void __launch_bounds__(kHist8Threads, 1)
k_whist_u8(const uint8_t *w, int64_t n, int skip, unsigned long long *hist)
{
    extern __shared__ uint32_t hs[];
    for (int i = threadIdx.x; i < (kHist8Threads / 32) * 256 * 32; i += blockDim.x) hs[i] = 0;
    __syncthreads();
    uint32_t *mine = hs + (threadIdx.x >> 5) * 256 * 32 + (threadIdx.x & 31);
    int64_t head = (int64_t)((16 - ((uintptr_t)w & 15)) & 15);
    if (head > n) head = n;
    // the whole 16-byte vectors read: with skip > 1, 32 of each 32 * skip
    const int64_t whole = (n - head) >> 4;
    const int64_t nv = skip == 1 ? whole : whole / (32 * skip) * 32;
    auto at = [&](int64_t q) -> int64_t { return skip == 1 ? q : (q >> 5) * (32 * skip) + (q & 31); };
    const uint4 *v = reinterpret_cast<const uint4 *>(w + head);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    auto add16 = [&](const uint4 &x) {
        const uint32_t wd[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int k = 0; k < 16; ++k)     // no-return adds: equal bytes do not serialise
            atomicAdd(&mine[((wd[k >> 2] >> (8 * (k & 3))) & 255u) * 32], 1u);
    };
    // few warps fit beside the private columns, so each thread keeps eight
    // 16-byte loads in flight
    constexpr int kU = 8;
    int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; q + (kU - 1) * stride < nv; q += kU * stride) {
        uint4 x[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) x[u] = __ldcs(v + at(q + u * stride));
        // all eight loads are issued before the first is consumed
#pragma unroll
        for (int u = 0; u < kU; ++u)
            asm volatile("" : "+r"(x[u].x), "+r"(x[u].y), "+r"(x[u].z), "+r"(x[u].w));
#pragma unroll
        for (int u = 0; u < kU; ++u) add16(x[u]);
    }
    for (; q < nv; q += stride) add16(__ldcs(v + at(q)));
    // the unaligned head and the ragged tail (< 32 bytes), by the first block
    if (blockIdx.x == 0 && skip == 1) {
        const int64_t tail0 = head + (nv << 4);
        const int64_t rest = head + (n - tail0);
        const int64_t t = threadIdx.x;
        if (t < rest) mine[(uint32_t)w[t < head ? t : tail0 + (t - head)] * 32] += 1;
    }
    __syncthreads();
    for (int b = threadIdx.x; b < 256; b += blockDim.x) {
        unsigned long long tot = 0;
        for (int wp = 0; wp < kHist8Threads / 32; ++wp)
            for (int l = 0; l < 32; ++l) tot += hs[(wp * 256 + b) * 32 + l];
        if (tot) atomicAdd(&hist[b], tot);
    }
}

// (skip > 1: of one in `skip` of the bytes, 512 of each 512 * skip)
static int launch_whist_u8(const uint8_t *w, int64_t n, unsigned long long *hist, cudaStream_t st,
                           int skip = 1)
{
    EACB_CUDA(allow_max_dyn_smem(k_whist_u8));
    k_whist_u8<<<grid_for((n / skip + 15) / 16, kHist8Threads, 148 * 3), kHist8Threads, kHist8Smem,
                 st>>>(w, n, skip, hist);
    EACB_CHECK_LAUNCH();
    return EACB_OK;
}

// Phase builds: the edges of a weight-bucket range (lo, hi] whose endpoints
// are in different components, appended to eout, with the first round's
// minimum-edge selection.  Output slots are reserved with one atomicAdd per
// block step (the identity phase) or per warp staging flush, which keeps the
// shared cursor off the critical path.  Edge order is not deterministic,
// results are: selection uses a strict total order.
// the final clustering merges its remaining weight phases once fewer than
// one component per this many points is left
constexpr int64_t kMergeBelow = 64;
constexpr int kPhThreads = 256;
constexpr int kPhWarps = kPhThreads / 32;

// Exclusive offsets of the block's per-warp counts in s_cnt and one
// reservation of mult * total slots.  A reservation that would pass `cap`
// (the output capacity) writes nothing and raises DEV_CAPACITY; it returns
// false to every thread of the block.
__device__ __forceinline__ bool phase_reserve(int64_t *s_cnt, unsigned long long *s_base,
                                              unsigned long long *cursor, int mult,
                                              unsigned long long cap, int *err)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t tot = 0;
        for (int w = 0; w < kPhWarps; ++w) {
            const int64_t c = s_cnt[w];
            s_cnt[w] = tot;
            tot += c;
        }
        const unsigned long long need = (unsigned long long)(mult * tot);
        const unsigned long long b = tot ? atomicAdd(cursor, need) : 0ull;
        *s_base = b;
        s_ok = b + need <= cap;
        if (!s_ok) set_err(err, DEV_CAPACITY);
    }
    __syncthreads();
    return s_ok != 0;
}

// Graph rows are short (degrees), so a warp takes 32 consecutive rows per
// block step, one row per lane for the row data.  When the 32 rows lie back
// to back in the CSR (the usual layout) and their entries fit the warp's
// row staging, the warp copies the whole range into shared memory with
// coalesced 16-byte loads and each lane then walks its own row there, with
// no per-entry row search: an inexpensive test records the kept entries,
// and a dense pass builds and offers their words (see kPhChunk).  A longer
// back-to-back range is walked as one flat
// range, 32 entries per step, each lane finding its entry's row among the
// lanes' row starts (a 5-step shuffle search).  Otherwise the warp walks
// the rows one by one.  Kept words are staged in shared memory.  In the
// identity phase (every row read) the block reserves once per step and
// copies them out coalesced; a later phase, which skips most rows, has no
// block barrier: each warp flushes its staging when it fills up and at the
// end.
constexpr int kPhStage = 256;            // staged words per warp
constexpr int kPhChunk = 8;              // entries per row between dense passes
constexpr int kPhRec = 32 * kPhChunk;    // kept-entry records per warp (dynamic shared memory)
constexpr size_t kPhRecBytes = (size_t)kPhWarps * kPhRec * sizeof(int32_t);
constexpr int kPhRowBytes = 3840;        // row staging per warp: entries x (4 + sizeof(WT))

template <typename WT>
struct RowCap {
    static constexpr int value = (kPhRowBytes / (4 + (int)sizeof(WT))) & ~15;
};

// Copies entries [e_begin, e_end) of src (E entries) into the warp's dst and
// returns the entry index that dst[0] holds: 16-byte vectors from the
// aligned vector at or before e_begin when src is 16-byte aligned (every
// vector read lies inside [0, E)), else one entry per lane.  The caller
// checks that e_end - e_begin + 16 / sizeof(T) - 1 <= CAP.
template <typename T, int CAP>
__device__ __forceinline__ int64_t warp_copy_range(const T *src, int64_t e_begin, int64_t e_end,
                                                   int64_t E, T *dst)
{
    constexpr int VEC = 16 / (int)sizeof(T);
    constexpr int NV = (CAP / VEC + 31) / 32;      // vectors per lane at most
    constexpr int NB = 3;                          // vectors in flight per lane
    const int lane = threadIdx.x & 31;
    if (((uintptr_t)src & 15) == 0) {
        const int64_t base = e_begin & ~(int64_t)(VEC - 1);
        const int nv = (int)((e_end - base + VEC - 1) / VEC);
#pragma unroll
        for (int k0 = 0; k0 < NV; k0 += NB) {
            if (lane + 32 * k0 >= nv) break;
            uint4 x[NB];
#pragma unroll
            for (int k = 0; k < NB; ++k) {
                const int i = lane + 32 * (k0 + k);
                const int64_t e = base + (int64_t)i * VEC;
                if (i < nv && e + VEC <= E) {
                    x[k] = __ldg(reinterpret_cast<const uint4 *>(src + e));
                } else {
                    T t[VEC];
#pragma unroll
                    for (int q = 0; q < VEC; ++q) t[q] = (i < nv && e + q < E) ? src[e + q] : T(0);
                    memcpy(&x[k], t, 16);
                }
            }
#pragma unroll
            for (int k = 0; k < NB; ++k) {
                const int i = lane + 32 * (k0 + k);
                if (i < nv) *reinterpret_cast<uint4 *>(dst + (int64_t)i * VEC) = x[k];
            }
        }
        return base;
    }
    for (int64_t i = lane; i < e_end - e_begin; i += 32) dst[i] = src[e_begin + i];
    return e_begin;
}

__device__ __forceinline__ void phase_flush_warp(const uint64_t *stage, int cnt, uint64_t *eout,
                                                 unsigned long long *cursor,
                                                 unsigned long long cap, int *err)
{
    const int lane = threadIdx.x & 31;
    unsigned long long b = 0;
    if (lane == 0) b = atomicAdd(cursor, (unsigned long long)cnt);
    b = __shfl_sync(0xffffffffu, b, 0);
    if (b + cnt > cap) {
        if (lane == 0) set_err(err, DEV_CAPACITY);
        return;
    }
    for (int i = lane; i < cnt; i += 32) eout[b + i] = stage[i];
}

// Appends one candidate per lane to the warp's staging (flushing first when
// it would overflow).
__device__ __forceinline__ void phase_stage(bool keep, uint64_t k, uint64_t *stage, int &cnt,
                                            uint64_t *eout, unsigned long long *cursor,
                                            unsigned long long cap, int *err)
{
    const int lane = threadIdx.x & 31;
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    const int nb = __popc(bal);
    if (cnt + nb > kPhStage) {
        __syncwarp();
        phase_flush_warp(stage, cnt, eout, cursor, cap, err);
        __syncwarp();
        cnt = 0;
    }
    if (keep) stage[cnt + __popc(bal & ((1u << lane) - 1u))] = k;
    cnt += nb;
}

// identity: the first phase (every vertex its own root: no label is read,
// and every entry is checked once for a destination out of range, and
// counted into sym[0] (u < v) or sym[1] (u > v): a symmetric graph has as
// many of each).  Its selection offers are reductions with no check load: a
// vertex is offered its own incident edges only.
// skip_root (device int, or null; -1 = none): a later phase skips the rows of
// that root -- the giant component the earlier phases built -- and emits
// both directions of each kept entry whose other end lies in it, so the
// giant still sees every edge it has to another component (each such edge is
// found once, from the row outside the giant).
template <int MODE, typename WT>
__global__ void __launch_bounds__(kPhThreads, 4)
k_phase_csr(const int32_t *first, const int32_t *deg, const int32_t *dest, const WT *weight,
            int32_t V, int64_t E, int wbits, int lo, int hi, const int *dev_lohi, int slot,
            int identity, const int32_t *skip_root, const int32_t *label, Pack pk,
            uint64_t *eout, unsigned long long *cursor, unsigned long long cap,
            unsigned long long *best, unsigned long long *sym, int *err)
{
    unsigned n_lt = 0, n_gt = 0;             // this lane's entries by direction (the warp sum is 32-bit)
    if (dev_lohi) {
        lo = dev_lohi[2 * slot];
        hi = dev_lohi[2 * slot + 1];
    }
    const int32_t skip = skip_root ? *skip_root : -1;
    constexpr int kCap = RowCap<WT>::value;
    __shared__ uint64_t stage_all[kPhWarps][kPhStage];
    __shared__ __align__(16) int32_t rdest_all[kPhWarps][kCap];
    __shared__ __align__(16) WT rw_all[kPhWarps][kCap];
    __shared__ int64_t s_cnt[kPhWarps];
    __shared__ unsigned long long s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t *stage = stage_all[warp];
    int32_t *rdest = rdest_all[warp];
    WT *rw = rw_all[warp];
    extern __shared__ int32_t ph_rec[];      // kPhWarps x kPhRec kept-entry records
    int32_t *rec = ph_rec + warp * kPhRec;
    const int64_t step = (int64_t)kPhWarps * 32;
    auto root_of = [&](int32_t v) -> int32_t { return identity ? v : label[v]; };
    // a kept entry u -> v (roots lu != lv) becomes one word for the
    // undirected edge: written from the row of its smaller end, or from the
    // only row read when v lies in the skipped giant; its key is offered to
    // both ends (MST: (weight, min, max); CC: (weight, other end's root))
    // (off: the entry's offset in row u, recorded when u is the smaller end)
    auto emit = [&](bool kept, uint32_t w, int32_t u, int32_t v, int32_t lu, int32_t lv,
                    int64_t off, int &cnt) {
        const bool keep = kept && (u < v || lv == skip);
        const uint64_t k =
            keep ? pk.make(w, (uint32_t)u, (uint32_t)v,
                           (u < v && (uint64_t)off < pk.omask) ? (uint64_t)off : pk.omask)
                 : 0ull;
        phase_stage(keep, k, stage, cnt, eout, cursor, cap, err);
        if (keep) {
            offer_min(&best[lu], MODE == SEL_MST ? (k >> 1) : (((uint64_t)w << 32) | (uint32_t)lv),
                      !identity);
            offer_min(&best[lv], MODE == SEL_MST ? (k >> 1) : (((uint64_t)w << 32) | (uint32_t)lu),
                      !identity);
        }
    };
    int cnt = 0;                         // staged words (carried across steps without identity)
    // the next step's row labels are loaded one step ahead (a later phase
    // spends most steps on this load alone: its rows are mostly skipped)
    auto row_label = [&](int64_t r) -> int32_t {
        const int64_t u = r + (int64_t)warp * 32 + lane;
        return (identity || u >= V) ? (int32_t)u : label[u];
    };
    int32_t lu_next = row_label((int64_t)blockIdx.x * step);
    for (int64_t r0 = (int64_t)blockIdx.x * step; r0 < V; r0 += (int64_t)gridDim.x * step) {
        const int64_t u0 = r0 + (int64_t)warp * 32;
        const int nrows = u0 >= V ? 0 : (int)(V - u0 < 32 ? V - u0 : 32);
        int64_t f = 0, d = 0;
        int32_t lu = 0;
        bool live = false;
        const int32_t lu_this = lu_next;
        lu_next = row_label(r0 + (int64_t)gridDim.x * step);
        if (lane < nrows) {
            lu = lu_this;
            live = lu != skip;
            if (live) {
                f = first[u0 + lane];
                d = deg[u0 + lane];
                if (f < 0 || d < 0 || f + d > E) {
                    set_err(err, DEV_BAD_INPUT);
                    f = 0;
                    d = 0;
                }
            }
        }
        if (__any_sync(0xffffffffu, live)) {
            // rows back to back?  (row l + 1 starts where row l ends; a
            // skipped row must not break the range, so it counts as empty
            // only when the whole warp is flat over the live rows)
            const int64_t f_next = __shfl_down_sync(0xffffffffu, f, 1);
            const bool nl = __shfl_down_sync(0xffffffffu, live, 1);
            const bool linked = lane + 1 >= nrows || !live || !nl || f_next == f + d;
            const unsigned lmask = __ballot_sync(0xffffffffu, live);
            const int lfirst = __ffs(lmask) - 1, llast = 31 - __clz(lmask);
            const int64_t e_begin = __shfl_sync(0xffffffffu, f, lfirst);
            const int64_t e_end = __shfl_sync(0xffffffffu, f + d, llast);
            const bool flat = __all_sync(0xffffffffu, linked) && lmask == (nrows >= 32 ? 0xffffffffu : ((1u << nrows) - 1u)) &&
                              e_end - e_begin < ((int64_t)1 << 30);
            // the whole range fits the row staging (with the slack of the
            // aligned first vector of either array)
            constexpr int kSlack = 16 / (int)(sizeof(WT) < 4 ? sizeof(WT) : 4) - 1;
            if (flat && e_end - e_begin + kSlack <= kCap) {
                const int64_t db = warp_copy_range<int32_t, kCap>(dest, e_begin, e_end, E, rdest);
                const int64_t wb = warp_copy_range<WT, kCap>(weight, e_begin, e_end, E, rw);
                __syncwarp();
                const int32_t od = (int32_t)(f - db), ow = (int32_t)(f - wb);
                const int32_t u = (int32_t)(u0 + lane);
                const int dl = (int)d;                  // 0 past the last row
                const int dmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)dl);
                const unsigned below = (1u << lane) - 1u;
                // kPhChunk entries of every row at a time: a cheap test of
                // each entry records the kept ones as (row lane, offset), then
                // a dense pass over the records builds, stages and offers
                // their words with every lane busy (a phase keeps a small
                // share of the entries).  The same words and offers as
                // emit(): one word per undirected edge, offered to both ends.
                for (int j0 = 0; j0 < dmax; j0 += kPhChunk) {
                    const int j1 = j0 + kPhChunk < dmax ? j0 + kPhChunk : dmax;
                    int nrec = 0;
                    for (int j = j0; j < j1; ++j) {
                        bool keep = false;
                        if (j < dl) {
                            const int32_t v = rdest[od + j];
                            if ((uint32_t)v >= (uint32_t)V) {
                                set_err(err, DEV_BAD_INPUT);
                            } else if (v != u) {
                                if (v > u) ++n_lt; else ++n_gt;
                                const int bk = (int)wbucket(wword(rw[ow + j]), wbits);
                                if (bk > lo && bk <= hi) {
                                    const int32_t lv = root_of(v);
                                    keep = lv != lu && (u < v || lv == skip);
                                }
                            }
                        }
                        const unsigned bal = __ballot_sync(0xffffffffu, keep);
                        if (keep) rec[nrec + __popc(bal & below)] = (lane << 16) | j;
                        nrec += __popc(bal);
                    }
                    __syncwarp();
                    for (int i0 = 0; i0 < nrec; i0 += 32) {
                        const bool ok = i0 + lane < nrec;
                        const int32_t rc = ok ? rec[i0 + lane] : 0;
                        const int r = rc >> 16, jr = rc & 0xffff;
                        const int32_t odr = __shfl_sync(0xffffffffu, od, r);
                        const int32_t owr = __shfl_sync(0xffffffffu, ow, r);
                        const int32_t lur = __shfl_sync(0xffffffffu, lu, r);
                        const int32_t ur = (int32_t)(u0 + r);
                        const int32_t v = ok ? rdest[odr + jr] : 0;
                        const uint32_t w = ok ? wword(rw[owr + jr]) : 0u;
                        const int32_t lv = ok ? root_of(v) : 0;
                        const uint64_t k =
                            ok ? pk.make(w, (uint32_t)ur, (uint32_t)v,
                                         (ur < v && (uint64_t)jr < pk.omask) ? (uint64_t)jr
                                                                             : pk.omask)
                               : 0ull;
                        phase_stage(ok, k, stage, cnt, eout, cursor, cap, err);
                        if (ok) {
                            offer_min(&best[lur],
                                      MODE == SEL_MST ? (k >> 1)
                                                      : (((uint64_t)w << 32) | (uint32_t)lv),
                                      !identity);
                            offer_min(&best[lv],
                                      MODE == SEL_MST ? (k >> 1)
                                                      : (((uint64_t)w << 32) | (uint32_t)lur),
                                      !identity);
                        }
                    }
                    __syncwarp();                       // the records are reused
                }
                __syncwarp();                           // the row staging is reused
            } else if (flat) {
                const int32_t frel = (int32_t)(f - e_begin);      // row starts, warp-relative
                // four 32-entry slices per step, the loads of all in flight together
                constexpr int S = 4;
                for (int64_t e0 = e_begin; e0 < e_end; e0 += 32 * S) {
                    int64_t e[S];
                    int r[S];
                    int32_t lr[S], v[S], eo[S];
                    uint32_t w[S];
                    bool in[S];
#pragma unroll
                    for (int q = 0; q < S; ++q) {
                        e[q] = e0 + 32 * q + lane;
                        in[q] = e[q] < e_end;
                        const int32_t erel = (int32_t)(e[q] - e_begin);
                        // row of entry e: the last row starting at or before e
                        int rr = 0;
#pragma unroll
                        for (int st = 16; st >= 1; st >>= 1) {
                            const int c = rr + st;
                            const int32_t fs = __shfl_sync(0xffffffffu, frel, c & 31);
                            if (c < nrows && fs <= erel) rr = c;
                        }
                        r[q] = rr;
                        lr[q] = __shfl_sync(0xffffffffu, lu, rr);
                        eo[q] = erel - __shfl_sync(0xffffffffu, frel, rr);   // offset in its row
                        v[q] = in[q] ? dest[e[q]] : -1;
                        w[q] = in[q] ? wword(weight[e[q]]) : 0u;
                    }
                    bool cand[S];
                    int32_t lv[S];
#pragma unroll
                    for (int q = 0; q < S; ++q) {
                        cand[q] = false;
                        if (in[q]) {
                            if (v[q] < 0 || v[q] >= V) {
                                set_err(err, DEV_BAD_INPUT);
                            } else if (v[q] != (int32_t)(u0 + r[q])) {
                                if (v[q] > (int32_t)(u0 + r[q])) ++n_lt; else ++n_gt;
                                const int bk = (int)wbucket(w[q], wbits);
                                cand[q] = bk > lo && bk <= hi;
                            }
                        }
                        lv[q] = cand[q] ? root_of(v[q]) : 0;
                    }
#pragma unroll
                    for (int q = 0; q < S; ++q)
                        emit(cand[q] && lv[q] != lr[q], w[q], (int32_t)(u0 + r[q]), v[q], lr[q],
                             lv[q], eo[q], cnt);
                }
            } else {
                for (int rr = 0; rr < nrows; ++rr) {
                    if (!((lmask >> rr) & 1u)) continue;
                    const int64_t fr = __shfl_sync(0xffffffffu, f, rr);
                    const int64_t dr = __shfl_sync(0xffffffffu, d, rr);
                    const int32_t lr = __shfl_sync(0xffffffffu, lu, rr);
                    const int32_t u = (int32_t)(u0 + rr);
                    for (int64_t e0 = fr; e0 < fr + dr; e0 += 32) {
                        const int64_t e = e0 + lane;
                        bool cand = false;
                        int32_t v = -1, lv = 0;
                        uint32_t w = 0;
                        if (e < fr + dr) {
                            v = dest[e];
                            if (v < 0 || v >= V) {
                                set_err(err, DEV_BAD_INPUT);
                            } else if (v != u) {
                                if (v > u) ++n_lt; else ++n_gt;
                                w = wword(weight[e]);
                                const int bk = (int)wbucket(w, wbits);
                                cand = bk > lo && bk <= hi;
                                if (cand) lv = root_of(v);
                            }
                        }
                        emit(cand && lv != lr, w, u, v, lr, lv, e - fr, cnt);
                    }
                }
            }
        }
        if (identity) {
            // identity is uniform over the grid, so every thread of the
            // block takes the reservation's barriers
            if (lane == 0) s_cnt[warp] = cnt;
            const bool fits = phase_reserve(s_cnt, &s_base, cursor, 1, cap, err);
            if (fits) {
                const unsigned long long at = s_base + (unsigned long long)s_cnt[warp];
                for (int i = lane; i < cnt; i += 32) eout[at + i] = stage[i];
            }
            __syncthreads();      // staging and s_cnt are reused by the next step
            cnt = 0;
        }
    }
    if (!identity && cnt > 0) {
        __syncwarp();
        phase_flush_warp(stage, cnt, eout, cursor, cap, err);
    }
    if (sym) {
        n_lt = __reduce_add_sync(0xffffffffu, (unsigned)n_lt);
        n_gt = __reduce_add_sync(0xffffffffu, (unsigned)n_gt);
        if ((threadIdx.x & 31) == 0 && (n_lt | n_gt)) {
            atomicAdd(&sym[0], (unsigned long long)n_lt);
            atomicAdd(&sym[1], (unsigned long long)n_gt);
        }
    }
}

// The root holding most vertices (from a strided sample of 2048 vertices, in
// a shared-memory count table), or -1 when none holds a quarter of the
// sample: the rows a later weight phase may skip.
constexpr int kGiantSample = 2048;
__global__ void __launch_bounds__(1024)
k_pick_giant(const int32_t *label, int64_t V0, int32_t *out)
{
    constexpr int T = 2 * kGiantSample;
    __shared__ int32_t key[T];
    __shared__ int32_t cnt[T];
    __shared__ unsigned long long best;
    for (int i = threadIdx.x; i < T; i += blockDim.x) {
        key[i] = -1;
        cnt[i] = 0;
    }
    if (threadIdx.x == 0) best = 0ull;
    __syncthreads();
    const int64_t n = V0 < kGiantSample ? V0 : kGiantSample;
    for (int64_t j = threadIdx.x; j < n; j += blockDim.x) {
        const int32_t r = label[(j * V0) / n];
        unsigned slot = ((uint32_t)r * 2654435761u) % T;
        for (int probe = 0; probe < T; ++probe) {
            int32_t k = key[slot];
            if (k == -1) {
                k = atomicCAS(&key[slot], -1, r);
                if (k == -1) k = r;
            }
            if (k == r) {
                atomicAdd(&cnt[slot], 1);
                break;
            }
            slot = (slot + 1) % T;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < T; i += blockDim.x)
        if (cnt[i]) atomicMax(&best, ((unsigned long long)cnt[i] << 32) | (uint32_t)key[i]);
    __syncthreads();
    if (threadIdx.x == 0) {
        const int64_t c = (int64_t)(best >> 32);
        *out = (n > 0 && 4 * c >= n) ? (int32_t)(uint32_t)best : -1;
    }
}

// Same for an upper-triangle CSR with uint8 weights: one word per kept entry,
// offered to both ends.  Co-association rows are long (thousands of entries)
// and a phase keeps few of them, so the work is split in two.  A scan reads
// the weights, tests them against the phase's range four bytes at once and
// records the candidates' entry numbers in shared memory; when a warp's
// records fill, a dense pass with a record per lane reads their columns and
// labels, checks the entries (j > i, j < n), updates the selection slots and
// the per-weight counts, and writes the kept ones' words with one cursor
// atomic.  Records are carried from row to row, so both halves run with full
// warps, and the chains of dependent loads are paid per 256 records, not per
// row.  (One pass that handled its candidates as it found them spent 165
// instructions and four dependent L2 latencies on each 128 entries; the two
// sparse phases of 920M entries went from 2.26 and 1.60 to 0.50 and 0.53 ms,
// 1.8 TB/s of weights, bound by the instructions of the byte tests.)
struct UpArgs {
    const int64_t *indptr;
    const int32_t *indices;
    const uint8_t *w;
    int32_t n;
    int64_t nnz;
    int lo, hi;                      // weights in (lo, hi]
    int ident;                       // labels are the identity (nothing merged yet)
    int64_t row0, row1;
    const int32_t *label;
    Pack pk;
    uint64_t *eout;
    unsigned long long *cursor;
    unsigned long long cap;
    unsigned long long *best;
    unsigned long long *khist;       // kept entries per weight
    int *err;
};

constexpr int kUpRec = 256;          // records per warp, k_phase_upper
constexpr int kPairRec = 128;        // and k_pair_min

// the words w's bytes q in [L, H] as bits q, with c1 = (0x8000 - L) and c2 =
// (0x7fff - H) in both 16-bit halves: bytes 0, 2 and bytes 1, 3 are spread to
// 16-bit lanes, where bit 15 of x + c1 is x >= L and bit 15 of x + c2 is x > H
__device__ __forceinline__ unsigned bytes_in_range(uint32_t w, uint32_t c1, uint32_t c2)
{
    const uint32_t e = __byte_perm(w, 0u, 0x4240), o = __byte_perm(w, 0u, 0x4341);
    const uint32_t me = (e + c1) & ~(e + c2), mo = (o + c1) & ~(o + c2);
    return ((me >> 15) & 1u) | ((mo >> 14) & 2u) | ((me >> 29) & 4u) | ((mo >> 28) & 8u);
}

// The warp's n records (entry numbers and their rows): checked, offered and
// written.  The kept words replace the records from the front (a batch's
// records are read before its words are written, and there are never more).
__device__ __forceinline__ void up_flush(const UpArgs &a, uint64_t *rec, const int32_t *rrow, int n,
                                      unsigned *s_kh)
{
    constexpr int U = 2;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    int out = 0;
    __syncwarp();
    for (int b = 0; b < n; b += 32 * U) {
        int64_t e[U];
        int32_t i[U], j[U], li[U], lj[U];
        uint32_t wq[U];
        uint64_t cj[U], ci[U];
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int t = b + 32 * u + lane;
            ok[u] = t < n;
            e[u] = ok[u] ? (int64_t)rec[t] : 0;
            i[u] = ok[u] ? rrow[t] : 0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            j[u] = ok[u] ? __ldg(a.indices + e[u]) : 0;
            wq[u] = ok[u] ? __ldg(a.w + e[u]) : 0u;
            li[u] = ok[u] && !a.ident ? a.label[i[u]] : i[u];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (ok[u] && (j[u] <= i[u] || j[u] >= a.n)) {
                set_err(a.err, DEV_BAD_INPUT);
                ok[u] = false;
            }
            lj[u] = ok[u] ? (a.ident ? j[u] : a.label[j[u]]) : li[u];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            ok[u] = ok[u] && lj[u] != li[u];
            cj[u] = ok[u] ? __ldcg(a.best + lj[u]) : 0ull;
            ci[u] = ok[u] ? __ldcg(a.best + li[u]) : 0ull;
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const unsigned bal = __ballot_sync(0xffffffffu, ok[u]);
            if (!bal) continue;
            const uint64_t k = a.pk.make(wq[u], (uint32_t)i[u], (uint32_t)j[u]);
            if (ok[u]) {
                atomicAdd(&s_kh[wq[u]], 1u);
                if ((k >> 1) < cj[u]) atomicMin(a.best + lj[u], (unsigned long long)(k >> 1));
                rec[out + __popc(bal & below)] = k;
            }
            // (a row's records are consecutive: one reduction for each run)
            if (__any_sync(0xffffffffu, ok[u] && (k >> 1) < ci[u]))
                seg_min_atomic(ok[u], li[u], k >> 1, a.best);
            out += __popc(bal);
        }
        __syncwarp();
    }
    if (out == 0) return;
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(a.cursor, (unsigned long long)out);
    at = __shfl_sync(0xffffffffu, at, 0);
    if (at + (unsigned long long)out > a.cap) {
        if (lane == 0) set_err(a.err, DEV_CAPACITY);
    } else {
        for (int t = lane; t < out; t += 32) a.eout[at + t] = rec[t];
    }
    __syncwarp();                    // the records are written again
}

// Appends to the warp's records the entries of row i that the lanes' bits m
// name: bit q is entry e + q of the lane's first load, and every PER bits a
// load of the warp's further on.  More than CAP at once go 4 bits at a time.
template <int CAP, int PER, typename Flush>
__device__ __forceinline__ void up_record(unsigned m, int64_t e, int32_t i, uint64_t *rec,
                                          int32_t *rrow, int &nrec, Flush flush)
{
    static_assert(CAP >= 4 * 32, "a piece of 4 bits fits");
    const int lane = threadIdx.x & 31;
    if (!__any_sync(0xffffffffu, m != 0u)) return;
    unsigned rest = m;
    int piece = 32;
    while (true) {
        const unsigned now = piece < 32 ? rest & ((1u << piece) - 1u) : rest;
        int incl = __popc(now);
        int p = -incl;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += o;
        }
        const int tot = __shfl_sync(0xffffffffu, incl, 31);
        if (tot > CAP) {
            piece = 4;
            continue;
        }
        if (nrec + tot > CAP) {
            flush(nrec);
            nrec = 0;
        }
        p += nrec + incl;
        for (unsigned t = now; t; t &= t - 1u, ++p) {
            const int q = __ffs(t) - 1;
            rec[p] = (uint64_t)(e + q + (q / PER) * (31 * PER));
            rrow[p] = i;
        }
        nrec += tot;
        rest &= ~now;
        if (piece == 32) break;
        piece += 4;
        if (piece > 32 || !__any_sync(0xffffffffu, rest != 0u)) break;
    }
}

// bits q of m kept for the entries e + q of N that lie in [s, e_end)
template <int N>
__device__ __forceinline__ unsigned up_clip(unsigned m, int64_t e, int64_t s, int64_t e_end)
{
    if (e >= s && e + N <= e_end) return m;
    const int64_t a = s - e, b = e_end - e;
    const int qa = a < 0 ? 0 : (a > N ? N : (int)a);
    const int qb = b < 0 ? 0 : (b > N ? N : (int)b);
    constexpr unsigned all = (1u << N) - 1u;
    return m & (all << qa) & (all >> (N - qb));
}

// the 16 weights from entry e on, zero outside the array
__device__ __noinline__ uint4 up_edge_bytes(const uint8_t *w, int64_t e, int64_t nnz)
{
    uint32_t t[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int q = 0; q < 16; ++q)
        if (e + q >= 0 && e + q < nnz) t[q >> 2] |= (uint32_t)w[e + q] << (8 * (q & 3));
    return make_uint4(t[0], t[1], t[2], t[3]);
}

// A warp per row, 16 weights per lane and load, two loads in flight with the
// next row's extent; any order and any alignment of the arrays.
__global__ void __launch_bounds__(kPhThreads, 4)
k_phase_upper(const __grid_constant__ UpArgs a)
{
    constexpr int G = 2;
    __shared__ unsigned s_kh[256];           // kept entries per weight, this block
    __shared__ uint64_t rec_all[kPhWarps][kUpRec];
    __shared__ int32_t row_all[kPhWarps][kUpRec];
    for (int b = threadIdx.x; b < 256; b += blockDim.x) s_kh[b] = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    uint64_t *rec = rec_all[threadIdx.x >> 5];
    int32_t *rrow = row_all[threadIdx.x >> 5];
    int nrec = 0;
    const uint32_t c1 = 0x00010001u * (uint32_t)(0x8000 - (a.lo + 1));
    const uint32_t c2 = 0x00010001u * (uint32_t)(0x7fff - a.hi);
    const int mis = (int)((uintptr_t)a.w & 15);
    const int64_t nwarps = (int64_t)gridDim.x * kPhWarps;
    int64_t i = a.row0 + (int64_t)blockIdx.x * kPhWarps + (threadIdx.x >> 5);
    int64_t s1 = 0, e1 = 0;
    if (i < a.row1) {
        s1 = a.indptr[i];
        e1 = a.indptr[i + 1];
    }
    for (; i < a.row1; i += nwarps) {
        const int64_t s = s1, e_end = e1;
        if (i + nwarps < a.row1) {
            s1 = a.indptr[i + nwarps];
            e1 = a.indptr[i + nwarps + 1];
        }
        if (s < 0 || e_end < s || e_end > a.nnz) {
            if (lane == 0) set_err(a.err, DEV_BAD_INPUT);
            continue;
        }
        // groups start on 16-byte boundaries of the weights (the first may
        // start before the array: its loads are made byte by byte)
        for (int64_t g = s - ((s + mis) & 15); g < e_end; g += 512 * G) {
            uint4 v[G];
#pragma unroll
            for (int u = 0; u < G; ++u) {
                const int64_t e = g + 512 * u + 16 * lane;
                v[u] = make_uint4(0u, 0u, 0u, 0u);
                if (e >= e_end) continue;
                v[u] = e >= 0 && e + 15 < a.nnz ? __ldg(reinterpret_cast<const uint4 *>(a.w + e))
                                                : up_edge_bytes(a.w, e, a.nnz);
            }
            unsigned m = 0u;
#pragma unroll
            for (int u = 0; u < G; ++u) {
                const unsigned x =
                    bytes_in_range(v[u].x, c1, c2) | bytes_in_range(v[u].y, c1, c2) << 4 |
                    bytes_in_range(v[u].z, c1, c2) << 8 | bytes_in_range(v[u].w, c1, c2) << 12;
                m |= up_clip<16>(x, g + 512 * u + 16 * lane, s, e_end) << (16 * u);
            }
            up_record<kUpRec, 16>(m, g + 16 * lane, (int32_t)i, rec, rrow, nrec,
                                  [&](int c) { up_flush(a, rec, rrow, c, s_kh); });
        }
    }
    up_flush(a, rec, rrow, nrec, s_kh);
    __syncthreads();
    for (int b = threadIdx.x; b < 256; b += blockDim.x)
        if (s_kh[b]) atomicAdd(&a.khist[b], (unsigned long long)s_kh[b]);
}

// The last phase: all the weights left, once the components are few.  Of the
// entries between two components only the least can be in the forest, so
// none is written: pairs[c * V + d] receives the least key between rows of
// component c and columns of component d (V of them, numbered in cid), and
// k_pair_emit makes one word of each pair.  Nearly every entry joins a
// component to itself, and telling so by gathering the other end's component
// takes an L2 access per entry (920M entries of 300,000 rows: 4.9 ms, most
// of it L1 misses; this kernel takes 1.5, 3.1 TB/s of the 5 bytes per entry).  Here the rows are taken component by component (ord,
// the components of at least kPairMin vertices first): a block holds the
// component's members as a bitmap in shared memory, an entry costs one
// shared-memory read, and those that leave the component become records,
// whose pass offers them to the block's least keys per component.  The rows
// of the smaller components offer every entry to the pairs themselves.
// Blocks take shares of the row list that are equal in entries (pre: the
// rows' first entries in list order), several for each block: a share whose
// rows mostly leave their component takes up to 2.5 times as long.
constexpr int kPairThreads = 1024;
constexpr int kPairWarps = kPairThreads / 32;
constexpr int kPairMax = 2048;       // components at most
constexpr int64_t kPairOuter = (int64_t)1 << 21;   // entries between components at most, beside
constexpr int64_t kPairOuterShare = 16;            // one in this many of all
constexpr int kOuterSample = 1 << 14;              // estimated from as many
constexpr int kPairNarrow = 3;                     // times that other phases are tried first
constexpr int kPairMin = 32;         // vertices from which a bitmap is worth its making
constexpr int kPairBlocks = 148;     // one per SM
// shares per block at most, of at least kPairShareMin entries: fewer leave a
// tail, more wait at more barriers (100,000 points x 50 partitions 2.12, 2.18
// and 2.29 ms with 3, 5 and 8; 300,000 x 30 4.72, 4.51, 4.63)
constexpr int kPairShares = 5;
constexpr int64_t kPairShareMin = (int64_t)1 << 17;
constexpr size_t kPairRecBytes = (size_t)kPairWarps * kPairRec * (sizeof(uint64_t) + sizeof(int32_t));
constexpr size_t kPairMaxSmem = 220 << 10;

static size_t pair_smem(int32_t n, int V)
{
    return kPairRecBytes + (size_t)V * sizeof(uint64_t) + (size_t)(((int64_t)n + 31) / 32) * 4;
}

struct PairArgs {
    const int32_t *ord;              // rows, component by component
    const int64_t *pre;              // n + 1: entries of the rows before
    const int32_t *size;             // vertices per root
    const int32_t *off;              // first list place per root of a large component
    int *share;                      // zeroed: shares taken
    int shares;
    const uint16_t *cid;             // component number per vertex
    unsigned long long *pairs;       // V x V
    int V;
};

// The warp's n records: checked, offered to the block's least keys (rows of
// one component) or, with least null, to the pairs.
__device__ __noinline__ void pair_flush(const UpArgs &a, const PairArgs &o,
                                        unsigned long long *least, const uint64_t *rec,
                                        const int32_t *rrow, int n)
{
    constexpr int U = 4;
    const int lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int u = 0; u < U; ++u) {
        static_assert(kPairRec == 32 * U, "one pass");
        const int t = 32 * u + lane;
        if (t >= n) continue;
        const int64_t e = (int64_t)rec[t];
        const int32_t i = rrow[t], j = __ldg(a.indices + e);
        const uint32_t w = __ldg(a.w + e);
        if (j <= i || j >= a.n) {
            set_err(a.err, DEV_BAD_INPUT);
            continue;
        }
        const unsigned long long k = a.pk.make(w, (uint32_t)i, (uint32_t)j) >> 1;
        const int d = o.cid[j];
        if (least) {
            if (k < *(volatile unsigned long long *)(least + d)) atomicMin(least + d, k);
        } else {
            const int c = o.cid[i];
            if (c != d) min_if_lower(o.pairs + (int64_t)c * o.V + d, k);
        }
    }
    __syncwarp();                    // the records are written again
}

__global__ void __launch_bounds__(kPairThreads, 1)
k_pair_min(const __grid_constant__ UpArgs a, const __grid_constant__ PairArgs o)
{
    constexpr int G = 4;
    extern __shared__ __align__(16) uint8_t pair_smem_raw[];
    uint64_t *rec_all = reinterpret_cast<uint64_t *>(pair_smem_raw);
    unsigned long long *least = reinterpret_cast<unsigned long long *>(rec_all + kPairWarps * kPairRec);
    int32_t *row_all = reinterpret_cast<int32_t *>(least + o.V);
    uint32_t *bm = reinterpret_cast<uint32_t *>(row_all + kPairWarps * kPairRec);
    __shared__ int s_next, s_share;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t *rec = rec_all + warp * kPairRec;
    int32_t *rrow = row_all + warp * kPairRec;
    const uint32_t c1 = 0x00010001u * (uint32_t)(0x8000 - (a.lo + 1));
    const uint32_t c2 = 0x00010001u * (uint32_t)(0x7fff - a.hi);
    const int shares = o.shares;
    // where share b begins: the first row whose first entry lies in it
    auto first_row = [&](int b) -> int {
        if (b >= shares) return a.n;
        const int64_t tot = o.pre[a.n];
        const int64_t t = tot / shares * b + tot % shares * b / shares;
        int lo = 0, hi = a.n;
        while (lo < hi) {                    // 32 probes at a time
            const int at = lo + (int)((int64_t)(hi - lo) * lane / 32);
            const int c = __popc(__ballot_sync(0xffffffffu, o.pre[at] < t));
            const int last = __shfl_sync(0xffffffffu, at, c ? c - 1 : 0);
            const int next = __shfl_sync(0xffffffffu, at, c < 32 ? c : 31);
            if (c < 32) hi = next;
            if (c) lo = last + 1;
        }
        return lo;
    };
    const int words = (a.n + 31) / 32;
    while (true) {
        if (threadIdx.x == 0) s_share = atomicAdd(o.share, 1);
        __syncthreads();
        const int share = shares - 1 - s_share;    // (the small components' rows first)
        if (share < 0) break;
        int x = first_row(share);
        const int x1 = first_row(share + 1);
        while (x < x1) {
            // the share's rows of one component, or those of small ones
            const int32_t v0 = o.ord[x], root = a.label[v0];
            const int members = o.size[root], c0 = o.off[root], row = o.cid[v0];
            const bool own = members >= kPairMin;
            const int xe = own ? min(x1, c0 + members) : x1;
            auto flush = [&](int c) { pair_flush(a, o, own ? least : nullptr, rec, rrow, c); };
            if (threadIdx.x == 0) s_next = x;
            if (own) {
                for (int b = threadIdx.x; b < words; b += kPairThreads) bm[b] = 0u;
                for (int b = threadIdx.x; b < o.V; b += kPairThreads) least[b] = kNone;
                __syncthreads();
                for (int y = threadIdx.x; y < members; y += kPairThreads) {
                    const int32_t v = o.ord[c0 + y];
                    atomicOr(&bm[v >> 5], 1u << (v & 31));
                }
            }
            __syncthreads();
            // rows by a counter, the next one's extent loaded ahead
            auto take = [&](int32_t &i, int64_t &s, int64_t &e) -> bool {
                int y = 0;
                if (lane == 0) y = atomicAdd(&s_next, 1);
                y = __shfl_sync(0xffffffffu, y, 0);
                if (y >= xe) return false;
                i = o.ord[y];
                s = a.indptr[i];
                e = a.indptr[i + 1];
                return true;
            };
            int nrec = 0;
            int32_t i = 0, i1 = 0;
            int64_t s = 0, e_end = 0, s1 = 0, e1 = 0;
            bool more = take(i, s, e_end);
            while (more) {
                more = take(i1, s1, e1);
                if (s < 0 || e_end < s || e_end > a.nnz) {
                    if (lane == 0) set_err(a.err, DEV_BAD_INPUT);
                    s = e_end = 0;
                }
                const uint32_t span = (uint32_t)(a.n - 1 - i);
                for (int64_t g = s & ~(int64_t)3; g < e_end; g += 128 * G) {
                    uint32_t wv[G];
                    int4 jv[G];
#pragma unroll
                    for (int u = 0; u < G; ++u) {
                        const int64_t e = g + 128 * u + 4 * lane;
                        wv[u] = 0u;
                        jv[u] = make_int4(0, 0, 0, 0);
                        if (e >= e_end) continue;
                        if (e + 3 < a.nnz) {
                            wv[u] = __ldg(reinterpret_cast<const uint32_t *>(a.w + e));
                            jv[u] = __ldg(reinterpret_cast<const int4 *>(a.indices + e));
                        } else {
                            int32_t t[4] = {0, 0, 0, 0};
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                if (e + q >= a.nnz) continue;
                                wv[u] |= (uint32_t)a.w[e + q] << (8 * q);
                                t[q] = a.indices[e + q];
                            }
                            jv[u] = make_int4(t[0], t[1], t[2], t[3]);
                        }
                    }
                    unsigned m = 0u;
#pragma unroll
                    for (int u = 0; u < G; ++u) {
                        unsigned x = up_clip<4>(bytes_in_range(wv[u], c1, c2), g + 128 * u + 4 * lane, s, e_end);
                        const int32_t jj[4] = {jv[u].x, jv[u].y, jv[u].z, jv[u].w};
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            // (a column outside (i, n) is recorded: the records'
                            // pass reports it)
                            const bool in = (uint32_t)(jj[q] - i - 1) < span;
                            const int32_t j = in ? jj[q] : i;
                            if (own && in && ((bm[j >> 5] >> (j & 31)) & 1u)) x &= ~(1u << q);
                        }
                        m |= x << (4 * u);
                    }
                    up_record<kPairRec, 4>(m, g + 4 * lane, i, rec, rrow, nrec, flush);
                }
                i = i1;
                s = s1;
                e_end = e1;
            }
            flush(nrec);
            __syncthreads();
            if (own)
                for (int b = threadIdx.x; b < o.V; b += kPairThreads)
                    if (least[b] != kNone) min_if_lower(o.pairs + (int64_t)row * o.V + b, least[b]);
            __syncthreads();                     // the bitmap, least and the counters start anew
            x = xe;
        }
        __syncthreads();
    }
}

// One word per pair of components with an entry between them, offered to both.
__global__ void k_pair_emit(const unsigned long long *pairs, int V, const int32_t *roots,
                            uint64_t *eout, unsigned long long *cursor, unsigned long long *best)
{
    const int c = blockIdx.x;
    for (int d = c + 1 + threadIdx.x; d < V; d += blockDim.x) {
        const uint64_t x = pairs[(int64_t)c * V + d], y = pairs[(int64_t)d * V + c];
        const uint64_t m = x < y ? x : y;
        if (m == kNone) continue;
        eout[atomicAdd(cursor, 1ull)] = m << 1;
        min_if_lower(best + roots[c], m);
        min_if_lower(best + roots[d], m);
    }
}

// The row list of k_pair_min: vertices per root; the components' numbers and
// the large ones' sizes (a scan then places them); the list with its rows'
// lengths.
// (Lanes with the same root share an atomic: the components are few.)
__global__ void k_pair_count(const int32_t *label, int32_t n, int32_t *size)
{
    for (int64_t vb = (int64_t)blockIdx.x * blockDim.x; vb < n; vb += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = vb + threadIdx.x;
        const int32_t r = v < n ? label[v] : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, r);
        if (r >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&size[r], __popc(peers));
    }
}

// (found: zeroed; V: the components there are)
__global__ void k_pair_number(const int32_t *size, int32_t n, int V, int32_t *large, int32_t *number,
                              int32_t *roots, int32_t *found)
{
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n;
         r += (int64_t)gridDim.x * blockDim.x) {
        large[r] = size[r] >= kPairMin ? size[r] : 0;
        if (size[r] == 0) continue;
        const int c = atomicAdd(found, 1);
        if (c < V) roots[c] = (int32_t)r;
        number[r] = min(c, V - 1);
    }
}

// given: zeroed, the places given out per root; *others likewise for the
// small components' rows, which come after the *n_large others.  A
// component's rows come in about ascending order, so that later rows' keys
// are seldom the lower ones.
__global__ void k_pair_place(const int64_t *indptr, const int32_t *label, int32_t n, int64_t nnz,
                             const int32_t *size, const int32_t *off, const int64_t *n_large,
                             const int32_t *number, int32_t *given, int32_t *others, int32_t *ord,
                             int32_t *len, uint16_t *cid)
{
    const int lane = threadIdx.x & 31;
    for (int64_t vb = (int64_t)blockIdx.x * blockDim.x; vb < n; vb += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = vb + threadIdx.x;
        const int32_t r = v < n ? label[v] : -1;
        const bool large = r >= 0 && size[r] >= kPairMin;
        const unsigned peers = __match_any_sync(0xffffffffu, large ? r : r >= 0 ? -2 : -1);
        const int lead = __ffs(peers) - 1, cnt = __popc(peers);
        int base = 0;
        if (lane == lead && r >= 0)
            base = large ? off[r] + atomicAdd(&given[r], cnt)
                         : (int)*n_large + atomicAdd(others, cnt);
        base = __shfl_sync(0xffffffffu, base, lead);
        if (v < n) {
            const int at = base + __popc(peers & ((1u << lane) - 1u));
            const int64_t s = indptr[v], e = indptr[v + 1];
            ord[at] = (int32_t)v;
            // (a bad extent counts as empty here; its row reports it)
            len[at] = (s < 0 || e < s || e > nnz || e - s > 0x7fffffff) ? 0 : (int32_t)(e - s);
            cid[v] = (uint16_t)number[r];
        }
    }
}

// One phase: the entries with weight bucket in (lo, hi] of rows [r0, r1);
// with slot >= 0 the range is read on the device from the plan's slot.
struct Phase {
    int lo, hi;
    int64_t r0, r1;
    int slot;
    int ident;            // the labels are still the identity (no merges yet)
    int pairs = 0;        // components, in the phase that takes their pairs (k_pair_min)
};

// Phase ranges (lo, hi] of weight buckets: cut the bucket histogram at the
// given cumulative fractions of the entries.
__host__ __device__ static int phase_ranges(const unsigned long long *hist, const double *fracs,
                                            int nf, int *lo, int *hi)
{
    unsigned long long tot = 0;
    for (int b = 0; b < 256; ++b) tot += hist[b];
    int np = 0, prev = -1;
    unsigned long long acc = 0;
    int b = 0;
    for (int f = 0; f < nf; ++f) {
        const double target = fracs[f] * (double)tot;
        while (b < 255 && (double)(acc + hist[b]) < target) acc += hist[b++];
        const int cut = (f == nf - 1) ? 255 : b;
        if (cut > prev) {
            lo[np] = prev;
            hi[np] = cut;
            np++;
            prev = cut;
        }
        if (cut == 255) break;
        acc += hist[b];
        b++;
    }
    if (prev < 255) {
        lo[np] = prev;
        hi[np] = 255;
        np++;
    }
    return np;
}

// The weight phases of an MST on the device (no host read): ranges (lo, hi]
// at cumulative fractions p1 (per mille of the entries; a tuning-table
// knob, default a quarter) and 1 of the histogram, one slot each in lohi
// (an unused slot holds the empty range (255, 255]).
constexpr int kPhaseSlots = 2;
__global__ void k_phase_plan(const unsigned long long *hist, int *lohi, int p1_permille)
{
    __shared__ unsigned long long h[256];
    for (int b = threadIdx.x; b < 256; b += blockDim.x) h[b] = hist[b];
    __syncthreads();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double fracs[kPhaseSlots] = {p1_permille / 1000.0, 1.0};
    int lo[8], hi[8];
    const int np = phase_ranges(h, fracs, kPhaseSlots, lo, hi);
    for (int q = 0; q < kPhaseSlots; ++q) {
        lohi[2 * q] = q < np ? lo[q] : 255;
        lohi[2 * q + 1] = q < np ? hi[q] : 255;
    }
}

constexpr int kMaxRounds = 96;   // Boruvka rounds per phase (halving: 96 is never reached)

// Round state kept on the device (int64 words), so that the phases of an MST
// can be queued back to back without a host read:
enum : int {
    C_V = 0,          // supervertices at the start of the next round
    C_E = 1,          // edge words in the round kernel's input buffer
    C_NMST = 2,       // forest edges emitted so far (all phases)
    C_CURSOR = 3,     // phase-build output cursor
    C_ROUNDS = 4,     // rounds run by the last round kernel
    C_DONE = 5,       // how the last round kernel ended (see k_rounds)
    C_ROUNDS_ALL = 6, // rounds run since the engine's reset (all phases)
    C_EBUF = 7,       // edge buffer holding the last round's survivors (0 or 1)
    C_AUX0 = 8,       // scratch totals of single-pass kernels
    C_AUX1 = 9,
    C_SYM_LT = 10,    // CSR entries u -> v with u < v (symmetry check)
    C_SYM_GT = 11,    // ... with u > v
    C_PLAN = 12,      // the final clustering's CutPlan (four words)
    C_COUNT = 16
};

// ---------------------------------------------------------------------------
// Boruvka rounds: all rounds of a phase in ONE persistent kernel.
//
// Supervertices are named by an original vertex, their root: `parent` is a
// union-find forest over the original vertices (a root points to itself), so
// a round never renumbers anything and never sweeps all original vertices;
// an edge endpoint or a key endpoint finds its supervertex by following
// parent pointers (and shortens the path it walked).  Only the ACTIVE roots
// -- those with an edge to another supervertex -- are visited, from a list
// kept in increasing id order.
//
// The participants are either every block of a cooperative grid (all blocks
// resident at once, so they may wait on one another) or a single block.
// Each participant owns a contiguous chunk of the original vertices (its
// part of the active list) and a contiguous segment of the phase's edge
// words; both shrink in place.  Between the steps of a round the
// participants meet at a barrier: a bounded spin on an arrival counter for
// the grid, __syncthreads for one block.  Once few active roots and edges are
// left, the grid's other blocks leave and block 0 runs the remaining rounds
// alone for every participant's chunk and segment (no grid barriers).
// A round is
//   A. per active root s: its successor t (the root of the other end of its
//      selected key); a mutual pick (t's successor is s) is broken towards
//      the larger id, so the smaller one stays a root
//      (MyML/MyML/graph/mst.py:283-305); color[s] = t, or s.
//   B. in list order: each non-root emits its key as a forest edge (slots in
//      root-id order, from the participants' counts), finds its new root
//      (bounded chase with compare-and-swap path halving over color) and
//      points its parent there; the roots that still have an edge stay in the
//      list, and their selection slots are cleared.
//   D. contraction fused with the next round's minimum-edge selection: each
//      edge word whose endpoints now have different roots stays in its
//      segment (compacted in place: a tile's words are in registers before
//      any of the tile's survivors is written, and survivors never move past
//      their tile) and is offered to both its roots' slots (one atomicMin per
//      run of equal first root in a warp, and one for the other root).  Edge order does not matter:
//      selection uses total orders, so every result is independent of it.
// Three barriers per round.  After the last one every participant reads the
// same sizes and takes the same decision to stop:
//   C_DONE = 1 converged (no edge left), 2 no contraction (not a valid
//   graph), 3 round cap, 4 a device error.
// Root ids keep the reference's choices: its renumbering is order-preserving,
// so "smaller id" and "smallest destination" compare the same way, and its
// final component number is the rank of the root id (k_rank_roots).
// The steps handle several elements per thread at a time with all loads of
// one level issued together: they are chains of dependent gathers, so the
// independent chains in flight, not bandwidth, set their speed.
// ---------------------------------------------------------------------------
constexpr int kRT = 1024;                       // round-kernel threads per block
constexpr int kRItems = 4;                      // edge words per thread per tile
constexpr int kRV = 4;                          // vertices per thread per step
constexpr int64_t kRTile = (int64_t)kRT * kRItems;
constexpr int kRWarps = kRT / 32;
constexpr int kMaxTeam = 148 * 8;               // participants (blocks) at most
constexpr long long kBarrierSpins = 1ll << 21;  // about a second of waiting
constexpr int64_t kSoloActive = 1024;           // block 0 alone below these sizes
constexpr int64_t kSoloEdges = 8192;
constexpr int kFindLimit = 1 << 20;             // parent-chain steps (a forest is shorter)
// bits for the active roots beside a count of edge words: a word holds 8 bits
// of weight or more, two vertices and a spare bit, so there are at most 2^27
// roots, which leaves the words 2^35 (with 31 bits for the roots, 2^32 words
// -- a phase of 17 million points can keep as many -- turned the count negative)
constexpr int kActiveBits = 28;
static_assert((64 - 1 - 8) / 2 < kActiveBits, "every root counts");

struct GridBarrier {
    unsigned count;       // arrivals since the launch began (never reset inside one)
    unsigned pad;
};

// Grid-wide barrier of a cooperative launch.  Thread 0 of each block adds
// its arrival to a counter that only grows, with no return value, and waits
// until the counter reaches (barriers passed + 1) x blocks: no block resets
// anything, so the last arrival is the only write the others wait for.  The
// counter starts at zero (the host clears it before each launch).  The wait
// gives up after about a second (DEV_SPIN_LIMIT), or as soon as any block
// has raised an error, so a block that left early never holds the others.
// Returns false when it gave up.  The arrival is a release and the polling
// load an acquire (gpu scope); with the block barriers around them they
// order every thread's writes before the arrival and its reads after the
// wait.  The data exchanged between blocks is read with L1-bypassing loads.
__device__ __forceinline__ bool grid_barrier(GridBarrier *b, unsigned &passed, int *err)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned target = (passed + 1u) * gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&b->count) : "memory");
        auto count_now = [&]() -> unsigned {
            unsigned c;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(&b->count) : "memory");
            return c;
        };
        int ok = 1;
        long long spins = 0;
        while ((int)(count_now() - target) < 0) {
            if (*(volatile int *)err) {
                ok = 0;
                break;
            }
            if (++spins > kBarrierSpins) {
                set_err(err, DEV_SPIN_LIMIT);
                ok = 0;
                break;
            }
            if (spins > 256) __nanosleep(32);
        }
        s_ok = ok;
    }
    __syncthreads();
    ++passed;
    return s_ok != 0;
}

struct RoundArgs {
    Pack pk;
    int64_t V0;
    uint64_t *e;                  // edge words of the phase (compacted per segment)
    int32_t *parent;              // V0: union-find parent (a root points to itself)
    unsigned long long *best;     // V0: selection slot per root
    int32_t *color;               // V0: successor, then new root, per active root
    int32_t *act;                 // V0: active roots, per participant chunk
    uint64_t *mst;                // forest keys, appended at cnt[C_NMST] (MST mode)
    int32_t *part;                // 2 x kMaxTeam: per participant (emits, merges)
    int32_t *alen;                // kMaxTeam: active roots per participant
    int64_t *seg;                 // kMaxTeam: edge words per participant segment
    int64_t *cnt;                 // C_* round state
    int64_t *trace;               // 3 x kMaxRounds: (V, E, active) per round
    GridBarrier *bar;
    int *err;
    int max_rounds;
    int from_cursor;              // edge count = cnt[C_CURSOR] (a queued phase's build)
    int first_phase;              // supervertex count = V0
};

// Roots of N vertices at once (all parent loads of one level issued
// together); each vertex whose first parent was not its root is pointed at
// the root (a benign race: every writer writes the same root).  Negative
// ids (empty lanes) are left alone: they must not all walk and rewrite the
// path of one real vertex.
// The parent loads may be served by L1: late rounds send most finds to the
// few roots left, and L2-only loads of those few lines from every SM
// serialise (a 20x slower contraction measured on a 16-NN graph).  The
// entries a round rewrites (merged roots, step B) were written before the
// barrier that precedes the finds, whose acquire fence orders the later
// loads after them; within a step the only writes are path compressions,
// so a stale value is an older ancestor and the walk still ends at the root.
template <int N>
__device__ __forceinline__ void find_batch(int32_t *parent, int32_t (&x)[N], int *err)
{
    int32_t r[N], first[N];
    bool go[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        r[i] = x[i] >= 0 ? parent[x[i]] : x[i];
        first[i] = r[i];
        go[i] = r[i] != x[i];
    }
    for (int step = 0;; ++step) {
        int32_t up[N];
        bool any = false;
#pragma unroll
        for (int i = 0; i < N; ++i) up[i] = go[i] ? parent[r[i]] : r[i];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if (go[i] && up[i] != r[i]) {
                r[i] = up[i];
                any = true;
            } else {
                go[i] = false;
            }
        }
        if (!any) break;
        if (step > kFindLimit) {
            set_err(err, DEV_CHASE_LIMIT);
            break;
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (first[i] != x[i] && first[i] != r[i]) parent[x[i]] = r[i];
        x[i] = r[i];
    }
}

// Successors of up to kRV active roots at once (s[i] < 0: none): the root of
// the other end of each selected key, or the root itself when it selected
// nothing.
// b receives the selected keys.
template <int MODE>
__device__ __forceinline__ void succ_batch(const RoundArgs &a, const int32_t (&s)[kRV],
                                           int32_t (&t)[kRV], uint64_t (&b)[kRV])
{
#pragma unroll
    for (int i = 0; i < kRV; ++i) b[i] = s[i] >= 0 ? __ldcg(a.best + s[i]) : kNone;
    if constexpr (MODE == SEL_CC) {
#pragma unroll
        for (int i = 0; i < kRV; ++i) t[i] = b[i] == kNone ? s[i] : (int32_t)(uint32_t)b[i];
    } else {
    int32_t e[2 * kRV];
#pragma unroll
    for (int i = 0; i < kRV; ++i) {
        const bool ok = b[i] != kNone;
        e[2 * i] = ok ? (int32_t)a.pk.sel_a(b[i]) : -1;
        e[2 * i + 1] = ok ? (int32_t)a.pk.sel_b(b[i]) : -1;
    }
    find_batch<2 * kRV>(a.parent, e, a.err);
#pragma unroll
    for (int i = 0; i < kRV; ++i)
        t[i] = b[i] == kNone ? s[i] : (e[2 * i] == s[i] ? e[2 * i + 1] : e[2 * i]);
    }
}

template <int MODE, bool GRID>
__global__ void __launch_bounds__(kRT, 1)
k_rounds(RoundArgs a)
{
    __shared__ int s_off[kRItems][kRWarps];
    __shared__ int s_base;
    __shared__ int s_err;
    const int64_t P = GRID ? (int64_t)gridDim.x : 1, p = GRID ? (int64_t)blockIdx.x : 0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    bool solo = !GRID;                  // one block does all the work
    int64_t Pe = P;                     // participants whose chunks and segments are in use
    unsigned passed = 0;                // grid barriers passed (the same in every block)
    auto sync = [&]() -> bool {
        if (!solo) return grid_barrier(a.bar, passed, a.err);
        __syncthreads();
        return true;
    };
    // a queued weight phase starts from its build's cursor and the previous
    // phase's supervertex count (V0 for the first phase)
    int64_t V = a.first_phase ? a.V0 : __ldcg(a.cnt + C_V);
    int64_t E = __ldcg(a.cnt + (a.from_cursor ? C_CURSOR : C_E));
    int64_t nmst = __ldcg(a.cnt + C_NMST);
    const int64_t E0 = E;
    const int64_t seg_stride = (E0 + P - 1) / P;     // edge segment of participant q
    const int64_t vchunk = (a.V0 + P - 1) / P;       // vertex chunk of participant q
    auto ebase = [&](int64_t q) { return min(E0, q * seg_stride); };
    auto vbase = [&](int64_t q) { return min(a.V0, q * vchunk); };

    // ---- active list: the roots with a selection, in id order -------------
    // (kRV consecutive vertices per thread: the loads of all in flight, one
    // block scan per kRT * kRV vertices)
    for (int64_t q = solo ? 0 : p; q < (solo ? P : p + 1); ++q) {
        const int64_t v0 = vbase(q), v1 = min(a.V0, v0 + vchunk);
        int64_t kept = 0;
        for (int64_t xb = v0; xb < v1; xb += (int64_t)kRT * kRV) {
            const int64_t x0 = xb + (int64_t)tid * kRV;
            int32_t par[kRV];
            uint64_t sel[kRV];
#pragma unroll
            for (int i = 0; i < kRV; ++i) {
                const bool in = x0 + i < v1;
                par[i] = in ? __ldcg(a.parent + x0 + i) : -1;
                sel[i] = in ? __ldcg(a.best + x0 + i) : kNone;
            }
            int c = 0;
            bool on[kRV];
#pragma unroll
            for (int i = 0; i < kRV; ++i) {
                on[i] = par[i] == (int32_t)(x0 + i) && sel[i] != kNone;
                c += on[i] ? 1 : 0;
            }
            int64_t ttot;
            int64_t at = v0 + kept + block_excl_sum_shfl<kRT>(c, ttot);
#pragma unroll
            for (int i = 0; i < kRV; ++i)
                if (on[i]) a.act[at++] = (int32_t)(x0 + i);
            kept += ttot;
        }
        const int64_t e0 = ebase(q);
        if (tid == 0) {
            a.alen[q] = (int32_t)kept;
            a.seg[q] = min(E0, e0 + seg_stride) - e0;
        }
    }
    if (tid == 0) s_err = *(volatile int *)a.err;
    __syncthreads();
    int round = 0, done = s_err ? 4 : ((E == 0 || V <= 1) ? 1 : 0);
    if (!done && !sync()) done = 4;
    int64_t Aact = 0;                                 // active roots this round
    if (!done) {
        int64_t x = 0;
        for (int64_t j = tid; j < P; j += kRT) x += __ldcg(a.alen + j);
        block_excl_sum_shfl<kRT>(x, Aact);
    }
    while (!done) {
        const int64_t q0 = solo ? 0 : p, q1 = solo ? Pe : p + 1;
        // ---- A: successors, mutual picks, per-participant counts ---------
        for (int64_t q = q0; q < q1; ++q) {
            const int32_t *al = a.act + vbase(q);
            const int64_t n = __ldcg(a.alen + q);
            int64_t mine = 0;                   // (forest edges << 32) | merges
            for (int64_t ib = tid; ib < n; ib += (int64_t)kRT * kRV) {
                int32_t s[kRV], t[kRV];
                uint64_t b[kRV], bt[kRV];
#pragma unroll
                for (int i = 0; i < kRV; ++i) {
                    const int64_t j = ib + (int64_t)i * kRT;
                    s[i] = j < n ? __ldcg(al + j) : -1;
                }
                succ_batch<MODE>(a, s, t, b);
                // mutual pick: only a smaller s with a successor needs t's
                // selection.  CC keys name the other end; MST keys are one
                // per edge word and every word is offered to both its ends,
                // so two roots pick each other exactly when their keys are
                // the same (no root has to be found again)
#pragma unroll
                for (int i = 0; i < kRV; ++i)
                    bt[i] = (s[i] >= 0 && s[i] < t[i]) ? __ldcg(a.best + t[i]) : kNone;
#pragma unroll
                for (int i = 0; i < kRV; ++i) {
                    if (s[i] < 0) continue;
                    const bool mutual =
                        MODE == SEL_MST ? bt[i] != kNone && bt[i] == b[i]
                                        : bt[i] != kNone && (int32_t)(uint32_t)bt[i] == s[i];
                    const bool keep = t[i] != s[i] && !mutual;
                    a.color[s[i]] = keep ? t[i] : s[i];
                    mine += keep ? ((MODE == SEL_MST ? (1ll << 32) : 0ll) | 1ll) : 0ll;
                }
            }
            int64_t btot;
            block_excl_sum_shfl<kRT>(mine, btot);
            if (tid == 0) {
                a.part[q] = (int32_t)(btot >> 32);             // forest edges
                a.part[kMaxTeam + q] = (int32_t)(btot & 0xffffffffll);   // merges
            }
        }
        if (!sync()) break;

        // ---- B: forest edges, new roots, the next active list -----------
        int64_t merges = 0, epre = 0;           // all merges; forest edges before q0
        {
            // both below 2^31 (at most V0 each): one scan of (merges << 32) | edges
            int64_t x = 0, tot = 0;
            for (int64_t j = tid; j < Pe; j += kRT) {
                x += (int64_t)__ldcg(a.part + kMaxTeam + j) << 32;
                if (j < q0) x += __ldcg(a.part + j);
            }
            block_excl_sum_shfl<kRT>(x, tot);
            merges = tot >> 32;
            epre = tot & 0xffffffffll;
        }
        for (int64_t q = q0; q < q1; ++q) {
            int32_t *al = a.act + vbase(q);
            const int64_t n = __ldcg(a.alen + q);
            int64_t kept = 0;
            for (int64_t base = 0; base < n; base += (int64_t)kRT * kRV) {
                // thread tid takes kRV consecutive entries, so the block scans
                // keep list order
                int32_t s[kRV], c[kRV];
                bool root[kRV], act[kRV], stay[kRV];
                int64_t fl = 0;                 // (forest edges << 32) | staying roots
                const int64_t jb = base + (int64_t)tid * kRV;
#pragma unroll
                for (int i = 0; i < kRV; ++i) {
                    const bool in = jb + i < n;
                    s[i] = in ? __ldcg(al + jb + i) : 0;
                }
#pragma unroll
                for (int i = 0; i < kRV; ++i) {
                    const bool in = jb + i < n;
                    c[i] = in ? __ldcg(a.color + s[i]) : 0;
                    root[i] = in && c[i] == s[i];
                    act[i] = in && !root[i];
                    // a root stays active only while it has an edge
                    stay[i] = root[i] && __ldcg(a.best + s[i]) != kNone;
                    fl += ((act[i] && MODE == SEL_MST) ? (1ll << 32) : 0ll) | (stay[i] ? 1ll : 0ll);
                }
                int64_t ttot;
                int64_t ex = block_excl_sum_shfl<kRT>(fl, ttot);
                __syncthreads();                // every entry of the tile is read
                int64_t ep = epre + (ex >> 32), kp = kept + (ex & 0xffffffffll);
#pragma unroll
                for (int i = 0; i < kRV; ++i) {
                    if (stay[i]) al[kp++] = s[i];
                    if (act[i] && MODE == SEL_MST) a.mst[nmst + ep++] = __ldcg(a.best + s[i]);
                }
                // new roots of the non-roots: chases interleaved
                for (int64_t guard = 0;; ++guard) {
                    bool any = false;
                    int32_t up[kRV], g[kRV];
#pragma unroll
                    for (int i = 0; i < kRV; ++i) up[i] = act[i] ? __ldcg(a.color + c[i]) : 0;
#pragma unroll
                    for (int i = 0; i < kRV; ++i) {
                        if (act[i] && up[i] == c[i]) {
                            act[i] = false;
                            a.color[s[i]] = c[i];
                            a.parent[s[i]] = c[i];
                        }
                        g[i] = act[i] ? __ldcg(a.color + up[i]) : 0;
                    }
#pragma unroll
                    for (int i = 0; i < kRV; ++i) {
                        if (!act[i]) continue;
                        if (g[i] != up[i]) atomicCAS(a.color + c[i], up[i], g[i]);
                        c[i] = g[i];
                        any = true;
                    }
                    if (!any) break;
                    if (guard > V + 64) {
                        set_err(a.err, DEV_CHASE_LIMIT);
                        break;
                    }
                }
#pragma unroll
                for (int i = 0; i < kRV; ++i)
                    if (stay[i]) a.best[s[i]] = kNone;
                kept += ttot & 0xffffffffll;
                epre += ttot >> 32;
            }
            if (tid == 0) a.alen[q] = (int32_t)kept;
        }
        if (!sync()) break;

        // ---- D: contraction of the segments, in place ---------------------
        for (int64_t q = q0; q < q1; ++q) {
            uint64_t *seg = a.e + ebase(q);
            const int64_t elen = __ldcg(a.seg + q);
            int64_t out = 0;                    // survivors written so far
            for (int64_t base = 0; base < elen; base += kRTile) {
                uint64_t k[kRItems];
#pragma unroll
                for (int it = 0; it < kRItems; ++it) {
                    const int64_t i = base + (int64_t)it * kRT + tid;
                    k[it] = i < elen ? __ldcg(seg + i) : kNone;
                }
                // dead words (self loops left by a CSR load) have a == b
                int32_t ep[2 * kRItems];
                bool ok[kRItems];
#pragma unroll
                for (int it = 0; it < kRItems; ++it) {
                    ok[it] = k[it] != kNone && a.pk.a(k[it]) < (uint64_t)a.V0 &&
                             a.pk.b(k[it]) < (uint64_t)a.V0;
                    ep[2 * it] = ok[it] ? (int32_t)a.pk.a(k[it]) : -1;
                    ep[2 * it + 1] = ok[it] ? (int32_t)a.pk.b(k[it]) : -2;
                }
                find_batch<2 * kRItems>(a.parent, ep, a.err);
                bool keep[kRItems];
                unsigned bal[kRItems];
#pragma unroll
                for (int it = 0; it < kRItems; ++it) {
                    const int32_t su = ep[2 * it], sv = ep[2 * it + 1];
                    keep[it] = ok[it] && su != sv;
                    bal[it] = __ballot_sync(0xffffffffu, keep[it]);
                    if (lane == 0) s_off[it][warp] = __popc(bal[it]);
                    // one word per undirected edge: offered to both ends
                    const uint64_t sel = MODE == SEL_MST
                                             ? (k[it] >> 1)
                                             : (((uint64_t)a.pk.w(k[it]) << 32) | (uint32_t)sv);
                    seg_min_atomic(keep[it], su, sel, a.best);
                    if (keep[it])
                        min_if_lower(&a.best[sv],
                                     MODE == SEL_MST
                                         ? (k[it] >> 1)
                                         : (((uint64_t)a.pk.w(k[it]) << 32) | (uint32_t)su));
                }
                __syncthreads();                // the tile's words are all read
                if (warp == 0) {
                    // exclusive scan of the per-(item, warp) counts in
                    // (item, warp) order
                    constexpr int N = kRItems * kRWarps;
                    constexpr int PER = N / 32;
                    int cc[PER];
                    int sum = 0;
#pragma unroll
                    for (int j = 0; j < PER; ++j) {
                        const int idx = lane * PER + j;
                        cc[j] = s_off[idx / kRWarps][idx % kRWarps];
                        sum += cc[j];
                    }
                    int incl = sum;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const int o = __shfl_up_sync(0xffffffffu, incl, d);
                        if (lane >= d) incl += o;
                    }
                    int r = incl - sum;
#pragma unroll
                    for (int j = 0; j < PER; ++j) {
                        const int idx = lane * PER + j;
                        s_off[idx / kRWarps][idx % kRWarps] = r;
                        r += cc[j];
                    }
                    if (lane == 31) s_base = incl;
                }
                __syncthreads();
                const unsigned lt = (1u << lane) - 1u;
#pragma unroll
                for (int it = 0; it < kRItems; ++it)
                    if (keep[it]) seg[out + s_off[it][warp] + __popc(bal[it] & lt)] = k[it];
                out += s_base;
                __syncthreads();                // s_off and s_base are reused
            }
            if (tid == 0) a.seg[q] = out;
        }
        if (!sync()) break;

        // ---- E: the next round's sizes, the same in every participant ----
        int64_t En = 0, An = 0;
        {
            // the error flag is read beside the counts; the scans' block
            // barriers publish s_err
            const int e_now = tid == 0 ? *(volatile int *)a.err : 0;
            // one scan of (edge words << kActiveBits) | active roots
            int64_t x = 0, tot = 0;
            for (int64_t j = tid; j < Pe; j += kRT)
                x += (__ldcg(a.seg + j) << kActiveBits) + __ldcg(a.alen + j);
            if (tid == 0) s_err = e_now;
            block_excl_sum_shfl<kRT>(x, tot);
            En = tot >> kActiveBits;
            An = tot & (((int64_t)1 << kActiveBits) - 1);
        }
        if (p == 0 && tid == 0 && round < kMaxRounds) {
            a.trace[3 * round] = V;
            a.trace[3 * round + 1] = E;
            a.trace[3 * round + 2] = Aact;
        }
        ++round;
        nmst += MODE == SEL_MST ? merges : 0;
        if (s_err) done = 4;
        else if (En == 0) done = 1;
        else if (merges == 0) done = 2;
        else if (round >= a.max_rounds) done = 3;
        V -= merges;
        E = En;
        Aact = An;
        __syncthreads();                        // s_err is rewritten next round
        if (!done && !solo && An <= kSoloActive && En <= kSoloEdges) {
            // every block decides alike: the others leave, and block 0 moves
            // all active roots and edge words to the front of its own chunk
            // and segment, in participant order (list order = id order is
            // kept).  The participants' counts are read at once and their
            // exclusive prefixes kept in shared memory; the copy then runs
            // over the concatenated elements, kRT at a time, each element
            // finding its participant by binary search.  A destination never
            // passes its source, so each chunk is read before it is written.
            solo = true;
            if (p != 0) return;
            static_assert(2 * kRT >= kMaxTeam, "two participants per thread");
            __shared__ int64_t s_apre[kMaxTeam + 1], s_epre[kMaxTeam + 1];
            {
                const int64_t j0 = 2 * (int64_t)tid;
                const int64_t a0 = j0 < Pe ? (int64_t)__ldcg(a.alen + j0) : 0;
                const int64_t a1 = j0 + 1 < Pe ? (int64_t)__ldcg(a.alen + j0 + 1) : 0;
                const int64_t m0 = j0 < Pe ? __ldcg(a.seg + j0) : 0;
                const int64_t m1 = j0 + 1 < Pe ? __ldcg(a.seg + j0 + 1) : 0;
                int64_t at, mt;
                const int64_t ax = block_excl_sum_shfl<kRT>(a0 + a1, at);
                const int64_t mx = block_excl_sum_shfl<kRT>(m0 + m1, mt);
                if (j0 < Pe) {
                    s_apre[j0] = ax;
                    s_epre[j0] = mx;
                }
                if (j0 + 1 < Pe) {
                    s_apre[j0 + 1] = ax + a0;
                    s_epre[j0 + 1] = mx + m0;
                }
                if (tid == 0) {
                    s_apre[Pe] = at;
                    s_epre[Pe] = mt;
                }
            }
            __syncthreads();
            const int64_t ao = s_apre[Pe], eo = s_epre[Pe];
            // the participant holding concatenated element i: the last q < Pe
            // with pre[q] <= i (pre[0] = 0)
            auto owner = [&](const int64_t *pre, int64_t i) -> int64_t {
                int64_t lo = 0, hi = Pe - 1;
                while (lo < hi) {
                    const int64_t mid = (lo + hi + 1) >> 1;
                    if (pre[mid] <= i) lo = mid;
                    else hi = mid - 1;
                }
                return lo;
            };
            for (int64_t c = 0; c < ao; c += kRT) {
                const int64_t i = c + tid;
                int32_t v = 0;
                if (i < ao) {
                    const int64_t q = owner(s_apre, i);
                    v = __ldcg(a.act + vbase(q) + (i - s_apre[q]));
                }
                __syncthreads();
                if (i < ao) a.act[i] = v;
                __syncthreads();
            }
            for (int64_t c = 0; c < eo; c += kRT) {
                const int64_t i = c + tid;
                uint64_t v = 0;
                if (i < eo) {
                    const int64_t q = owner(s_epre, i);
                    v = __ldcg(a.e + ebase(q) + (i - s_epre[q]));
                }
                __syncthreads();
                if (i < eo) a.e[i] = v;
                __syncthreads();
            }
            if (tid == 0) {
                a.alen[0] = (int32_t)ao;
                a.seg[0] = eo;
            }
            Pe = 1;
            __syncthreads();
        }
    }
    if (p == 0 && tid == 0) {
        a.cnt[C_V] = V;
        a.cnt[C_E] = E;
        a.cnt[C_NMST] = nmst;
        a.cnt[C_ROUNDS] = round;
        a.cnt[C_ROUNDS_ALL] += round;
        a.cnt[C_DONE] = done;
        if (done == 2 || done == 3) set_err(a.err, DEV_CHASE_LIMIT);
    }
}

// Points every original vertex at its root (the next phase's builds and the
// final labels read roots directly).
// With next_best set, it also readies the next weight phase of a queued MST:
// every selection slot empty, the build cursor and the round kernel's barrier
// at zero (the round kernel that precedes it has ended).
__global__ void k_flatten(int32_t *parent, int64_t V0, int *err, unsigned long long *next_best,
                          int64_t *cnt, GridBarrier *bar)
{
    if (next_best && blockIdx.x == 0 && threadIdx.x == 0) {
        cnt[C_CURSOR] = 0;
        bar->count = 0;
    }
    const int64_t stride = (int64_t)gridDim.x * blockDim.x * 4;
    for (int64_t xb = (int64_t)blockIdx.x * blockDim.x * 4 + threadIdx.x; xb < V0; xb += stride) {
        int32_t r[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t v = xb + (int64_t)i * blockDim.x;
            r[i] = v < V0 ? (int32_t)v : -1;
            if (next_best && v < V0) next_best[v] = kNone;
        }
        find_batch<4>(parent, r, err);
    }
}

// Engine state for a new run: no error, the round state, weight histogram
// and barrier at zero, every selection slot empty, and every vertex its own
// root (parent) and its own successor (color; a root that no round visits
// keeps color[s] == s).
__global__ void k_engine_reset(int *err, int64_t *cnt, unsigned long long *hist, GridBarrier *bar,
                               unsigned long long *best, int32_t *parent, int32_t *color,
                               int64_t n)
{
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            *err = 0;
            bar->count = 0;
        }
        for (int i = threadIdx.x; i < C_COUNT; i += blockDim.x) cnt[i] = 0;
        for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0ull;
    }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        best[i] = kNone;
        parent[i] = (int32_t)i;
        color[i] = (int32_t)i;
    }
}

// Sizes of a round-kernel run started from the host (E < 0: the edge words a
// filter kept, cnt[C_AUX0]), and its barrier at zero.
// outer: null, or 256 words to zero.
__global__ void k_set_sizes(int64_t *cnt, int64_t V, int64_t E, GridBarrier *bar,
                            unsigned long long *outer)
{
    if (outer)
        for (int i = threadIdx.x; i < 256; i += blockDim.x) outer[i] = 0ull;
    if (threadIdx.x == 0) {
        cnt[C_V] = V;
        cnt[C_E] = E < 0 ? cnt[C_AUX0] : E;
        bar->count = 0;
    }
}

// Component numbers = rank of the root id among all roots: the reference's
// numbering (its per-round renumbering keeps root order).  flag/pos: V0
// int32 scratch; labels may alias parent.
__global__ void k_root_flags(const int32_t *parent, int64_t V0, int32_t *flag)
{
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < V0;
         x += (int64_t)gridDim.x * blockDim.x)
        flag[x] = parent[x] == (int32_t)x;
}

__global__ void k_rank_roots(const int32_t *parent, const int32_t *pos, int64_t V0,
                             int32_t *labels)
{
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < V0;
         x += (int64_t)gridDim.x * blockDim.x)
        labels[x] = pos[parent[x]];
}

// Round-kernel launch shape.  Test hooks: g_round_cap lowers the rounds a
// phase may run (reaching it is an error, as for the built-in cap), and
// g_round_team forces the number of participants (1 = one block).
static int g_round_cap = 0;
static int g_round_team = 0;
// A host thread may cap the participants of the round kernels it launches
// (set_thread_round_team): the batched path runs many small instances side
// by side, each best served by a single block instead of the whole GPU.
static thread_local int t_round_team_cap = 0;

template <int MODE>
static int round_team_max(int *out)
{
    static int cached = 0;
    if (!cached) {
        int dev = 0, sms = 0, per_sm = 0;
        EACB_CUDA(cudaGetDevice(&dev));
        EACB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        EACB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_rounds<MODE, true>,
                                                                kRT, 0));
        int m = sms * (per_sm > 2 ? 2 : per_sm);
        cached = m < 1 ? 1 : (m > kMaxTeam ? kMaxTeam : m);
    }
    *out = cached;
    return EACB_OK;
}

// Participants for a graph of V0 vertices and about E edge words: one per
// 4096 vertices or 16K edge words, up to the resident maximum.
template <int MODE>
static int round_team(int64_t V0, int64_t E, int kind, int *team)
{
    int mx = 1;
    int s = round_team_max<MODE>(&mx);
    if (s) return s;
    const int64_t work = std::max((V0 + 4095) / 4096, (E + 16383) / 16384);
    int t = g_round_team > 0 ? g_round_team : (int)std::min<int64_t>(work, mx);
    const int64_t cap = g_round_team > 0 ? 0 : tune_get(TUNE_ROUND_TEAM, kind, V0, 0);
    if (cap > 0) t = (int)std::min<int64_t>(t, cap);
    if (t_round_team_cap > 0) t = std::min(t, t_round_team_cap);
    *team = std::max(1, std::min(t, mx));
    return EACB_OK;
}

// MST selection key -> index of its entry in row min(u,v) of a symmetric CSR
// (the smallest index with the key's destination and weight).  A key whose
// build recorded the entry's offset in that row (the word's spare bits) is
// one load of the row start.  Otherwise one thread per key scans the row,
// with the loads of a step in flight together: graph rows are short, and a
// thread per key keeps every key's dependent loads (key -> row extent ->
// entries) overlapping with all the others.
// The number of keys is read on the device (cnt[C_NMST]); after an error of
// an earlier kernel the keys are not complete and none is looked up.
template <typename WT>
__global__ void k_key2eid(const uint64_t *keys, const int64_t *cnt, const int32_t *first,
                          const int32_t *deg, const int32_t *dest, const WT *weight, Pack pk,
                          int32_t *out, int *err)
{
    if (*(volatile int *)err) return;
    const int64_t n_keys = cnt[C_NMST];
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n_keys;
         q += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t s = keys[q];
        const int32_t a = (int32_t)pk.sel_a(s), b = (int32_t)pk.sel_b(s);
        const uint32_t w = pk.sel_w(s);
        const uint64_t off = pk.sel_off(s);
        const int64_t f = first[a];
        if (off != pk.omask) {
            // the build recorded where the entry sits in row a: the first
            // such entry, since a parallel entry of the row with a smaller
            // offset has the smaller selection key
            out[q] = (int32_t)(f + (int64_t)off);
            continue;
        }
        const int64_t d = deg[a];
        int64_t found = -1;
        // the first 16 entries in one batch of loads (most rows of a k-NN
        // graph end there), the rest 8 at a time: a row of 20,000 entries
        // takes 1.23 ms with one loop for both, 1.37 with the number of keys
        // read here, 0.72 with two loops
        auto batch = [&](int64_t e0, auto count) {
            constexpr int N = decltype(count)::value;
            int32_t v[N];
            uint32_t ww[N];
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const bool in = e0 + i < f + d;
                v[i] = in ? __ldg(dest + e0 + i) : -1;
                ww[i] = in ? wword(__ldg(weight + e0 + i)) : 0u;
            }
#pragma unroll
            for (int i = N - 1; i >= 0; --i)
                if (v[i] == b && ww[i] == w) found = e0 + i;
        };
        batch(f, std::integral_constant<int, 16>());
        for (int64_t e0 = f + 16; e0 < f + d && found < 0; e0 += 8)
            batch(e0, std::integral_constant<int, 8>());
        if (found < 0) set_err(err, DEV_BAD_INPUT);   // graph not symmetric
        out[q] = (int32_t)found;
    }
}

// Adds to outer, per weight, those of kOuterSample entries, evenly spread, that
// join two components; nothing with more than vmax components, or one.
__global__ void __launch_bounds__(256)
k_outer_sample(const int64_t *indptr, const int32_t *indices, const uint8_t *w, int32_t n, int64_t nnz,
               const int32_t *label, const int64_t *cnt, int64_t vmax, unsigned long long *outer)
{
    __shared__ unsigned s_h[256];
    if (cnt[C_V] > vmax || cnt[C_V] <= 1) return;
    s_h[threadIdx.x] = 0u;
    __syncthreads();
    const int t = blockIdx.x * 256 + threadIdx.x;
    const int64_t e = nnz / kOuterSample * t + nnz % kOuterSample * t / kOuterSample;
    int a = 0, b = n;                              // indptr[a] <= e < indptr[b]
    while (b - a > 1) {
        const int m = a + (b - a) / 2;
        if (indptr[m] <= e) a = m; else b = m;
    }
    const int32_t j = indices[e];
    if (j >= 0 && j < n && label[a] != label[j]) atomicAdd(&s_h[w[e]], 1u);
    __syncthreads();
    if (s_h[threadIdx.x]) atomicAdd(&outer[threadIdx.x], (unsigned long long)s_h[threadIdx.x]);
}

// Every column of an upper-triangle CSR (16-byte aligned): i < j < n in row i.
// A warp per row; HBM-bound, 4 bytes per entry.
__global__ void __launch_bounds__(kPhThreads)
k_check_columns(const int64_t *indptr, const int32_t *indices, int32_t n, int64_t nnz, int *err)
{
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = (int64_t)gridDim.x * kPhWarps;
    bool bad = false;
    for (int64_t i = (int64_t)blockIdx.x * kPhWarps + (threadIdx.x >> 5); i < n; i += nwarps) {
        const int64_t s = indptr[i], e = indptr[i + 1];
        if (s < 0 || e < s || e > nnz) {
            bad = true;
            continue;
        }
        const uint32_t span = (uint32_t)(n - 1 - (int32_t)i);
        auto off = [&](int32_t j) { return (uint32_t)(j - (int32_t)i - 1) >= span; };
        const int64_t v0 = (s + 3) >> 2, v1 = e >> 2;          // whole vectors
        if (v0 > v1) {
            for (int64_t t = s + lane; t < e; t += 32) bad = bad || off(indices[t]);
            continue;
        }
        if (s + lane < 4 * v0) bad = bad || off(indices[s + lane]);
        if (4 * v1 + lane < e) bad = bad || off(indices[4 * v1 + lane]);
        const int4 *v = reinterpret_cast<const int4 *>(indices);
        constexpr int U = 4;
        for (int64_t t = v0 + lane; t < v1; t += 32 * U) {
            int4 x[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                x[u] = t + 32 * u < v1 ? __ldcs(v + t + 32 * u) : __ldcs(v + t);
#pragma unroll
            for (int u = 0; u < U; ++u)
                bad = bad || off(x[u].x) || off(x[u].y) || off(x[u].z) || off(x[u].w);
        }
    }
    if (bad) set_err(err, DEV_BAD_INPUT);
}

// ---------------------------------------------------------------------------
// Host-side engine
// ---------------------------------------------------------------------------
struct Engine {
    int *err;
    int64_t *cnt;             // round state (C_*)
    uint64_t *ea;             // edge words: phase builds write them, the rounds compact them
    int32_t *label;           // union-find parent; after each phase every vertex's root
    unsigned long long *best;
    int32_t *color, *flag, *pos, *act;
    uint64_t *mst;
    unsigned long long *hist; // 256 weight buckets
    unsigned long long *outer; // and those of sampled entries between components
    int *lohi;                // the device phase plan (k_phase_plan)
    int32_t *giant;           // root whose rows a later phase skips (k_pick_giant)
    int32_t *part;            // per-participant counts of the round kernel
    int32_t *alen;            // per-participant active roots
    int64_t *seg;             // per-participant surviving edge words
    int64_t *trace;
    GridBarrier *bar;
    ScanScratch scan;
    int32_t V0;
    int64_t Emax;
    int kind = 0;             // 0 graph MST/CC, 1 EAC final clustering (tuning shape)

    static Engine carve(Carver &c, int32_t V0, int64_t Emax)
    {
        Engine g;
        // the error word and the counts, read by the host in one copy (with
        // the sampled weights where they are wanted)
        g.err = (int *)c.take<int64_t>(1 + C_COUNT + 256);
        g.cnt = (int64_t *)g.err + 1;
        g.outer = (unsigned long long *)(g.cnt + C_COUNT);
        g.hist = c.take<unsigned long long>(256);
        g.lohi = c.take<int>(2 * kPhaseSlots);
        g.giant = c.take<int32_t>(1);
        g.bar = c.take<GridBarrier>(1);
        g.seg = c.take<int64_t>(kMaxTeam);
        g.trace = c.take<int64_t>(3 * kMaxRounds);
        g.part = c.take<int32_t>(2 * kMaxTeam);
        g.alen = c.take<int32_t>(kMaxTeam);
        g.V0 = V0;
        // the edge words (compacted in place by the rounds); they also hold
        // the two directions of a forest (at most 2 V0 words)
        g.Emax = std::max<int64_t>(Emax, 2 * (int64_t)V0);
        g.ea = c.take<uint64_t>(g.Emax);
        g.label = c.take<int32_t>(V0);
        g.best = c.take<unsigned long long>(V0);
        g.color = c.take<int32_t>(V0);
        g.flag = c.take<int32_t>(V0);
        g.pos = c.take<int32_t>(V0);
        g.act = c.take<int32_t>(V0);
        g.mst = c.take<uint64_t>(V0);
        g.scan = ScanScratch::carve(c, g.Emax, g.err);
        return g;
    }

    // (oh: null, or receives outer as well)
    int read_counts(cudaStream_t st, int64_t h[C_COUNT], unsigned long long *oh = nullptr)
    {
        int64_t both[1 + C_COUNT + 256];
        EACB_CUDA(cudaMemcpyAsync(both, err, (1 + C_COUNT + (oh ? 256 : 0)) * sizeof(int64_t),
                                  cudaMemcpyDeviceToHost, st));
        EACB_CUDA(cudaStreamSynchronize(st));
        std::copy(both + 1, both + 1 + C_COUNT, h);
        if (oh) std::copy(both + 1 + C_COUNT, both + 1 + C_COUNT + 256, oh);
        int e;
        memcpy(&e, both, sizeof(e));
        return dev_err_to_status(e);
    }

    int read_hist(cudaStream_t st, unsigned long long h[256])
    {
        EACB_CUDA(cudaMemcpyAsync(h, hist, 256 * sizeof(unsigned long long),
                                  cudaMemcpyDeviceToHost, st));
        EACB_CUDA(cudaStreamSynchronize(st));
        return EACB_OK;
    }

    int reset(cudaStream_t st)
    {
        k_engine_reset<<<grid_for(V0, 256), 256, 0, st>>>(err, cnt, hist, bar, best, label, color,
                                                         V0);
        EACB_CHECK_LAUNCH();
        return EACB_OK;
    }

    // Runs the rounds of one phase: input edges in ea (cnt[C_E] of them, or
    // cnt[C_CURSOR] with from_cursor), supervertices [0, cnt[C_V]) (V0 with
    // first_phase) with their selection in best; the barrier is at zero (the
    // reset, k_set_sizes or the previous phase's k_flatten cleared it).  One
    // launch; with profiling on it is timed, and its algorithmic bytes come
    // from the per-round sizes the kernel records.  With next_phase set, the
    // flattening after it readies the next queued phase.
    template <int MODE>
    int rounds(Pack pk, cudaStream_t st, int64_t e_hint, int from_cursor = 0,
               int first_phase = 0, bool next_phase = false)
    {
        int team = 1;
        int s = round_team<MODE>(V0, e_hint, kind, &team);
        if (s) return s;
        RoundArgs a;
        a.pk = pk;
        a.V0 = V0;
        a.e = ea;
        a.parent = label;
        a.best = best;
        a.color = color;
        a.act = act;
        a.mst = mst;
        a.part = part;
        a.alen = alen;
        a.seg = seg;
        a.cnt = cnt;
        a.trace = trace;
        a.bar = bar;
        a.err = err;
        a.max_rounds = g_round_cap > 0 ? std::min(g_round_cap, kMaxRounds) : kMaxRounds;
        a.from_cursor = from_cursor;
        a.first_phase = first_phase;
        ProfScope ps(PROF_ROUNDS, st);
        if (team == 1) {
            k_rounds<MODE, false><<<1, kRT, 0, st>>>(a);
            EACB_CHECK_LAUNCH();
        } else {
            void *args[] = {(void *)&a};
            EACB_CUDA(cudaLaunchCooperativeKernel((const void *)k_rounds<MODE, true>, dim3(team),
                                                  dim3(kRT), args, 0, st));
            count_launch();
        }
        if (ps.on) {
            // per round: each edge word read and (if it survives) written
            // back, 8 B each, with its two endpoints' parents (8 B); per
            // active root its list entry, selection slot, successor and
            // parent (20 B)
            int64_t h[C_COUNT], tr[3 * kMaxRounds];
            EACB_CUDA(cudaMemcpyAsync(h, cnt, sizeof(h), cudaMemcpyDeviceToHost, st));
            EACB_CUDA(cudaMemcpyAsync(tr, trace, sizeof(tr), cudaMemcpyDeviceToHost, st));
            EACB_CUDA(cudaStreamSynchronize(st));
            double bytes = 0.0;
            const int64_t nr = std::min<int64_t>(h[C_ROUNDS], kMaxRounds);
            for (int64_t r = 0; r < nr; ++r) {
                const double En = r + 1 < nr ? (double)tr[3 * r + 4] : (double)h[C_E];
                bytes += 16.0 * (double)tr[3 * r + 1] + 8.0 * En + 20.0 * (double)tr[3 * r + 2];
            }
            ps.done(bytes);
        }
        // every vertex to its root, for the next phase's builds and the labels
        k_flatten<<<grid_for(V0, 256 * 4, 148 * 8), 256, 0, st>>>(
            label, V0, err, next_phase ? best : nullptr, cnt, bar);
        EACB_CHECK_LAUNCH();
        return EACB_OK;
    }

    // MST by weight phases (see k_phase_csr), all queued back to back with no
    // host read in between, right after reset(): build(ph) appends a phase's
    // edges to ea through cnt[C_CURSOR] with their selection in best; the
    // round kernel takes its edge count from the cursor, and the flattening
    // after it clears the slots, the cursor and the barrier for the next
    // phase.  Nothing is read: the forest size and any error stay on the
    // device.
    template <typename Build>
    int run_phased(Pack pk, const std::vector<Phase> &plan, Build build, cudaStream_t st)
    {
        for (size_t q = 0; q < plan.size(); ++q) {
            Phase ph = plan[q];
            ph.ident = q == 0;                 // no round has merged anything yet
            int s = build(ph);
            if (s) return s;
            if ((s = rounds<SEL_MST>(pk, st, Emax, 1, q == 0 ? 1 : 0, q + 1 < plan.size())))
                return s;
        }
        return EACB_OK;
    }

    // Phases in order with a host read after each build (the final
    // clustering): the edge array holds a phase's usual output, and a phase
    // whose kept entries overflow it is discarded and redone as the pieces
    // split() cuts from the build's per-weight kept counts, in order.  From
    // at most pair_max components on, one phase takes the rest by pairs of
    // components -- unless that phase would see many entries between
    // components, which it is slow on (11 ps each against 1.6 for an entry
    // inside one).  Then the next phase ends where some 16 of them per point
    // are lighter, which usually join the components; sample() queues the
    // estimate of their weights (outer), and check() looks at the columns that
    // no phase reads then.  (Blocks of equal size, entries
    // between all: 11,600 points, 300 blocks 1.87 -> 0.66 ms, 2 blocks 1.02 ->
    // 0.84; 5,000 points, 100 blocks 0.73 -> 0.52; 30,000 points, 100 blocks 4.6
    // -> 1.4; 0.88, 1.82, 0.67 and 5.8 with ordinary phases alone.)
    template <typename Build, typename Split, typename Sample, typename Check>
    int run_phased_retry(Pack pk, std::vector<Phase> plan, Build build, Split split, Sample sample,
                         Check check, int64_t nnz, int64_t pair_max, cudaStream_t st)
    {
        int64_t V = V0, n_mst = 0;
        size_t q = 0;
        bool merged = false;
        int narrow = 0;
        while (q < plan.size()) {
            Phase ph = plan[q];
            ph.ident = !merged;                // no round has merged anything yet
            EACB_CUDA(cudaMemsetAsync(best, 0xff, sizeof(uint64_t) * V, st));
            EACB_CUDA(cudaMemsetAsync(&cnt[C_CURSOR], 0, sizeof(int64_t), st));
            EACB_CUDA(cudaMemsetAsync(hist, 0, 256 * sizeof(unsigned long long), st));
            int s = build(ph);
            if (s) return s;
            int64_t h[C_COUNT];
            const int e = read_counts(st, h);
            const int64_t Ep = h[C_CURSOR];
            if (e == dev_err_to_status(DEV_CAPACITY)) {
                // the build still counted every kept entry, per weight, in
                // hist: the pieces are cut from those counts
                unsigned long long kh[256];
                EACB_CUDA(cudaMemcpyAsync(kh, hist, sizeof(kh), cudaMemcpyDeviceToHost, st));
                EACB_CUDA(cudaStreamSynchronize(st));
                std::vector<Phase> pieces;
                if ((s = split(ph, kh, pieces))) return s;
                EACB_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
                plan.erase(plan.begin() + (ptrdiff_t)q);
                plan.insert(plan.begin() + (ptrdiff_t)q, pieces.begin(), pieces.end());
                continue;
            }
            if (e) return e;
            if (Ep > Emax) return EACB_ERR_INTERNAL;
            if (prof().enabled) prof().bytes[PROF_PHASE] += 8.0 * (double)Ep;   // words written
            int64_t nc = 0;
            unsigned long long oh[256];
            const bool ask = pair_max && q + 1 < plan.size() && narrow < kPairNarrow;
            if ((s = run<SEL_MST>(pk, Ep, V, st, &n_mst, &nc, sample, ask ? oh : nullptr))) return s;
            merged = merged || nc < V;
            V = nc;
            ++q;
            if (V <= 1) return narrow && q < plan.size() ? check() : EACB_OK;
            // Few components left: the rest of the weights in one phase.
            // Each phase walks the whole matrix, and once the components are
            // few most entries join a component to itself, so the remaining
            // phases would keep few words each; a merged phase that does
            // overflow the edge array is redone in pieces like any other.
            if (q == plan.size()) break;
            bool full = true;
            for (size_t r = q; r < plan.size(); ++r)
                full = full && plan[r].r0 == 0 && plan[r].r1 == V0;
            if (!full) continue;
            const int lo = plan[q].lo, hi = plan.back().hi;
            const bool pairs = V <= pair_max && 2 * V * V <= Emax;
            int cut = hi;
            if (pairs && ask) {
                const double each = (double)nnz / kOuterSample;
                double all = 0.0, light = 0.0;
                for (int w = lo + 1; w <= hi; ++w) all += each * (double)oh[w];
                if (all > (double)(kPairOuter + nnz / kPairOuterShare)) {
                    for (cut = lo; cut < hi && light < 16.0 * (double)V0;)
                        light += each * (double)oh[++cut];
                    if (light > 0.5 * (double)Emax) cut = hi;      // (not to be redone in pieces)
                }
            }
            if (cut < hi) {
                ++narrow;
                plan.resize(q);
                plan.push_back(Phase{lo, cut, 0, V0, -1, 0});
                plan.push_back(Phase{cut, hi, 0, V0, -1, 0});
            } else if (pairs || (q + 1 < plan.size() && V * kMergeBelow <= V0)) {
                plan.resize(q);
                plan.push_back(Phase{lo, hi, 0, V0, -1, 0, pairs ? (int)V : 0});
            }
        }
        return EACB_OK;
    }

    template <int MODE, typename Src>
    int filter(const Src &src, int64_t n_in, uint64_t *out, cudaStream_t st)
    {
        if (n_in == 0) {
            EACB_CUDA(cudaMemsetAsync(&cnt[C_AUX0], 0, sizeof(int64_t), st));
            return EACB_OK;
        }
        const int64_t ntiles = (n_in + kETile - 1) / kETile;
        if (ntiles > scan.max_tiles) return EACB_ERR_WORKSPACE;
        EACB_CUDA(scan.clear(ntiles, false, st));
        k_edge_tile<MODE, Src><<<(unsigned)ntiles, kET, 0, st>>>(
            src, n_in, out, best, scan.status, scan.counter, &cnt[C_AUX0], err);
        EACB_CHECK_LAUNCH();
        return EACB_OK;
    }

    // Rounds from E0 edge words in ea (selection already in best) over
    // supervertices [0, V_start).  On return: label = component of every
    // vertex, *n_comp_out = number of components, *n_mst_total = forest
    // edges emitted since the engine's reset.  With oh set, sample() is queued
    // behind the rounds and its counts by weight are read with the others.
    template <int MODE, typename Sample>
    int run(Pack pk, int64_t E0, int64_t V_start, cudaStream_t st, int64_t *n_mst_total,
            int64_t *n_comp_out, Sample sample, unsigned long long *oh)
    {
        k_set_sizes<<<1, 32, 0, st>>>(cnt, V_start, E0, bar, oh ? outer : nullptr);
        EACB_CHECK_LAUNCH();
        int s = rounds<MODE>(pk, st, E0);
        if (s) return s;
        if (oh && (s = sample())) return s;
        int64_t h[C_COUNT];
        if ((s = read_counts(st, h, oh))) return s;
        if (h[C_DONE] != 1) return EACB_ERR_NOT_CONVERGED;
        *n_mst_total = h[C_NMST];
        *n_comp_out = h[C_V];
        return EACB_OK;
    }
};

template <typename WT>
static int csr_graph_run(int mode, const int32_t *dest, const WT *weight, int wbits,
                         const int32_t *first, const int32_t *deg, int32_t V, int64_t E,
                         int32_t *mst_out, int64_t *host_n_mst, int32_t *labels_out,
                         int64_t *host_n_comp, void *ws, size_t ws_bytes, cudaStream_t st)
{
    Pack pk;
    int s = make_pack(V, wbits, pk, mode == SEL_MST);
    if (s) return s;
    Carver c(ws, ws_bytes);
    Engine g = Engine::carve(c, V, E);
    if (c.overflow) return EACB_ERR_WORKSPACE;
    if ((s = g.reset(st))) return s;
    int64_t h[C_COUNT];
    const unsigned gr = grid_for((int64_t)V * 32, 256);
    const unsigned gph = grid_for(V, kPhThreads, 148 * 4);   // phase builds: grid-stride rows
    if (mode == SEL_MST) {
        // weight phases over the bucket histogram of the entries (the reset
        // cleared it)
        if (E > 0) {
            if (sizeof(WT) == 1) {
                if ((s = launch_whist_u8((const uint8_t *)weight, E, g.hist, st))) return s;
            } else {
                k_whist_csr<WT><<<grid_for(E, kHistThreads, 148 * 8), kHistThreads, 0, st>>>(
                    weight, E, wbits, g.hist);
            }
            EACB_CHECK_LAUNCH();
        }
        // the phase plan stays on the device: the whole MST is queued without
        // a host read until its end
        const int p1 = (int)std::min<int64_t>(999, std::max<int64_t>(
                           1, tune_get(TUNE_MST_PHASE1, 0, V, 250)));
        k_phase_plan<<<1, 256, 0, st>>>(g.hist, g.lohi, p1);
        EACB_CHECK_LAUNCH();
        std::vector<Phase> plan;
        for (int q = 0; q < kPhaseSlots; ++q) plan.push_back(Phase{0, 0, 0, V, q});
        // a phase holds a subset of the E entries: the edge array always fits.
        // The first phase reads every row with identity labels; the later one
        // skips the rows of the giant component the first phase built
        auto build = [&](const Phase &ph) -> int {
            if (E == 0) return EACB_OK;
            if (ph.slot > 0) {
                k_pick_giant<<<1, 1024, 0, st>>>(g.label, V, g.giant);
                EACB_CHECK_LAUNCH();
            }
            ProfScope ps(PROF_PHASE, st);
            // the first phase reads every row and needs many warps to keep
            // its loads in flight; the skipping phase touches few rows
            // the kept-entry records (dynamic) on top of the static staging pass 48 KB
            EACB_CUDA((allow_max_dyn_smem(k_phase_csr<SEL_MST, WT>)));
            k_phase_csr<SEL_MST, WT><<<ph.slot == 0 ? gr : gph, kPhThreads, kPhRecBytes, st>>>(
                first, deg, dest, weight, V, E, wbits, 0, 0, g.lohi, ph.slot, ph.slot == 0 ? 1 : 0,
                ph.slot > 0 ? g.giant : nullptr, g.label, pk, g.ea,
                (unsigned long long *)&g.cnt[C_CURSOR], (unsigned long long)g.Emax, g.best,
                ph.slot == 0 ? (unsigned long long *)&g.cnt[C_SYM_LT] : nullptr, g.err);
            EACB_CHECK_LAUNCH();
            // compulsory reads: row extents and labels (12 B per row), dest and
            // weight (4 + sizeof(WT) B per entry); the written words follow
            ps.done(12.0 * V + (4.0 + sizeof(WT)) * (double)E);
            return EACB_OK;
        };
        if ((s = g.run_phased(pk, plan, build, st))) return s;
        if (V > 1) {
            k_key2eid<WT><<<grid_for(V - 1, 256), 256, 0, st>>>(g.mst, g.cnt, first, deg, dest,
                                                                  weight, pk, mst_out, g.err);
            EACB_CHECK_LAUNCH();
        }
        if ((s = g.read_counts(st, h))) return s;
        if (h[C_SYM_LT] != h[C_SYM_GT]) return EACB_ERR_BAD_INPUT;   // not symmetric
        *host_n_mst = h[C_NMST];
    } else {
        // every entry with identity labels: one word per undirected edge and
        // each vertex's first selection (the reference's round one)
        if (E > 0) {
            EACB_CUDA((allow_max_dyn_smem(k_phase_csr<SEL_CC, WT>)));
            k_phase_csr<SEL_CC, WT><<<gr, kPhThreads, kPhRecBytes, st>>>(
                first, deg, dest, weight, V, E, wbits, -1, 255, nullptr, 0, 1, nullptr, g.label, pk,
                g.ea, (unsigned long long *)&g.cnt[C_CURSOR], (unsigned long long)g.Emax, g.best,
                (unsigned long long *)&g.cnt[C_SYM_LT], g.err);
            EACB_CHECK_LAUNCH();
        }
        // the rounds take the words' count from the build's cursor (one word
        // per undirected edge); everything is queued up to one read
        if ((s = g.rounds<SEL_CC>(pk, st, E / 2, 1, 1))) return s;
        // the reference's component numbers: ranks of the root ids
        const unsigned gv = grid_for(V, 256);
        k_root_flags<<<gv, 256, 0, st>>>(g.label, V, g.flag);
        EACB_CHECK_LAUNCH();
        if ((s = scan_launch<int32_t, int32_t>(g.flag, g.pos, V, 0, &g.cnt[C_AUX1], g.scan, st)))
            return s;
        k_rank_roots<<<gv, 256, 0, st>>>(g.label, g.pos, V, labels_out);
        EACB_CHECK_LAUNCH();
        if ((s = g.read_counts(st, h))) return s;
        if (h[C_SYM_LT] != h[C_SYM_GT]) return EACB_ERR_BAD_INPUT;   // not symmetric
        if (h[C_DONE] != 1) return EACB_ERR_NOT_CONVERGED;
        if (h[C_AUX1] != h[C_V]) return EACB_ERR_INTERNAL;
        *host_n_comp = h[C_V];
    }
    return EACB_OK;
}

static int csr_dispatch(int mode, const int32_t *dest, const void *weight, int dt,
                        const int32_t *first, const int32_t *deg, int32_t V, int64_t E,
                        int32_t *mst_out, int64_t *host_n_mst, int32_t *labels,
                        int64_t *host_n_comp, void *ws, size_t ws_bytes, uintptr_t stream)
{
    if (V <= 0 || E < 0 || !first || !deg || (E > 0 && (!dest || !weight)) || !ws)
        return EACB_ERR_BAD_ARGUMENT;
    cudaStream_t st = as_stream(stream);
    const int wb = dtype_bits(dt);
    switch (dt) {
    case EACB_U8:
        return csr_graph_run<uint8_t>(mode, dest, (const uint8_t *)weight, wb, first, deg, V, E,
                                      mst_out, host_n_mst, labels, host_n_comp, ws, ws_bytes, st);
    case EACB_U16:
        return csr_graph_run<uint16_t>(mode, dest, (const uint16_t *)weight, wb, first, deg, V, E,
                                       mst_out, host_n_mst, labels, host_n_comp, ws, ws_bytes, st);
    case EACB_I32:
        return csr_graph_run<int32_t>(mode, dest, (const int32_t *)weight, wb, first, deg, V, E,
                                      mst_out, host_n_mst, labels, host_n_comp, ws, ws_bytes, st);
    case EACB_U32:
        return csr_graph_run<uint32_t>(mode, dest, (const uint32_t *)weight, wb, first, deg, V, E,
                                       mst_out, host_n_mst, labels, host_n_comp, ws, ws_bytes, st);
    case EACB_F32:
        return csr_graph_run<float>(mode, dest, (const float *)weight, wb, first, deg, V, E,
                                    mst_out, host_n_mst, labels, host_n_comp, ws, ws_bytes, st);
    default:
        return EACB_ERR_BAD_ARGUMENT;
    }
}

// ---------------------------------------------------------------------------
// Final clustering helpers
// ---------------------------------------------------------------------------
__global__ void k_weight_hist(const uint64_t *keys, const int64_t *cnt, Pack pk, int64_t *hist)
{
    const int64_t n = cnt[C_NMST];
    __shared__ int64_t h[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        atomicAdd((unsigned long long *)&h[pk.sel_w(keys[i]) & 255], 1ull);
    __syncthreads();
    for (int i = threadIdx.x; i < 256; i += blockDim.x)
        if (h[i]) atomicAdd((unsigned long long *)&hist[i], (unsigned long long)h[i]);
}

struct CutPlan {
    int64_t status;      // 0 ok, else an eacb status
    int64_t n_clusters;  // nc_stable
    int64_t wmax;        // keep forest edges with weight <= wmax (-1: none)
    int64_t need_labels;
};

// The lifetime rule of MyML/MyML/EAC/eac.py:366-391 and the cut decision of
// :220-265, evaluated on the 256-bin histogram of the uint8 MST weights
// (sorted weights are the bins expanded in order).
// (d_n_mst: the number of weights on the device, or null: n_mst)
__global__ void k_cut_plan(const int64_t *hist, int64_t n_mst, const int64_t *d_n_mst, int32_t n,
                           int32_t max_dist, int32_t n_clusters, CutPlan *plan)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    if (d_n_mst) n_mst = *d_n_mst;
    CutPlan p{0, 0, 255, 0};
    const int64_t n_disc = (int64_t)n - n_mst;
    int64_t nc;
    int64_t thr = 255;
    if (n_clusters == 0) {
        if (n_mst < 2) { p.status = EACB_ERR_VALUE; *plan = p; return; }
        // lifetimes = differences of consecutive sorted weights; zero ones
        // exist iff some bin holds two or more edges
        bool has_zero = false;
        int prev = -1, wlast = 0;
        int best_gap = 0, m_w = -1;
        for (int b = 0; b < 256; ++b) {
            int64_t c = hist[b];
            if (!c) continue;
            if (c >= 2) has_zero = true;
            if (prev >= 0 && b - prev > best_gap) { best_gap = b - prev; m_w = prev; }
            prev = b;
            wlast = b;
        }
        if (!has_zero) { p.status = EACB_ERR_VALUE; *plan = p; return; }
        int first_w = -1;
        for (int b = 0; b < 256; ++b) if (hist[b]) { first_w = b; break; }
        if (m_w < 0) m_w = first_w;          // all lifetimes zero: argmax = 0
        int64_t above = 0;
        for (int b = m_w + 1; b < 256; ++b) above += hist[b];
        int64_t cont = above == 0 ? 1 : above + 1;
        // th < 2 * min(zero lifetimes) never holds once a zero lifetime exists
        if (n_disc > 1) {
            int64_t disc_life = (int64_t)max_dist + 1 + 1 - wlast;
            if ((int64_t)best_gap > disc_life) cont += n_disc - 1;
            else cont = n_disc;
        }
        nc = cont;
        thr = m_w;    // the cut removes exactly the edges heavier than w[m]
    } else {
        nc = n_clusters;
        if (nc > n_disc) {
            // cut the (nc - n_disc) heaviest forest edges; supported when that
            // boundary falls between two weight bins (no tie to split)
            const int64_t n_cuts = nc - n_disc;
            int64_t acc = 0;
            thr = 255;
            for (int b = 255; b >= 0 && acc < n_cuts; --b) {
                if (acc + hist[b] > n_cuts) { p.status = EACB_ERR_UNSUPPORTED; *plan = p; return; }
                acc += hist[b];
                thr = b - 1;
            }
        }
    }
    p.n_clusters = nc;
    p.wmax = (nc > n_disc) ? thr : 255;
    p.need_labels = nc > 1;
    *plan = p;
}

__global__ void k_comp_min(const int32_t *label, int32_t n, int32_t *cmin)
{
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n;
         x += (int64_t)gridDim.x * blockDim.x)
        atomicMin(&cmin[label[x]], (int32_t)x);
}

__global__ void k_first_flag(const int32_t *label, const int32_t *cmin, int32_t n, int32_t *flag)
{
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n;
         x += (int64_t)gridDim.x * blockDim.x)
        flag[x] = cmin[label[x]] == (int32_t)x;
}

__global__ void k_canon(const int32_t *label, const int32_t *cmin, const int32_t *pos, int32_t n,
                        int32_t *out)
{
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n;
         x += (int64_t)gridDim.x * blockDim.x)
        out[x] = pos[cmin[label[x]]];
}

}  // namespace eacb

using namespace eacb;

// Test hooks of the Boruvka round kernel (see k_rounds): the rounds a phase
// may run (0 = the built-in cap; reaching a lower cap is reported as
// EACB_ERR_NOT_CONVERGED, like the built-in one) and its participants
// (0 = automatic, 1 = one block, more = that many cooperative blocks, at
// most the resident maximum).  Process-wide; set them only between calls.
namespace eacb {
void set_thread_round_team(int blocks) { t_round_team_cap = blocks > 0 ? blocks : 0; }
}  // namespace eacb

extern "C" void eacb_debug_set_round_cap(int rounds) { g_round_cap = rounds > 0 ? rounds : 0; }
extern "C" void eacb_debug_set_round_team(int blocks) { g_round_team = blocks > 0 ? blocks : 0; }

extern "C" size_t eacb_boruvka_workspace_size(int32_t n_vertices, int64_t n_edges)
{
    Carver c(nullptr, 0);
    Engine::carve(c, n_vertices, n_edges);
    return c.off;
}

extern "C" int eacb_boruvka_mst(const int32_t *dest, const void *weight, int weight_dtype,
                                const int32_t *first_edge, const int32_t *out_degree,
                                int32_t n_vertices, int64_t n_edges, int32_t *mst_out,
                                int64_t *host_n_mst, void *ws, size_t ws_bytes, uintptr_t stream)
{
    if (!host_n_mst || (!mst_out && n_vertices > 1)) return EACB_ERR_BAD_ARGUMENT;
    int64_t dummy = 0;
    return csr_dispatch(SEL_MST, dest, weight, weight_dtype, first_edge, out_degree, n_vertices,
                        n_edges, mst_out, host_n_mst, nullptr, &dummy, ws, ws_bytes, stream);
}

extern "C" int eacb_connected_components(const int32_t *dest, const void *weight,
                                         int weight_dtype, const int32_t *first_edge,
                                         const int32_t *out_degree, int32_t n_vertices,
                                         int64_t n_edges, int32_t *labels, int64_t *host_n_comps,
                                         void *ws, size_t ws_bytes, uintptr_t stream)
{
    if (!labels || !host_n_comps) return EACB_ERR_BAD_ARGUMENT;
    int64_t dummy = 0;
    return csr_dispatch(SEL_CC, dest, weight, weight_dtype, first_edge, out_degree, n_vertices,
                        n_edges, nullptr, &dummy, labels, host_n_comps, ws, ws_bytes, stream);
}

// Matrices of up to this many entries get an edge word for every entry, so
// no phase can overflow and all phases are queued with no host read between
// them (the many small matrices of batched EAC); larger ones keep the
// bounded edge array below and may redo an overflowing phase in pieces.
constexpr int64_t kFinalQueuedEntries = (int64_t)1 << 26;

// The phases of such a larger matrix are planned from an eighth of its
// weights (8M or more), spread evenly: the plan only chooses where the phases
// end.  (920M entries: 355 us for all the weights, 53 for the sample.)
constexpr int kWhistSkip = 8;

// Edge words of the final clustering (one per kept entry): every entry when
// the matrix is small, else 256 words per point (at least 2^20): room for
// the usual output of a phase, not its worst case (a phase that overflows is
// redone in pieces), so a matrix of thousands of entries per row does not
// need an edge array of its own size.
static int64_t final_edge_cap(int32_t n, int64_t nnz)
{
    const int64_t all = nnz > (int64_t)n ? nnz : (int64_t)n;
    if (all <= kFinalQueuedEntries) return all;       // nothing can overflow
    const int64_t usual = 256 * (int64_t)n > ((int64_t)1 << 20) ? 256 * (int64_t)n : ((int64_t)1 << 20);
    return all < usual ? all : usual;
}

// Phases of the final clustering, lightest weights first: the weight ranges
// whose cumulative entry counts reach 8n, 32n, 128n, 512n, 2048n and all
// entries.  A co-association matrix holds thousands of entries per row, and
// the lightest few per point already join most points: later phases keep
// only entries between different components, so they write few edges, and a
// phase over a narrow range reads little more than the weights.
//
// h may be of a sample of the entries: every weight lies in some range, and
// which one changes the phases' sizes only.
static void plan_final_phases(const unsigned long long h[256], int32_t n, int64_t nnz,
                              std::vector<Phase> &plan)
{
    const double t = nnz ? (double)nnz : 1.0;
    double fracs[6];
    for (int f = 0; f < 5; ++f) fracs[f] = std::min(1.0, (double)(8 << (2 * f)) * n / t);
    fracs[5] = 1.0;
    int lo[8], hi[8];
    const int np = phase_ranges(h, fracs, 6, lo, hi);
    for (int q = 0; q < np; ++q) plan.push_back(Phase{lo[q], hi[q], 0, n, -1});
}

// Pieces of a phase whose kept entries did not fit the edge array, from the
// kept entries per weight that its build counted (kh; upper bounds for the
// pieces, whose components only merge): consecutive weights while their
// kept entries fit, and a weight that alone does not fit split into row
// ranges of equal entry counts (the order (w, a, b) keeps a row range of one
// weight contiguous).  Host row pointers are fetched on the first row split.
static int split_final_phase(const Phase &ph, const unsigned long long kh[256], int64_t cap_entries,
                             const int64_t *d_indptr, int32_t n, std::vector<int64_t> &ip,
                             cudaStream_t st, std::vector<Phase> &out)
{
    const unsigned long long cap = (unsigned long long)(cap_entries / 8 * 7);
    if (ph.r0 != 0 || ph.r1 != n) {
        // a row range of one weight: halve the rows
        if (ph.r1 - ph.r0 < 2) return EACB_ERR_INTERNAL;
        const int64_t m = ph.r0 + (ph.r1 - ph.r0) / 2;
        out.push_back(Phase{ph.lo, ph.hi, ph.r0, m, -1});
        out.push_back(Phase{ph.lo, ph.hi, m, ph.r1, -1});
        return EACB_OK;
    }
    int start = ph.lo;
    unsigned long long acc = 0;
    for (int w = ph.lo + 1; w <= ph.hi; ++w) {
        if (kh[w] <= cap && acc + kh[w] <= cap) {
            acc += kh[w];
            continue;
        }
        if (w - 1 > start) out.push_back(Phase{start, w - 1, 0, n, -1});
        if (kh[w] <= cap) {                    // w opens the next piece
            start = w - 1;
            acc = kh[w];
            continue;
        }
        // weight w alone: rows in pieces of about equal entry counts
        if (ip.empty()) {
            ip.resize((size_t)n + 1);
            EACB_CUDA(cudaMemcpyAsync(ip.data(), d_indptr, sizeof(int64_t) * ((size_t)n + 1),
                                      cudaMemcpyDeviceToHost, st));
            EACB_CUDA(cudaStreamSynchronize(st));
        }
        const int64_t parts = (int64_t)((kh[w] + cap - 1) / cap);
        const double piece = (double)ip[n] / (double)parts;
        int64_t r = 0;
        while (r < n) {
            int64_t e = r + 1;
            while (e < n && (double)(ip[e + 1] - ip[r]) <= piece) ++e;
            out.push_back(Phase{w - 1, w, r, e, -1});
            r = e;
        }
        start = w;
        acc = 0;
    }
    if (ph.hi > start) out.push_back(Phase{start, ph.hi, 0, n, -1});
    if (out.size() == 1 && out[0].lo == ph.lo && out[0].hi == ph.hi) {
        // the counts say it fits (it cannot have overflowed): split anyway
        out.clear();
        if (ph.hi - ph.lo < 2) return EACB_ERR_INTERNAL;
        const int m = ph.lo + (ph.hi - ph.lo) / 2;
        out.push_back(Phase{ph.lo, m, 0, n, -1});
        out.push_back(Phase{m, ph.hi, 0, n, -1});
    }
    return EACB_OK;
}

// Matrices of this many entries read the number of components after each
// phase, to end with a phase by pairs of components (k_pair_min: its rows'
// members are a bitmap in shared memory, up to about 1.2 million points);
// smaller ones queue all phases with no read between them.  (1.7M entries:
// 0.65 ms queued, 0.70 by pairs; 4.2M: 0.77 either way; 12.6M: 1.14 and
// 0.95.)
constexpr int64_t kPairEntries = (int64_t)1 << 22;

static bool pair_phase(int32_t n, int64_t nnz)
{
    return nnz >= kPairEntries && pair_smem(n, kPairMax) <= kPairMaxSmem;
}

struct PairList {
    int32_t *ord, *len, *roots, *found;
    int64_t *pre;
    uint16_t *cid;
};

static void carve_final(Carver &c, int32_t n, int64_t nnz, Engine *g, int64_t **hist,
                        int32_t **cmin, PairList *pl)
{
    *g = Engine::carve(c, n, final_edge_cap(n, nnz));
    *hist = c.take<int64_t>(256);
    *cmin = c.take<int32_t>(n);
    *pl = PairList{};
    if (!pair_phase(n, nnz)) return;
    pl->ord = c.take<int32_t>(n);
    pl->len = c.take<int32_t>(n);
    pl->roots = c.take<int32_t>(kPairMax);
    pl->found = c.take<int32_t>(3);      // components numbered, small ones' rows, shares taken
    pl->pre = c.take<int64_t>((int64_t)n + 1);
    pl->cid = c.take<uint16_t>(n);
}

extern "C" size_t eacb_final_clustering_workspace_size(int32_t n, int64_t nnz)
{
    Carver c(nullptr, 0);
    Engine g;
    int64_t *h;
    int32_t *m;
    PairList pl;
    carve_final(c, n, nnz, &g, &h, &m, &pl);
    return c.off;
}

extern "C" int eacb_final_clustering(const int64_t *indptr, const int32_t *indices,
                                     const uint8_t *diassoc, int32_t n, int64_t nnz,
                                     int32_t max_dist, int32_t n_clusters, int32_t *labels,
                                     int64_t *host_n_fclusts, int32_t *host_labels_valid,
                                     void *ws, size_t ws_bytes, uintptr_t stream)
{
    if (n <= 0 || nnz < 0 || !indptr || (nnz > 0 && (!indices || !diassoc)) || !labels ||
        !host_n_fclusts || !host_labels_valid || !ws || n_clusters < 0)
        return EACB_ERR_BAD_ARGUMENT;
    cudaStream_t st = as_stream(stream);
    Pack pk;
    int s = make_pack(n, 8, pk);
    if (s) return s;
    Carver c(ws, ws_bytes);
    Engine g;
    int64_t *hist;
    int32_t *cmin;
    PairList pl;
    carve_final(c, n, nnz, &g, &hist, &cmin, &pl);
    if (c.overflow) return EACB_ERR_WORKSPACE;
    g.kind = 1;
    if ((s = g.reset(st))) return s;
    // 1. minimum spanning forest of the dissimilarity graph, by weight phases
    //    (the reset cleared the histogram)
    if (nnz > 0) {
        if ((s = launch_whist_u8(diassoc, nnz, g.hist, st,
                                 nnz > kFinalQueuedEntries ? kWhistSkip : 1)))
            return s;
    }
    unsigned long long wh[256];
    if ((s = g.read_hist(st, wh))) return s;
    std::vector<Phase> phases;
    plan_final_phases(wh, n, nnz, phases);
    auto build = [&](const Phase &ph) -> int {
        if (nnz == 0) return EACB_OK;
        ProfScope ps(PROF_PHASE, st);
        const UpArgs ua{indptr, indices, diassoc, n, nnz, ph.lo, ph.hi, ph.ident, ph.r0, ph.r1,
                        g.label, pk, g.ea, (unsigned long long *)&g.cnt[C_CURSOR],
                        (unsigned long long)g.Emax, g.best, g.hist, g.err};
        if (ph.pairs) {
            const unsigned gn = grid_for(n, 256, 148 * 8);
            const int64_t V = ph.pairs;
            // the pairs at the end of the edge array, their words at its start
            unsigned long long *pairs = (unsigned long long *)g.ea + (g.Emax - V * V);
            EACB_CUDA(cudaMemsetAsync(pairs, 0xff, sizeof(uint64_t) * V * V, st));
            EACB_CUDA(cudaMemsetAsync(g.flag, 0, sizeof(int32_t) * n, st));
            EACB_CUDA(cudaMemsetAsync(pl.found, 0, 3 * sizeof(int32_t), st));
            k_pair_count<<<gn, 256, 0, st>>>(g.label, n, g.flag);
            EACB_CHECK_LAUNCH();
            k_pair_number<<<gn, 256, 0, st>>>(g.flag, n, (int)V, g.act, cmin, pl.roots, pl.found);
            EACB_CHECK_LAUNCH();
            int t = scan_launch<int32_t, int32_t>(g.act, g.pos, n, 0, &g.cnt[C_AUX1], g.scan, st);
            if (t) return t;
            EACB_CUDA(cudaMemsetAsync(g.act, 0, sizeof(int32_t) * n, st));
            k_pair_place<<<gn, 256, 0, st>>>(indptr, g.label, n, nnz, g.flag, g.pos, &g.cnt[C_AUX1],
                                            cmin, g.act, pl.found + 1, pl.ord, pl.len, pl.cid);
            EACB_CHECK_LAUNCH();
            if ((t = scan_launch<int32_t, int64_t>(pl.len, pl.pre, n, 0, &pl.pre[n], g.scan, st)))
                return t;
            EACB_CUDA(allow_max_dyn_smem(k_pair_min));
            const int shares = (int)std::min<int64_t>(
                kPairBlocks * kPairShares, std::max<int64_t>(kPairBlocks, nnz / kPairShareMin));
            k_pair_min<<<kPairBlocks, kPairThreads, pair_smem(n, (int)V), st>>>(
                ua, PairArgs{pl.ord, pl.pre, g.flag, g.pos, pl.found + 2, shares, pl.cid, pairs, (int)V});
            EACB_CHECK_LAUNCH();
            k_pair_emit<<<(unsigned)V, 256, 0, st>>>(pairs, (int)V, pl.roots, g.ea,
                                                     (unsigned long long *)&g.cnt[C_CURSOR], g.best);
        } else {
            k_phase_upper<<<grid_for((ph.r1 - ph.r0) * 32, kPhThreads, 148 * 4), kPhThreads, 0, st>>>(ua);
        }
        EACB_CHECK_LAUNCH();
        // compulsory reads: row pointers and labels (12 B per row), column and
        // weight (5 B per entry; a row-range phase is counted in proportion to
        // its rows); the written words follow
        const double rows = (double)(ph.r1 - ph.r0);
        ps.done(12.0 * rows + 5.0 * (double)nnz * (rows / (double)n));
        return EACB_OK;
    };
    std::vector<int64_t> hip;
    auto split = [&](const Phase &ph, const unsigned long long kh[256], std::vector<Phase> &out) {
        return split_final_phase(ph, kh, g.Emax, indptr, n, hip, st, out);
    };
    auto sample = [&]() -> int {
        k_outer_sample<<<kOuterSample / 256, 256, 0, st>>>(indptr, indices, diassoc, n, nnz, g.label,
                                                          g.cnt, kPairMax, g.outer);
        EACB_CHECK_LAUNCH();
        return EACB_OK;
    };
    auto check = [&]() -> int {
        k_check_columns<<<grid_for((int64_t)n * 32, kPhThreads, 148 * 8), kPhThreads, 0, st>>>(
            indptr, indices, n, nnz, g.err);
        EACB_CHECK_LAUNCH();
        return EACB_OK;
    };
    // (the pairs' phase and the check read the arrays in 4-entry vectors)
    const bool vec = ((uintptr_t)indices & 15) == 0 && ((uintptr_t)diassoc & 3) == 0;
    if (g.Emax >= nnz && !pl.ord) {
        if ((s = g.run_phased(pk, phases, build, st))) return s;
    } else {
        if ((s = g.run_phased_retry(pk, phases, build, split, sample, check, nnz,
                                    pl.ord && vec ? kPairMax : 0, st))) return s;
    }
    // 2. lifetime rule on the weight histogram
    static_assert(sizeof(CutPlan) == (C_COUNT - C_PLAN) * sizeof(int64_t), "the plan is read with the counts");
    EACB_CUDA(cudaMemsetAsync(hist, 0, 256 * sizeof(int64_t), st));
    k_weight_hist<<<grid_for(n, 256, 148 * 4), 256, 0, st>>>(g.mst, g.cnt, pk, hist);
    EACB_CHECK_LAUNCH();
    k_cut_plan<<<1, 32, 0, st>>>(hist, 0, &g.cnt[C_NMST], n, max_dist, n_clusters,
                                  (CutPlan *)&g.cnt[C_PLAN]);
    EACB_CHECK_LAUNCH();
    int64_t h[C_COUNT];
    if ((s = g.read_counts(st, h))) return s;
    const int64_t n_mst = h[C_NMST];
    CutPlan hp;
    memcpy(&hp, &h[C_PLAN], sizeof(hp));
    if (hp.status) return (int)hp.status;
    *host_n_fclusts = hp.n_clusters;
    if (!hp.need_labels) {
        *host_labels_valid = 0;
        *host_n_fclusts = 1;
        return EACB_OK;
    }
    // 3. components of the forest without the cut edges: the kept forest
    //    keys go from mst into ea, then the rounds
    if ((s = g.reset(st))) return s;
    SrcForest sf{g.mst, n_mst, hp.wmax, pk};
    if ((s = g.filter<SEL_CC>(sf, n_mst, g.ea, st))) return s;
    k_set_sizes<<<1, 32, 0, st>>>(g.cnt, n, -1, g.bar, nullptr);      // the filter's count
    EACB_CHECK_LAUNCH();
    if ((s = g.rounds<SEL_CC>(pk, st, n_mst))) return s;
    // 4. number components by their smallest member
    EACB_CUDA(cudaMemsetAsync(cmin, 0x7f, sizeof(int32_t) * n, st));
    const unsigned gn = grid_for(n, 256);
    k_comp_min<<<gn, 256, 0, st>>>(g.label, n, cmin);
    EACB_CHECK_LAUNCH();
    k_first_flag<<<gn, 256, 0, st>>>(g.label, cmin, n, g.flag);
    EACB_CHECK_LAUNCH();
    if ((s = scan_launch<int32_t, int32_t>(g.flag, g.pos, n, 0, &g.cnt[C_AUX1], g.scan, st)))
        return s;
    k_canon<<<gn, 256, 0, st>>>(g.label, cmin, g.pos, n, labels);
    EACB_CHECK_LAUNCH();
    if ((s = g.read_counts(st, h))) return s;
    if (h[C_DONE] != 1) return EACB_ERR_NOT_CONVERGED;
    *host_n_fclusts = h[C_AUX1];
    *host_labels_valid = 1;
    return EACB_OK;
}

// ---------------------------------------------------------------------------
// The final clustering's two steps as separate calls.
// ---------------------------------------------------------------------------
__global__ void k_check_labels(const int32_t *labels, int32_t n, int *err)
{
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n;
         x += (int64_t)gridDim.x * blockDim.x)
        if (labels[x] < 0 || labels[x] >= n) set_err(err, DEV_BAD_INPUT);
}

extern "C" size_t eacb_lifetime_cut_workspace_size(void)
{
    Carver c(nullptr, 0);
    c.take<unsigned long long>(256);
    c.take<CutPlan>(1);
    return c.off;
}

// lifetime_n_clusters (MyML/MyML/EAC/eac.py:366-391) and the cut decision of
// sp_sl_lifetime (:220-265) on the uint8 weights of a minimum spanning forest
// of n points (any order).  *host_n_clusters receives the number of clusters;
// *host_threshold the largest forest weight kept (-1: none, 255: all).
extern "C" int eacb_lifetime_cut(const uint8_t *mst_weights, int64_t n_mst, int32_t n,
                                 int32_t max_dist, int32_t n_clusters, int64_t *host_n_clusters,
                                 int32_t *host_threshold, void *ws, size_t ws_bytes,
                                 uintptr_t stream)
{
    if (n <= 0 || n_mst < 0 || n_mst >= n || (n_mst > 0 && !mst_weights) || n_clusters < 0 ||
        !host_n_clusters || !host_threshold || !ws)
        return EACB_ERR_BAD_ARGUMENT;
    cudaStream_t st = as_stream(stream);
    Carver c(ws, ws_bytes);
    unsigned long long *hist = c.take<unsigned long long>(256);
    CutPlan *plan = c.take<CutPlan>(1);
    if (c.overflow) return EACB_ERR_WORKSPACE;
    EACB_CUDA(cudaMemsetAsync(hist, 0, 256 * sizeof(unsigned long long), st));
    if (n_mst > 0) {
        const int s = launch_whist_u8(mst_weights, n_mst, hist, st);
        if (s) return s;
    }
    k_cut_plan<<<1, 32, 0, st>>>((const int64_t *)hist, n_mst, nullptr, n, max_dist, n_clusters,
                                  plan);
    EACB_CHECK_LAUNCH();
    CutPlan hp;
    EACB_CUDA(cudaMemcpyAsync(&hp, plan, sizeof(CutPlan), cudaMemcpyDeviceToHost, st));
    EACB_CUDA(cudaStreamSynchronize(st));
    if (hp.status) return (int)hp.status;
    *host_n_clusters = hp.n_clusters;
    *host_threshold = (int32_t)hp.wmax;
    return EACB_OK;
}

extern "C" size_t eacb_relabel_canonical_workspace_size(int32_t n)
{
    Carver c(nullptr, 0);
    c.take<int>(1);
    c.take<int64_t>(1);
    c.take<int32_t>(n);
    c.take<int32_t>(n);
    c.take<int32_t>(n);
    ScanScratch::carve(c, n);
    return c.off;
}

// Numbers the groups of a labelling by their smallest member (the group of
// point 0 is 0, the next group to appear is 1, ...): the numbering scipy's
// connected_components gives, which the final labels use.  labels_in holds
// n group ids in [0, n); labels_out may equal labels_in.
extern "C" int eacb_relabel_canonical(const int32_t *labels_in, int32_t n, int32_t *labels_out,
                                      int64_t *host_n_groups, void *ws, size_t ws_bytes,
                                      uintptr_t stream)
{
    if (!labels_in || n <= 0 || !labels_out || !host_n_groups || !ws) return EACB_ERR_BAD_ARGUMENT;
    cudaStream_t st = as_stream(stream);
    Carver c(ws, ws_bytes);
    int *err = c.take<int>(1);
    int64_t *total = c.take<int64_t>(1);
    int32_t *cmin = c.take<int32_t>(n);
    int32_t *flag = c.take<int32_t>(n);
    int32_t *pos = c.take<int32_t>(n);
    ScanScratch scan = ScanScratch::carve(c, n, err);
    if (c.overflow) return EACB_ERR_WORKSPACE;
    EACB_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
    EACB_CUDA(cudaMemsetAsync(cmin, 0x7f, sizeof(int32_t) * n, st));
    const unsigned gn = grid_for(n, 256);
    k_check_labels<<<gn, 256, 0, st>>>(labels_in, n, err);
    EACB_CHECK_LAUNCH();
    int e = 0;
    EACB_CUDA(cudaMemcpyAsync(&e, err, sizeof(int), cudaMemcpyDeviceToHost, st));
    EACB_CUDA(cudaStreamSynchronize(st));
    if (e) return dev_err_to_status(e);
    k_comp_min<<<gn, 256, 0, st>>>(labels_in, n, cmin);
    EACB_CHECK_LAUNCH();
    k_first_flag<<<gn, 256, 0, st>>>(labels_in, cmin, n, flag);
    EACB_CHECK_LAUNCH();
    int s = scan_launch<int32_t, int32_t>(flag, pos, n, 0, total, scan, st);
    if (s) return s;
    k_canon<<<gn, 256, 0, st>>>(labels_in, cmin, pos, n, labels_out);
    EACB_CHECK_LAUNCH();
    int64_t ng = 0;
    EACB_CUDA(cudaMemcpyAsync(&ng, total, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    EACB_CUDA(cudaMemcpyAsync(&e, err, sizeof(int), cudaMemcpyDeviceToHost, st));
    EACB_CUDA(cudaStreamSynchronize(st));
    if (e) return dev_err_to_status(e);
    *host_n_groups = ng;
    return EACB_OK;
}
