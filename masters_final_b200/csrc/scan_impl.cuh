// Scan kernels shared by the scan entry points and by the graph/coassoc code.
#pragma once
#include "eacb_common.cuh"

namespace eacb {

// Tile shape.  Bound by HBM (one read and one write of the stream), and
// before that by the look-back: with the status words of neighbouring tiles
// in one line, the polls of every block in flight met on a few lines and a
// tile took 25-40 ns whatever its size (64 Mi int32: 186 us with 6,144
// elements per tile, 1 word apart; 170 us with 16,384).  So each tile has a
// line of its own (kStatusStride), and 128 bytes per thread keep the tiles
// few and the loads many.  A warp owns consecutive elements and each of its
// 16-byte loads and stores covers 512 consecutive bytes, so every line is
// touched once.  64 Mi int32: 110 us (4.9 TB/s); 135 us with the wide tiles
// alone, 118 with status words 32 bytes apart.
constexpr int kScanThreads = 512;
constexpr int kScanWarps = kScanThreads / 32;
// elements per thread: 128 bytes of the wider type, or 64 while that leaves
// SMs without a tile
template <typename TIn, typename TOut>
constexpr int kScanWide = 128 / (int)(sizeof(TIn) > sizeof(TOut) ? sizeof(TIn) : sizeof(TOut));
template <typename TIn, typename TOut> constexpr int kScanNarrow = kScanWide<TIn, TOut> / 2;
constexpr int64_t kScanWideMin = 148;     // wide tiles from one per SM
constexpr int64_t scan_tile(int items) { return (int64_t)kScanThreads * items; }
// up to this many elements one block scans the stream by itself
constexpr int kScanSmallThreads = 1024;
constexpr int kScanSmallItems = 16;
constexpr int64_t kScanSmallStep = (int64_t)kScanSmallThreads * kScanSmallItems;
constexpr int64_t kScanSmallMax = 2 * kScanSmallStep;     // (see scan_launch)

struct ScanScratch {
    uint64_t *status;      // kStatusStride words per tile, from the counter's line on
    int *counter;          // tile counter
    int *err;              // its own sits in the line before the counter's
    int64_t max_tiles;
    // lines: [own error word] [counter] [tile 0] [tile 1] ...
    static ScanScratch carve(Carver &c, int64_t n, int *err = nullptr)
    {
        ScanScratch s;
        // sized for the smallest tile any single-pass kernel uses (2048)
        s.max_tiles = (n + 2047) / 2048 + 1;
        uint64_t *w = c.take<uint64_t>((size_t)(s.max_tiles + 2) * kStatusStride);
        s.err = err ? err : (int *)w;
        s.counter = (int *)(w + kStatusStride);
        s.status = w + 2 * kStatusStride;
        return s;
    }
    // zeroes the tile counter and `tiles` status lines (and, with_err, the
    // scratch's own error word) in one memset
    cudaError_t clear(int64_t tiles, bool with_err, cudaStream_t st) const
    {
        const size_t line = kStatusStride * sizeof(uint64_t);
        char *p = (char *)counter - (with_err ? line : 0);
        return cudaMemsetAsync(p, 0, (size_t)((char *)status - p) + (size_t)tiles * line, st);
    }
};

template <typename T> struct Vec16;
template <> struct Vec16<int32_t> { typedef int4 type; static constexpr int n = 4; };
template <> struct Vec16<int64_t> { typedef longlong2 type; static constexpr int n = 2; };

// a 16-byte input vector's outputs in one store: 16 bytes, or 32 where int32
// widens to int64 (two 16-byte stores would each write half sectors)
__device__ __forceinline__ void store_vec(int32_t *p, const int32_t (&o)[4])
{
    __stcs(reinterpret_cast<int4 *>(p), make_int4(o[0], o[1], o[2], o[3]));
}
__device__ __forceinline__ void store_vec(int64_t *p, const int64_t (&o)[2])
{
    __stcs(reinterpret_cast<longlong2 *>(p), make_longlong2(o[0], o[1]));
}
__device__ __forceinline__ void store_vec(int64_t *p, const int64_t (&o)[4])
{
    asm volatile("st.global.cs.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(o[0]), "l"(o[1]),
                 "l"(o[2]), "l"(o[3])
                 : "memory");
}

// Prefixes inside a tile: int32 outputs are stored modulo 2^32, so theirs are
// scanned in 32 bits; totals and the tiles' prefixes are always 64-bit.
template <typename TOut> struct ScanAcc { typedef int64_t type; };
template <> struct ScanAcc<int32_t> { typedef uint32_t type; };

__device__ __forceinline__ uint32_t warp_incl(uint32_t v)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += o;
    }
    return v;
}
__device__ __forceinline__ int64_t warp_incl(int64_t v) { return warp_incl_sum(v); }

// exact warp sum of values below 2^47 in magnitude (two 32-bit reductions)
__device__ __forceinline__ int64_t warp_sum_47(int64_t v)
{
    const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)(v & 0xffffff));
    const int hi = __reduce_add_sync(0xffffffffu, (int)(v >> 24));
    return ((int64_t)hi << 24) + (int64_t)lo;
}

// A thread's share of a step: ITEMS elements as ITEMS / VN groups of VN
// consecutive ones (VN: elements of a 16-byte input vector), group j of lane
// l at first + (j * 32 + l) * VN.
template <typename TIn, typename TOut, bool VEC, int ITEMS>
struct ScanItems {
    typedef typename ScanAcc<TOut>::type Acc;
    static constexpr int VN = Vec16<TIn>::n;
    static constexpr int NG = ITEMS / VN;
    static constexpr int64_t kWarpSpan = 32 * ITEMS;
    TIn v[ITEMS];
    Acc pre[NG];               // sum of the warp's elements before the group

    // elements of [first, n); the rest read as zero
    __device__ __forceinline__ void load(const TIn *in, int64_t first, int64_t n, bool full)
    {
        const int lane = threadIdx.x & 31;
        if (VEC && full) {
            typedef typename Vec16<TIn>::type V;
            const V *p = reinterpret_cast<const V *>(in + first) + lane;
#pragma unroll
            for (int j = 0; j < NG; ++j) {
                const V x = __ldcs(p + j * 32);
                memcpy(&v[j * VN], &x, sizeof(V));
            }
        } else {
#pragma unroll
            for (int q = 0; q < ITEMS; ++q) {
                const int64_t e = first + (int64_t)((q / VN) * 32 + lane) * VN + q % VN;
                v[q] = e < n ? in[e] : TIn(0);
            }
        }
    }

    // prefixes of the groups within the warp; returns the warp's exact total
    __device__ __forceinline__ int64_t scan_warp()
    {
        Acc run = 0;
        int64_t exact = 0;
#pragma unroll
        for (int j = 0; j < NG; ++j) {
            int64_t s = 0;
#pragma unroll
            for (int e = 0; e < VN; ++e) s += (int64_t)v[j * VN + e];
            exact += s;
            const Acc inc = warp_incl((Acc)s);
            pre[j] = run + inc - (Acc)s;
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
        // a 64-bit running sum is the total already; a 32-bit one has lost
        // the high part (a lane's 32 int32 values stay below 2^37)
        if (sizeof(Acc) == 8) return (int64_t)run;
        return warp_sum_47(exact);
    }

    __device__ __forceinline__ void store(TOut *out, int64_t first, int64_t n, bool full,
                                          int64_t base) const
    {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int j = 0; j < NG; ++j) {
            Acc run = (Acc)base + pre[j];
            TOut o[VN];
#pragma unroll
            for (int e = 0; e < VN; ++e) {
                o[e] = (TOut)run;
                run += (Acc)v[j * VN + e];
            }
            const int64_t e0 = first + (int64_t)(j * 32 + lane) * VN;
            if (VEC && full) {
                store_vec(out + e0, o);
            } else {
#pragma unroll
                for (int e = 0; e < VN; ++e)
                    if (e0 + e < n) out[e0 + e] = o[e];
            }
        }
    }
};

template <typename TIn, typename TOut, bool VEC, int ITEMS>
__global__ void __launch_bounds__(kScanThreads, 2)
k_scan(const TIn *__restrict__ in, TOut *__restrict__ out, int64_t n, int64_t init,
       uint64_t *status, int *counter, int64_t *total, int *err)
{
    typedef ScanItems<TIn, TOut, VEC, ITEMS> Items;
    constexpr int64_t kTile = scan_tile(ITEMS);
    __shared__ int s_tile;
    __shared__ int64_t s_warp[kScanWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1);
    __syncthreads();
    const int64_t tile = s_tile;
    const int64_t first = tile * kTile + (int64_t)warp * Items::kWarpSpan;
    const bool full = (tile + 1) * kTile <= n;
    Items it;
    it.load(in, first, n, full);
    const int64_t wt = it.scan_warp();
    if (lane == 0) s_warp[warp] = wt;
    __syncthreads();
    if (warp == 0) {
        // the warps' totals become their prefixes in the whole stream
        const int64_t x = lane < kScanWarps ? s_warp[lane] : 0;
        const int64_t inc = warp_incl_sum(x);
        const int64_t agg = __shfl_sync(0xffffffffu, inc, 31);
        const int64_t pre = lookback(status, tile, agg, init, err);
        if (lane < kScanWarps) s_warp[lane] = pre + inc - x;
        if (lane == 0 && (tile + 1) * kTile >= n && total) *total = pre + agg;
    }
    __syncthreads();
    it.store(out, first, n, full, s_warp[warp]);
}

// A short stream on one block: no tile state to clear and no look-back.
// clear_err: an error word to zero on the way (null: leave it).
template <typename TIn, typename TOut, bool VEC>
__global__ void __launch_bounds__(kScanSmallThreads)
k_scan_small(const TIn *__restrict__ in, TOut *__restrict__ out, int64_t n, int64_t init,
             int64_t *total, int *clear_err)
{
    typedef ScanItems<TIn, TOut, VEC, kScanSmallItems> Items;
    __shared__ int64_t s_warp[2][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int64_t run = init;
    int ph = 0;
    for (int64_t base = 0; base < n; base += kScanSmallStep, ph ^= 1) {
        const int64_t first = base + (int64_t)warp * Items::kWarpSpan;
        const bool full = base + kScanSmallStep <= n;
        Items it;
        it.load(in, first, n, full);
        const int64_t wt = it.scan_warp();
        if (lane == 0) s_warp[ph][warp] = wt;      // the other half was read one barrier ago
        __syncthreads();
        const int64_t x = s_warp[ph][lane];
        const int64_t inc = warp_incl_sum(x);
        it.store(out, first, n, full, run + __shfl_sync(0xffffffffu, inc - x, warp));
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (threadIdx.x == 0) {
        if (total) *total = run;
        if (clear_err) *clear_err = 0;
    }
}

__global__ void k_set_i64(int64_t *p, int64_t v);

template <typename TIn, typename TOut, int ITEMS>
inline int scan_launch_tiles(const TIn *in, TOut *out, int64_t n, int64_t init, int64_t *d_total,
                             const ScanScratch &s, cudaStream_t st, bool clear_err, bool vec)
{
    const int64_t ntiles = (n + scan_tile(ITEMS) - 1) / scan_tile(ITEMS);
    if (ntiles > (int64_t)0x7fffffff) return EACB_ERR_UNSUPPORTED;
    if (ntiles > s.max_tiles) return EACB_ERR_WORKSPACE;
    EACB_CUDA(s.clear(ntiles, clear_err, st));
    if (vec)
        k_scan<TIn, TOut, true, ITEMS><<<(unsigned)ntiles, kScanThreads, 0, st>>>(
            in, out, n, init, s.status, s.counter, d_total, s.err);
    else
        k_scan<TIn, TOut, false, ITEMS><<<(unsigned)ntiles, kScanThreads, 0, st>>>(
            in, out, n, init, s.status, s.counter, d_total, s.err);
    EACB_CHECK_LAUNCH();
    return EACB_OK;
}

// clear_err: also zero the scratch's own error word (the one in the line
// before the counter).  One block takes a stream of one step, and of two where
// they move 8 bytes per element in whole vectors: there the clearing memset and
// the look-back cost as much as the second step.  Device time of 20,011 and
// 32,768 elements, one block against tiles: int32 6.2, 6.0 / 6.2, 6.2 us; off
// the 16-byte boundary 10.3, 13.6 / 8.2, 8.3; int32 to int64 8.1, 8.9 / 8.2,
// 6.3, unaligned 16.4, 23.1 / 8.2, 8.2; int64 9.7, 10.8 / 7.9, 6.9.
template <typename TIn, typename TOut>
inline int scan_launch(const TIn *in, TOut *out, int64_t n, int64_t init, int64_t *d_total,
                       const ScanScratch &s, cudaStream_t st, bool clear_err = false)
{
    if (n == 0) {
        if (d_total) {
            k_set_i64<<<1, 1, 0, st>>>(d_total, init);
            EACB_CHECK_LAUNCH();
        }
        return EACB_OK;
    }
    // 16-byte input vectors, and as many outputs as one holds in one store
    const bool vec = ((uintptr_t)in % 16 == 0) &&
                     ((uintptr_t)out % (16 / sizeof(TIn) * sizeof(TOut)) == 0);
    if (n <= (vec && sizeof(TIn) + sizeof(TOut) == 8 ? kScanSmallMax : kScanSmallStep)) {
        int *ce = clear_err ? s.err : nullptr;
        if (vec)
            k_scan_small<TIn, TOut, true><<<1, kScanSmallThreads, 0, st>>>(in, out, n, init,
                                                                          d_total, ce);
        else
            k_scan_small<TIn, TOut, false><<<1, kScanSmallThreads, 0, st>>>(in, out, n, init,
                                                                           d_total, ce);
        EACB_CHECK_LAUNCH();
        return EACB_OK;
    }
    constexpr int kWide = kScanWide<TIn, TOut>, kNarrow = kScanNarrow<TIn, TOut>;
    if (n < kScanWideMin * scan_tile(kWide))
        return scan_launch_tiles<TIn, TOut, kNarrow>(in, out, n, init, d_total, s, st, clear_err,
                                                     vec);
    return scan_launch_tiles<TIn, TOut, kWide>(in, out, n, init, d_total, s, st, clear_err, vec);
}

}  // namespace eacb
