// Cluster member lists by a stable counting sort (shared by the
// co-association build and the k-means centroid update).
//
// For a label matrix labels[p*n + i] in [0, K) (-1 = none), the member list of
// cluster (p, c) is the ascending list of points with that label.  Lists are
// laid out back to back in (partition, cluster) order: a tile histogram
// cnt[(p*K + c)*ntiles + tile] is scanned (exclusive, int64) into S, so that
// S[(p*K + c)*ntiles + tile] is where tile `tile`'s members of (p, c) start and
// [S[(p*K+c)*ntiles], S[(p*K+c+1)*ntiles]) is the whole list.
#pragma once
#include "eacb_common.cuh"

namespace eacb {

constexpr int kMLTile = 4096;          // points per tile in the counting sort

// ---------------------------------------------------------------- step 1 --
static __global__ void __launch_bounds__(256)
k_ml_count(const int32_t *labels, int32_t n, int32_t K, int64_t ntiles, int32_t *cnt, int *err)
{
    extern __shared__ int hist[];
    const int64_t p = blockIdx.x / ntiles, tile = blockIdx.x % ntiles;
    for (int c = threadIdx.x; c < K; c += blockDim.x) hist[c] = 0;
    __syncthreads();
    const int64_t i0 = tile * kMLTile;
    const int32_t *lp = labels + p * n;
    for (int64_t i = i0 + threadIdx.x; i < i0 + kMLTile && i < n; i += blockDim.x) {
        int32_t l = lp[i];
        if (l >= K) { set_err(err, DEV_BAD_INPUT); continue; }
        if (l >= 0) atomicAdd(&hist[l], 1);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < K; c += blockDim.x)
        cnt[((int64_t)p * K + c) * ntiles + tile] = hist[c];
}

// One block per (partition, tile), a warp per contiguous share of the tile:
// the warp ranks its points among its own equals (32 at a time, in index
// order, counts per cluster in shared memory), the block turns the warps'
// counts into offsets, and every point's place is its cluster's place for
// the tile plus its warp's offset plus its rank.  Bound by the chain of
// 32-point steps (match, count read, count write): one warp took a whole
// tile in 128 of them, 60 us whatever the number of tiles (1,000,000
// points); 18 us with 16.
constexpr int kMLWarps = 8;
constexpr int kMLSteps = kMLTile / (32 * kMLWarps);
static inline size_t ml_place_smem(int32_t K)
{
    return (size_t)K * (sizeof(int32_t) + kMLWarps * sizeof(uint16_t));
}

static __global__ void __launch_bounds__(kMLWarps * 32)
k_ml_place(const int32_t *labels, int32_t n, int32_t K, int64_t ntiles, const int64_t *S,
           int32_t *members, int32_t *mypos)
{
    extern __shared__ int32_t ml_base[];       // K places, then a row of K counts per warp
    uint16_t *cnt = reinterpret_cast<uint16_t *>(ml_base + K);
    const int64_t p = blockIdx.x / ntiles, tile = blockIdx.x % ntiles;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = threadIdx.x; c < K; c += blockDim.x) {
        ml_base[c] = (int32_t)S[((int64_t)p * K + c) * ntiles + tile];    // below P n < 2^31
        for (int w = 0; w < kMLWarps; ++w) cnt[w * K + c] = 0;
    }
    const int32_t *lp = labels + p * n;
    const int64_t i0 = tile * kMLTile + (int64_t)warp * (32 * kMLSteps) + lane;
    int32_t l[kMLSteps];
#pragma unroll
    for (int s = 0; s < kMLSteps; ++s) {
        const int64_t i = i0 + 32 * s;
        l[s] = i < n ? lp[i] : -1;
        if (l[s] >= K) l[s] = -1;
    }
    __syncthreads();
    uint16_t *mine = cnt + (int64_t)warp * K;
    const unsigned lt = (1u << lane) - 1u;
    uint16_t rank[kMLSteps];
#pragma unroll
    for (int s = 0; s < kMLSteps; ++s) {
        const unsigned peers = __match_any_sync(0xffffffffu, l[s] >= 0 ? l[s] : -1 - lane);
        const int before = l[s] >= 0 ? mine[l[s]] : 0;
        __syncwarp();
        rank[s] = (uint16_t)(before + __popc(peers & lt));
        if (l[s] >= 0 && lane == 31 - __clz(peers)) mine[l[s]] = (uint16_t)(before + __popc(peers));
        __syncwarp();
    }
    __syncthreads();
    for (int c = threadIdx.x; c < K; c += blockDim.x) {
        int run = 0;
#pragma unroll
        for (int w = 0; w < kMLWarps; ++w) {
            const int v = cnt[w * K + c];
            cnt[w * K + c] = (uint16_t)run;
            run += v;
        }
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < kMLSteps; ++s) {
        const int64_t i = i0 + 32 * s;
        if (i >= n) break;
        int32_t pos = -1;
        if (l[s] >= 0) {
            pos = ml_base[l[s]] + mine[l[s]] + rank[s];
            members[pos] = (int32_t)i;
        }
        mypos[p * n + i] = pos;
    }
}

static int launch_ml_place(cudaStream_t st, const int32_t *labels, int32_t n, int32_t P, int32_t K,
                           int64_t ntiles, const int64_t *S, int32_t *members, int32_t *mypos)
{
    const size_t smem = ml_place_smem(K);
    if (smem > 48 * 1024) EACB_CUDA(allow_max_dyn_smem(k_ml_place));
    k_ml_place<<<(unsigned)(P * ntiles), kMLWarps * 32, smem, st>>>(labels, n, K, ntiles, S, members,
                                                                   mypos);
    EACB_CHECK_LAUNCH();
    return EACB_OK;
}

// non-empty clusters per partition, then the processing order
static __global__ void k_ncl(const int64_t *S, int32_t K, int64_t ntiles, int32_t *ncl, int *maxsize)
{
    __shared__ int tot, big;
    if (threadIdx.x == 0) tot = big = 0;
    __syncthreads();
    const int64_t p = blockIdx.x;
    int mine = 0, mbig = 0;
    for (int c = threadIdx.x; c < K; c += blockDim.x) {
        int64_t a = S[(p * K + c) * ntiles], b = S[(p * K + c + 1) * ntiles];
        mine += b > a;
        mbig = max(mbig, (int)(b - a));
    }
    atomicAdd(&tot, mine);
    atomicMax(&big, mbig);
    __syncthreads();
    if (threadIdx.x == 0) {
        ncl[p] = tot;
        atomicMax(maxsize, big);
    }
}

static __global__ void k_order(const int32_t *ncl, int32_t P, int32_t *order)
{
    if (threadIdx.x != 0) return;
    int first = 0;
    for (int p = 1; p < P; ++p)
        if (ncl[p] < ncl[first]) first = p;
    order[0] = first;
    int q = 1;
    for (int p = 0; p < P; ++p)
        if (p != first) order[q++] = p;
}

}  // namespace eacb
