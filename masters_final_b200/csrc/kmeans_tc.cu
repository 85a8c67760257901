// K-means label pass on tcgen05 tensor cores.
//
// dist(x, c) = |x|^2 - 2 x.c + |c|^2 on data centred near its mean.  The dot
// products run as ONE BF16 GEMM with FP32 accumulation in tensor memory:
// each float32 operand is split into three BF16 parts (h + m + l, ~24
// significant bits) and the K dimension holds the six products that matter
// (see put_row), the large h*h group last.  The epilogue (8 warps, one point
// row per thread, half the columns per warp) reads the accumulator tile
// from TMEM with tcgen05.ld, forms the screened distances and keeps the best
// two of the minima of four columns per point, with the winner's four.  Those
// four are compared by direct float32 distances; a point whose other three, or
// whose least column outside them, are not certainly behind is re-labelled in
// the reference's arithmetic; every other point gets its winner's exact
// reference distance.  Labels therefore equal the reference's
// (MyML/MyML/cluster/KMeans.py:453-490) for any input.  2,000,000 x 8, ten
// partitions of about 1,000: 7.8 ms a pass with an index and a runner-up per
// column (six instructions), 6.25 now (two and a half).
//
// Shapes: M = 128 points per CTA, N <= 128 centroids per MMA tile, K = 6d
// padded to a multiple of 16 (<= 192).  Operands are pre-arranged in global
// memory in the UMMA K-major no-swizzle core-matrix layout (8 rows x 16
// bytes per core matrix, LBO = 128 B along K, SBO = 128 B * K/8 along M/N),
// so each tile is one contiguous cp.async.bulk copy into shared memory.
// One thread issues the MMAs; TMEM holds one 128 x 128 FP32 accumulator per
// CTA (128 columns), four CTAs per SM share the 512 columns and overlap each
// other's MMA and epilogue.  Every wait is bounded and reports an error.
#include "kmeans_common.cuh"
#include "tcgen05.cuh"
#include <cuda_bf16.h>

#include <algorithm>

namespace eacb {

constexpr int kTM = 128;           // points per CTA tile
constexpr int kTN = kTcCentPad;    // centroids per MMA tile
constexpr int kTThreads = 256;     // 8 warps: 4 TMEM lane quarters x 2 column halves
constexpr int kTColGroups = kTThreads / kTM;
constexpr int kTColsPer = kTN / kTColGroups;
constexpr int kTmemCols = kTN;

// instruction descriptor: BF16 x BF16 -> FP32, both K-major, M x N
__host__ __device__ constexpr uint32_t umma_idesc(int M, int N)
{
    return (1u << 4)                       // D format F32
           | (1u << 7)                     // A format BF16
           | (1u << 10)                    // B format BF16
           | ((uint32_t)(N >> 3) << 17)    // N
           | ((uint32_t)(M >> 4) << 24);   // M
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                         uint32_t idesc, uint32_t accumulate)
{
    const uint32_t z = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(
            tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(z), "r"(z), "r"(z), "r"(z));
}

__host__ __device__ __forceinline__ uint32_t sbo_b(int Kp) { return 128u * (uint32_t)(Kp >> 3); }

// byte offset of element (row, k) inside a blocked K-major tile with Kp columns
__host__ __device__ __forceinline__ uint32_t core_off(int row, int k, int Kp)
{
    const int g = row >> 3, rr = row & 7, q = k >> 3, kk = k & 7;
    return (uint32_t)((((g * (Kp >> 3) + q) << 3) + rr) * 16 + kk * 2);
}

// ------------------------------------------------------------ preparation --
// About the mean of at most kMeanRows rows, evenly spread: float64 partials per
// block (one thread per dimension and row lane, consecutive addresses), which
// k_mean puts together.  Reading all of 2,000,000 x 8 took 383 us.
constexpr int kMeanRows = 65536;
constexpr int kMeanBlocks = 296;
__global__ void __launch_bounds__(256)
k_colsum(const float *X, int32_t n, int32_t D, int32_t m, double *part)
{
    __shared__ double s[256];
    const int per = 256 / D;                           // row lanes
    const int d = threadIdx.x % D, r = threadIdx.x / D;
    double acc = 0.0;
    if (r < per)
        for (int64_t j = (int64_t)blockIdx.x * per + r; j < m; j += (int64_t)gridDim.x * per)
            acc += (double)X[j * n / m * D + d];
    s[threadIdx.x] = acc;
    __syncthreads();
    if (r == 0) {
        double t = 0.0;
        for (int q = 0; q < per; ++q) t += s[q * D + d];
        part[(int64_t)blockIdx.x * 32 + d] = t;
    }
}

// The rows in 32 parts (lane l: blocks l, l + 32, ...), and the median of the
// parts' means: a few rows far out, or not finite, move one part's mean but
// not the centre, which would put all other points far from it and leave them
// to the re-check (200,000 x 32 with ten rows at 10^6: 2.4 -> 0.8 ms a pass).
__global__ void k_mean(const double *part, int nblocks, int32_t m, int32_t D, float *mu)
{
    const int lane = threadIdx.x & 31, d = threadIdx.x >> 5;
    if (d >= D) return;
    const int per = 256 / D;                           // as in k_colsum
    const int64_t cycle = (int64_t)nblocks * per, rest = m % cycle;
    double t = 0.0;
    int64_t rows = 0;
    for (int b = lane; b < nblocks; b += 32) {
        t += part[(int64_t)b * 32 + d];
        const int64_t r = rest - (int64_t)b * per;
        rows += m / cycle * per + (r < 0 ? 0 : (r < per ? r : per));
    }
    const float v = rows ? (float)(t / (double)rows) : 0.f;
    const bool ok = rows && fabsf(v) <= 3.4e38f;
    const unsigned all = __ballot_sync(0xffffffffu, ok);
    int rank = 0;
#pragma unroll
    for (int o = 0; o < 32; ++o) {
        const float w = __shfl_sync(0xffffffffu, v, o);
        rank += ((all >> o) & 1u) && (w < v || (w == v && o < lane)) ? 1 : 0;
    }
    if (ok && rank == __popc(all) / 2) mu[d] = v;
    if (all == 0u && lane == 0) mu[d] = 0.f;
}

int data_mean(const float *X, int32_t n, int32_t D, TcScratch &s, cudaStream_t st)
{
    if (s.mean_ready) return EACB_OK;
    const int32_t m = std::min(n, kMeanRows);
    k_colsum<<<kMeanBlocks, 256, 0, st>>>(X, n, D, m, s.part);
    EACB_CHECK_LAUNCH();
    k_mean<<<1, 1024, 0, st>>>(s.part, kMeanBlocks, m, D, s.mu);
    EACB_CHECK_LAUNCH();
    s.mean_ready = true;
    return EACB_OK;
}

// Rows of one operand, centred and split into three BF16 parts
// v = h + m + l (each part the BF16 rounding of the remainder, so |m| <=
// 2^-8 |v|, |l| <= 2^-16 |v| and the rest is below 2^-24 |v|).  The K axis
// holds six groups of D products, smallest first so that the large h*h
// products are accumulated last:
//   group      0    1    2    3    4    5
//   point      l    m    h    m    h    h
//   centroid   h    m    l    h    m    h
// Their sum is x.c up to the dropped l*m, m*l, l*l terms (< 3 * 2^-24 |x||c|).
__device__ __forceinline__ void put_row(const float *v, const float *mu, int D, int Kp, int row,
                                       uint8_t *tile, bool point_side, float &norm)
{
    constexpr int kPointPart[6] = {2, 1, 0, 1, 0, 0};      // 0 = h, 1 = m, 2 = l
    constexpr int kCentPart[6] = {0, 1, 2, 0, 1, 0};
    float nrm = 0.f;
    for (int k = 0; k < Kp; ++k) {
        __nv_bfloat16 b = __float2bfloat16_rn(0.f);
        if (k < 6 * D) {
            const int d = k % D, grp = k / D;
            const float xc = __fsub_rn(v[d], mu[d]);
            const __nv_bfloat16 h = __float2bfloat16_rn(xc);
            const float r1 = __fsub_rn(xc, __bfloat162float(h));
            const __nv_bfloat16 m = __float2bfloat16_rn(r1);
            const __nv_bfloat16 l = __float2bfloat16_rn(__fsub_rn(r1, __bfloat162float(m)));
            const int part = point_side ? kPointPart[grp] : kCentPart[grp];
            b = part == 0 ? h : (part == 1 ? m : l);
            if (grp == 0) nrm = fmaf(xc, xc, nrm);
        }
        *reinterpret_cast<__nv_bfloat16 *>(tile + core_off(row, k, Kp)) = b;
    }
    norm = nrm;
}

__global__ void k_prep_points(const float *X, int32_t n, int32_t D, int32_t Kp, const float *mu,
                              uint8_t *A, float *nx, int64_t n_pad)
{
    const int64_t tile_bytes = (int64_t)kTM * Kp * 2;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_pad;
         i += (int64_t)gridDim.x * blockDim.x) {
        uint8_t *tile = A + (i / kTM) * tile_bytes;
        float v[32];
        for (int d = 0; d < D; ++d) v[d] = i < n ? X[i * D + d] : mu[d];
        float nrm;
        put_row(v, mu, D, Kp, (int)(i % kTM), tile, true, nrm);
        nx[i] = nrm;
    }
}

__global__ void k_prep_centroids(const float *C, const int32_t *kk, int32_t kmax, int32_t P,
                                 int32_t D, int32_t Kp, int32_t kt_max, const float *mu,
                                 const int32_t *active, uint8_t *B, float *nc, float *cmax2)
{
    const int64_t tile_bytes = (int64_t)kTN * Kp * 2;
    const int64_t per_p = (int64_t)kt_max * kTN;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < (int64_t)P * per_p;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int p = (int)(e / per_p);
        if (!active[p]) continue;
        const int c = (int)(e % per_p);
        uint8_t *tile = B + ((int64_t)p * kt_max + c / kTN) * tile_bytes;
        float v[32];
        const bool real = c < kk[p];
        for (int d = 0; d < D; ++d) v[d] = real ? C[((int64_t)p * kmax + c) * D + d] : mu[d];
        float nrm;
        put_row(v, mu, D, Kp, c % kTN, tile, false, nrm);
        nc[e] = real ? nrm : __int_as_float(0x7f800000);
        // a NaN norm (which no screen may judge) counts only at centroid 0:
        // there the reference keeps it, elsewhere it never compares as smaller
        if (real && (nrm == nrm || c == 0))
            atomicMax(reinterpret_cast<int *>(&cmax2[p]),
                      nrm == nrm ? __float_as_int(nrm) : 0x7fffffff);
    }
}

template <int DM>
__device__ __forceinline__ float screen_dist(const float (&x)[DM], const float (&c)[DM], int D)
{
    float acc = 0.f;
#pragma unroll
    for (int d = 0; d < DM; ++d)
        if (d < D) {
            const float diff = __fsub_rn(x[d], c[d]);
            acc = __fmaf_rn(diff, diff, acc);
        }
    return acc;
}

// ---------------------------------------------------------------- labels --
// columns of which only the least score is kept: the winner's chunk is
// compared again at the end, a row of D floats per column (with eight columns
// the rows cost more than the scores saved)
constexpr int kTcChunk = 4;

// DM: D rounded up to 4, 8, 16 or 32; VEC: D equals DM and the rows of X and C
// can be read as 16-byte vectors
template <int DM, bool VEC>
__global__ void __launch_bounds__(kTThreads, 4)
k_label_tc(const float *__restrict__ X, int32_t n, int32_t D, int32_t Kp, const float *__restrict__ C,
           const int32_t *__restrict__ kk, int32_t kmax, int32_t kt_max, int32_t P, int32_t ppc,
           const int32_t *__restrict__ active, const uint8_t *__restrict__ A,
           const float *__restrict__ nx, const uint8_t *__restrict__ B,
           const float *__restrict__ nc, const float *__restrict__ cmax2, float E, int nbuf,
           int32_t *labels, float *dists, int32_t *amb, int *namb, int *err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t bar_a, bar_b[2], bar_mma;
    __shared__ uint32_t tmem_slot;
    __shared__ float s_b1[kTColGroups - 1][kTM], s_b2[kTColGroups - 1][kTM];
    __shared__ int s_i1[kTColGroups - 1][kTM];
    __shared__ int s_fail;
    const uint32_t a_bytes = (uint32_t)kTM * Kp * 2, b_bytes = (uint32_t)kTN * Kp * 2;
    uint8_t *sA = smem;
    // two centroid-tile buffers when they fit (prefetch overlaps the MMA),
    // else one (prefetch overlaps the epilogue)
    uint8_t *sB[2] = {smem + a_bytes, nbuf == 2 ? smem + a_bytes + b_bytes : smem + a_bytes};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the MMA issuer: a thread of the last warp, which has no per-partition
    // tail, so the next MMA starts while the first warps finish a partition
    const bool issuer = threadIdx.x == kTThreads - 32;
    const int64_t tile0 = blockIdx.x;
    const uint8_t *Ap = A + tile0 * a_bytes;
    // the tiles in order: every centroid tile of every active partition of
    // this CTA's share [pb, pe) of the partitions
    const int pb = blockIdx.y * ppc, pe = min(P, pb + ppc);
    auto ntiles = [&](int q) -> int { return active[q] ? (kk[q] + kTN - 1) / kTN : 0; };
    auto first_from = [&](int q) -> int {
        while (q < pe && ntiles(q) == 0) ++q;
        return q < pe ? q : P;
    };
    auto btile = [&](int q, int t) -> const uint8_t * {
        return B + ((int64_t)q * kt_max + t) * b_bytes;
    };

    int p = first_from(pb);
    if (p >= P) return;                          // uniform: nothing to label
    if (threadIdx.x == 0) {
        s_fail = 0;
        mbar_init(&bar_a, 1);
        mbar_init(&bar_b[0], 1);
        mbar_init(&bar_b[1], 1);
        mbar_init(&bar_mma, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_addr(&tmem_slot)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    if (issuer) {
        mbar_expect_tx(&bar_a, a_bytes);
        bulk_g2s(sA, Ap, a_bytes, &bar_a);
        mbar_expect_tx(&bar_b[0], b_bytes);
        bulk_g2s(sB[0], btile(p, 0), b_bytes, &bar_b[0]);
    }
    // epilogue ownership: row = 32*(warp%4) + lane (the TMEM lanes warp w may
    // read), columns [64*(warp/4), +64) of the 128-column tile
    const int row = 32 * (warp & 3) + lane;
    const int cgrp = warp >> 2, colh = kTColsPer * cgrp;
    const int64_t i = tile0 * kTM + row;
    const float xn = (i < n) ? nx[i] : 0.f;
    float b1 = __int_as_float(0x7f800000), b2 = b1;
    int i1 = 0;
    const uint32_t lbo = 128, sbo = 128u * (uint32_t)(Kp >> 3);
    uint32_t ph_b[2] = {0, 0}, ph_mma = 0;
    int pend = -1;                               // buffer with a copy in flight (issuer)
    int mma_ph = -1;                             // phase of an MMA not yet seen complete
    bool ok = true;
    int t = 0, tiles = ntiles(p);
    for (int64_t j = 0; p < P; ++j) {
        // the tile after (p, t): its copy is issued while this one is used
        int pn = p, tn = t + 1;
        if (tn == tiles) {
            pn = first_from(p + 1);
            tn = 0;
        }
        const int buf = nbuf == 2 ? (int)(j & 1) : 0;
        const int nvalid = min(kTN, kk[p] - t * kTN);
        const int N = (nvalid + 15) & ~15;
        if (issuer) {
            bool got = (j == 0 ? mbar_wait(&bar_a, 0) : true) && mbar_wait(&bar_b[buf], ph_b[buf]);
            if (!got) {
                set_err(err, DEV_SPIN_LIMIT);
                s_fail = 1;
            } else {
                pend = -1;
                tc_fence_after();
                const uint32_t idesc = umma_idesc(kTM, N);
                for (int s = 0; s < (Kp >> 4); ++s) {
                    const uint64_t ad = umma_desc(sA + s * 256, lbo, sbo);
                    const uint64_t bd = umma_desc(sB[buf] + s * 256, lbo, sbo_b(Kp));
                    mma_bf16(tmem, ad, bd, idesc, s > 0 ? 1u : 0u);
                }
                mma_commit(&bar_mma);
                mma_ph = (int)ph_mma;
                if (nbuf == 2 && pn < P) {
                    // the other buffer's last reader (the previous MMA) completed
                    mbar_expect_tx(&bar_b[buf ^ 1], b_bytes);
                    bulk_g2s(sB[buf ^ 1], btile(pn, tn), b_bytes, &bar_b[buf ^ 1]);
                    pend = buf ^ 1;
                }
            }
        }
        ph_b[buf] ^= 1;
        __syncthreads();
        if (s_fail) { ok = false; break; }
        if (!mbar_wait(&bar_mma, ph_mma)) {
            set_err(err, DEV_SPIN_LIMIT);
            s_fail = 1;
        } else if (issuer) {
            mma_ph = -1;
            if (nbuf == 1 && pn < P) {
                // single buffer: this tile's MMA has finished reading it
                mbar_expect_tx(&bar_b[0], b_bytes);
                bulk_g2s(sB[0], btile(pn, tn), b_bytes, &bar_b[0]);
                pend = 0;
            }
        }
        ph_mma ^= 1;
        tc_fence_after();
        const float *ncp = nc + ((int64_t)p * kt_max + t) * kTN;
        const int c_lo = colh, c_hi = min(colh + kTColsPer, nvalid);
        // 32 columns at a time (a 64-column share; past the tile's valid
        // columns the norms are +inf, so those columns never win)
        for (int c0 = c_lo; c0 < c_hi; c0 += 32) {
            float v[32], ncv[32];
            tmem_ld32(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c0, v);
            // the 32 centroid norms, the same for every lane: eight 16-byte loads
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float4 f = __ldg(reinterpret_cast<const float4 *>(ncp + c0) + q);
                ncv[4 * q] = f.x;
                ncv[4 * q + 1] = f.y;
                ncv[4 * q + 2] = f.z;
                ncv[4 * q + 3] = f.w;
            }
            // the screened distance less the row's |x|^2 (the same for every
            // column, so the order and the gaps are those of the distance):
            // one rounding, where adding |x|^2 first would take two
            constexpr int CK = kTcChunk;
            const int gb = (t * kTN + c0) / CK;
            const uint64_t m2 = pack2(-2.f, -2.f);
#pragma unroll
            for (int g = 0; g < 32 / CK; ++g) {
                float sc[CK];
#pragma unroll
                for (int h = 0; h < CK; h += 2)      // ncp[c] = +inf past K
                    unpack2(ffma2(m2, pack2(v[CK * g + h], v[CK * g + h + 1]),
                                  pack2(ncv[CK * g + h], ncv[CK * g + h + 1])),
                            sc[h], sc[h + 1]);
                top2_chunks(min4(sc[0], sc[1], sc[2], sc[3]), gb + g, b1, b2, i1);
            }
        }
        tc_fence_before();
        __syncthreads();                         // the accumulator is free again
        if (s_fail) { ok = false; break; }
        if (t + 1 == tiles) {
            // the partition is done: merge the column groups of each row, in
            // column order
            if (cgrp > 0) {
                s_b1[cgrp - 1][row] = b1;
                s_b2[cgrp - 1][row] = b2;
                s_i1[cgrp - 1][row] = i1;
            }
            __syncthreads();
            if (cgrp == 0 && i < n) {
                // the lower index wins equal screened values; equal values are
                // a near tie anyway and go to the exact re-check
                float w1 = b1, w2 = b2;
                int wi = i1;
#pragma unroll
                for (int q = 0; q < kTColGroups - 1; ++q) {
                    const float o1 = s_b1[q][row], o2 = s_b2[q][row];
                    if (o1 < w1) {
                        w2 = fminf(w1, o2);
                        w1 = o1;
                        wi = s_i1[q][row];
                    } else {
                        w2 = fminf(w2, o1);
                    }
                }
                const float inf = __int_as_float(0x7f800000), cm2 = cmax2[p];
                constexpr int CK = kTcChunk;
                // inside the chunk: direct float32 distances, within (D + 2)
                // 2^-24 of the reference's (relative), so the least is
                // certain when the next is beyond four times that
                const int64_t row0 = (int64_t)p * kmax;
                float xv[DM], cv[DM];
                load_row<DM, VEC>(X + i * D, D, xv);
                float bd = inf, bd2 = inf;
                int w = -1;
#pragma unroll
                for (int c = 0; c < CK; ++c) {
                    if (CK * wi + c >= kk[p]) break;
                    load_row<DM, VEC>(C + (row0 + CK * wi + c) * D, D, cv);
                    const float d32 = screen_dist<DM>(xv, cv, DM);
                    w = d32 < bd ? CK * wi + c : w;
                    bd2 = fminf(bd2, fmaxf(bd, d32));
                    bd = fminf(bd, d32);
                }
                const float thr = __fadd_ru(__fmul_ru(bd, 1.f + 4.f * (float)(D + 2) * 5.9604645e-8f),
                                            1e-38f);
                const int64_t o = (int64_t)p * n + i;
                // No column outside the chunk comes before w either, when the
                // least of their screened distances, w2 + |x|^2, is beyond w's
                // by more than its error: column c's is within e(c) = E/2
                // (|x|^2 + |c|^2) of the exact one, and a c* that the exact
                // arithmetic could rank at or before w has |x - c*|^2 <= thr,
                // so |c*| <= |x| + sqrt(thr), and at most the partition's
                // largest norm.  (The bound is taken 5% wide for the rounding
                // of w2 + |x|^2, at most 2^-24 of 2 (|x|^2 + |c*|^2) where 5%
                // of e(c*) are 2.5 2^-24 of half of that or more, with an
                // absolute part for products that underflow: 6 D of them,
                // below 2^-126 each.)
                const float rc = sqrtf(xn) + sqrtf(thr);
                const float bound = 0.525f * E * (xn + fminf(rc * rc, cm2)) + 1e-35f;
                if (w2 + xn > __fadd_ru(thr, bound) && bd2 > thr && w >= 0 && cm2 == cm2) {
                    load_row<DM, VEC>(C + (row0 + w) * D, D, cv);
                    labels[o] = w;
                    dists[o] = (float)exact_dist<DM>(xv, cv, D);
                } else {
                    amb[atomicAdd(namb, 1)] = (int32_t)o;
                }
            }
            b1 = b2 = __int_as_float(0x7f800000);
            i1 = 0;
        }
        p = pn;
        t = tn;
        if (tn == 0 && pn < P) tiles = ntiles(pn);
    }
    if (!ok && issuer) {
        // leave no copy or MMA writing into this CTA's memory (bounded waits)
        if (pend >= 0) mbar_wait(&bar_b[pend], ph_b[pend]);
        if (mma_ph >= 0) mbar_wait(&bar_mma, (uint32_t)mma_ph);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(kTmemCols));
}

__device__ __forceinline__ void exact_label_point(const float *__restrict__ X, int32_t n, int32_t D,
                                                  const float *__restrict__ C,
                                                  const int32_t *__restrict__ kk, int32_t kmax,
                                                  int64_t o, int32_t *labels, float *dists)
{
    const int64_t p = o / n, i = o - p * n;
    const int K = kk[p];
    const float *x = X + i * D;
    const float *Cp = C + p * kmax * D;
    double best = 0.0;
    int bl = 0;
    for (int k = 0; k < K; ++k) {
        double dist = 0.0;
        for (int d = 0; d < D; ++d) {
            const float diff = __fsub_rn(x[d], Cp[(int64_t)k * D + d]);
            dist = __dadd_rn(dist, (double)__fmul_rn(diff, diff));
        }
        if (k == 0 || dist < best) {
            best = dist;
            bl = k;
        }
    }
    labels[o] = bl;
    dists[o] = (float)best;
}

// if a tile gave up waiting, relabel every active point with the exact loop
// (never expected; keeps the result correct and the error reported)
__global__ void k_exact_all(const float *__restrict__ X, int32_t n, int32_t D,
                            const float *__restrict__ C, const int32_t *__restrict__ kk,
                            int32_t kmax, int32_t P, const int32_t *active, const int *err,
                            int32_t *labels, float *dists)
{
    if (*err == 0) return;
    for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < (int64_t)P * n;
         o += (int64_t)gridDim.x * blockDim.x)
        if (active[o / n]) exact_label_point(X, n, D, C, kk, kmax, o, labels, dists);
}

// The reference's distance sum_d (double) fl(fl(x_d - c_d)^2) and the FP32
// sum of the same squares by fused multiply-adds differ by at most (D + 2)
// 2^-24 of either (the squares round once, the chain once per term; the
// double sum adds < D 2^-53), plus subnormal rounding far below 1e-38.  So
// every centroid that can hold the reference's minimum -- and every one tied
// with it -- has an FP32 sum within (1 + 4 (D + 2) 2^-24) of the smallest
// FP32 sum, with a factor 2 to spare.
constexpr int kExactThreads = 256;
constexpr int kExactCacheK = 2048;     // FP32 sums kept in shared memory up to this k

// One warp per ambiguous point, lane l over centroids l, l + 32, ...: an FP32
// pass finds the smallest sum (keeping each sum in shared memory when k is at
// most kExactCacheK), a second pass evaluates the reference's arithmetic only
// for the centroids within the bound above, and the warp keeps the smallest
// distance, the smallest index among equal ones (the reference loop's first
// minimum).
template <int DM, bool VEC>
__global__ void __launch_bounds__(kExactThreads)
k_label_exact_tc(const float *__restrict__ X, int32_t n, int32_t D, const float *__restrict__ C,
                 const int32_t *__restrict__ kk, int32_t kmax, int32_t P,
                 const int32_t *__restrict__ amb, const int *__restrict__ namb,
                 const int *__restrict__ err, int32_t *labels, float *dists)
{
    extern __shared__ float s_sum[];
    if (err && *err != 0) return;               // k_exact_all did every point
    const int64_t cap = (int64_t)P * n;
    const int m = (int)min((int64_t)*namb, cap);
    const float grow = 1.f + 4.f * (float)(D + 2) * 5.9604645e-8f;     // 2^-24
    const bool cached = kmax <= kExactCacheK;
    float *mine = s_sum + (threadIdx.x >> 5) * (cached ? kmax : 0);
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < m; t += nw) {
        const int64_t o = amb[t];
        const int64_t p = o / n, i = o - p * n;
        const int K = kk[p];
        float xv[DM], cv[DM];
        load_row<DM, VEC>(X + i * D, D, xv);
        const float *Cp = C + p * kmax * D;
        float mn = __int_as_float(0x7f800000);
        for (int k = lane; k < K; k += 32) {
            load_row<DM, VEC>(Cp + (int64_t)k * D, D, cv);
            const float d32 = screen_dist<DM>(xv, cv, D);
            if (cached) mine[k] = d32;
            mn = fminf(mn, d32);
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, off));
        const float thr = __fadd_ru(__fmul_ru(mn, grow), 1e-38f);
        double best = 0.0;
        int bl = 0x7fffffff, nan0 = 0;
        for (int k = lane; k < K; k += 32) {
            float d32;
            if (cached) {
                d32 = mine[k];
            } else {
                load_row<DM, VEC>(Cp + (int64_t)k * D, D, cv);
                d32 = screen_dist<DM>(xv, cv, D);
            }
            if (d32 > thr) continue;
            load_row<DM, VEC>(Cp + (int64_t)k * D, D, cv);
            const double dist = exact_dist<DM>(xv, cv, D);
            // a NaN never compares as smaller, so the reference keeps one
            // only from centroid 0, and then to the end
            if (dist != dist) {
                if (k == 0) nan0 = 1;
                continue;
            }
            if (bl == 0x7fffffff || dist < best) {
                best = dist;
                bl = k;
            }
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, off);
            const int ok = __shfl_xor_sync(0xffffffffu, bl, off);
            if (ok != 0x7fffffff && (bl == 0x7fffffff || ob < best || (ob == best && ok < bl))) {
                best = ob;
                bl = ok;
            }
        }
        if (lane == 0) {
            labels[o] = nan0 ? 0 : bl;
            dists[o] = nan0 ? __int_as_float(0x7fffffff) : (float)best;
        }
        __syncwarp();                           // the sums are rewritten by the next point
    }
}

TcScratch TcScratch::carve(Carver &c, int32_t n, int32_t D, int32_t P, int32_t kmax)
{
    TcScratch s;
    s.Kp = ((6 * D + 15) / 16) * 16;
    s.n_pad = ((int64_t)n + kTM - 1) / kTM * kTM;
    s.kt_max = (kmax + kTN - 1) / kTN;
    s.A = c.take<uint8_t>((size_t)s.n_pad * s.Kp * 2);
    s.nx = c.take<float>((size_t)s.n_pad);
    s.B = c.take<uint8_t>((size_t)P * s.kt_max * kTN * s.Kp * 2);
    s.nc = c.take<float>((size_t)P * s.kt_max * kTN);
    s.cmax2 = c.take<float>((size_t)P + 2);
    s.nblk = (int *)(s.cmax2 + P);
    s.namb = s.nblk + 1;
    s.blk = c.take<int32_t>((size_t)P * (((int64_t)n + kLabelPts - 1) / kLabelPts));
    s.mu = c.take<float>(32);
    s.part = c.take<double>((size_t)32 * kMeanBlocks);
    s.err = c.take<int>(1);
    s.points_ready = s.mean_ready = false;
    return s;
}

int label_exact_points(const float *X, int32_t n, int32_t D, int32_t P, const float *C,
                       const int32_t *kk, int32_t kmax, int32_t *labels, float *dists,
                       const int32_t *amb, const int *namb, const int *err, cudaStream_t st)
{
    const size_t esmem = kmax <= kExactCacheK
                             ? (size_t)(kExactThreads / 32) * kmax * sizeof(float) : 0;
    int es = EACB_OK;
    auto exact = [&](auto kern) {
        if (esmem > 48 * 1024 && allow_max_dyn_smem(kern) != cudaSuccess)
            es = EACB_ERR_CUDA;
        else
            kern<<<148 * 8, kExactThreads, esmem, st>>>(X, n, D, C, kk, kmax, P, amb, namb, err,
                                                        labels, dists);
    };
    // 16-byte row loads when every row is exactly DM floats on a 16-byte boundary
    const bool al = ((uintptr_t)X % 16 == 0) && ((uintptr_t)C % 16 == 0);
    if (D == 4 && al) exact(k_label_exact_tc<4, true>);
    else if (D <= 4) exact(k_label_exact_tc<4, false>);
    else if (D == 8 && al) exact(k_label_exact_tc<8, true>);
    else if (D <= 8) exact(k_label_exact_tc<8, false>);
    else if (D == 16 && al) exact(k_label_exact_tc<16, true>);
    else if (D <= 16) exact(k_label_exact_tc<16, false>);
    else if (D == 32 && al) exact(k_label_exact_tc<32, true>);
    else exact(k_label_exact_tc<32, false>);
    if (es) return es;
    EACB_CHECK_LAUNCH();
    return EACB_OK;
}

int label_pass_tc(const float *X, int32_t n, int32_t D, int32_t P, const float *C,
                  const int32_t *kk, int32_t kmax, const int32_t *active, int32_t *labels,
                  float *dists, int32_t *amb, TcScratch &s, cudaStream_t st)
{
    if (!s.points_ready) {
        int r = data_mean(X, n, D, s, st);
        if (r) return r;
        k_prep_points<<<grid_for(s.n_pad, 128), 128, 0, st>>>(X, n, D, s.Kp, s.mu, s.A, s.nx,
                                                              s.n_pad);
        EACB_CHECK_LAUNCH();
        s.points_ready = true;
    }
    EACB_CUDA(cudaMemsetAsync(s.cmax2, 0, sizeof(float) * ((size_t)P + 2), st));   // and namb
    k_prep_centroids<<<grid_for((int64_t)P * s.kt_max * kTN, 128), 128, 0, st>>>(
        C, kk, kmax, P, D, s.Kp, s.kt_max, s.mu, active, s.B, s.nc, s.cmax2);
    EACB_CHECK_LAUNCH();
    // Error model of the screened distance, doubled for margin.  The dot
    // product: the three-way split drops < 3 * 2^-24 |x||c|; the MMA adds
    // the h*h group last, so its accumulation error is at most
    // (16 ceil(D/16) + 3) 2^-23 of sum|x_d c_d| (<= |x||c|), the earlier,
    // 2^8-times smaller groups add less than one more 2^-23.  Norms and the
    // epilogue: (D + 6) 2^-24 of |x|^2 + |c|^2.  With 2|x||c| <= |x|^2 +
    // |c|^2 the screened distance is within E (|x|^2 + max|c|^2) / 2.
    const double dot_err = 3.0 * ldexp(1.0, -24) +
                           (16.0 * ((D + 15) / 16) + 4.0) * ldexp(1.0, -23);
    const float E = 2.f * (float)(dot_err + (D + 6) * ldexp(1.0, -24));
    const size_t a_bytes = (size_t)kTM * s.Kp * 2, b_bytes = (size_t)kTN * s.Kp * 2;
    // CTAs per SM (each holds 128 TMEM columns): four by default, fewer when
    // their operand tiles do not fit four to an SM
    int ctas = (int)tune_get(TUNE_TC_CTAS_PER_SM, D, n, 4);
    ctas = ctas >= 4 ? 4 : (ctas >= 2 ? 2 : 1);
    while (ctas > 1 && a_bytes + b_bytes > (size_t)(220 / ctas) * 1024) ctas /= 2;
    const size_t cap_bytes = (size_t)(220 / ctas) * 1024;
    int nbuf = (a_bytes + 2 * b_bytes <= cap_bytes) ? 2 : 1;
    nbuf = (int)std::min<int64_t>(nbuf, std::max<int64_t>(1, tune_get(TUNE_TC_BUFFERS, D, n, nbuf)));
    const size_t smem = a_bytes + nbuf * b_bytes;
    // a floor on the request so that no more CTAs than asked share an SM
    const size_t floor_bytes = (size_t)(228 / (ctas + 1) + 2) * 1024;
    const size_t smem_req = smem < floor_bytes ? floor_bytes : smem;
    // one CTA per 128-point tile and share of the partitions: all partitions
    // (the tile's operands load once) unless that leaves fewer than two
    // CTAs per SM slot in flight
    const int64_t ptiles = s.n_pad / kTM;
    const int64_t want = 2 * 148 * ctas;
    const int groups = (int)std::min<int64_t>(P, std::max<int64_t>(1, (want + ptiles - 1) / ptiles));
    const int ppc = (P + groups - 1) / groups;
    dim3 grid((unsigned)ptiles, (unsigned)((P + ppc - 1) / ppc));
    ProfScope ps(PROF_KMEANS, st);
    cudaError_t ce = cudaSuccess;
    auto go = [&](auto kern) {
        if ((ce = allow_max_dyn_smem(kern)) != cudaSuccess) return;
        kern<<<grid, kTThreads, smem_req, st>>>(X, n, D, s.Kp, C, kk, kmax, s.kt_max, P, ppc, active,
                                                s.A, s.nx, s.B, s.nc, s.cmax2, E, nbuf, labels, dists,
                                                amb, s.namb, s.err);
    };
    const bool al = ((uintptr_t)X % 16 == 0) && ((uintptr_t)C % 16 == 0);
    if (D == 4 && al) go(k_label_tc<4, true>);
    else if (D <= 4) go(k_label_tc<4, false>);
    else if (D == 8 && al) go(k_label_tc<8, true>);
    else if (D <= 8) go(k_label_tc<8, false>);
    else if (D == 16 && al) go(k_label_tc<16, true>);
    else if (D <= 16) go(k_label_tc<16, false>);
    else if (D == 32 && al) go(k_label_tc<32, true>);
    else go(k_label_tc<32, false>);
    EACB_CUDA(ce);
    EACB_CHECK_LAUNCH();
    ps.done(0.0);
    k_exact_all<<<296, 256, 0, st>>>(X, n, D, C, kk, kmax, P, active, s.err, labels, dists);
    EACB_CHECK_LAUNCH();
    return label_exact_points(X, n, D, P, C, kk, kmax, labels, dists, amb, s.namb, s.err, st);
}

}  // namespace eacb
