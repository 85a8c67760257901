// Batched K-Means (Lloyd) ensemble generation with the reference's exact
// arithmetic.
//
// Reference: MyML/MyML/cluster/KMeans.py -- fit :117-189, _init_centroids
// :191-201, numba_label / _cu_label_kernel_dists :453-490 / :586-629,
// numba_recompute_centroids :709-754; MyML/MyML/utils/sorting.py:9-47
// (arg_k_select); MyML/MyML/utils/partition.py:88-124 (generateEnsemble).
//
// Exactness: a label is argmin_k of sum_d float64(float32((x_d - c_kd)^2))
// with the first index winning ties, the stored distance is float32 of it,
// centroids are float32(float64(float32 sequential sum) / count), the
// inertia is numpy's float32 pairwise sum of the distances and a partition
// stops early when it changes by at most tol.  The float32 label passes below
// screen all centroids and keep the best two; when the runner-up is outside
// the screening error bound of the winner only the winner's exact distance
// is computed, otherwise the point is re-labelled in the reference's
// arithmetic.  The labels are therefore identical to the reference's for any
// input.
//
// Batching: all P partitions of an ensemble (each with its own k) advance
// together; every kernel takes the partition from its grid and partitions
// that stopped early are skipped on the device.
#include "eacb_common.cuh"
#include "scan_impl.cuh"
#include "members.cuh"
#include "kmeans_common.cuh"

#include <cooperative_groups.h>

#include <type_traits>

namespace eacb {

template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES)
                     : "memory");
}

// ------------------------------------------------- float32 label pass --
// The screen works on data centred near its mean, where |x - c|^2 = |x|^2 +
// 2 (|c|^2 / 2 - x.c): a centroid's score is its half norm less the dot
// product, one fused multiply-add per dimension in the centroid's row order,
// two points at a time (fma.rn.f32x2).  A thread holds 2 NP points in
// registers and reads each centroid row (the half norm, then the values
// negated) from shared memory as a broadcast, a vector ahead of its use.
// Per point the best two chunk minima and the winner's chunk are kept (chunks
// of four or eight centroids); the runner-up inside that chunk is found at
// the end from the same scores.
//
// Error: with S = |x|^2 + |c|^2 (centred, u = 2^-24), centring both sides
// moves the distance by at most 4 u S, the half norm and the chain of D
// products by (3 D + 1) u S, and the reference's own float32 squares by 6 u S:
// a screened distance is within e(c) = (3 D + 12) u S of the reference's.  A
// point whose runner-up is not certainly behind its winner is open: a block's
// few open points go to the exact re-check, a block with many to
// k_label_direct, because S is large against the distances' gaps for all
// points of a blob that lies far from the mean.
//
// Bound by the FMA pipe (half of its cycles) and the shared-memory reads.
// One pass: 500,000 x 16 points, 20 partitions of 530: 20.5 ms with a
// subtract and a multiply-add per dimension and an index per centroid; 6.4
// with scalar row loads and re-reads of the winner's group at the end (a
// lane per row: D loads of 32 sectors each); 3.7 with vector loads, 3.5 with
// chunk minima.  32 dimensions, 10 partitions: 6.3 -> 3.9.  1,000,000 x 2,
// k 1,024: 0.90 -> 0.15 ms.
constexpr int kLT = 128;               // label threads per block

template <int DM> struct LabelRow {
    static constexpr int RF = (DM + 4) & ~3;             // floats of a staged centroid
    static constexpr int CH = 128;                       // centroids per staging buffer
};

// staged centroid rows: the half norm, then -c; rows past k get an infinite
// half norm and never win
template <int DM>
__global__ void k_prep_label_f32(const float *__restrict__ C, const int32_t *__restrict__ kk,
                                 int32_t kmax, int32_t kpad, int32_t P, int32_t D,
                                 const float *__restrict__ mu, const int32_t *__restrict__ active,
                                 float *__restrict__ rows, float *cmax2)
{
    constexpr int RF = LabelRow<DM>::RF;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < (int64_t)P * kpad; e += stride) {
        const int p = (int)(e / kpad), c = (int)(e % kpad);
        if (!active[p]) continue;
        const bool real = c < kk[p];
        float *row = rows + e * RF;
        float nrm = 0.f;
#pragma unroll
        for (int d = 0; d < DM; ++d) {
            const float v = real && d < D ? __fsub_rn(C[((int64_t)p * kmax + c) * D + d], mu[d]) : 0.f;
            nrm = fmaf(v, v, nrm);
            row[1 + d] = -v;
        }
        row[0] = real ? 0.5f * nrm : __int_as_float(0x7f800000);
        // a NaN norm (which no screen may judge) counts only at centroid 0:
        // there the reference keeps it, elsewhere it never compares as smaller
        if (real && (nrm == nrm || c == 0))
            atomicMax(reinterpret_cast<int *>(&cmax2[p]),
                      nrm == nrm ? __float_as_int(nrm) : 0x7fffffff);
    }
}

// The thread's 2 NP points as pairs (point q: i0 + q kLT; past the last one
// its row again, never written), CENTRED less mu with their norms in xn, or
// as they are.
template <int DM, int NP, bool VEC, bool CENTRED>
__device__ __forceinline__ void label_points(const float *__restrict__ X, int32_t n, int32_t D,
                                             int64_t i0, const float *__restrict__ mu,
                                             uint64_t (&x)[DM][NP], float (&xn)[2 * NP])
{
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        float v[2][DM];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t i = min((int64_t)n - 1, i0 + (2 * j + h) * kLT);
            load_row<DM, VEC>(X + i * D, D, v[h]);
            if (CENTRED) xn[2 * j + h] = 0.f;
        }
#pragma unroll
        for (int d = 0; d < DM; ++d) {
            if (CENTRED) {
                const float m = VEC || d < D ? mu[d] : 0.f;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    v[h][d] = __fsub_rn(v[h][d], m);
                    xn[2 * j + h] = fmaf(v[h][d], v[h][d], xn[2 * j + h]);
                }
            }
            x[d][j] = pack2(v[0][d], v[1][d]);
        }
    }
}

// One dimension's part of a score: of the centred rows less the product, of
// the rows as they are (DIRECT) the square of the difference.
template <bool DIRECT>
__device__ __forceinline__ uint64_t score_step2(uint64_t x, uint64_t w, uint64_t acc)
{
    if (!DIRECT) return ffma2(x, w, acc);
    const uint64_t t = fadd2(x, w);
    return ffma2(t, t, acc);
}

// The best two chunk minima of every point's scores and the winner's chunk,
// over K rows; stage(dst, c0) begins to bring rows c0 to c0 + CH - 1 (padded
// to whole chunks) into a buffer.
template <int DM, int NP, int CK, bool DIRECT, typename Stage>
__device__ __forceinline__ void
label_sweep(float (&cs)[2][(LabelRow<DM>::CH + 4) * LabelRow<DM>::RF], int K,
            const uint64_t (&x)[DM][NP], float (&b1)[2 * NP], float (&b2)[2 * NP],
            int (&i1)[2 * NP], Stage stage)
{
    constexpr int RF = LabelRow<DM>::RF, CH = LabelRow<DM>::CH, Q = 2 * NP;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        b1[q] = b2[q] = __int_as_float(0x7f800000);
        i1[q] = 0;
    }
    stage(cs[0], 0);
    int buf = 0;
    for (int c0 = 0; c0 < K; c0 += CH, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                         // this buffer is there, the other one is free
        if (c0 + CH < K) stage(cs[buf ^ 1], c0 + CH);
        const int g1 = min(CH, (K - c0 + CK - 1) / CK * CK) >> 2;    // groups of four
        float cmin[Q];                           // the chunk's least scores
        // the four rows' next 16-byte vectors are read while the current ones
        // are used (past the last group they are read and dropped)
        const float *row = cs[buf];
        float4 f[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) f[c] = *reinterpret_cast<const float4 *>(row + c * RF);
        for (int g = 0; g < g1; ++g, row += 4 * RF) {
            uint64_t acc[4][NP];
#pragma unroll
            for (int v = 0; v < RF / 4; ++v) {
                float4 nx[4];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    nx[c] = *reinterpret_cast<const float4 *>(
                        row + (4 * v + 4 < RF ? c * RF + 4 * v + 4 : (4 + c) * RF));
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int d = 4 * v + k - 1;
                    if (d >= DM) continue;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float e = k == 0 ? f[c].x : k == 1 ? f[c].y : k == 2 ? f[c].z : f[c].w;
                        const uint64_t w = twice(e);
#pragma unroll
                        for (int j = 0; j < NP; ++j)
                            acc[c][j] = d < 0 ? w : score_step2<DIRECT>(x[d < 0 ? 0 : d][j], w, acc[c][j]);
                    }
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) f[c] = nx[c];
            }
            const bool first = CK == 4 || (g & 1) == 0, ends = CK == 4 || (g & 1) == 1;
            const int id = (c0 + 4 * g) / CK;
#pragma unroll
            for (int j = 0; j < NP; ++j) {
                float s[4][2];
#pragma unroll
                for (int c = 0; c < 4; ++c) unpack2(acc[c][j], s[c][0], s[c][1]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int q = 2 * j + h;
                    const float m = min4(s[0][h], s[1][h], s[2][h], s[3][h]);
                    cmin[q] = first ? m : fminf(cmin[q], m);
                    if (ends) top2_chunks(cmin[q], id, b1[q], b2[q], i1[q]);
                }
            }
        }
    }
}

// The block's points without a certain label (open: the thread's), by all its
// threads: up to one in eight go to the list that label_exact_points takes,
// which is a warp and a read of every centroid's row for each.  More stay, and
// the block has to go on with them (false).
template <int Q>
__device__ __forceinline__ bool label_listed(unsigned open, int64_t o0, int *s_open, int32_t *amb,
                                             int *namb)
{
    const int mine = (int)__reduce_add_sync(0xffffffffu, (unsigned)__popc(open));
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(s_open, mine);
    __syncthreads();
    if (amb ? *s_open * 8 > Q * kLT : *s_open > 0) return false;
    for (unsigned t = open; t; t &= t - 1u)
        amb[atomicAdd(namb, 1)] = (int32_t)(o0 + (int64_t)(__ffs(t) - 1) * kLT);
    return true;
}

// a certain label and the reference's distance to its centroid
template <int DM, bool VEC>
__device__ __forceinline__ void label_settle(const float *__restrict__ xrow,
                                             const float *__restrict__ crow, int32_t D, int w,
                                             int32_t *label, float *dist)
{
    float xv[DM], cv[DM];
    load_row<DM, VEC>(xrow, D, xv);
    load_row<DM, VEC>(crow, D, cv);
    *label = w;
    *dist = (float)exact_dist<DM>(xv, cv, D);
}

// CK: centroids per chunk; VEC: D equals DM and the rows of X and C can be
// read as vectors
template <int DM, int NP, int CK, bool VEC>
__global__ void __launch_bounds__(kLT, 4)
k_label_f32(const float *__restrict__ X, int32_t n, int32_t D, const float *__restrict__ C,
            const float *__restrict__ rows, const int32_t *__restrict__ kk, int32_t kmax,
            int32_t kpad, const int32_t *__restrict__ active, const float *__restrict__ mu,
            const float *__restrict__ cmax2, float E, int32_t *__restrict__ labels,
            float *__restrict__ dists, int32_t *__restrict__ amb, int *__restrict__ namb,
            int32_t *__restrict__ blk, int *__restrict__ nblk)
{
    constexpr int RF = LabelRow<DM>::RF, CH = LabelRow<DM>::CH, Q = 2 * NP;
    __shared__ __align__(16) float cs[2][(CH + 4) * RF];
    __shared__ int s_open;
    static_assert(CH % CK == 0 && kTcCentPad % CK == 0, "whole chunks");
    const int p = blockIdx.y;
    if (!active[p]) return;
    const int K = kk[p];
    const float inf = __int_as_float(0x7f800000), cmax = cmax2[p];
    const int64_t i0 = (int64_t)blockIdx.x * (Q * kLT) + threadIdx.x;    // point q: i0 + q kLT
    if (threadIdx.x == 0) s_open = 0;
    uint64_t x[DM][NP];
    float xn[Q], b1[Q], b2[Q];
    int i1[Q];
    label_points<DM, NP, VEC, true>(X, n, D, i0, mu, x, xn);
    const float *src = rows + (int64_t)p * kpad * RF;
    label_sweep<DM, NP, CK, false>(cs, K, x, b1, b2, i1, [&](float *dst, int c0) {
        for (int e = threadIdx.x; e < CH * RF / 4; e += kLT)     // kpad is a multiple of CH
            cp_async<16>(dst + 4 * e, src + (int64_t)c0 * RF + 4 * e);
        asm volatile("cp.async.commit_group;" ::: "memory");
    });
    unsigned open = 0;                           // points that are not certain
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int64_t i = i0 + q * kLT;
        if (i >= n) continue;
        // the winner and the runner-up inside its chunk, by the same scores
        const float *rg = src + (int64_t)CK * i1[q] * RF;
        int bi = -1;
        float ncw = 0.f, best = inf;
#pragma unroll
        for (int c = 0; c < CK; ++c) {
            float e[RF];
            load_row<RF, true>(rg + c * RF, RF, e);
            float s = e[0];
#pragma unroll
            for (int d = 0; d < DM; ++d) {
                float v[2];
                unpack2(x[d][q / 2], v[0], v[1]);
                s = fmaf(v[q & 1], e[1 + d], s);
            }
            if (s < best) {
                bi = c;
                ncw = 2.f * e[0];
            }
            b2[q] = fminf(b2[q], fmaxf(best, s));
            best = fminf(best, s);
        }
        const int w = CK * i1[q] + bi;
        // Only a centroid within |x| + sqrt(winner's distance and error) of
        // the origin can be the reference's choice instead of the winner, so
        // its norm -- and with it its error -- is bounded through the
        // winner's distance (capped by the partition's largest norm).  The
        // bound is 1% wide for this arithmetic's rounding, with an absolute
        // part for products that underflow.
        // (A winner whose squared distance may pass the largest float is not
        // judged: the reference's squares are then infinite, and it keeps the
        // first of the centroids that far.)
        const float ew = E * (xn[q] + ncw);
        const float far = xn[q] + 2.f * b1[q] + ew;
        const float rc = sqrtf(xn[q]) + sqrtf(fmaxf(0.f, far));
        const float bound = 1.01f * (ew + E * (xn[q] + fminf(rc * rc, cmax))) + 1e-36f;
        if (2.f * (b2[q] - b1[q]) > bound && bi >= 0 && far < 3e38f && cmax == cmax)
            label_settle<DM, VEC>(X + i * D, C + ((int64_t)p * kmax + w) * D, D, w,
                                  labels + (int64_t)p * n + i, dists + (int64_t)p * n + i);
        else
            open |= 1u << q;
    }
    if (!label_listed<Q>(open, (int64_t)p * n + i0, &s_open, amb, namb) && threadIdx.x == 0)
        blk[atomicAdd(nblk, 1)] = p * (int)gridDim.x + (int)blockIdx.x;
}

// The blocks of k_label_f32 that were left with many open points (pts points
// each, nb blocks per partition): their points lie far from the mean compared
// with the gaps between their centroids, or are tied.  Or every block (blk
// null), where the work is too small for the mean, the centred rows and the
// launches that k_label_f32 needs.  Scores are the float32 squared distances,
// whose error is relative to the distance -- within (D + 2) 2^-24 of the
// reference's -- so a winner is certain when the next is beyond four times
// that.  Where more than one point in eight is open even so (ties; any point
// at all without a list), a last sweep takes every centroid within that bound
// in the reference's arithmetic and order.
//
// Bound by the FMA pipe: an addition and a multiply-add per dimension.  Blobs
// 1,000 standard deviations apart, 500,000 x 16 points, 4 partitions of 530:
// 8.9 ms a pass with a warp per open point, 2.35 now (5.06 with scalar
// differences for every point); 800,000 x 32 in 300: 7.7 -> 1.3.
template <int DM, int NP, bool VEC>
__global__ void __launch_bounds__(kLT, 4)
k_label_direct(const float *__restrict__ X, int32_t n, int32_t D, const float *__restrict__ C,
               const int32_t *__restrict__ kk, int32_t kmax, int32_t P,
               const int32_t *__restrict__ active, int32_t *__restrict__ labels,
               float *__restrict__ dists, int32_t *__restrict__ amb, int *__restrict__ namb,
               const int32_t *__restrict__ blk, const int *__restrict__ nblk, int pts, int nb)
{
    constexpr int RF = LabelRow<DM>::RF, CH = LabelRow<DM>::CH, Q = 2 * NP, CK = 4;
    __shared__ __align__(16) float cs[2][(CH + 4) * RF];
    __shared__ int s_open;
    const float inf = __int_as_float(0x7f800000);
    const float grow = 1.f + 4.f * (float)(D + 2) * 5.9604645e-8f;       // 2^-24
    const int per = pts / (Q * kLT);             // steps per block
    const int64_t steps = (blk ? (int64_t)*nblk : (int64_t)P * nb) * per;
    for (int64_t t = blockIdx.x; t < steps; t += gridDim.x) {
        const int b = blk ? blk[t / per] : (int)(t / per), p = b / nb;
        const int64_t first = (int64_t)(b - p * nb) * pts + (t % per) * (Q * kLT);
        if (first >= n || !active[p]) continue;  // uniform across the block
        const int K = kk[p];
        const int64_t i0 = first + threadIdx.x, o0 = (int64_t)p * n + i0;
        const float *Cp = C + (int64_t)p * kmax * D;
        // rows as in k_prep_label_f32, with a zero for the half norm
        auto stage = [&](float *dst, int c0) {
            const int m = min(CH, (K - c0 + CK - 1) / CK * CK);
            for (int e = threadIdx.x; e < m * RF; e += kLT) {
                const int c = e / RF, d = e % RF - 1;
                const bool real = c0 + c < K;
                float v = real || d >= 0 ? 0.f : inf;
                if (real && d >= 0 && d < D) v = -__ldg(Cp + (int64_t)(c0 + c) * D + d);
                dst[e] = v;
            }
        };
        uint64_t x[DM][NP];
        float b1[Q], b2[Q], thr[Q];
        int i1[Q];
        label_points<DM, NP, VEC, false>(X, n, D, i0, nullptr, x, thr);
        // a NaN centroid 0 keeps every point in the reference: none is certain
        bool nan_first = false;
        for (int d = 0; d < D; ++d) nan_first |= !(__ldg(Cp + d) == __ldg(Cp + d));
        __syncthreads();                         // the last step's rows and count are done with
        if (threadIdx.x == 0) s_open = 0;
        label_sweep<DM, NP, CK, true>(cs, K, x, b1, b2, i1, stage);
        unsigned open = 0;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            // the winner and the runner-up inside its chunk, by the same scores
            int w = -1;
            float best = inf;
#pragma unroll
            for (int c = 0; c < CK; ++c) {
                if (CK * i1[q] + c >= K) break;
                float e[DM], s = 0.f;
                load_row<DM, VEC>(Cp + (int64_t)(CK * i1[q] + c) * D, D, e);
#pragma unroll
                for (int d = 0; d < DM; ++d) {
                    float v[2];
                    unpack2(x[d][q / 2], v[0], v[1]);
                    const float diff = __fsub_rn(v[q & 1], e[d]);
                    s = fmaf(diff, diff, s);
                }
                w = s < best ? CK * i1[q] + c : w;
                b2[q] = fminf(b2[q], fmaxf(best, s));
                best = fminf(best, s);
            }
            // (the absolute part: subnormal squares, D 2^-149 at most)
            thr[q] = __fadd_ru(__fmul_ru(best, grow), 1e-42f);
            if (i0 + q * kLT >= n) continue;
            if (b2[q] > thr[q] && w >= 0 && !nan_first)
                label_settle<DM, VEC>(X + (i0 + q * kLT) * D, Cp + (int64_t)w * D, D, w,
                                      labels + o0 + q * kLT, dists + o0 + q * kLT);
            else
                open |= 1u << q;
        }
        if (label_listed<Q>(open, o0, &s_open, amb, namb)) continue;
        // (a NaN distance never compares as smaller: the reference keeps one
        // only from centroid 0, and then to the end)
        double bd[Q];
        int bl[Q];
        unsigned nan0 = 0;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            bd[q] = 0.0;
            bl[q] = -1;
        }
        for (int c0 = 0; c0 < K; c0 += CH) {
            __syncthreads();
            stage(cs[0], c0);
            __syncthreads();
            const int cn = min(CH, K - c0);
            for (int c = 0; c < cn; ++c) {
                const float *row = cs[0] + c * RF;
                uint64_t acc[NP];
#pragma unroll
                for (int j = 0; j < NP; ++j) acc[j] = 0ull;
#pragma unroll
                for (int d = 0; d < DM; ++d) {
                    const uint64_t w = twice(row[1 + d]);
#pragma unroll
                    for (int j = 0; j < NP; ++j) acc[j] = score_step2<true>(x[d][j], w, acc[j]);
                }
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    float s[2];
                    unpack2(acc[q / 2], s[0], s[1]);
                    if (!((open >> q) & 1u) || s[q & 1] > thr[q]) continue;
                    double dist = 0.0;
#pragma unroll
                    for (int d = 0; d < DM; ++d) {
                        float v[2];
                        unpack2(x[d][q / 2], v[0], v[1]);
                        const float diff = __fadd_rn(v[q & 1], row[1 + d]);
                        dist = __dadd_rn(dist, (double)__fmul_rn(diff, diff));
                    }
                    if (dist != dist) {
                        if (c0 + c == 0) nan0 |= 1u << q;
                    } else if (bl[q] < 0 || dist < bd[q]) {
                        bd[q] = dist;
                        bl[q] = c0 + c;
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            if (!((open >> q) & 1u)) continue;
            const bool nan = ((nan0 >> q) & 1u) != 0u;
            labels[o0 + q * kLT] = nan ? 0 : bl[q];
            dists[o0 + q * kLT] = nan ? __int_as_float(0x7fffffff) : (float)bd[q];
        }
    }
}

// numpy float32 add.reduce of a contiguous array: pairwise summation, blocks
// of at most 128 summed with 8 partial sums; a node longer than 128 splits at
// n/2 rounded down to a multiple of 8 and adds (left, right).
__device__ __forceinline__ float np_pairwise_leaf(const float *a, int64_t n)
{
    if (n < 8) {
        float r = -0.0f;
        for (int64_t i = 0; i < n; ++i) r = __fadd_rn(r, a[i]);
        return r;
    }
    float r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = a[j];
    int64_t i = 8;
    for (; i < n - (n % 8); i += 8)
#pragma unroll
        for (int j = 0; j < 8; ++j) r[j] = __fadd_rn(r[j], a[i + j]);
    float res = __fadd_rn(__fadd_rn(__fadd_rn(r[0], r[1]), __fadd_rn(r[2], r[3])),
                          __fadd_rn(__fadd_rn(r[4], r[5]), __fadd_rn(r[6], r[7])));
    for (; i < n; ++i) res = __fadd_rn(res, a[i]);
    return res;
}

// The split tree's levels are even: nodes of one depth differ by at most 30
// elements, so down to the depth where some node gets short (at most 128)
// every node splits.  Node q of that depth -- the leaf level, up to a second
// split -- is found from the root by q's bits.
__host__ __device__ __forceinline__ void np_split(int64_t len, int64_t &left)
{
    left = len / 2;
    left -= left % 8;
}
// depth of the leaf level: 2^depth nodes (the leftmost path is the shortest)
static inline int np_leaf_depth(int64_t n)
{
    int depth = 0;
    for (int64_t len = n; len > 128; ++depth) np_split(len, len);
    return depth;
}

// Sum of [a, a + n) by eight lanes in numpy's order: lane j holds its partial
// sum r[j], combined pairwise (additions commute), the ragged tail in order.
__device__ __forceinline__ float np_leaf_8(const float *a, int64_t n, unsigned mask)
{
    const int j = threadIdx.x & 7;
    if (n < 8) return np_pairwise_leaf(a, n);
    float r = a[j];
    const int64_t m = n - n % 8;
#pragma unroll 4
    for (int64_t i = 8; i < m; i += 8) r = __fadd_rn(r, a[i + j]);
    r = __fadd_rn(r, __shfl_xor_sync(mask, r, 1));
    r = __fadd_rn(r, __shfl_xor_sync(mask, r, 2));
    r = __fadd_rn(r, __shfl_xor_sync(mask, r, 4));
    for (int64_t i = m; i < n; ++i) r = __fadd_rn(r, a[i]);
    return r;
}

// Inertia, first part: the sums of the leaf level's nodes, eight lanes each
// (their loads share 32-byte sectors).  HBM-bound: the distances are read
// once.  One block per partition summed 256 subtrees of 7,800 elements each
// on one thread: 660 us for 10 x 2,000,000 distances; 29 us here and 18 for
// the levels above.
constexpr int kInertiaThreads = 256;
__global__ void __launch_bounds__(kInertiaThreads)
k_inertia_leaves(const float *dists, int32_t n, const int32_t *active, int depth, float *part)
{
    const int p = blockIdx.y;
    if (!active[p]) return;                    // uniform across the block
    const float *a = dists + (int64_t)p * n;
    const int64_t nodes = (int64_t)1 << depth;
    const unsigned mask = 0xffu << (threadIdx.x & 24);
    const int64_t q = ((int64_t)blockIdx.x * kInertiaThreads + threadIdx.x) >> 3;
    if (q >= nodes) return;                    // uniform across the eight lanes
    int64_t off = 0, len = n;
    for (int b = depth - 1; b >= 0; --b) {
        int64_t left;
        np_split(len, left);
        if ((q >> b) & 1) {
            off += left;
            len -= left;
        } else {
            len = left;
        }
    }
    float s;
    if (len <= 128) {
        s = np_leaf_8(a + off, len, mask);
    } else {
        int64_t left;
        np_split(len, left);
        s = np_leaf_8(a + off, left, mask);
        s = __fadd_rn(s, np_leaf_8(a + off + left, len - left, mask));
    }
    if ((threadIdx.x & 7) == 0) part[(int64_t)p * nodes + q] = s;
}

// Second part: the tree above the leaf level, one block per partition, level
// by level in place, and the convergence test of the iteration
// (KMeans.py:158-180).
__global__ void __launch_bounds__(1024)
k_inertia(float *part, int depth, int32_t *active, float *inertia, int32_t *iters, float tol)
{
    const int p = blockIdx.x;
    if (!active[p]) return;                    // uniform across the block
    float *v = part + ((int64_t)p << depth);
    // a thread's 2^sub consecutive nodes first, then the levels across threads
    const int sub = depth > 10 ? depth - 10 : 0, top = depth - sub;
    __shared__ float s_val[1024];
    const int t = threadIdx.x;
    if (t < (1 << top)) {
        float *m = v + ((int64_t)t << sub);
        for (int d = sub; d > 0; --d)
            for (int q = 0; q < 1 << (d - 1); ++q) m[q] = __fadd_rn(m[2 * q], m[2 * q + 1]);
        s_val[t] = m[0];
    }
    __syncthreads();
    for (int c = 1 << top; c > 1; c >>= 1) {
        float x = 0.f;
        if (t < c / 2) x = __fadd_rn(s_val[2 * t], s_val[2 * t + 1]);
        __syncthreads();
        if (t < c / 2) s_val[t] = x;
        __syncthreads();
    }
    if (t == 0) {
        const float I = s_val[0];
        const float err = fabsf(__fsub_rn(I, inertia[p]));
        inertia[p] = I;
        iters[p] += 1;
        if (err <= tol) active[p] = 0;
    }
}

static int launch_inertia(cudaStream_t st, const float *dists, int32_t n, int32_t P, float *part,
                          int32_t *active, float *inertia, int32_t *iters, float tol)
{
    const int depth = np_leaf_depth(n);
    const int64_t nodes = (int64_t)1 << depth;
    const dim3 grid((unsigned)((nodes * 8 + kInertiaThreads - 1) / kInertiaThreads), (unsigned)P);
    k_inertia_leaves<<<grid, kInertiaThreads, 0, st>>>(dists, n, active, depth, part);
    EACB_CHECK_LAUNCH();
    k_inertia<<<P, 1024, 0, st>>>(part, depth, active, inertia, iters, tol);
    EACB_CHECK_LAUNCH();
    return EACB_OK;
}

// float32 (reference) or float64 sums of each cluster's members in point
// order, one warp per cluster.  The sums are sequential in member order (the
// reference's order), so a cluster's sum is a chain as long as the cluster
// and the largest cluster sets the kernel's time.  All lanes copy the
// members' rows ahead into a ring of staging buffers (cp.async; three
// batches of rows in flight, the batches' member ids further ahead in a ring
// of their own), and lane d adds dimension d from shared memory, where the
// chain is the additions alone.  A pass, against a lane per (cluster,
// dimension) with 16 loads in flight: 2,000,000 x 8, 10 x 1,000 clusters 720
// -> 380 us; 500,000 x 16, 20 x 530 clusters 485 -> 330; 1,000,000 x 2, 1,024
// clusters 165 -> 33.
constexpr int kCentWarps = 4;                     // warps per block
constexpr int kCentRing = 4;                      // row buffers per warp
constexpr int kCentIds = 2 * kCentRing;           // id buffers per warp
constexpr int kCentFloats = 1024;                 // floats per row buffer
constexpr int kCentBatch = 128;                   // members per buffer at most
struct CentStage {
    float row[kCentRing][kCentFloats];
    int32_t id[kCentIds][kCentBatch];
};
constexpr size_t kCentSmem = kCentWarps * sizeof(CentStage);

// CH: floats per copy (4, 2 or 1: the largest that divides D and that X's
// alignment allows)
template <bool F64, int CH>
__global__ void __launch_bounds__(kCentWarps * 32)
k_centroids(const float *__restrict__ X, int32_t D, const int32_t *__restrict__ members,
            const int64_t *__restrict__ S, int32_t K, int64_t ntiles,
            const int32_t *__restrict__ kk, int32_t kmax, const int32_t *__restrict__ active,
            float *C, int32_t *nempty)
{
    extern __shared__ __align__(16) uint8_t cent_smem[];
    const int p = blockIdx.y;
    if (!active[p]) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * kCentWarps + warp;
    if (c >= kk[p]) return;
    CentStage &st = reinterpret_cast<CentStage *>(cent_smem)[warp];
    const int64_t s0 = S[((int64_t)p * K + c) * ntiles], s1 = S[((int64_t)p * K + c + 1) * ntiles];
    const int cnt = (int)(s1 - s0);
    if (cnt == 0) {
        if (lane == 0) atomicAdd(&nempty[p], 1);
        return;
    }
    const int batch = min(kCentBatch, kCentFloats / D);
    const int nb = (cnt + batch - 1) / batch;
    const int32_t *mem = members + s0;
    // a row is `per` copies: lane l takes copy l % per of members l / per, ...
    const int per = D / CH, mstep = 32 / per, m_of = lane / per, ch = (lane - m_of * per) * CH;
    auto ids = [&](int b) {
        if (b >= nb) return;
        const int nm = min(batch, cnt - b * batch);
        for (int m = lane; m < nm; m += 32)
            cp_async<4>(&st.id[b % kCentIds][m], mem + (int64_t)b * batch + m);
    };
    auto rows = [&](int b) {
        if (b >= nb || m_of >= mstep) return;
        const int nm = min(batch, cnt - b * batch);
        const int32_t *id = st.id[b % kCentIds];
        float *buf = st.row[b % kCentRing] + ch;
#pragma unroll 4
        for (int m = m_of; m < nm; m += mstep)
            cp_async<4 * CH>(buf + m * D, X + (int64_t)id[m] * D + ch);
    };
    auto commit = []() { asm volatile("cp.async.commit_group;" ::: "memory"); };
    for (int b = 0; b < kCentRing; ++b) ids(b);
    commit();
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    // group b: the rows of batch b and the ids of batch b + kCentRing
    for (int b = 0; b < kCentRing - 1; ++b) {
        rows(b);
        ids(b + kCentRing);
        commit();
    }
    using Acc = typename std::conditional<F64, double, float>::type;
    Acc acc = 0;
    for (int b = 0; b < nb; ++b) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kCentRing - 2) : "memory");
        __syncwarp();                             // batch b is there; batch b - 1 is summed
        rows(b + kCentRing - 1);
        ids(b + 2 * kCentRing - 1);
        commit();
        const int nm = min(batch, cnt - b * batch);
        if (lane < D) {
            const float *v = st.row[b % kCentRing] + lane;
#pragma unroll 8
            for (int m = 0; m < nm; ++m, v += D) {
                if (F64) acc += (double)*v;
                else acc = (Acc)__fadd_rn((float)acc, *v);
            }
        }
    }
    if (lane >= D) return;
    float *out = C + ((int64_t)p * kmax + c) * D + lane;
    if (F64) *out = __double2float_rn((double)acc / (double)cnt);
    else *out = __double2float_rn(__ddiv_rn((double)acc, (double)cnt));
}

// The same sums with a lane per (cluster, dimension), 32 / D clusters per warp
// and 16 members' loads in flight: for small clusters, whose members fit a few
// of those batches (a warp and its buffers for each of them cost more than the
// sums), and for rows that k_centroids would copy singly.
constexpr int kCentDepth = 16;       // members in flight per lane

template <bool F64>
__global__ void __launch_bounds__(256)
k_centroids_lanes(const float *__restrict__ X, int32_t D, const int32_t *__restrict__ members,
                  const int64_t *__restrict__ S, int32_t K, int64_t ntiles,
                  const int32_t *__restrict__ kk, int32_t kmax, const int32_t *__restrict__ active,
                  float *C, int32_t *nempty)
{
    const int p = blockIdx.y;
    if (!active[p]) return;
    const int lane = threadIdx.x & 31;
    const int G = 32 / D;                       // clusters per warp
    const int g = lane / D, d = lane - g * D;
    const int c = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * G + g;
    if (g >= G || c >= kk[p]) return;
    const int64_t s0 = S[((int64_t)p * K + c) * ntiles], s1 = S[((int64_t)p * K + c + 1) * ntiles];
    const int64_t cnt = s1 - s0;
    if (cnt == 0) {
        if (d == 0) atomicAdd(&nempty[p], 1);
        return;
    }
    using Acc = typename std::conditional<F64, double, float>::type;
    Acc acc = 0;
    auto add = [&](float v) {
        if (F64) acc += (double)v;
        else acc = (Acc)__fadd_rn((float)acc, v);
    };
    // the next batch's ids load while this batch's coordinates do
    int64_t m = s0;
    if (m + kCentDepth <= s1) {
        int32_t id[kCentDepth];
#pragma unroll
        for (int q = 0; q < kCentDepth; ++q) id[q] = members[m + q];
        for (; m + kCentDepth <= s1; m += kCentDepth) {
            float v[kCentDepth];
#pragma unroll
            for (int q = 0; q < kCentDepth; ++q) v[q] = X[(int64_t)id[q] * D + d];
            const bool more = m + 2 * kCentDepth <= s1;
#pragma unroll
            for (int q = 0; q < kCentDepth; ++q) id[q] = more ? members[m + kCentDepth + q] : 0;
#pragma unroll
            for (int q = 0; q < kCentDepth; ++q) add(v[q]);
        }
    }
    for (; m < s1; ++m) add(X[(int64_t)members[m] * D + d]);
    C[((int64_t)p * kmax + c) * D + d] =
        F64 ? __double2float_rn((double)acc / (double)cnt)
            : __double2float_rn(__ddiv_rn((double)acc, (double)cnt));
}

// k_centroids_lanes up to this many points per cluster on average (a pass of
// 50 x 100 clusters, 16 dimensions: 8 points 6 us against 14, 32 points 11
// against 18, 64 points 23 against 25, 256 points 76 against 58), and where a
// copy instruction of k_centroids takes too few rows to keep up with the
// additions: one, or two with float64 sums (a cluster of 92,000 points: 31
// dimensions 3.3 ms against 4.4, float64 2.5 against 4.8).
constexpr int kCentSmall = 48;

static int launch_centroids(cudaStream_t st, bool f64, const float *X, int32_t n, int32_t D,
                            int32_t P, const int32_t *members, const int64_t *S, int32_t K,
                            int64_t ntiles, const int32_t *kk, int32_t kmax, const int32_t *active,
                            float *C, int32_t *nempty)
{
    const int ch = D % 4 == 0 && (uintptr_t)X % 16 == 0 ? 4
                   : D % 2 == 0 && (uintptr_t)X % 8 == 0 ? 2 : 1;
    const int rows = 32 / (D / ch);               // per copy instruction
    if ((int64_t)n < (int64_t)kCentSmall * kmax || rows < (f64 ? 3 : 2)) {
        const int G = 32 / D, warps = (kmax + G - 1) / G;
        const dim3 lg((unsigned)((warps * 32 + 255) / 256), (unsigned)P);
        if (f64)
            k_centroids_lanes<true><<<lg, 256, 0, st>>>(X, D, members, S, K, ntiles, kk, kmax, active,
                                                        C, nempty);
        else
            k_centroids_lanes<false><<<lg, 256, 0, st>>>(X, D, members, S, K, ntiles, kk, kmax, active,
                                                         C, nempty);
        EACB_CHECK_LAUNCH();
        return EACB_OK;
    }
    const dim3 grid((unsigned)((kmax + kCentWarps - 1) / kCentWarps), (unsigned)P);
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kern) {
        if ((e = allow_max_dyn_smem(kern)) != cudaSuccess) return;
        kern<<<grid, kCentWarps * 32, kCentSmem, st>>>(X, D, members, S, K, ntiles, kk, kmax,
                                                       active, C, nempty);
    };
    if (f64) {
        if (ch == 4) go(k_centroids<true, 4>);
        else if (ch == 2) go(k_centroids<true, 2>);
        else go(k_centroids<true, 1>);
    } else {
        if (ch == 4) go(k_centroids<false, 4>);
        else if (ch == 2) go(k_centroids<false, 2>);
        else go(k_centroids<false, 1>);
    }
    EACB_CUDA(e);
    EACB_CHECK_LAUNCH();
    return EACB_OK;
}

// Empty clusters take the points arg_k_select returns for their number
// (KMeans.py:727-750, MyML/MyML/utils/sorting.py:9-47): the reference's
// quickselect on (distance, index) pairs, one thread-block cluster per
// partition, with the distances permuted in place (key[r] is the reference's
// a[args[r]]; the distances are not needed again before the next label pass).
//
// One partition step of the reference on [lo, hi] with pivot mid moves the
// element at r to the back (swapping in the element at w) when it is >= mid,
// and otherwise advances r.  Its result has a closed form that a cluster can
// compute in parallel.  Count positions t from lo; "big" means >= mid, NS is
// the number of the others ("small").  The step reads the range from the
// front and from the back, and the two readings meet behind position x: x is
// NS - 1 when the element at position NS is small (or there is none), else
// NS.  The element read last is the one at x (read from the front) when that
// completes the reading, else the one at x + 1:
//   x = NS - 1: at x when it is small, else at x + 1;
//   x = NS:     at x when x is the end or the element at x + 1 is small,
//               else at x + 1.
// It stays at r.  With A the bigs at positions <= x (from the front) and B
// the smalls behind x (from the back), every other element lands at:
//   a front small           -> its own position,
//   the m-th front big      -> one before B's (m-1)-th position (the end for m = 1),
//   the m-th back small     -> A's m-th position,
//   a back big              -> one position further front,
// and r = lo + NS, less one if the last element is small.
//
// The reference goes on in [lo, r] when its target k is at most r, and only
// those positions are read again: then the step is just "B's m-th element
// replaces A's m-th" (k is the number of empty clusters, so nearly every step
// is one).  Otherwise all elements move.
//
// Bound by the passes over the range (two reads of the keys and one of the
// lists, halving from step to step) and a cluster barrier between them: with
// one block per partition and all elements moved in each step a 2,000,000
// point partition took 18.4 ms, all of it one SM; eight blocks take 0.77 ms.
// Ranges up to kFillSeqMax elements finish with the reference's loop on one
// thread in shared memory.
constexpr int kFillThreads = 1024;
constexpr int kFillItems = 8;
constexpr int kFillTile = kFillThreads * kFillItems;
constexpr int kFillSeqMax = 256;
// steps of that loop at most.  A step whose pivot is the least of the range
// only rotates the range by one place, so the range may stand still while
// copies of that value pass the middle (fewer than its length) before it
// shrinks: at most length x length steps (two values, 256 keys: 257).
constexpr int kFillSeqSteps = kFillSeqMax * kFillSeqMax;
constexpr int kFillRounds = 1 << 15;     // steps shrink the range; equal keys take one per cluster
// blocks per partition: a cluster from this many points on (below, one
// block's passes cost no more than the cluster's barriers)
constexpr int kFillCluster = 8;
constexpr int kFillClusterMin = 16384;

// Walks [t0, t1) in ascending tiles, calling f(t, big, before) for every
// position; before packs the front bigs (high half) and back smalls (low
// half) of the walk before t, on top of `base`.  x splits front and back.
template <typename F>
__device__ __forceinline__ void fill_walk(const float *key, int t0, int t1, float mid, int x,
                                          int64_t base, F f)
{
    for (int64_t b = t0; b < t1; b += kFillTile) {
        const int64_t p0 = b + (int64_t)threadIdx.x * kFillItems;
        unsigned mask = 0;
        int64_t c = 0;
#pragma unroll
        for (int q = 0; q < kFillItems; ++q) {
            const int64_t t = p0 + q;
            if (t < t1) {
                const bool big = key[t] >= mid;
                mask |= (big ? 1u : 0u) << q;
                c += big ? (t <= x ? (1ll << 32) : 0ll) : (t > x ? 1ll : 0ll);
            }
        }
        int64_t tot;
        int64_t before = base + block_excl_sum_shfl<kFillThreads>(c, tot);
#pragma unroll
        for (int q = 0; q < kFillItems; ++q) {
            const int64_t t = p0 + q;
            if (t < t1) {
                const bool big = (mask >> q) & 1u;
                f((int)t, big, before);
                before += big ? (t <= x ? (1ll << 32) : 0ll) : (t > x ? 1ll : 0ll);
            }
        }
        base += tot;
    }
}

// smalls among [t0, t1), summed over the block
__device__ __forceinline__ int fill_smalls(const float *key, int t0, int t1, float mid)
{
    int c = 0;
#pragma unroll 8
    for (int64_t t = (int64_t)t0 + threadIdx.x; t < t1; t += kFillThreads) c += !(key[t] >= mid);
    int64_t tot;
    block_excl_sum_shfl<kFillThreads>(c, tot);
    return (int)tot;
}

__global__ void __launch_bounds__(kFillThreads, 1)
k_fill_empty(const float *X, int32_t n, int32_t D, float *dists, const int64_t *S, int32_t K,
             int64_t ntiles, const int32_t *kk, int32_t kmax, const int32_t *active,
             const int32_t *nempty, int32_t *args_all, int32_t *sel_all, float *okey_all,
             int32_t *oarg_all, float *C, int *err)
{
    namespace cg = cooperative_groups;
    const cg::cluster_group cl = cg::this_cluster();
    const int CL = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    // (a block alone: with many equal keys a step settles one point and is
    // mostly its barriers; 16,000 points of four distances, 984 empty clusters
    // 16.6 ms with cluster barriers, 12.7 with the block's)
    auto sync = [&]() {
        if (CL > 1) cl.sync();
        else __syncthreads();
    };
    __shared__ int s_small[2], s_fb[2], s_bs[2];       // this block's counts, by step parity
    __shared__ float s_key[kFillSeqMax];
    __shared__ int32_t s_arg[kFillSeqMax];
    const int p = (int)blockIdx.x / CL;
    if (!active[p] || nempty[p] == 0) return;          // uniform across the cluster
    const int k = nempty[p];
    float *key0 = dists + (int64_t)p * n;
    int32_t *args0 = args_all + (int64_t)p * n;
    int32_t *sel = sel_all + (int64_t)p * n;           // positions of A, then of B
    const int gt = rank * kFillThreads + (int)threadIdx.x, gs = CL * kFillThreads;
    for (int64_t i = gt; i < n; i += gs) args0[i] = (int32_t)i;
    sync();
    int lo = 0, hi = n - 1;
    for (int step = 0; hi - lo + 1 > kFillSeqMax; ++step) {
        if (step > kFillRounds) {                      // a NaN pivot does not shrink the range
            if (gt == 0) set_err(err, DEV_CHASE_LIMIT);
            return;
        }
        const int L = hi - lo + 1, ph = step & 1;
        float *key = key0 + lo;
        int32_t *args = args0 + lo;
        const float mid = key[(int)(((int64_t)lo + hi) / 2 - lo)];
        const int cs = (L + CL - 1) / CL;
        const int c0 = (int)min((int64_t)L, (int64_t)rank * cs);
        const int c1 = (int)min((int64_t)L, (int64_t)c0 + cs);
        // the smalls of the range
        const int mine = fill_smalls(key, c0, c1, mid);
        if (threadIdx.x == 0) s_small[ph] = mine;
        sync();
        int NS = 0;
        for (int q = 0; q < CL; ++q) NS += *cl.map_shared_rank(&s_small[ph], q);
        // where the two readings meet and which element is read last
        const bool has = NS < L && key[NS] >= mid;     // a big at position NS
        const int x = NS == L ? L - 1 : (has ? NS : NS - 1);
        bool at_x;
        if (NS == L) at_x = true;
        else if (!has) at_x = x >= 0 && !(key[x] >= mid);
        else at_x = x == L - 1 || !(key[x + 1] >= mid);
        const int last = at_x ? x : x + 1;
        const float klast = key[last];
        const int32_t alast = args[last];
        const int Sm = NS - (klast >= mid ? 0 : 1);
        const int r = lo + Sm - (klast > mid ? 1 : 0);
        // front bigs and back smalls before each block's share
        int fb = 0, bs = 0;
        if (c1 <= x + 1) {
            fb = (c1 - c0) - mine;
        } else if (c0 > x) {
            bs = mine;
        } else {
            const int sf = fill_smalls(key, c0, x + 1, mid);
            fb = (x + 1 - c0) - sf;
            bs = mine - sf;
        }
        if (threadIdx.x == 0) {
            s_fb[ph] = fb;
            s_bs[ph] = bs;
        }
        sync();
        int64_t base = 0;
        int nA = 0, M = 0;
        for (int q = 0; q < CL; ++q) {
            const int f = *cl.map_shared_rank(&s_fb[ph], q), b = *cl.map_shared_rank(&s_bs[ph], q);
            if (q < rank) base += ((int64_t)f << 32) + b;
            nA += f;
            M += b;
        }
        fill_walk(key, c0, c1, mid, x, base, [&](int t, bool big, int64_t before) {
            if (t <= x) {
                if (big) sel[before >> 32] = t;
            } else if (!big) {
                sel[nA + M - 1 - (int)(before & 0xffffffffll)] = t;
            }
        });
        sync();
        if (k <= r) {
            for (int64_t m = gt; m < M; m += gs) {
                const int a = sel[m], b = sel[nA + m];
                key[a] = key[b];
                args[a] = args[b];
            }
            if (gt == 0 && r == lo + NS && !at_x) {    // it equals mid and comes from x + 1
                key[NS] = klast;
                args[NS] = alast;
            }
            hi = r;
        } else {
            float *okey = okey_all + (int64_t)p * n + lo;
            int32_t *oarg = oarg_all + (int64_t)p * n + lo;
            fill_walk(key, c0, c1, mid, x, base, [&](int t, bool big, int64_t before) {
                int dst;
                if (t == last) dst = Sm;
                else if (t <= x) {
                    const int m = (int)(before >> 32);           // front bigs before
                    dst = !big ? t : (m == 0 ? L : sel[nA + m - 1]) - 1;
                } else {
                    dst = big ? t - 1 : sel[M - 1 - (int)(before & 0xffffffffll)];
                }
                okey[dst] = key[t];
                oarg[dst] = args[t];
            });
            sync();
            for (int64_t t = gt; t < L; t += gs) {
                key[t] = okey[t];
                args[t] = oarg[t];
            }
            lo = r + 1;
        }
        sync();
    }
    if (rank != 0) return;
    const int L = hi - lo + 1;
    for (int t = (int)threadIdx.x; t < L; t += kFillThreads) {
        s_key[t] = key0[lo + t];
        s_arg[t] = args0[lo + t];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int a = 0, b = L - 1, steps = 0;
        while (a < b) {
            if (++steps > kFillSeqSteps) {             // a NaN pivot does not shrink the range
                set_err(err, DEV_CHASE_LIMIT);
                break;
            }
            int r = a, w = b;
            const float mid = s_key[(int)((2 * (int64_t)lo + a + b) / 2 - lo)];
            float kr = s_key[r];
            while (r < w) {
                if (kr >= mid) {
                    const float kw = s_key[w];
                    const int32_t t = s_arg[w];
                    s_key[w] = kr;
                    s_arg[w] = s_arg[r];
                    s_key[r] = kw;
                    s_arg[r] = t;
                    kr = kw;
                    w--;
                } else {
                    kr = s_key[++r];
                }
            }
            if (s_key[r] > mid) r--;
            if (k <= lo + r) b = r; else a = r + 1;
        }
    }
    __syncthreads();
    for (int t = (int)threadIdx.x; t < L; t += kFillThreads) args0[lo + t] = s_arg[t];
    __syncthreads();
    // the empty clusters, in order, take the points of args[0, k)
    const int Kp = kk[p];
    int e = 0;
    for (int b = 0; b < Kp; b += kFillThreads) {
        const int c = b + (int)threadIdx.x;
        const bool empty = c < Kp && S[((int64_t)p * K + c + 1) * ntiles] == S[((int64_t)p * K + c) * ntiles];
        int64_t tot;
        const int at = e + (int)block_excl_sum_shfl<kFillThreads>(empty, tot);
        if (empty) {
            const int32_t src = args0[at];
            for (int d = 0; d < D; ++d) C[((int64_t)p * kmax + c) * D + d] = X[(int64_t)src * D + d];
        }
        e += (int)tot;
    }
}

static int launch_fill_empty(cudaStream_t st, const float *X, int32_t n, int32_t D, int32_t P,
                             float *dists, const int64_t *S, int32_t K, int64_t ntiles,
                             const int32_t *kk, int32_t kmax, const int32_t *active,
                             const int32_t *nempty, int32_t *args, int32_t *sel, float *okey,
                             int32_t *oarg, float *C, int *err)
{
    const unsigned cl = n >= kFillClusterMin ? kFillCluster : 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)P * cl);
    cfg.blockDim = dim3(kFillThreads);
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = cl;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    EACB_CUDA(cudaLaunchKernelEx(&cfg, k_fill_empty, X, n, D, dists, S, K, ntiles, kk, kmax, active,
                                 nempty, args, sel, okey, oarg, C, err));
    EACB_CHECK_LAUNCH();
    return EACB_OK;
}

__global__ void k_init_centroids(const float *X, int32_t D, const int32_t *init, const int32_t *kk,
                                 int32_t kmax, int32_t P, float *C, int32_t *active, float *inertia,
                                 int32_t *iters, int32_t n, int *err)
{
    const int64_t total = (int64_t)P * kmax * D;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = e / ((int64_t)kmax * D);
        const int64_t r = e - p * kmax * D;
        const int c = (int)(r / D), d = (int)(r % D);
        if (c >= kk[p]) continue;
        const int32_t src = init[p * kmax + c];
        if (src < 0 || src >= n) { set_err(err, DEV_BAD_INPUT); continue; }
        C[e] = X[(int64_t)src * D + d];
        if (c == 0 && d == 0) {
            active[p] = 1;
            inertia[p] = __int_as_float(0x7f800000);
            iters[p] = 0;
        }
    }
}

struct KMWS {
    int *err;
    float *dists;
    int32_t *active, *iters, *nempty, *amb;
    float *inertia;
    int32_t *members, *mypos, *cnt, *args;
    int64_t *S;
    int32_t *ncl, *order;
    int *maxsize;
    ScanScratch scan;
    TcScratch tc;
    int64_t ntiles;
    static KMWS carve(Carver &c, int32_t n, int32_t D, int32_t P, int32_t kmax)
    {
        KMWS w;
        w.err = c.take<int>(1);
        const int64_t pn = (int64_t)P * n;
        w.ntiles = ((int64_t)n + kMLTile - 1) / kMLTile;
        const int64_t m = (int64_t)P * kmax * w.ntiles;
        w.dists = c.take<float>(pn);
        w.active = c.take<int32_t>(P);
        w.iters = c.take<int32_t>(P);
        w.nempty = c.take<int32_t>(P);
        w.inertia = c.take<float>(P);
        w.amb = c.take<int32_t>(pn);
        w.members = c.take<int32_t>(pn);
        w.mypos = c.take<int32_t>(pn);
        w.args = c.take<int32_t>(pn);
        w.cnt = c.take<int32_t>(m + 1);
        w.S = c.take<int64_t>(m + 1);
        w.ncl = c.take<int32_t>(P);
        w.order = c.take<int32_t>(P);
        w.maxsize = c.take<int>(1);
        w.scan = ScanScratch::carve(c, m + 1, w.err);
        w.tc = TcScratch::carve(c, n, D, P, kmax);
        w.tc.err = w.err;         // tensor-core failures report through the same word
        return w;
    }
};

// few: k_label_direct alone, for every point
template <int DM, int NP, int CK>
static int launch_label(cudaStream_t st, bool few, const float *X, int32_t n, int32_t D, int32_t P,
                        const float *C, const int32_t *kk, int32_t kmax, const int32_t *active,
                        int32_t *labels, float *dists, int32_t *amb, const TcScratch &s)
{
    constexpr int ND = NP < 2 ? NP : 2;           // (k_label_direct has no registers for more)
    static_assert(kTcCentPad % LabelRow<DM>::CH == 0, "whole staging buffers of rows");
    constexpr int pts = 2 * NP * kLT;
    static_assert(pts >= kLabelPts, "the block list is sized for blocks of that many points");
    const int nb = (n + pts - 1) / pts;
    // rows as vectors where their length and place allow it
    const uintptr_t at = (uintptr_t)X | (uintptr_t)C;
    const bool vec = D == DM && at % (DM % 4 == 0 ? 16 : 8) == 0;
    ProfScope ps(PROF_KMEANS, st);
    if (!few) {
        const int32_t kpad = (int32_t)s.kt_max * kTcCentPad;
        if (LabelRow<DM>::RF * sizeof(float) > (size_t)2 * s.Kp) return EACB_ERR_INTERNAL;
        float *rows = reinterpret_cast<float *>(s.B);
        k_prep_label_f32<DM><<<grid_for((int64_t)P * kpad, 128), 128, 0, st>>>(
            C, kk, kmax, kpad, P, D, s.mu, active, rows, s.cmax2);
        EACB_CHECK_LAUNCH();
        const float E = (float)((3 * D + 12) * ldexp(1.0, -24));
        const dim3 grid((unsigned)nb, (unsigned)P);
        if (vec)
            k_label_f32<DM, NP, CK, true><<<grid, kLT, 0, st>>>(
                X, n, D, C, rows, kk, kmax, kpad, active, s.mu, s.cmax2, E, labels, dists, amb,
                s.namb, s.blk, s.nblk);
        else
            k_label_f32<DM, NP, CK, false><<<grid, kLT, 0, st>>>(
                X, n, D, C, rows, kk, kmax, kpad, active, s.mu, s.cmax2, E, labels, dists, amb,
                s.namb, s.blk, s.nblk);
        EACB_CHECK_LAUNCH();
    }
    const unsigned gd = (unsigned)std::min<int64_t>((int64_t)nb * P * (NP / ND), 148 * 4 * (few ? 4 : 1));
    int32_t *list = few ? nullptr : amb;
    const int32_t *blk = few ? nullptr : s.blk;
    if (vec)
        k_label_direct<DM, ND, true><<<gd, kLT, 0, st>>>(X, n, D, C, kk, kmax, P, active, labels, dists,
                                                         list, s.namb, blk, s.nblk, pts, nb);
    else
        k_label_direct<DM, ND, false><<<gd, kLT, 0, st>>>(X, n, D, C, kk, kmax, P, active, labels, dists,
                                                          list, s.namb, blk, s.nblk, pts, nb);
    EACB_CHECK_LAUNCH();
    ps.done(0.0);
    return EACB_OK;
}

// k_label_direct alone up to this many centroids, or this many float32
// differences (points x centroids x dimensions) in all: it costs twice the
// arithmetic of k_label_f32 and saves some 20 us of kernels around it.  One
// pass over 400,000 points: 5 dimensions, 16 centroids 20 us (40 with
// k_label_f32), 128 centroids 48 (61); 16 dimensions, 16 centroids 41 (57);
// 32 dimensions, 200 centroids, above the line, 299 and 220.
constexpr int kLabelFewK = 32;
constexpr double kLabelFewWork = (double)(1 << 28);

int label_pass_f32(const float *X, int32_t n, int32_t D, int32_t P, const float *C,
                   const int32_t *kk, int32_t kmax, const int32_t *active, int32_t *labels,
                   float *dists, int32_t *amb, TcScratch &s, cudaStream_t st)
{
    int r;
    const bool few = kmax <= kLabelFewK || (double)n * P * kmax * D <= kLabelFewWork;
    if (!few) {
        if ((r = data_mean(X, n, D, s, st))) return r;
        // (and nblk, namb)
        EACB_CUDA(cudaMemsetAsync(s.cmax2, 0, sizeof(float) * ((size_t)P + 2), st));
    }
    // more points per thread (fewer reads of the staged rows per distance)
    // while that leaves every SM four blocks
    auto many = [&](int np) {
        return ((int64_t)n + 2 * np * kLT - 1) / (2 * np * kLT) * P >= 148 * 4;
    };
    // chunks of eight for few dimensions and many centroids, where the min
    // operations cost more than the eight rows compared at the end (2
    // dimensions, 1,000,000 points, k 1,024: 153 us, 250 with the runner-up
    // tracked throughout; 100 x 10,000, k 75: 39 us against 26 with four)
    const bool wide = kmax >= 256;
#define EACB_LABEL(DM, NPW, CKW)                                                                 \
    (!many(NPW) ? launch_label<DM, 1, 4>(st, few, X, n, D, P, C, kk, kmax, active, labels, dists, \
                                         amb, s)                                                  \
     : wide     ? launch_label<DM, NPW, CKW>(st, few, X, n, D, P, C, kk, kmax, active, labels,    \
                                             dists, amb, s)                                       \
                : launch_label<DM, NPW, 4>(st, few, X, n, D, P, C, kk, kmax, active, labels,      \
                                           dists, amb, s))
    if (D <= 2) r = EACB_LABEL(2, 4, 8);
    else if (D <= 4) r = EACB_LABEL(4, 4, 8);
    else if (D <= 6) r = EACB_LABEL(6, 4, 4);
    else if (D <= 8) r = EACB_LABEL(8, 4, 4);
    else if (D <= 12) r = EACB_LABEL(12, 2, 4);
    else if (D <= 16) r = EACB_LABEL(16, 2, 4);
    else if (D <= 24) r = EACB_LABEL(24, 1, 4);
    else r = EACB_LABEL(32, 1, 4);
#undef EACB_LABEL
    if (r || few) return r;
    return label_exact_points(X, n, D, P, C, kk, kmax, labels, dists, amb, s.namb, nullptr, st);
}

}  // namespace eacb

using namespace eacb;

extern "C" size_t eacb_kmeans_workspace_size(int32_t n, int32_t d, int32_t P, int32_t kmax)
{
    Carver c(nullptr, 0);
    KMWS::carve(c, n, d, P, kmax);
    (void)d;
    return c.off;
}

extern "C" int eacb_kmeans_ensemble(const float *X, int32_t n, int32_t d, int32_t P,
                                    const int32_t *k, int32_t kmax, const int32_t *init,
                                    int32_t max_iter, float tol, int32_t label_mode,
                                    int32_t centroid_mode, int32_t *labels, float *centroids,
                                    float *dists_out, int32_t *iters_out, float *inertia_out,
                                    void *ws, size_t ws_bytes, uintptr_t stream)
{
    if (!X || n <= 0 || d <= 0 || P <= 0 || !k || kmax <= 0 || !init || max_iter <= 0 ||
        !labels || !centroids || !ws)
        return EACB_ERR_BAD_ARGUMENT;
    if (d > 32 || kmax > 8192) return EACB_ERR_UNSUPPORTED;
    if (label_mode != 0 && label_mode != 1) return EACB_ERR_BAD_ARGUMENT;
    if ((int64_t)P * n >= ((int64_t)1 << 31)) return EACB_ERR_UNSUPPORTED;
    cudaStream_t st = as_stream(stream);
    Carver c(ws, ws_bytes);
    KMWS w = KMWS::carve(c, n, d, P, kmax);
    if (c.overflow) return EACB_ERR_WORKSPACE;
    EACB_CUDA(cudaMemsetAsync(w.err, 0, sizeof(int), st));
    k_init_centroids<<<grid_for((int64_t)P * kmax * d, 256), 256, 0, st>>>(
        X, d, init, k, kmax, P, centroids, w.active, w.inertia, w.iters, n, w.err);
    EACB_CHECK_LAUNCH();
    const int64_t nt = w.ntiles;
    const int64_t m = (int64_t)P * kmax * nt;
    for (int it = 0;; ++it) {
        int s;
        if (label_mode == 1)
            s = label_pass_tc(X, n, d, P, centroids, k, kmax, w.active, labels, w.dists, w.amb,
                              w.tc, st);
        else
            s = label_pass_f32(X, n, d, P, centroids, k, kmax, w.active, labels, w.dists, w.amb,
                               w.tc, st);
        if (s) return s;
        // the member scratch is free here: at most n / 32 node sums per partition
        if ((s = launch_inertia(st, w.dists, n, P, (float *)w.args, w.active, w.inertia, w.iters,
                                tol)))
            return s;
        if (it + 1 >= max_iter) break;
        // centroids of the partitions still running
        k_ml_count<<<(unsigned)(P * nt), 256, kmax * sizeof(int), st>>>(labels, n, kmax, nt, w.cnt,
                                                                        w.err);
        EACB_CHECK_LAUNCH();
        if ((s = scan_launch<int32_t, int64_t>(w.cnt, w.S, m, 0, &w.S[m], w.scan, st))) return s;
        if ((s = launch_ml_place(st, labels, n, P, kmax, nt, w.S, w.members, w.mypos))) return s;
        EACB_CUDA(cudaMemsetAsync(w.nempty, 0, sizeof(int32_t) * P, st));
        if ((s = launch_centroids(st, centroid_mode == 1, X, n, d, P, w.members, w.S, kmax, nt, k, kmax,
                                  w.active, centroids, w.nempty)))
            return s;
        // amb, mypos and members are free here (the centroids are done) and
        // serve as the quickselect's scratch
        if ((s = launch_fill_empty(st, X, n, d, P, w.dists, w.S, kmax, nt, k, kmax, w.active,
                                   w.nempty, w.args, w.amb, (float *)w.mypos, w.members,
                                   centroids, w.err)))
            return s;
    }
    if (dists_out)
        EACB_CUDA(cudaMemcpyAsync(dists_out, w.dists, sizeof(float) * (size_t)P * n,
                                  cudaMemcpyDeviceToDevice, st));
    if (iters_out)
        EACB_CUDA(cudaMemcpyAsync(iters_out, w.iters, sizeof(int32_t) * P, cudaMemcpyDeviceToDevice,
                                  st));
    if (inertia_out)
        EACB_CUDA(cudaMemcpyAsync(inertia_out, w.inertia, sizeof(float) * P,
                                  cudaMemcpyDeviceToDevice, st));
    int e = 0;
    EACB_CUDA(cudaMemcpyAsync(&e, w.err, sizeof(int), cudaMemcpyDeviceToHost, st));
    EACB_CUDA(cudaStreamSynchronize(st));
    return dev_err_to_status(e);
}

extern "C" int eacb_kmeans_label(const float *X, int32_t n, int32_t d, const float *C, int32_t k,
                                 int32_t label_mode, int32_t *labels, float *dists, void *ws,
                                 size_t ws_bytes, uintptr_t stream)
{
    if (!X || n <= 0 || d <= 0 || !C || k <= 0 || !labels || !dists || !ws)
        return EACB_ERR_BAD_ARGUMENT;
    if (d > 32) return EACB_ERR_UNSUPPORTED;
    cudaStream_t st = as_stream(stream);
    Carver c(ws, ws_bytes);
    int *err = c.take<int>(1);
    int32_t *kk = c.take<int32_t>(1);
    int32_t *active = c.take<int32_t>(1);
    int32_t *amb = c.take<int32_t>(n);
    TcScratch tc = TcScratch::carve(c, n, d, 1, k);
    tc.err = err;
    if (c.overflow) return EACB_ERR_WORKSPACE;
    EACB_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
    k_set2<<<1, 1, 0, st>>>(kk, active, k, 1);
    EACB_CHECK_LAUNCH();
    if (label_mode == 1)
        return label_pass_tc(X, n, d, 1, C, kk, k, active, labels, dists, amb, tc, st);
    return label_pass_f32(X, n, d, 1, C, kk, k, active, labels, dists, amb, tc, st);
}

extern "C" size_t eacb_kmeans_label_workspace_size(int32_t n, int32_t d, int32_t k)
{
    Carver c(nullptr, 0);
    c.take<int>(1);
    c.take<int32_t>(1);
    c.take<int32_t>(1);
    c.take<int>(1);
    c.take<int32_t>(n);
    TcScratch::carve(c, n, d, 1, k);
    return c.off;
}

// The label step with its arithmetic path fixed by name.
extern "C" int eacb_kmeans_label_fp32(const float *X, int32_t n, int32_t d, const float *C,
                                      int32_t k, int32_t *labels, float *dists, void *ws,
                                      size_t ws_bytes, uintptr_t stream)
{
    return eacb_kmeans_label(X, n, d, C, k, 0, labels, dists, ws, ws_bytes, stream);
}

extern "C" int eacb_kmeans_label_bf16tc(const float *X, int32_t n, int32_t d, const float *C,
                                        int32_t k, int32_t *labels, float *dists, void *ws,
                                        size_t ws_bytes, uintptr_t stream)
{
    return eacb_kmeans_label(X, n, d, C, k, 1, labels, dists, ws, ws_bytes, stream);
}

// Workspace of one centroid update (the ensemble's second half for P = 1).
struct CentWS {
    int *err;
    int32_t *kk, *active, *nempty;
    int32_t *cnt, *members, *mypos, *args, *sel, *oarg;
    float *key, *okey;
    int64_t *S;
    ScanScratch scan;
    int64_t ntiles;
    static CentWS carve(Carver &c, int32_t n, int32_t k)
    {
        CentWS w;
        w.err = c.take<int>(1);
        w.kk = c.take<int32_t>(1);
        w.active = c.take<int32_t>(1);
        w.nempty = c.take<int32_t>(1);
        w.ntiles = ((int64_t)n + kMLTile - 1) / kMLTile;
        const int64_t m = (int64_t)k * w.ntiles;
        w.cnt = c.take<int32_t>(m + 1);
        w.S = c.take<int64_t>(m + 1);
        w.members = c.take<int32_t>(n);
        w.mypos = c.take<int32_t>(n);
        w.args = c.take<int32_t>(n);
        w.sel = c.take<int32_t>(n);
        w.oarg = c.take<int32_t>(n);
        w.key = c.take<float>(n);
        w.okey = c.take<float>(n);
        w.scan = ScanScratch::carve(c, m + 1, w.err);
        return w;
    }
};

extern "C" size_t eacb_kmeans_centroids_workspace_size(int32_t n, int32_t d, int32_t k)
{
    Carver c(nullptr, 0);
    CentWS::carve(c, n, k);
    (void)d;
    return c.off;
}

extern "C" int eacb_kmeans_centroids(const float *X, int32_t n, int32_t d, const int32_t *labels,
                                     const float *dists, int32_t k, int32_t centroid_mode,
                                     float *C, void *ws, size_t ws_bytes, uintptr_t stream)
{
    if (!X || n <= 0 || d <= 0 || !labels || !dists || k <= 0 || !C || !ws)
        return EACB_ERR_BAD_ARGUMENT;
    if (centroid_mode != 0 && centroid_mode != 1) return EACB_ERR_BAD_ARGUMENT;
    if (d > 32 || k > 8192) return EACB_ERR_UNSUPPORTED;
    cudaStream_t st = as_stream(stream);
    Carver c(ws, ws_bytes);
    CentWS w = CentWS::carve(c, n, k);
    if (c.overflow) return EACB_ERR_WORKSPACE;
    const int64_t nt = w.ntiles;
    const int64_t m = (int64_t)k * nt;
    EACB_CUDA(cudaMemsetAsync(w.err, 0, sizeof(int), st));
    EACB_CUDA(cudaMemsetAsync(w.nempty, 0, sizeof(int32_t), st));
    k_set2<<<1, 1, 0, st>>>(w.kk, w.active, k, 1);
    EACB_CHECK_LAUNCH();
    k_ml_count<<<(unsigned)nt, 256, k * sizeof(int), st>>>(labels, n, k, nt, w.cnt, w.err);
    EACB_CHECK_LAUNCH();
    int s = scan_launch<int32_t, int64_t>(w.cnt, w.S, m, 0, &w.S[m], w.scan, st);
    if (s) return s;
    if ((s = launch_ml_place(st, labels, n, 1, k, nt, w.S, w.members, w.mypos))) return s;
    if ((s = launch_centroids(st, centroid_mode == 1, X, n, d, 1, w.members, w.S, k, nt, w.kk, k,
                              w.active, C, w.nempty)))
        return s;
    // the quickselect permutes its keys: it works on a copy of the distances
    EACB_CUDA(cudaMemcpyAsync(w.key, dists, sizeof(float) * (size_t)n, cudaMemcpyDeviceToDevice, st));
    if ((s = launch_fill_empty(st, X, n, d, 1, w.key, w.S, k, nt, w.kk, k, w.active, w.nempty,
                               w.args, w.sel, w.okey, w.oarg, C, w.err)))
        return s;
    int e = 0;
    EACB_CUDA(cudaMemcpyAsync(&e, w.err, sizeof(int), cudaMemcpyDeviceToHost, st));
    EACB_CUDA(cudaStreamSynchronize(st));
    return dev_err_to_status(e);
}
