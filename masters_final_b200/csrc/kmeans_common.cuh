// Pieces shared by the float32 and the tensor-core k-means label passes.
#pragma once
#include "eacb_common.cuh"

namespace eacb {

// The reference's distance (MyML/MyML/cluster/KMeans.py:463-466): float32
// difference, float32 square, float64 running sum in dimension order.
template <int DM>
__device__ __forceinline__ double exact_dist(const float *x, const float *c, int D)
{
    double dist = 0.0;
#pragma unroll
    for (int d = 0; d < DM; ++d) {
        if (d < D) {
            const float diff = __fsub_rn(x[d], c[d]);
            dist = __dadd_rn(dist, (double)__fmul_rn(diff, diff));
        }
    }
    return dist;
}

__device__ __forceinline__ uint64_t pack2(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t twice(float a) { return pack2(a, a); }
__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t fadd2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float min3(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Folds the least score of a chunk of centroids into the best two chunk
// minima and the winner's chunk.  The runner-up inside the winner's chunk is
// looked for once, at the end: per centroid this takes 1.6 (chunks of four)
// or 1.1 (eight) operations of the half-rate ALU pipe that bounds the label
// passes, where keeping the best two of all centroids took 3.5 and an index
// per centroid 5.
__device__ __forceinline__ void top2_chunks(float m, int id, float &b1, float &b2, int &i1)
{
    i1 = m < b1 ? id : i1;
    b2 = fminf(b2, fmaxf(b1, m));
    b1 = fminf(b1, m);
}
__device__ __forceinline__ float min4(float a, float b, float c, float d)
{
    return fminf(min3(a, b, c), d);
}

// a row of D floats into registers (zeros past D): with VEC -- D equals DM
// and rows start on 16-byte (DM a multiple of four) or 8-byte boundaries --
// four or two floats at a time
template <int DM, bool VEC>
__device__ __forceinline__ void load_row(const float *c, int D, float (&v)[DM])
{
    if (VEC && DM % 4 == 0) {
#pragma unroll
        for (int d = 0; d + 3 < DM; d += 4) {
            const float4 f = __ldg(reinterpret_cast<const float4 *>(c + d));
            v[d] = f.x;
            v[d + 1] = f.y;
            v[d + 2] = f.z;
            v[d + 3] = f.w;
        }
    } else if (VEC) {
#pragma unroll
        for (int d = 0; d + 1 < DM; d += 2) {
            const float2 f = __ldg(reinterpret_cast<const float2 *>(c + d));
            v[d] = f.x;
            v[d + 1] = f.y;
        }
    } else {
#pragma unroll
        for (int d = 0; d < DM; ++d) v[d] = d < D ? __ldg(c + d) : 0.f;
    }
}

static __global__ void k_set2(int32_t *a, int32_t *b, int32_t va, int32_t vb)
{
    *a = va;
    *b = vb;
}

// Scratch of the label passes.  Tensor cores: operands in the UMMA layout.
// Float32: B holds the staged centroid rows (up to 4 (D + 4) bytes each, D
// rounded up to the kernel's, which fit the 2 Kp bytes of a tile row).
constexpr int kTcCentPad = 128;      // centroid rows are padded to tiles of this many
constexpr int kLabelPts = 256;       // points per block of the float32 pass at least
struct TcScratch {
    int Kp;              // 6d rounded up to a multiple of 16
    int64_t n_pad;       // points rounded up to the 128-point tile
    int kt_max;          // kTcCentPad-centroid tiles per partition
    uint8_t *A;          // point tiles
    float *nx;           // |x - mu|^2
    uint8_t *B;          // centroid tiles
    float *nc;           // |c - mu|^2 (+inf for padding)
    float *cmax2;        // per partition max |c - mu|^2
    int *nblk;           // (behind cmax2) blocks of the float32 pass left with many open points
    int *namb;           // (behind it) points left to the exact re-check
    int32_t *blk;        // and which
    float *mu;           // the centre (data_mean)
    double *part;        // column-sum partials
    int *err;
    bool points_ready;   // A / nx depend on X only
    bool mean_ready;     // and so do part / mu
    static TcScratch carve(Carver &c, int32_t n, int32_t D, int32_t P, int32_t kmax);
};

// Label pass on tcgen05 tensor cores (kmeans_tc.cu); same contract as the
// float32 pass: every point of every active partition gets the reference's
// label and distance.
int label_pass_tc(const float *X, int32_t n, int32_t D, int32_t P, const float *C,
                  const int32_t *kk, int32_t kmax, const int32_t *active, int32_t *labels,
                  float *dists, int32_t *amb, TcScratch &s, cudaStream_t st);

// A point amid the data (the median of the means of 32 parts of a strided
// sample), once per scratch: the label passes centre on it, which keeps their
// error bounds small; their results do not depend on it.
int data_mean(const float *X, int32_t n, int32_t D, TcScratch &s, cudaStream_t st);

// The reference's label and distance for the *namb listed (partition, point)
// pairs; err (may be null): nonzero means they are done already.
int label_exact_points(const float *X, int32_t n, int32_t D, int32_t P, const float *C,
                       const int32_t *kk, int32_t kmax, int32_t *labels, float *dists,
                       const int32_t *amb, const int *namb, const int *err, cudaStream_t st);

}  // namespace eacb
