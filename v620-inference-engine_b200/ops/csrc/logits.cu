// Reductions over a vocabulary shard of logits: (max, argmax with ties to the lowest index) and
// (max, sum exp) per row (roles of the reference's src/kernels/logits.hip:7-70).  Results of the
// shards are merged by merge_argmax / on the host.
#include "common.cuh"

#include <cooperative_groups.h>

namespace qw {

// A row is reduced by a cluster of eight CTAs, each with an eighth of the columns: its own maximum first, the sum of exponentials
// around it from a second pass (L1 / L2), and rank 0 puts the eight parts together.  One CTA per row took 32 us for 248,320
// logits (one SM's loads in flight); eight take 7.  grid 8 M, 512 threads.  out_val[m], out_idx[m] (index offset by idx0); lse
// parts: out_max[m], out_sum[m].
constexpr int RR_CTAS = 8, RR_THREADS = 512;
__global__ void __cluster_dims__(RR_CTAS, 1, 1) __launch_bounds__(RR_THREADS) row_reduce_kernel(const float *logits, int ld, int V, int idx0,
                                                                                               float *out_val, int *out_idx, float *out_max,
                                                                                               float *out_sum) {
    namespace cg = cooperative_groups;
    __shared__ float sv[32], scratch[32];
    __shared__ int si[32];
    __shared__ float part_max[RR_CTAS], part_sum[RR_CTAS];          // rank 0's: every CTA's (max, sum, index)
    __shared__ int part_idx[RR_CTAS];
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();          // every CTA of the cluster runs: rank 0's memory may be written (before the wait for the logits, which is longer)
    pdl_wait();
    const int m = blockIdx.x / RR_CTAS, rank = blockIdx.x % RR_CTAS, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float *l = logits + (long long)m * ld;
    const int per = ((V + RR_CTAS - 1) / RR_CTAS + 3) & ~3, c0 = rank * per, c1 = min(V, c0 + per);
    const bool vec = ((uintptr_t)l & 15) == 0;
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    const int v1 = vec ? c0 + max(0, c1 - c0) / 4 * 4 : c0;          // columns c0 .. v1 in 16-byte pieces
#pragma unroll 4
    for (int i = c0 + threadIdx.x * 4; i < v1; i += RR_THREADS * 4) {
        const float4 v = *reinterpret_cast<const float4 *>(l + i);
        if (v.x > bv) { bv = v.x; bi = i; }       // ascending columns: keeps the lowest index among equals
        if (v.y > bv) { bv = v.y; bi = i + 1; }
        if (v.z > bv) { bv = v.z; bi = i + 2; }
        if (v.w > bv) { bv = v.w; bi = i + 3; }
    }
    for (int i = v1 + threadIdx.x; i < c1; i += RR_THREADS)
        if (l[i] > bv) { bv = l[i]; bi = i; }
    auto best = [&](int lanes) {
        for (int o = lanes / 2; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
    };
    best(32);
    if (lane == 0) { sv[w] = bv; si[w] = bi; }
    __syncthreads();
    if (w == 0) {
        bv = lane < RR_THREADS / 32 ? sv[lane] : -INFINITY;
        bi = lane < RR_THREADS / 32 ? si[lane] : 0x7fffffff;
        best(32);
        if (lane == 0) { sv[0] = bv; si[0] = bi; }
    }
    __syncthreads();
    const float mx = sv[0];
    float z = 0.f;
    if (out_sum) {
        const float at = mx == -INFINITY ? 0.f : mx;                 // nothing but -inf (or NaN) in this eighth: its sum is 0 (NaN)
#pragma unroll 4
        for (int i = c0 + threadIdx.x * 4; i < v1; i += RR_THREADS * 4) {
            const float4 v = *reinterpret_cast<const float4 *>(l + i);
            z += (__expf(v.x - at) + __expf(v.y - at)) + (__expf(v.z - at) + __expf(v.w - at));
        }
        for (int i = v1 + threadIdx.x; i < c1; i += RR_THREADS) z += __expf(l[i] - at);
        z = block_sum<RR_THREADS>(z, scratch);
    }
    if (threadIdx.x == 0) {
        *cl.map_shared_rank(&part_max[rank], 0) = mx;
        *cl.map_shared_rank(&part_idx[rank], 0) = si[0];
        *cl.map_shared_rank(&part_sum[rank], 0) = z;
    }
    cl.sync();
    if (rank == 0 && threadIdx.x == 0) {
        float M = part_max[0];
        int at = part_idx[0];
        for (int r = 1; r < RR_CTAS; ++r)                            // ranks hold ascending columns: a later equal one does not win
            if (part_max[r] > M) { M = part_max[r]; at = part_idx[r]; }
        if (out_val) out_val[m] = M;
        if (out_idx) out_idx[m] = at + idx0;
        if (out_sum) {
            float t = 0.f;
            for (int r = 0; r < RR_CTAS; ++r) t += part_sum[r] * __expf(part_max[r] - M);
            out_max[m] = M;
            out_sum[m] = t;
        }
    }
}

// Merge per-rank (value, index) pairs: parts[r][m]; ties to the lowest index.  One thread per row.
__global__ void merge_argmax_kernel(const float *vals, const int *idx, int ranks, int M, int stride, int *out_idx,
                                    float *out_val) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    for (int r = 0; r < ranks; ++r) {
        const float v = vals[r * stride + m];
        const int i = idx[r * stride + m];
        if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; }
    }
    out_idx[m] = bi;
    if (out_val) out_val[m] = bv;
}

// Chained decoding: the sampled token of each row becomes the row's next input, its position
// advances and the n-gram context shifts, all on the device, so consecutive steps need no host
// round trip (the reference chains its draft steps the same way, src/engine/decode.hip:293-334).
__global__ void advance_rows_kernel(int *tokens, int *pos, int *ctx3, const int *next, int M) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    const int t = next[m];
    ctx3[3 * m + 2] = ctx3[3 * m + 1];
    ctx3[3 * m + 1] = ctx3[3 * m];
    ctx3[3 * m] = t;
    tokens[m] = t;
    pos[m] += 1;
}

// Vocabulary-parallel argmax: every rank packs its (value, index) per row into its column pair of the
// gathered matrix; after the all-gather every rank picks the best pair (ties to the lowest index).
__global__ void amax_pack_kernel(const float *val, const int *idx, float *pairs, int M, int rank, int ranks) {
    pdl_wait();
    pdl_trigger();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    pairs[(long long)m * ranks * 2 + rank * 2] = val[m];
    pairs[(long long)m * ranks * 2 + rank * 2 + 1] = __int_as_float(idx[m]);
}
__global__ void amax_merge_kernel(const float *pairs, int M, int ranks, int *out_idx, float *out_val) {
    pdl_wait();
    pdl_trigger();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    for (int r = 0; r < ranks; ++r) {
        const float v = __ldcg(pairs + (long long)m * ranks * 2 + r * 2);
        const int i = __float_as_int(__ldcg(pairs + (long long)m * ranks * 2 + r * 2 + 1));
        if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; }
    }
    out_idx[m] = bi;
    if (out_val) out_val[m] = bv;
}

}  // namespace qw

using namespace qw;

QW_API int qwk_amax_pack(const float *val, const int *idx, float *pairs, int M, int rank, int ranks, cudaStream_t s) {
    return launch_pdl(amax_pack_kernel, dim3((M + 63) / 64), dim3(64), 0, s, val, idx, pairs, M, rank, ranks) == cudaSuccess ? 0 : -2;
}
QW_API int qwk_amax_merge(const float *pairs, int M, int ranks, int *out_idx, float *out_val, cudaStream_t s) {
    return launch_pdl(amax_merge_kernel, dim3((M + 63) / 64), dim3(64), 0, s, pairs, M, ranks, out_idx, out_val) == cudaSuccess ? 0 : -2;
}


QW_API int qwk_advance_rows(int *tokens, int *pos, int *ctx3, const int *next, int M, cudaStream_t s) {
    advance_rows_kernel<<<(M + 63) / 64, 64, 0, s>>>(tokens, pos, ctx3, next, M);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

QW_API int qwk_row_reduce(const float *logits, int ld, int V, int idx0, int M, float *out_val, int *out_idx,
                          float *out_max, float *out_sum, cudaStream_t s) {
    if (M <= 0) return 0;
    return launch_pdl(row_reduce_kernel, dim3((unsigned)(RR_CTAS * (long long)M)), dim3(RR_THREADS), 0, s, logits, ld, V, idx0, out_val, out_idx, out_max, out_sum) ==
                   cudaSuccess ? 0 : -2;
}

QW_API int qwk_merge_argmax(const float *vals, const int *idx, int ranks, int M, int stride, int *out_idx,
                            float *out_val, cudaStream_t s) {
    merge_argmax_kernel<<<(M + 63) / 64, 64, 0, s>>>(vals, idx, ranks, M, stride, out_idx, out_val);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
