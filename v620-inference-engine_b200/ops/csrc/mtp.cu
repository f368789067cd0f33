// MTP head plumbing kernels: the input of the MTP layer is, per stream, fc_hidden(norm(hidden stream)) +
// fc_embedding(gemma_norm(embedding of the next token)), where `norm` is ONE RMS norm over all hc*H values
// of the backbone's pre-final-mixer state (roles of the reference's src/kernels/mtp.hip:7-54;
// math in docs/MODEL.md:221-231).
#include "common.cuh"

namespace qw {

// grid M.  hidden [M][hc][H] fp32 -> hn bf16 [(m*hc + s)][H] = hidden * rsqrt(mean over all) * nh1;
// en bf16 [m][H] = gemma_norm(embed[token m]) with ne1 = 1 + w.  V columns per thread and step.
constexpr int MN_THREADS = 1024;      // a row of 10,240 values is 2.5 pieces of four per thread (with 256 threads and scalar loads 29 us a row, now 7)
template <int V>
__global__ void __launch_bounds__(MN_THREADS) mtp_norm_kernel(const float *hidden, const int *tokens, const bf16 *embed, int vocab,
                                                              const float *nh1, const float *ne1, int H, int hc, float eps, bf16 *hn,
                                                              bf16 *en) {
    __shared__ float scratch[32];
    const int m = blockIdx.x, n = hc * H;
    pdl_wait();
    pdl_trigger();
    int t = tokens[m];
    if (t < 0 || t >= vocab) t = 0;
    const bf16 *e = embed + (long long)t * H;
    const float *x = hidden + (long long)m * n;
    float ss = 0.f, es = 0.f;
#pragma unroll 3
    for (int i = threadIdx.x * V; i < n; i += MN_THREADS * V) {
        float v[V];
        ld_cols<V>(x + i, v);
#pragma unroll
        for (int k = 0; k < V; ++k) ss = fmaf(v[k], v[k], ss);
    }
    for (int i = threadIdx.x; i < H; i += MN_THREADS) {
        const float v = __bfloat162float(e[i]);
        es = fmaf(v, v, es);
    }
    ss = block_sum<MN_THREADS>(ss, scratch);
    es = block_sum<MN_THREADS>(es, scratch);
    const float r = rsqrtf(ss / float(n) + eps), re = rsqrtf(es / float(H) + eps);
#pragma unroll 3
    for (int i = threadIdx.x * V; i < n; i += MN_THREADS * V) {
        float v[V], w[V];
        ld_cols<V>(x + i, v);
        ld_cols<V>(nh1 + i, w);
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] = v[k] * r * w[k];
        st_cols<V>(hn + (long long)m * n + i, v);
    }
    for (int i = threadIdx.x; i < H; i += MN_THREADS) en[(long long)m * H + i] = __float2bfloat16(__bfloat162float(e[i]) * re * ne1[i]);
}

// X[m][s][c] = fh[(m*hc + s)][c] + fe[m][c]
__global__ void mtp_add_kernel(const float *fh, const float *fe, int H, int hc, float *X, long long total) {
    pdl_wait();
    pdl_trigger();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const long long m = i / ((long long)hc * H);
    const int c = (int)(i % H);
    X[i] = fh[i] + fe[m * H + c];
}

}  // namespace qw

using namespace qw;

QW_API int qwk_mtp_norm(const float *hidden, const int *tokens, const void *embed, int vocab, const float *nh1, const float *ne1,
                        int H, int hc, float eps, void *hn, void *en, int M, cudaStream_t s) {
    const bool vec = (hc * H & 3) == 0 && aligned16(hidden, nh1, (bf16 *)hn);
    return launch_pdl(vec ? mtp_norm_kernel<4> : mtp_norm_kernel<1>, dim3(M), dim3(MN_THREADS), 0, s, hidden, tokens, (const bf16 *)embed, vocab, nh1, ne1, H, hc, eps,
                      (bf16 *)hn, (bf16 *)en) == cudaSuccess ? 0 : -2;
}
QW_API int qwk_mtp_add(const float *fh, const float *fe, int H, int hc, float *X, int M, cudaStream_t s) {
    const long long total = (long long)M * hc * H;
    return launch_pdl(mtp_add_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, s, fh, fe, H, hc, X, total) == cudaSuccess ? 0 : -2;
}
