// Vision tower (Qwen3-VL ViT) kernels: everything between the tower's GEMMs (which run on the tcgen05 GEMM of
// gemm_tc.cu).  Residual stream fp32, GEMM operands bf16.
//
//   vit_embed          x = patch_gemm + bias + bilinear interpolation of the learned 48x48 position table
//   vit_layernorm      bf16(LayerNorm(x) * w + b)
//   vit_bias_rope      qkv += bias, then 2-D rotary on q and k (pairs (t, t+36); first 18 frequencies by row,
//                      last 18 by column)
//   (attention: vit_attn.cu)
//   vit_bias_gelu      y = gelu(y + bias), tanh or erf form
//   vit_residual_add   x += y + bias        vit_bias_out   out = y + bias
// (Role of the reference's src/kernels/vision.hip:33-217.)
#include "common.cuh"

namespace qw {

constexpr int VHD = 72;          // head dim
constexpr int VHALF = 36;
constexpr int VNF = 18;

__global__ void __launch_bounds__(256) vit_embed_kernel(float *x, const float *y, const float *bias, const float *table,
                                                        const int *idx, const float *wts, int D) {
    const int n = blockIdx.x;
    const int i0 = idx[n * 4], i1 = idx[n * 4 + 1], i2 = idx[n * 4 + 2], i3 = idx[n * 4 + 3];
    const float w0 = wts[n * 4], w1 = wts[n * 4 + 1], w2 = wts[n * 4 + 2], w3 = wts[n * 4 + 3];
    for (int c = threadIdx.x; c < D; c += 256) {
        const float p = w0 * table[(long long)i0 * D + c] + w1 * table[(long long)i1 * D + c] +
                        w2 * table[(long long)i2 * D + c] + w3 * table[(long long)i3 * D + c];
        x[(long long)n * D + c] = y[(long long)n * D + c] + bias[c] + p;
    }
}

__global__ void __launch_bounds__(256) vit_layernorm_kernel(const float *x, const float *w, const float *b, int D, float eps,
                                                            bf16 *out) {
    __shared__ float scratch[32];
    const int n = blockIdx.x;
    const float *row = x + (long long)n * D;
    float s = 0.f;
    for (int c = threadIdx.x; c < D; c += 256) s += row[c];
    const float mean = block_sum<256>(s, scratch) / float(D);
    float v = 0.f;
    for (int c = threadIdx.x; c < D; c += 256) {
        const float d = row[c] - mean;
        v = fmaf(d, d, v);
    }
    const float rstd = rsqrtf(block_sum<256>(v, scratch) / float(D) + eps);
    for (int c = threadIdx.x; c < D; c += 256) out[(long long)n * D + c] = __float2bfloat16((row[c] - mean) * rstd * w[c] + b[c]);
}

// one block per patch: bias on the whole row, rotary on q and k
__global__ void __launch_bounds__(256) vit_bias_rope_kernel(bf16 *qkv, const float *bias, const int *pos_hw, int heads) {
    const int n = blockIdx.x;
    const int D = heads * VHD;
    bf16 *row = qkv + (long long)n * 3 * D;
    for (int c = 2 * D + threadIdx.x; c < 3 * D; c += 256) row[c] = __float2bfloat16(__bfloat162float(row[c]) + bias[c]);
    const float pr = float(pos_hw[n * 2]), pc = float(pos_hw[n * 2 + 1]);
    for (int i = threadIdx.x; i < 2 * heads * VHALF; i += 256) {
        const int t = i % VHALF, hh = i / VHALF;          // hh over q heads then k heads
        const int f = t % VNF;
        const float inv = exp2f(-2.f * float(f) / float(VHALF) * 13.287712379549449f);      // 10000^(-2f/36)
        float sn, cs;
        sincosf((t < VNF ? pr : pc) * inv, &sn, &cs);
        const int base = hh * VHD;
        const float a = __bfloat162float(row[base + t]) + bias[base + t];
        const float b = __bfloat162float(row[base + t + VHALF]) + bias[base + t + VHALF];
        row[base + t] = __float2bfloat16(a * cs - b * sn);
        row[base + t + VHALF] = __float2bfloat16(b * cs + a * sn);
    }
}

__global__ void vit_bias_gelu_kernel(bf16 *y, const float *bias, long long total, int D, int tanh_form) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= total) return;
    const float v = __bfloat162float(y[i]) + bias[i % D];
    const float g = tanh_form ? 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)))
                              : 0.5f * v * (1.f + erff(v * 0.7071067811865476f));
    y[i] = __float2bfloat16(g);
}

__global__ void vit_residual_add_kernel(float *x, const float *y, const float *bias, long long total, int D, int assign) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= total) return;
    const float v = y[i] + bias[i % D];
    x[i] = assign ? v : x[i] + v;
}

}  // namespace qw

using namespace qw;

static inline unsigned blocks_for(long long n) { return (unsigned)((n + 255) / 256); }

QW_API int qwk_vit_embed(float *x, const float *y, const float *bias, const float *table, const int *idx, const float *wts,
                         int L, int D, cudaStream_t s) {
    vit_embed_kernel<<<L, 256, 0, s>>>(x, y, bias, table, idx, wts, D);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

QW_API int qwk_vit_layernorm(const float *x, const float *w, const float *b, int L, int D, float eps, void *out,
                             cudaStream_t s) {
    vit_layernorm_kernel<<<L, 256, 0, s>>>(x, w, b, D, eps, (bf16 *)out);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

QW_API int qwk_vit_bias_rope(void *qkv, const float *bias, const int *pos_hw, int L, int heads, cudaStream_t s) {
    vit_bias_rope_kernel<<<L, 256, 0, s>>>((bf16 *)qkv, bias, pos_hw, heads);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

QW_API int qwk_vit_bias_gelu(void *y, const float *bias, int L, int D, int tanh_form, cudaStream_t s) {
    const long long total = (long long)L * D;
    vit_bias_gelu_kernel<<<blocks_for(total), 256, 0, s>>>((bf16 *)y, bias, total, D, tanh_form);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// assign = 0: x += y + bias; assign = 1: x = y + bias.
QW_API int qwk_vit_residual_add(float *x, const float *y, const float *bias, int L, int D, int assign, cudaStream_t s) {
    const long long total = (long long)L * D;
    vit_residual_add_kernel<<<blocks_for(total), 256, 0, s>>>(x, y, bias, total, D, assign);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
