// Vision tower (Qwen3-VL ViT) kernels: everything between the tower's GEMMs (which run on the tcgen05 GEMM of
// gemm_tc.cu).  Residual stream fp32, GEMM operands bf16.
//
//   vit_embed          x = patch_gemm + bias + bilinear interpolation of the learned 48x48 position table
//   vit_layernorm      bf16(LayerNorm(x) * w + b), after x += y + bias where a residual add precedes it
//   vit_rope_table     cos | sin of every patch's 36 angles
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

// A warp per row, the row in registers: with `y` the residual add x += y + ybias comes first and x is written back, so a block's
// add and the next norm are one pass (at 3520 x 1152, 29 us as two kernels of one block per row and scalar accesses, 12 as one).
constexpr int VLN_MAX = 12;      // float4 per lane: D <= 1536
__device__ __forceinline__ float4 vit_ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__global__ void __launch_bounds__(128) vit_layernorm_kernel(float *x, const float *y, const float *ybias, const float *w, const float *b,
                                                            int L, int D, float eps, bf16 *out) {
    const int n = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (n >= L) return;
    float *row = x + (long long)n * D;
    float4 v[VLN_MAX];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VLN_MAX; ++i) {
        const int c = (i * 32 + lane) * 4;
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c >= D) continue;
        v[i] = vit_ld4(row + c);
        if (y) {
            const float4 a = vit_ld4(y + (long long)n * D + c), e = vit_ld4(ybias + c);
            v[i].x += a.x + e.x; v[i].y += a.y + e.y; v[i].z += a.z + e.z; v[i].w += a.w + e.w;
            *reinterpret_cast<float4 *>(row + c) = v[i];
        }
        s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
    }
    const float mean = warp_sum(s) / float(D);
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < VLN_MAX; ++i) {
        if ((i * 32 + lane) * 4 >= D) continue;
        v[i].x -= mean; v[i].y -= mean; v[i].z -= mean; v[i].w -= mean;
        q = fmaf(v[i].x, v[i].x, q); q = fmaf(v[i].y, v[i].y, q); q = fmaf(v[i].z, v[i].z, q); q = fmaf(v[i].w, v[i].w, q);
    }
    const float rstd = rsqrtf(warp_sum(q) / float(D) + eps);
#pragma unroll
    for (int i = 0; i < VLN_MAX; ++i) {
        const int c = (i * 32 + lane) * 4;
        if (c >= D) continue;
        const float4 ww = vit_ld4(w + c), bb = vit_ld4(b + c);
        uint2 pk;
        pk.x = pack_bf16(fmaf(v[i].x * rstd, ww.x, bb.x), fmaf(v[i].y * rstd, ww.y, bb.y));
        pk.y = pack_bf16(fmaf(v[i].z * rstd, ww.z, bb.z), fmaf(v[i].w * rstd, ww.w, bb.w));
        *reinterpret_cast<uint2 *>(out + (long long)n * D + c) = pk;
    }
}

// The same for any width and address: a block per row.
__global__ void __launch_bounds__(256) vit_layernorm_any_kernel(float *x, const float *y, const float *ybias, const float *w, const float *b,
                                                                int D, float eps, bf16 *out) {
    __shared__ float scratch[32];
    float *row = x + (long long)blockIdx.x * D;
    const float *add = y ? y + (long long)blockIdx.x * D : nullptr;
    float s = 0.f;
    for (int c = threadIdx.x; c < D; c += 256) {
        if (y) row[c] += add[c] + ybias[c];
        s += row[c];
    }
    const float mean = block_sum<256>(s, scratch) / float(D);
    float q = 0.f;
    for (int c = threadIdx.x; c < D; c += 256) q = fmaf(row[c] - mean, row[c] - mean, q);
    const float rstd = rsqrtf(block_sum<256>(q, scratch) / float(D) + eps);
    for (int c = threadIdx.x; c < D; c += 256) out[(long long)blockIdx.x * D + c] = __float2bfloat16((row[c] - mean) * rstd * w[c] + b[c]);
}

// cos | sin of the 36 angles of every patch (first 18 by row, last 18 by column): [L][2][36], once per slice instead of once per
// block, head and tensor.
__global__ void __launch_bounds__(256) vit_rope_table_kernel(const int *pos_hw, int L, float *tab) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= L * VHALF) return;
    const int n = i / VHALF, t = i - n * VHALF, f = t % VNF;
    const float inv = exp2f(-2.f * float(f) / float(VHALF) * 13.287712379549449f);      // 10000^(-2f/36)
    float sn, cs;
    sincosf(float(pos_hw[n * 2 + (t < VNF ? 0 : 1)]) * inv, &sn, &cs);
    tab[(long long)n * 2 * VHALF + t] = cs;
    tab[(long long)n * 2 * VHALF + VHALF + t] = sn;
}

// One block per patch: bias on the whole row, rotary on q and k, V values (of each half of a head) per step: four, or one where a
// pointer does not allow it.
template <int V>
__global__ void __launch_bounds__(256) vit_bias_rope_kernel(bf16 *qkv, const float *bias, const float *tab, int heads) {
    const int n = blockIdx.x, D = heads * VHD;
    bf16 *row = qkv + (long long)n * 3 * D;
    const float *cs = tab + (long long)n * 2 * VHALF, *sn = cs + VHALF;
    const int rot = 2 * heads * (VHALF / V), total = rot + D / V;
    for (int i = threadIdx.x; i < total; i += 256) {
        float a[V], e[V];
        if (i >= rot) {
            const int c = 2 * D + (i - rot) * V;
            ld_cols<V>(row + c, a);
            ld_cols<V>(bias + c, e);
#pragma unroll
            for (int k = 0; k < V; ++k) a[k] += e[k];
            st_cols<V>(row + c, a);
            continue;
        }
        const int hh = i / (VHALF / V), t = (i - hh * (VHALF / V)) * V, c = hh * VHD + t;      // hh over q heads then k heads
        float b[V], f[V], co[V], si[V], o[V], p[V];
        ld_cols<V>(row + c, a);
        ld_cols<V>(row + c + VHALF, b);
        ld_cols<V>(bias + c, e);
        ld_cols<V>(bias + c + VHALF, f);
        ld_cols<V>(cs + t, co);
        ld_cols<V>(sn + t, si);
#pragma unroll
        for (int k = 0; k < V; ++k) {
            a[k] += e[k];
            b[k] += f[k];
            o[k] = a[k] * co[k] - b[k] * si[k];
            p[k] = b[k] * co[k] + a[k] * si[k];
        }
        st_cols<V>(row + c, o);
        st_cols<V>(row + c + VHALF, p);
    }
}

__device__ __forceinline__ float vit_gelu(float v, int tanh_form) {
    return tanh_form ? 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)))
                     : 0.5f * v * (1.f + erff(v * 0.7071067811865476f));
}
constexpr int VG_ROWS = 8;
// Eight columns per thread (their bias in registers) down eight rows: 16-byte accesses.  At 3520 x 4304 53 us with two-byte
// accesses, a division per value for its column; 21 now.
__global__ void __launch_bounds__(128) vit_bias_gelu8_kernel(bf16 *y, const float *bias, int L, int D, int tanh_form) {
    const int c = (blockIdx.y * 128 + threadIdx.x) * 8;
    if (c >= D) return;
    float e[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) e[k] = bias[c + k];
    const int n0 = blockIdx.x * VG_ROWS, n1 = min(L, n0 + VG_ROWS);
#pragma unroll 4
    for (int n = n0; n < n1; ++n) {
        uint4 *p = reinterpret_cast<uint4 *>(y + (long long)n * D + c);
        const uint4 u = *p;
        const uint32_t in[4] = {u.x, u.y, u.z, u.w};
        uint32_t o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = pack_bf16(vit_gelu(bf16_lo(in[k]) + e[2 * k], tanh_form), vit_gelu(bf16_hi(in[k]) + e[2 * k + 1], tanh_form));
        *p = make_uint4(o[0], o[1], o[2], o[3]);
    }
}
// Any width.
__global__ void vit_bias_gelu_kernel(bf16 *y, const float *bias, long long total, int D, int tanh_form) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < total) y[i] = __float2bfloat16(vit_gelu(__bfloat162float(y[i]) + bias[i % D], tanh_form));
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

// out = bf16(LayerNorm(x) * w + b); with y (null: none) x += y + ybias first.
QW_API int qwk_vit_layernorm(float *x, const float *y, const float *ybias, const float *w, const float *b, int L, int D, float eps,
                             void *out, cudaStream_t s) {
    if ((D & 3) == 0 && D <= VLN_MAX * 128 && aligned16(x, y, y ? ybias : nullptr, w, b, (float *)out))
        vit_layernorm_kernel<<<(L + 3) / 4, 128, 0, s>>>(x, y, ybias, w, b, L, D, eps, (bf16 *)out);
    else
        vit_layernorm_any_kernel<<<L, 256, 0, s>>>(x, y, ybias, w, b, D, eps, (bf16 *)out);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// tab [L][2][36] fp32: cos | sin of every patch's rotary angles.
QW_API int qwk_vit_rope_table(const int *pos_hw, int L, float *tab, cudaStream_t s) {
    vit_rope_table_kernel<<<blocks_for((long long)L * VHALF), 256, 0, s>>>(pos_hw, L, tab);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

QW_API int qwk_vit_bias_rope(void *qkv, const float *bias, const float *tab, int L, int heads, cudaStream_t s) {
    if (aligned16((bf16 *)qkv, bias, tab)) vit_bias_rope_kernel<4><<<L, 256, 0, s>>>((bf16 *)qkv, bias, tab, heads);
    else vit_bias_rope_kernel<1><<<L, 256, 0, s>>>((bf16 *)qkv, bias, tab, heads);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

QW_API int qwk_vit_bias_gelu(void *y, const float *bias, int L, int D, int tanh_form, cudaStream_t s) {
    if ((D & 7) == 0 && ((uintptr_t)y & 15) == 0) {
        dim3 grid((L + VG_ROWS - 1) / VG_ROWS, (D / 8 + 127) / 128);
        vit_bias_gelu8_kernel<<<grid, 128, 0, s>>>((bf16 *)y, bias, L, D, tanh_form);
    } else {
        const long long total = (long long)L * D;
        vit_bias_gelu_kernel<<<blocks_for(total), 256, 0, s>>>((bf16 *)y, bias, total, D, tanh_form);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// assign = 0: x += y + bias; assign = 1: x = y + bias.
QW_API int qwk_vit_residual_add(float *x, const float *y, const float *bias, int L, int D, int assign, cudaStream_t s) {
    const long long total = (long long)L * D;
    vit_residual_add_kernel<<<blocks_for(total), 256, 0, s>>>(x, y, bias, total, D, assign);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
