// PLE (per-layer n-gram embedding) kernels for row batches: device-side n-gram hashing and the
// 16-row gather straight out of the host-resident table (pinned, mapped memory), the gate
// statistics, the gated value / normalised conv input, the dilated causal conv and its ring
// (roles of the reference's src/core/ple.cpp:86-125,184-211 on the host and
// src/kernels/ple.hip:8-215 on the device; math in docs/MODEL.md:185-219).
#include "common.cuh"

namespace qw {

constexpr int MAX_NGRAM_HEADS = 32;

struct NgramConst {
    unsigned long long mult[4];
    unsigned long long sizes[MAX_NGRAM_HEADS];
    long long offsets[MAX_NGRAM_HEADS];
    int ngram, heads, eos;
};
__constant__ NgramConst c_ng;
__constant__ float c_f8_lut[256];

enum PleLayout { PLE_F8 = 0, PLE_BF16 = 1, PLE_INT8 = 2, PLE_INT4 = 3 };

struct PleGatherArgs {
    const int *ctx;              // [M][3]: token at the row's position, the one before, two before (-1 = none)
    const void *const *shards;   // per shard: value rows
    const void *const *scales;   // per shard: fp16 scales (int8 / int4 layouts)
    long long rows_per_shard, rows;
    int layout, width;
    bf16 *e;                     // [M][heads*width]
    long long *ids_out;          // optional [M][heads]
};

// Row id of head h for a token and its predecessors.
__device__ __forceinline__ long long ple_row_id(const PleGatherArgs &a, int m, int h) {
    const int eos = c_ng.eos;
    const int t0 = a.ctx[m * 3], c1 = a.ctx[m * 3 + 1], c2 = a.ctx[m * 3 + 2];
    const int t1 = c1 >= 0 ? c1 : eos;
    const int t2 = (c2 >= 0 && t1 != eos) ? c2 : eos;
    const int order = 2 + h / (c_ng.heads / (c_ng.ngram - 1));
    unsigned long long mixed = (unsigned long long)t0 * c_ng.mult[0] ^ (unsigned long long)t1 * c_ng.mult[1];
    if (order >= 3) mixed ^= (unsigned long long)t2 * c_ng.mult[2];
    return ((long long)(mixed % c_ng.sizes[h]) + c_ng.offsets[h]) % a.rows;          // scaled-down synthetic tables wrap
}

// The byte layout in 16-byte pieces: half a warp per row (160 bytes: ten lanes), so a row crosses the host link as one or two
// requests instead of byte loads.  M * heads rows, 16 per block.
constexpr int PLE_G_ROWS = 16;
__global__ void __launch_bounds__(256) ple_gather_f8_kernel(PleGatherArgs a, int total, int heads) {
    const int i = blockIdx.x * PLE_G_ROWS + (threadIdx.x >> 4), lane = threadIdx.x & 15;
    if (i >= total) return;
    const int m = i / heads, h = i - m * heads;
    const long long id = ple_row_id(a, m, h);
    if (a.ids_out && lane == 0) a.ids_out[i] = id;
    const unsigned char *bytes = (const unsigned char *)a.shards[id / a.rows_per_shard] + id % a.rows_per_shard * a.width;
    if ((uintptr_t)bytes & 15) {                                     // a shard that does not start on 16 bytes
        for (int j = lane; j < a.width; j += 16) a.e[(long long)i * a.width + j] = __float2bfloat16(c_f8_lut[bytes[j]]);
        return;
    }
    const uint4 *row = reinterpret_cast<const uint4 *>(bytes);
    uint4 *out = reinterpret_cast<uint4 *>(a.e + (long long)i * a.width);
    for (int j = lane; j < a.width / 16; j += 16) {
        const uint4 v = row[j];
        const uint32_t b[4] = {v.x, v.y, v.z, v.w};
        uint32_t o[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            o[2 * k] = pack_bf16(c_f8_lut[b[k] & 255u], c_f8_lut[(b[k] >> 8) & 255u]);
            o[2 * k + 1] = pack_bf16(c_f8_lut[(b[k] >> 16) & 255u], c_f8_lut[b[k] >> 24]);
        }
        out[2 * j] = make_uint4(o[0], o[1], o[2], o[3]);
        out[2 * j + 1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
}

// Every layout, element by element.  grid (M, heads), 64 threads.
__global__ void ple_gather_kernel(PleGatherArgs a) {
    const int m = blockIdx.x, h = blockIdx.y;
    const long long id = ple_row_id(a, m, h);
    if (a.ids_out && threadIdx.x == 0) a.ids_out[m * c_ng.heads + h] = id;
    const long long sh = id / a.rows_per_shard, r = id % a.rows_per_shard;
    bf16 *out = a.e + ((long long)m * c_ng.heads + h) * a.width;
    const int W = a.width;
    if (a.layout == PLE_F8) {
        const unsigned char *row = (const unsigned char *)a.shards[sh] + r * W;
        for (int j = threadIdx.x; j < W; j += blockDim.x) out[j] = __float2bfloat16(c_f8_lut[row[j]]);
    } else if (a.layout == PLE_BF16) {
        const bf16 *row = (const bf16 *)a.shards[sh] + r * W;
        for (int j = threadIdx.x; j < W; j += blockDim.x) out[j] = row[j];
    } else if (a.layout == PLE_INT8) {
        const signed char *row = (const signed char *)a.shards[sh] + r * W;
        const __half *sc = (const __half *)a.scales[sh] + r * (W / 16);
        for (int j = threadIdx.x; j < W; j += blockDim.x) out[j] = __float2bfloat16(float(row[j]) * __half2float(sc[j / 16]));
    } else {
        const unsigned char *row = (const unsigned char *)a.shards[sh] + r * (W / 2);
        const __half *sc = (const __half *)a.scales[sh] + r * (W / 16);
        for (int j = threadIdx.x; j < W; j += blockDim.x) {
            const unsigned char b = row[j >> 1];
            const int q = (j & 1) ? (b >> 4) : (b & 0xf);
            out[j] = __float2bfloat16(float(q - 8) * __half2float(sc[j / 16]));
        }
    }
}

// grid (M, hc), 256 threads.  kv[m] = [ key (hc x SH) | value (SH) ] fp32.
// send[m][3s..3s+2] = sum k^2, sum x^2, sum k(1+wk) x(1+wq); send[m][3*hc] = sum v^2.
__global__ void __launch_bounds__(256) ple_stats_kernel(const float *kv, int ld_kv, const float *X, const float *nk1,
                                                        const float *nq1, int SH, int hc, float *send, int ld_send) {
    __shared__ float scratch[32];
    const int m = blockIdx.x, s = blockIdx.y;
    const float *k = kv + (long long)m * ld_kv + s * SH;
    const float *x = X + ((long long)m * hc + s) * SH;
    float kk = 0.f, xx = 0.f, kx = 0.f, vv = 0.f;
    for (int c = threadIdx.x; c < SH; c += 256) {
        const float kc = k[c], xc = x[c];
        kk = fmaf(kc, kc, kk);
        xx = fmaf(xc, xc, xx);
        kx = fmaf(kc * nk1[s * SH + c], xc * nq1[s * SH + c], kx);
        if (s == 0) {
            const float v = kv[(long long)m * ld_kv + hc * SH + c];
            vv = fmaf(v, v, vv);
        }
    }
    kk = block_sum<256>(kk, scratch);
    xx = block_sum<256>(xx, scratch);
    kx = block_sum<256>(kx, scratch);
    if (s == 0) vv = block_sum<256>(vv, scratch);
    if (threadIdx.x == 0) {
        float *o = send + (long long)m * ld_send;
        o[3 * s] = kk; o[3 * s + 1] = xx; o[3 * s + 2] = kx;
        if (s == 0) o[3 * hc] = vv;
    }
}

__device__ __forceinline__ float4 ple_ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// Gate, gated value gv and normalised conv input nc for the batch rows, V columns per thread.  grid (M, hc, ceil(SH / 256 V)).
template <int V>
__global__ void __launch_bounds__(256) ple_nc_kernel(const float *kv, int ld_kv, const float *red, int ld_red,
                                                     const float *nc1, int SH, int hc, int H, float eps, float *gv,
                                                     float *nc) {
    const int m = blockIdx.x, s = blockIdx.y, c = (blockIdx.z * 256 + threadIdx.x) * V;
    if (c >= SH) return;
    const float *r = red + (long long)m * ld_red;
    const float rk = rsqrtf(r[3 * s] / float(H) + eps), rq = rsqrtf(r[3 * s + 1] / float(H) + eps);
    const float gs = r[3 * s + 2] * rk * rq * rsqrtf(float(H));
    const float mag = sqrtf(fmaxf(fabsf(gs), 1e-6f));
    const float gate = sigmoidf_(gs < 0.f ? -mag : (gs > 0.f ? mag : 0.f));
    const float rn = rsqrtf(gate * gate * r[3 * hc] / float(H) + eps);
    float g[V], w[V];
    ld_cols<V>(kv + (long long)m * ld_kv + hc * SH + c, g);
    ld_cols<V>(nc1 + s * SH + c, w);
#pragma unroll
    for (int k = 0; k < V; ++k) {
        g[k] *= gate;
        w[k] = g[k] * rn * w[k];
    }
    const long long o = ((long long)m * hc + s) * SH + c;
    st_cols<V>(gv + o, g);
    st_cols<V>(nc + o, w);
}

// X += gv + silu(dilated conv of nc); taps at p-9, p-6, p-3, p from the batch or the ring.  Four columns and `rows_per` rows per
// thread: one row per block when there are few (a step of one row used four blocks and took 34 us, now 5), several with
// the taps' weights in registers when there are many (4096 rows: 300 us, now 150).  grid (ceil(M / rows_per), ceil(xw / 1024)).
constexpr int PLE_TAPS = 4;
__global__ void __launch_bounds__(256) ple_conv_kernel(const float *gv, const float *nc, const float *ring, const float *cw,
                                                       int xw, int dil, Rows rows, int rows_per, float *X) {
    const int col = (blockIdx.y * 256 + threadIdx.x) * 4;
    if (col >= xw) return;
    float w[4][PLE_TAPS];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 t = ple_ld4(cw + (col + i) * PLE_TAPS);
        w[i][0] = t.x; w[i][1] = t.y; w[i][2] = t.z; w[i][3] = t.w;
    }
    const int m1 = min(rows.M, (int)(blockIdx.x + 1) * rows_per);
    for (int m = blockIdx.x * rows_per; m < m1; ++m) {
        const int slot = rows.slot[m], pos = rows.pos[m], rs = rows.run_start[m];
        const float *rg = ring + (long long)slot * PLE_RING * xw;
        float4 v[PLE_TAPS];
#pragma unroll
        for (int k = 0; k < PLE_TAPS; ++k) {
            const int back = (PLE_TAPS - 1 - k) * dil, q = pos - back;
            if (m - back >= rs) v[k] = ple_ld4(nc + (long long)(m - back) * xw + col);
            else if (q >= 0) v[k] = ple_ld4(rg + (q % PLE_RING) * xw + col);
            else v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        float *xp = X + (long long)m * xw + col;
        float4 x = ple_ld4(xp);
        const float4 g = ple_ld4(gv + (long long)m * xw + col);
        float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < PLE_TAPS; ++k) {
            a[0] = fmaf(w[0][k], v[k].x, a[0]); a[1] = fmaf(w[1][k], v[k].y, a[1]);
            a[2] = fmaf(w[2][k], v[k].z, a[2]); a[3] = fmaf(w[3][k], v[k].w, a[3]);
        }
        x.x += g.x + siluf_(a[0]); x.y += g.y + siluf_(a[1]); x.z += g.z + siluf_(a[2]); x.w += g.w + siluf_(a[3]);
        *reinterpret_cast<float4 *>(xp) = x;
    }
}

// The same for any number of taps, width and address: a row and a column per thread.  grid (M, ceil(xw / 256)).
__global__ void __launch_bounds__(256) ple_conv_any_kernel(const float *gv, const float *nc, const float *ring, const float *cw,
                                                           int xw, int taps, int dil, Rows rows, float *X) {
    const int m = blockIdx.x, col = blockIdx.y * 256 + threadIdx.x;
    if (col >= xw) return;
    const int slot = rows.slot[m], pos = rows.pos[m], rs = rows.run_start[m];
    const float *rg = ring + (long long)slot * PLE_RING * xw;
    float acc = 0.f;
    for (int k = 0; k < taps; ++k) {
        const int back = (taps - 1 - k) * dil, q = pos - back;
        const float v = m - back >= rs ? nc[(long long)(m - back) * xw + col] : q >= 0 ? rg[(q % PLE_RING) * xw + col] : 0.f;
        acc = fmaf(cw[col * taps + k], v, acc);
    }
    X[(long long)m * xw + col] += gv[(long long)m * xw + col] + siluf_(acc);
}

// Stores the batch's last nc rows of every run in the ring (after ple_conv has read it).  grid (ceil(M / rows_per), ceil(xw / 256 V)).
template <int V>
__global__ void __launch_bounds__(256) ple_ring_kernel(const float *nc, float *ring, int xw, Rows rows, int rows_per) {
    const int col = (blockIdx.y * 256 + threadIdx.x) * V;
    if (col >= xw) return;
    const int m1 = min(rows.M, (int)(blockIdx.x + 1) * rows_per);
    for (int m = blockIdx.x * rows_per; m < m1; ++m) {
        const int rs = rows.run_start[m], len = rows.run_len[rs];
        if ((m - rs) < len - PLE_RING) continue;
        float v[V];
        ld_cols<V>(nc + (long long)m * xw + col, v);
        st_cols<V>(ring + ((long long)rows.slot[m] * PLE_RING + (rows.pos[m] % PLE_RING)) * xw + col, v);
    }
}

}  // namespace qw

using namespace qw;

QW_API int qwk_ple_init(const unsigned long long *mult, int ngram, const unsigned long long *sizes,
                        const long long *offsets, int heads, int eos, const float *f8_lut) {
    if (heads > MAX_NGRAM_HEADS || ngram > 4 || ngram < 2) return -1;
    NgramConst c;
    for (int i = 0; i < ngram; ++i) c.mult[i] = mult[i];
    for (int i = 0; i < heads; ++i) { c.sizes[i] = sizes[i]; c.offsets[i] = offsets[i]; }
    c.ngram = ngram; c.heads = heads; c.eos = eos;
    if (cudaMemcpyToSymbol(c_ng, &c, sizeof(c)) != cudaSuccess) return -2;
    if (f8_lut && cudaMemcpyToSymbol(c_f8_lut, f8_lut, 256 * sizeof(float)) != cudaSuccess) return -2;
    return 0;
}

QW_API int qwk_ple_gather(const int *ctx, const void *const *shards, const void *const *scales, long long rows_per_shard,
                          long long rows, int layout, int width, int heads, void *e, long long *ids_out, int M,
                          cudaStream_t s) {
    PleGatherArgs a;
    a.ctx = ctx; a.shards = shards; a.scales = scales; a.rows_per_shard = rows_per_shard; a.rows = rows;
    a.layout = layout; a.width = width; a.e = (bf16 *)e; a.ids_out = ids_out;
    if (layout == PLE_F8 && width % 16 == 0 && ((uintptr_t)e & 15) == 0) {
        const int total = M * heads;
        ple_gather_f8_kernel<<<(total + PLE_G_ROWS - 1) / PLE_G_ROWS, 256, 0, s>>>(a, total, heads);
    } else {
        dim3 grid(M, heads);
        ple_gather_kernel<<<grid, 64, 0, s>>>(a);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

QW_API int qwk_ple_stats(const float *kv, int ld_kv, const float *X, const float *nk1, const float *nq1, int SH, int hc,
                         float *send, int ld_send, int M, cudaStream_t s) {
    dim3 grid(M, hc);
    ple_stats_kernel<<<grid, 256, 0, s>>>(kv, ld_kv, X, nk1, nq1, SH, hc, send, ld_send);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

QW_API int qwk_ple_apply(const float *kv, int ld_kv, const float *red, int ld_red, const float *nc1, const float *cw,
                         int SH, int hc, int H, float eps, int taps, int dil, float *gv, float *nc, float *ring,
                         float *X, int M, const int *slot, const int *pos, const int *run_start, const int *run_len,
                         cudaStream_t s) {
    Rows rows{M, slot, pos, run_start, run_len};
    const int xw = hc * SH;
    if (((SH | ld_kv) & 3) == 0 && taps == PLE_TAPS && aligned16(kv, nc1, cw, gv, nc, ring, X)) {
        const int rows_per = M >= 256 ? 8 : 1, cb = (xw + 1023) / 1024, rb = (M + rows_per - 1) / rows_per;
        ple_nc_kernel<4><<<dim3(M, hc, (SH + 1023) / 1024), 256, 0, s>>>(kv, ld_kv, red, ld_red, nc1, SH, hc, H, eps, gv, nc);
        ple_conv_kernel<<<dim3(rb, cb), 256, 0, s>>>(gv, nc, ring, cw, xw, dil, rows, rows_per, X);
        ple_ring_kernel<4><<<dim3(rb, cb), 256, 0, s>>>(nc, ring, xw, rows, rows_per);
    } else {
        const int cb = (xw + 255) / 256;
        ple_nc_kernel<1><<<dim3(M, hc, (SH + 255) / 256), 256, 0, s>>>(kv, ld_kv, red, ld_red, nc1, SH, hc, H, eps, gv, nc);
        ple_conv_any_kernel<<<dim3(M, cb), 256, 0, s>>>(gv, nc, ring, cw, xw, taps, dil, rows, X);
        ple_ring_kernel<1><<<dim3(M, cb), 256, 0, s>>>(nc, ring, xw, rows, 1);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
