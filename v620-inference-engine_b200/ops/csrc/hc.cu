// Hyper-connection kernels for row batches (decode rows and prefill rows alike).
//
// The residual X has `hc` streams; a rank owns SH = H/ranks columns of each, X[m][s][c] fp32.
// A mixer is computed as
//   pre : X += pend * 2*sigmoid(inj/hc) (deferred combine of the previous block), y = bf16(X*(1+w)),
//         ssq[s] = sum_c X^2                                          (hc_pre)
//   down: part[s][j] = sum_c Wd[j][s,c] * y[s][c]                     (bf16 GEMV with column splits)
//   --- all-reduce of [ssq | part] over ranks ---
//   up  : r_s = rsqrt(ssq_s/H + eps); d_j = sum_s r_s part[s][j]; inj = d[rank..rank+hc);
//         u = silu(d/hc); g[s][c] = Wu[c][s] . u; block_in[c] = mean_s sigmoid(g) * y[s][c] * r_s   (hc_up_mix)
// which uses that the down projection is linear in the un-normalised y (the algebra of the
// reference's src/kernels/hc.hip:98-166 and src/engine/decode.hip:53-61).
#include "fuse.cuh"
#include "mma.cuh"

#include <cooperative_groups.h>

namespace qw {

// X[m][s][:] = embedding row of tokens[m] (this rank's columns) for every stream.  V columns per thread, grid (M, ceil(SH / 256 V)).
template <int V>
__global__ void __launch_bounds__(256) embed_rows_kernel(const int *tokens, const bf16 *table, int ld_table, int col0, int SH, int hc,
                                                         int vocab, float *X) {
    const int m = blockIdx.x, c = (blockIdx.y * 256 + threadIdx.x) * V;
    int t = tokens[m];
    QW_DCHECK(t >= 0 && t < vocab, 0x01000000u | (unsigned)(m & 0xffffff));          // token id outside the vocabulary (row m)
    if (t < 0 || t >= vocab) t = 0;
    if (c >= SH) return;
    float v[V];
    ld_cols<V>(table + (long long)t * ld_table + col0 + c, v);
    for (int s = 0; s < hc; ++s) st_cols<V>(X + ((long long)m * hc + s) * SH + c, v);
}

// V columns per thread and step.  grid (M, hc).  pend may be null (no deferred combine).  y and ssq may be null (combine only).
template <int V>
__global__ void __launch_bounds__(256) hc_pre_kernel(float *X, const float *pend, int ld_pend, const float *inj, int ld_inj,
                                                     const float *w1 /* (1+w) [hc][SH] */, int SH, int hc, bf16 *y,
                                                     float *ssq, int ld_ssq) {
    __shared__ float scratch[32];
    const int m = blockIdx.x, s = blockIdx.y;
    float *x = X + ((long long)m * hc + s) * SH;
    float coef = 0.f;
    if (pend) coef = 2.f * sigmoidf_(inj[(long long)m * ld_inj + s] / float(hc));
    float acc = 0.f;
#pragma unroll 3
    for (int c = threadIdx.x * V; c < SH; c += 256 * V) {
        float v[V];
        ld_cols<V>(x + c, v);
        if (pend) {
            float p[V];
            ld_cols<V>(pend + (long long)m * ld_pend + c, p);
#pragma unroll
            for (int k = 0; k < V; ++k) v[k] = fmaf(p[k], coef, v[k]);
            st_cols<V>(x + c, v);
        }
        if (y) {
            float w[V];
            ld_cols<V>(w1 + s * SH + c, w);
#pragma unroll
            for (int k = 0; k < V; ++k) w[k] *= v[k];
            st_cols<V>(y + ((long long)m * hc + s) * SH + c, w);
        }
#pragma unroll
        for (int k = 0; k < V; ++k) acc = fmaf(v[k], v[k], acc);
    }
    if (ssq) {
        acc = block_sum<256>(acc, scratch);
        if (threadIdx.x == 0) ssq[(long long)m * ld_ssq + s] = acc;
    }
}

constexpr int UP_ROWS = 4;     // rows per block of the fused hc_up_mix
constexpr int UP_MAXI = 5;     // 16-byte weight pieces per lane: covers mixer ranks up to 320

// FUSED: the form with the collectives inside (several ranks): waits for the all-reduce of the down projection, sends the all-gather.
// Otherwise: without them, for more low-rank and inject rows than hc_up_mma_kernel has threads.
// grid (ceil(SH/8), ceil(M/UPR)), 256 threads.  hc must be 4 (one 8-lane group per stream).
// y[s][c] = bf16(X[s][c] * w1[s][c]) is recomputed here exactly as hc_down_kernel computed it.
template <bool FUSED, int UPR>
__global__ void __launch_bounds__(256, 3) hc_up_mix_kernel(const float *red, int ld_red, const bf16 *Wu /* [SH][hc][R] */,
                                                        const float *X, const float *w1, int SH, int hc, int R, int hc_down,
                                                        float inv_H, float eps, int M, float *inj, int ld_inj, bf16 *bin,
                                                        int ld_bin, int bin_col0, FuseIn fi, FuseOut fo) {
    extern __shared__ float sm[];
    float *u = sm;                         // [UPR][R]
    float *rs = sm + UPR * R;          // [UPR][hc]
    const int m0 = blockIdx.y * UPR;
    const int nrow = min(UPR, M - m0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x * 8 + warp;
    const int s = lane >> 3, li = lane & 7;
    const int nch = R >> 3;
    // weights first: they do not depend on the predecessor
    uint4 w[UP_MAXI];
    if (c < SH) {
        const uint4 *wp = reinterpret_cast<const uint4 *>(Wu + ((long long)c * hc + s) * R);
#pragma unroll
        for (int i = 0; i < UP_MAXI; ++i)
            if (li + 8 * i < nch) w[i] = ld_stream(wp + li + 8 * i);
    }
    pdl_wait();
    pdl_trigger();
    // this lane's residual values times the norm weight: needed only at the very end, fetched now so that their L2
    // round trip overlaps the staging of the reduced vector
    float xw[UPR];
    {
        const float w1v = c < SH ? w1[s * SH + c] : 0.f;
#pragma unroll
        for (int mm = 0; mm < UPR; ++mm)
            xw[mm] = (c < SH && mm < nrow) ? __ldcg(X + ((long long)(m0 + mm) * hc + s) * SH + c) * w1v : 0.f;
    }
    // the reduced vector (FUSED: the ranks' words added in rank order), staged once per block into shared memory, with every
    // thread's loads in flight together
    float *reds = rs + UPR * hc;       // [UPR][ld_red]
    if constexpr (!FUSED) {
        const int used = hc + hc * hc_down;
        for (int i = threadIdx.x; i < nrow * used; i += 256) reds[i / used * ld_red + i % used] = __ldcg(red + (long long)(m0 + i / used) * ld_red + i % used);
    }
    const unsigned int seq_in = FUSED ? fuse_seq(fi) : 0u;
    // what this mixer's down projection wrote of each row (an even count), as pairs of words; a thread has
    // the loads of two pairs from four ranks in flight at once
    const int npair = (hc + hc * hc_down) >> 1, total = FUSED ? nrow * npair : 0;
    for (int p0 = threadIdx.x; p0 < total; p0 += 512) {
        const int p1 = p0 + 256;
        const bool two = p1 < total;
        const int mm0 = p0 / npair, j0 = (p0 - mm0 * npair) * 2;
        const int mm1 = two ? p1 / npair : mm0, j1 = two ? (p1 - mm1 * npair) * 2 : j0;
        float2 a, b;
        fuse_sum2x2(fi, seq_in, (long long)(m0 + mm0) * ld_red + j0, (long long)(m0 + mm1) * ld_red + j1, a, b);
        reds[mm0 * ld_red + j0] = a.x;
        reds[mm0 * ld_red + j0 + 1] = a.y;
        if (two) {
            reds[mm1 * ld_red + j1] = b.x;
            reds[mm1 * ld_red + j1 + 1] = b.y;
        }
    }
    __syncthreads();
    auto red_at = [&](long long i) -> float { return reds[i - (long long)m0 * ld_red]; };
    for (int i = threadIdx.x; i < nrow * hc; i += 256) {
        const int mm = i / hc, ss = i % hc;
        rs[mm * hc + ss] = rsqrtf(red_at((long long)(m0 + mm) * ld_red + ss) * inv_H + eps);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nrow * hc_down; i += 256) {
        const int mm = i / hc_down, j = i % hc_down;
        const long long p = (long long)(m0 + mm) * ld_red + hc + j;
        float d = 0.f;
        for (int ss = 0; ss < hc; ++ss) d = fmaf(rs[mm * hc + ss], red_at(p + ss * hc_down), d);
        if (j < R) u[mm * R + j] = siluf_(d / float(hc));
        else if (inj && blockIdx.x == 0) inj[(long long)(m0 + mm) * ld_inj + (j - R)] = d;
    }
    __syncthreads();
    if (c >= SH) return;
    const unsigned int seq_out = FUSED ? fuse_seq(fo) : 0u;
    float acc[UPR];
#pragma unroll
    for (int mm = 0; mm < UPR; ++mm) acc[mm] = 0.f;
#pragma unroll
    for (int i = 0; i < UP_MAXI; ++i) {
        const int ch = li + 8 * i;
        if (ch < nch) {
            const float wf[8] = {bf16_lo(w[i].x), bf16_hi(w[i].x), bf16_lo(w[i].y), bf16_hi(w[i].y),
                                 bf16_lo(w[i].z), bf16_hi(w[i].z), bf16_lo(w[i].w), bf16_hi(w[i].w)};
#pragma unroll
            for (int mm = 0; mm < UPR; ++mm) {
                if (mm < nrow) {
                    const float *uu = u + mm * R + ch * 8;
#pragma unroll
                    for (int k = 0; k < 8; ++k) acc[mm] = fmaf(wf[k], uu[k], acc[mm]);
                }
            }
        }
    }
#pragma unroll
    for (int mm = 0; mm < UPR; ++mm) {
        float g = acc[mm];
        g += __shfl_xor_sync(0xffffffffu, g, 1);
        g += __shfl_xor_sync(0xffffffffu, g, 2);
        g += __shfl_xor_sync(0xffffffffu, g, 4);
        float v = 0.f;
        if (mm < nrow) {
            const float yv = __bfloat162float(__float2bfloat16(xw[mm]));
            v = sigmoidf_(g) * yv * rs[mm * hc + s];
        }
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (lane == 0 && mm < nrow) {
            const bf16 o = __float2bfloat16(v / float(hc));
            if (FUSED) fuse_put_all(fo, seq_out, m0 + mm, c, (unsigned int)__bfloat16_as_ushort(o));      // fused all-gather
            else bin[(long long)(m0 + mm) * ld_bin + bin_col0 + c] = o;
        }
    }
}

// ------------------------------------------------------------------------------------------
// Fused mixer front end: deferred combine + per-stream sum of squares + down projection.
//   Xout[m][s][:] = Xin[m][s][:] + pend[m][:] * 2*sigmoid(inj_prev[m][s]/hc)     (when pend != null)
//   send[m][s]               = sum_c X^2
//   send[m][hc + s*down + j] = sum_c Wd[j][s][c] * bf16(X[s][c] * w1[s][c])
// Every block rebuilds the bf16 row slice it needs in shared memory (the residual is tiny and
// sits in L2); blocks with blockIdx.x == 0 also store X and the sums of squares.  X is written
// to a second buffer because other blocks still read the old one.
// grid (ceil(down/rpb), hc, ceil(M/8)), 256 threads, dynamic smem 8*SH bf16.
// ------------------------------------------------------------------------------------------
constexpr int DN_PF = 5;      // 16-byte weight pieces per lane fetched before the dependency wait (2560 columns / 2 warps / 32 lanes / 8)

struct HcDownArgs {
    const float *Xin;
    float *Xout;            // null: no combine, X stays where it is
    const float *pend;      // [M][ld_pend] or null
    int ld_pend;
    const float *inj_prev;  // [M][hc]
    const float *w1;        // [hc][SH]
    const bf16 *Wd;         // [down][hc][SH]
    float *send;            // [M][ld_send]
    int ld_send, SH, hc, down, M, wpr;
    FuseIn fi;              // fused reduce-scatter: `pend` is the sum of the ranks' slots
    FuseOut fo;             // fused all-reduce of `send`
};

// FUSED: the form with the collectives inside (several ranks).  Otherwise: without them, for rows that hc_down_mma_kernel has no room for.
template <bool FUSED>
__global__ void __launch_bounds__(256, 3) hc_down_kernel(HcDownArgs a) {
    extern __shared__ __align__(16) unsigned char smraw[];
    bf16 *ybuf = reinterpret_cast<bf16 *>(smraw);          // [8][SH]
    __shared__ float part[8][8];
    __shared__ float scratch[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s = blockIdx.y, m0 = blockIdx.z * 8;
    const int nrow = min(8, a.M - m0);
    const int wpr = a.wpr, rpb = 8 / wpr;
    const int j = blockIdx.x * rpb + warp / wpr, kw = warp % wpr;
    const int nchunk = a.SH >> 3;
    const bf16 *wrow = a.Wd + ((long long)j * a.hc + s) * a.SH;
    // weights first: prefetch this warp's share of its row into registers / L2
    uint4 w0[DN_PF];          // this warp's share of its weight row: all of it for the model's shapes, so no load is issued late
    const int stride = wpr * 32;
    if (j < a.down) {
#pragma unroll
        for (int u = 0; u < DN_PF; ++u) {
            const int c = kw * 32 + lane + u * stride;
            if (c < nchunk) w0[u] = ld_stream(reinterpret_cast<const uint4 *>(wrow) + c);
        }
    }
    pdl_wait();
    pdl_trigger();
    const bool scattered = FUSED && a.fi.active;
    const unsigned int seq_in = scattered ? fuse_seq(a.fi) : 0u;
    const unsigned int seq_out = FUSED ? fuse_seq(a.fo) : 0u;
    for (int r = 0; r < nrow; ++r) {           // the whole block builds each row slice: short dependent chains
        const int m = m0 + r;
        const float *xin = a.Xin + ((long long)m * a.hc + s) * a.SH;
        float coef = 0.f;
        if (a.pend) coef = 2.f * sigmoidf_(a.inj_prev[(long long)m * a.hc + s] / float(a.hc));
        float ss = 0.f;
        constexpr int CP = 1;                          // the ranks' words are in flight as well (SH is a shard)
        for (int c0 = threadIdx.x * 4; c0 < a.SH; c0 += 1024 * CP) {
            float4 xv[CP], pv[CP], wv[CP];
#pragma unroll
            for (int q = 0; q < CP; ++q) {
                const int c = c0 + q * 1024;
                if (c < a.SH) {
                    xv[q] = __ldcg(reinterpret_cast<const float4 *>(xin + c));
                    wv[q] = __ldg(reinterpret_cast<const float4 *>(a.w1 + s * a.SH + c));
                    if (a.pend && !scattered) pv[q] = __ldcg(reinterpret_cast<const float4 *>(a.pend + (long long)m * a.ld_pend + c));
                }
            }
#pragma unroll
            for (int q = 0; q < CP; ++q) {
                const int c = c0 + q * 1024;
                if (c < a.SH) {
                    float4 v = xv[q];
                    if (a.pend) {
                        // fused reduce-scatter: the ranks' parts of the block output, added in rank order
                        const float4 p = scattered ? fuse_sum4(a.fi, seq_in, (long long)m * a.ld_pend + c) : pv[q];
                        v.x = fmaf(p.x, coef, v.x); v.y = fmaf(p.y, coef, v.y);
                        v.z = fmaf(p.z, coef, v.z); v.w = fmaf(p.w, coef, v.w);
                        if (blockIdx.x == 0) *reinterpret_cast<float4 *>(a.Xout + ((long long)m * a.hc + s) * a.SH + c) = v;
                    }
                    ss = fmaf(v.x, v.x, ss); ss = fmaf(v.y, v.y, ss); ss = fmaf(v.z, v.z, ss); ss = fmaf(v.w, v.w, ss);
                    uint2 pk;
                    pk.x = pack_bf16(v.x * wv[q].x, v.y * wv[q].y);
                    pk.y = pack_bf16(v.z * wv[q].z, v.w * wv[q].w);
                    *reinterpret_cast<uint2 *>(ybuf + r * a.SH + c) = pk;
                }
            }
        }
        if (blockIdx.x == 0) {                 // block-uniform: only these blocks need the sum of squares
            ss = block_sum<256>(ss, scratch);
            if (threadIdx.x == 0) {
                if (FUSED) fuse_put_all(a.fo, seq_out, m, s, __float_as_uint(ss));      // fused all-reduce
                else a.send[(long long)m * a.ld_send + s] = ss;
            }
        }
    }
    __syncthreads();
    float acc[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) acc[m] = 0.f;
    if (j < a.down) {
        for (int c0 = kw * 32 + lane, first = 1; c0 < nchunk; c0 += DN_PF * stride, first = 0) {
            uint4 w[DN_PF];
#pragma unroll
            for (int u = 0; u < DN_PF; ++u) {
                const int c = c0 + u * stride;
                if (c < nchunk) w[u] = first ? w0[u] : ld_stream(reinterpret_cast<const uint4 *>(wrow) + c);
            }
#pragma unroll
            for (int u = 0; u < DN_PF; ++u) {
                const int c = c0 + u * stride;
                if (c < nchunk) {
#pragma unroll
                    for (int m = 0; m < 8; ++m)
                        if (m < nrow) acc[m] = dot8(w[u], *reinterpret_cast<const uint4 *>(ybuf + m * a.SH + c * 8), acc[m]);
                }
            }
        }
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) acc[m] = warp_sum(acc[m]);
    if (wpr > 1) {
        if (lane == 0) {
#pragma unroll
            for (int m = 0; m < 8; ++m) part[warp][m] = acc[m];
        }
        __syncthreads();
        if (kw == 0) {
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                float t = 0.f;
                for (int q = 0; q < wpr; ++q) t += part[warp + q][m];
                acc[m] = t;
            }
        }
    }
    if (kw == 0 && lane == 0 && j < a.down) {
#pragma unroll
        for (int m = 0; m < 8; ++m)
            if (m < nrow) {
                if (FUSED) fuse_put_all(a.fo, seq_out, m0 + m, a.hc + s * a.down + j, __float_as_uint(acc[m]));
                else a.send[(long long)(m0 + m) * a.ld_send + a.hc + s * a.down + j] = acc[m];
            }
    }
}

// ------------------------------------------------------------------------------------------
// The same two kernels without collectives, on the tensor cores (mma.sync m16n8k16): the rows of the step are the 16-row
// operand and eight weight rows the 8-column one, so up to 16 rows cost what one costs, and a row's sums do not depend on the
// rows beside it.  k is walked in an order that suits the loads (both operands agree): lane (g = lane / 4, q = lane % 4) takes the
// 16 bytes at k = 32 i + 8 q of row g, which are two MMAs' operand words.
// ------------------------------------------------------------------------------------------
// Two sums that the caller adds at the end: one chain of dependent MMAs would be twice as long.
__device__ __forceinline__ void mma_rows(float (&c)[2][4], const uint4 &r, const uint4 &r8, const uint4 &w) {
    mma_bf16(c[0], r.x, r8.x, r.y, r8.y, w.x, w.y);
    mma_bf16(c[1], r.z, r8.z, r.w, r8.w, w.z, w.w);
}

// Sum of N values in pairs: log2 N roundings on the way of each instead of up to N - 1.
template <int N, class F>
__device__ __forceinline__ float pair_sum(const F &at) {
    float v[N];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = at(k);
#pragma unroll
    for (int o = N / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < o; ++k) v[k] += v[k + o];
    return v[0];
}

constexpr int HM_THREADS = 512, HM_PAD = 32;      // padding of shared rows: their stride is 64 bytes off a multiple of 128
constexpr int HD_CL = 8, HD_J = 8, HD_W = HM_THREADS / 32, HD_ROWS = 8, HD_CLUSTER_MIN = 4;
// A CTA owns eight outputs j of one stream over all columns (its sixteen warps take every sixteenth chunk of 32).  The weights go
// to shared memory with cp.async before the dependency wait: no register waits for them, and 64 registers a thread let two CTAs
// share an SM with each other or with the previous kernel's.  The stream's bf16 rows are built eight at a time, in sixteen slices
// of the columns, with the same sums either way:
//   CLUSTER  eight CTAs build two slices each and write them into all eight shared memories; otherwise every CTA would rebuild every
//            row, which at 24 rows was most of the kernel's time
//   else     every CTA builds all slices, a warp each: fewer rows cost less than the cluster's two meetings
// In a chain of its own, us per launch, scalar products before and now: 1 row 6.5, 4.1; 2 rows 8.0, 5.4; 8 rows 19.2, 7.2; 24 rows 44, 20.
// The line between the forms: at 3 rows 6.4 (lone), at 4 rows 5.8 (cluster).
// Error of the sums against 64 bits: 7.8e-8 of their size, as the scalar products had it (running sums kept in the tensor core 1.1e-7,
// and 0.2 us less).
// grid (ceil(down / 8), rounded up to clusters, hc), 512 threads, dynamic smem (8 + min(M, 8)) x (SH + 32) bf16.
template <bool CLUSTER>
__global__ void __launch_bounds__(HM_THREADS, 2) hc_down_mma_kernel(HcDownArgs a) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ float red[HD_W][HD_ROWS][HD_J];
    __shared__ float sspart[HD_W][HD_ROWS];
    const cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int s = blockIdx.y, j0 = blockIdx.x * HD_J, ys = a.SH + HM_PAD;
    bf16 *ws = reinterpret_cast<bf16 *>(smraw), *y = ws + HD_J * ys;
    const int slice = CLUSTER ? (blockIdx.x % HD_CL) * 2 + (warp & 1) : warp;
    const int nch = (a.SH + 31) >> 5;
    const bool writes = blockIdx.x < (CLUSTER ? HD_CL : 1);      // this cluster (CTA) also stores X and the sums of squares
    {
        const int row = warp >> 1, pieces = a.SH >> 3;           // two warps per weight row
        const bf16 *src = a.Wd + ((long long)min(j0 + row, a.down - 1) * a.hc + s) * a.SH;
        for (int k = (warp & 1) * 32 + lane; k < pieces; k += 64) cp_async16(ws + row * ys + k * 8, src + k * 8);
        if (a.SH & 31) {                                         // the last chunk's columns past SH: zeros
            for (int i = tid; i < HD_J * HM_PAD; i += HM_THREADS) ws[i / HM_PAD * ys + a.SH + i % HM_PAD] = __float2bfloat16(0.f);
            for (int i = tid; i < min(a.M, HD_ROWS) * HM_PAD; i += HM_THREADS) y[i / HM_PAD * ys + a.SH + i % HM_PAD] = __float2bfloat16(0.f);
        }
    }
    const int per = ((a.SH >> 2) + HD_W - 1) / HD_W, f0 = slice * per, f1 = min(a.SH >> 2, f0 + per);
    if (CLUSTER) cl.sync();                                      // every CTA of the cluster runs: its memory may be written
    pdl_wait();
    pdl_trigger();
    for (int m0 = 0; m0 < a.M; m0 += HD_ROWS) {
        const int n = min(HD_ROWS, a.M - m0);
        if (CLUSTER && m0) cl.sync();                            // the rows before these are consumed everywhere
        for (int r = CLUSTER ? warp >> 1 : 0; r < n; r += CLUSTER ? HD_W / 2 : 1) {
            const int m = m0 + r;
            const long long row = ((long long)m * a.hc + s) * a.SH;
            float coef = 0.f, ss = 0.f;
            if (a.pend) coef = 2.f * sigmoidf_(a.inj_prev[(long long)m * a.hc + s] / float(a.hc));
            for (int fb = f0; fb < f1; fb += 64) {
                float4 xv[2], wv[2], pv[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int f = fb + lane + 32 * i;
                    if (f >= f1) continue;
                    xv[i] = __ldcg(reinterpret_cast<const float4 *>(a.Xin + row) + f);
                    wv[i] = __ldg(reinterpret_cast<const float4 *>(a.w1 + s * a.SH) + f);
                    if (a.pend) pv[i] = __ldcg(reinterpret_cast<const float4 *>(a.pend + (long long)m * a.ld_pend) + f);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int f = fb + lane + 32 * i;
                    if (f >= f1) continue;
                    float4 v = xv[i];
                    if (a.pend) {
                        v.x = fmaf(pv[i].x, coef, v.x); v.y = fmaf(pv[i].y, coef, v.y);
                        v.z = fmaf(pv[i].z, coef, v.z); v.w = fmaf(pv[i].w, coef, v.w);
                        if (writes) reinterpret_cast<float4 *>(a.Xout + row)[f] = v;
                    }
                    ss = fmaf(v.x, v.x, ss); ss = fmaf(v.y, v.y, ss); ss = fmaf(v.z, v.z, ss); ss = fmaf(v.w, v.w, ss);
                    const uint2 pk = make_uint2(pack_bf16(v.x * wv[i].x, v.y * wv[i].y), pack_bf16(v.z * wv[i].z, v.w * wv[i].w));
                    uint2 *dst = reinterpret_cast<uint2 *>(y + r * ys + f * 4);
                    if (!CLUSTER) {
                        *dst = pk;
                    } else {
#pragma unroll
                        for (int k = 0; k < HD_CL; ++k) *cl.map_shared_rank(dst, k) = pk;
                    }
                }
            }
            if (writes) {
                ss = warp_sum(ss);
                if (lane == 0) *(CLUSTER ? cl.map_shared_rank(&sspart[slice][r], 0) : &sspart[slice][r]) = ss;
            }
        }
        if (m0 == 0) cp_async_wait();
        if (CLUSTER) cl.sync();
        else __syncthreads();
        if (blockIdx.x == 0 && tid < n) {
            a.send[(long long)(m0 + tid) * a.ld_send + s] = pair_sum<HD_W>([&](int k) { return sspart[k][tid]; });
        }
        // operand rows past the last repeat it (and rows 8-15 the first eight): a result row depends on its own operand row alone
        float s0 = 0.f, s1 = 0.f;          // chunks are added with rounding: the tensor core's own running sum cuts off
        const bf16 *ya = y + min(g, n - 1) * ys + q * 8, *wa = ws + g * ys + q * 8;
#pragma unroll 5
        for (int chunk = warp; chunk < nch; chunk += HD_W) {
            const uint4 r = *reinterpret_cast<const uint4 *>(ya + chunk * 32);
            float c[2][4] = {};
            mma_rows(c, r, r, *reinterpret_cast<const uint4 *>(wa + chunk * 32));
            s0 += c[0][0] + c[1][0];
            s1 += c[0][1] + c[1][1];
        }
        *reinterpret_cast<float2 *>(&red[warp][g][2 * q]) = make_float2(s0, s1);
        __syncthreads();
        if (tid < HD_ROWS * HD_J && (tid >> 3) < n && j0 + (tid & 7) < a.down) {
            a.send[(long long)(m0 + (tid >> 3)) * a.ld_send + a.hc + s * a.down + j0 + (tid & 7)] =
                pair_sum<HD_W>([&](int k) { return red[k][tid >> 3][tid & 7]; });
        }
        __syncthreads();
    }
}

constexpr int HM_ROWS = 16;          // rows per pass of hc_up_mma_kernel
constexpr int HU_PAD = HM_PAD, HU_COLS = 16, HU_BATCH = 4, HU_CLUSTER_MIN = 3;
// Two warps own two columns x four streams = eight weight rows, every other chunk of 32 each; a block 16 columns.  The activated
// vector u (fp32) goes through the MMAs as three bf16 parts (24 bits of mantissa: the products and sums are those of fp32
// operands).  A block forms u itself from the down projection's parts (CLUSTER: eight blocks form every eighth row each and
// write it into all eight shared memories), once per 16 rows.  y[s][c] = bf16(X[s][c] * w1[s][c]) as hc_down_mma_kernel has it.
// In a chain of its own, us per launch, scalar products before and now: 1 row 5.4, 6.2 (with hc_down: 12.0, 10.1); 2 rows 8.0, 6.5;
// 8 rows 21.2, 8.3 (lone form 9.3); 24 rows 49.6, 17.9 (lone 21.2).  One row takes it as well, although the scalar kernel would be faster
// there: a row has to come out with the same bits alone and among others, or drafts that equal the model's choice are not accepted.
// grid ceil(SH / 16), rounded up to clusters, 512 threads; hc must be 4; dynamic smem (3 x 16 + 64) x (R rounded up to 32, + 32) bf16.
template <bool CLUSTER>
__global__ void __launch_bounds__(HM_THREADS, 2) hc_up_mma_kernel(const float *red, int ld_red, const bf16 *Wu /* [SH][hc][R] */, const float *X,
                                                           const float *w1, int SH, int R, int hc_down, float inv_H, float eps, int M,
                                                           float *inj, int ld_inj, bf16 *bin, int ld_bin, int bin_col0) {
    namespace cg = cooperative_groups;
    constexpr int hc = 4;
    extern __shared__ __align__(16) unsigned char smraw[];
    const cg::cluster_group cl = cg::this_cluster();
    __shared__ __align__(16) float rs[HM_ROWS][hc];
    __shared__ float4 other[8][32];
    bf16 *u = reinterpret_cast<bf16 *>(smraw);                   // [3][16][us]
    const int R32 = (R + 31) & ~31, us = R32 + HU_PAD, part = HM_ROWS * us;
    const int tid = threadIdx.x, pair = (tid >> 5) & 7, half = tid >> 8, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int c0 = blockIdx.x * HU_COLS + pair * 2;              // this pair's columns c0, c0 + 1; as operand: weight rows 4 c0 + g
    bf16 *ws = u + 3 * part;                                     // [64][us]: row 4 (column) + stream
    {
        // the block's 64 rows are one piece of memory; four rows per warp.  piece / (R / 8) by a multiplication (few and small)
        const int rp = R >> 3, inv = 65536 / rp + 1, row0 = (tid >> 5) * 4, rows = min(4 * HU_COLS, (SH - (int)blockIdx.x * HU_COLS) * hc);
        const bf16 *src = Wu + ((long long)blockIdx.x * HU_COLS * hc + row0) * R;
        for (int p = lane; p < 4 * rp; p += 32) {
            const int row = row0 + (p * inv >> 16);
            if (row < rows) cp_async16(ws + row * us + (p - (row - row0) * rp) * 8, src + p * 8);
        }
    }
    if (R32 != R)
        for (int i = tid; i < 4 * HU_COLS * (R32 - R); i += HM_THREADS) ws[i / (R32 - R) * us + R + i % (R32 - R)] = __float2bfloat16(0.f);
    if (R32 != R)
        for (int i = tid; i < 3 * HM_ROWS * (R32 - R); i += HM_THREADS) u[i / (R32 - R) * us + R + i % (R32 - R)] = __float2bfloat16(0.f);
    // in the result this lane holds rows g and g + 8 of streams s, s + 1 of column c
    const int c = c0 + (q >> 1), s = (2 * q) & 3;
    const bool c_ok = c < SH;
    const float wa = c_ok ? w1[s * SH + c] : 0.f, wb = c_ok ? w1[(s + 1) * SH + c] : 0.f;
    if (CLUSTER) cl.sync();                                      // every CTA of the cluster runs: its memory may be written
    pdl_wait();
    pdl_trigger();
    for (int m0 = 0; m0 < M; m0 += HM_ROWS) {
        const int n = min(HM_ROWS, M - m0);
        float xa[2], xb[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const bool ok = c_ok && g + 8 * h < n && half == 0;
            const float *x = X + ((long long)(m0 + g + 8 * h) * hc + s) * SH + c;
            xa[h] = ok ? __ldcg(x) * wa : 0.f;
            xb[h] = ok ? __ldcg(x + SH) * wb : 0.f;
        }
        // u: a thread per mixer row j, a few rows of the step per round (CLUSTER: every eighth row, for all eight CTAs); the first
        // round's loads are on their way while the rows' norms are formed
        if (CLUSTER && m0) cl.sync();                            // the rows before these are consumed everywhere
        constexpr int STEP = CLUSTER ? HD_CL : 1, BATCH = CLUSTER ? 2 : HU_BATCH;
        const int first = CLUSTER ? (int)cl.block_rank() : 0;
        for (int mb = first; mb < n || mb == first; mb += STEP * BATCH) {
            float v[BATCH][hc];
            const float *p = red + (long long)(m0 + mb) * ld_red + hc + tid;
#pragma unroll
            for (int b = 0; b < BATCH; ++b)
#pragma unroll
                for (int k = 0; k < hc; ++k) v[b][k] = tid < hc_down && mb + b * STEP < n ? __ldcg(p + b * STEP * ld_red + k * hc_down) : 0.f;
            if (mb == first) {
                if (tid < n * hc) rs[tid >> 2][tid & 3] = rsqrtf(__ldcg(red + (long long)(m0 + (tid >> 2)) * ld_red + (tid & 3)) * inv_H + eps);
                __syncthreads();
            }
#pragma unroll
            for (int b = 0; b < BATCH; ++b) {
                const int m = mb + b * STEP;
                if (m >= n) break;
                const float4 r = *reinterpret_cast<const float4 *>(rs[m]);
                const float d = fmaf(r.w, v[b][3], fmaf(r.z, v[b][2], fmaf(r.y, v[b][1], r.x * v[b][0])));
                const float f = siluf_(d * (1.f / float(hc)));
                const bf16 hi = __float2bfloat16(f);
                const float r1 = f - __bfloat162float(hi);
                const bf16 mid = __float2bfloat16(r1);
                const bf16 lo = __float2bfloat16(r1 - __bfloat162float(mid));
                bf16 *o = u + m * us + tid;
                if (!CLUSTER) {
                    if (tid < R) {
                        o[0] = hi;
                        o[part] = mid;
                        o[2 * part] = lo;
                    }
                } else {
                    // neighbours' values in one word: R is even, so a pair is written or not as a whole
                    uint32_t w[3] = {__bfloat16_as_ushort(hi), __bfloat16_as_ushort(mid), __bfloat16_as_ushort(lo)};
#pragma unroll
                    for (int k = 0; k < 3; ++k) w[k] |= __shfl_down_sync(0xffffffffu, w[k], 1) << 16;
                    if (tid < R && !(tid & 1))
#pragma unroll
                        for (int c = 0; c < HD_CL; ++c) {
                            bf16 *oc = cl.map_shared_rank(o, c);
#pragma unroll
                            for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t *>(oc + k * part) = w[k];
                        }
                }
                if (tid >= R && tid < hc_down && inj && blockIdx.x < STEP) inj[(long long)(m0 + m) * ld_inj + (tid - R)] = d;
            }
        }
        if (m0 == 0) cp_async_wait();
        if (CLUSTER) cl.sync();
        else __syncthreads();
        // operand rows past the last repeat it: a result row depends on its own operand row alone, and nobody reads theirs
        float c3[3][2][4] = {};
        const bf16 *ua = u + min(g, n - 1) * us + q * 8;
        const int row8 = (min(g + 8, n - 1) - min(g, n - 1)) * us;
        const bf16 *wa8 = ws + (pair * 8 + g) * us + q * 8;
#pragma unroll 5
        for (int k = half * 32; k < R; k += 64) {
            const uint4 wv = *reinterpret_cast<const uint4 *>(wa8 + k);
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const bf16 *row = ua + t * part + k;
                mma_rows(c3[t], *reinterpret_cast<const uint4 *>(row), *reinterpret_cast<const uint4 *>(row + row8), wv);
            }
        }
        float acc[4];          // the smallest part first
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] = ((c3[2][0][k] + c3[2][1][k]) + (c3[1][0][k] + c3[1][1][k])) + (c3[0][0][k] + c3[0][1][k]);
        float ra[2], rb[2];          // read before the meeting: behind it the next pass may write them
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            ra[h] = rs[g + 8 * h][s];
            rb[h] = rs[g + 8 * h][s + 1];
        }
        if (half) other[pair][lane] = make_float4(acc[0], acc[1], acc[2], acc[3]);
        __syncthreads();
        if (half) continue;
        const float4 o = other[pair][lane];
        acc[0] += o.x; acc[1] += o.y; acc[2] += o.z; acc[3] += o.w;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = g + 8 * h;
            float v = 0.f;
            if (r < n)
                v = sigmoidf_(acc[2 * h]) * __bfloat162float(__float2bfloat16(xa[h])) * ra[h] +
                    sigmoidf_(acc[2 * h + 1]) * __bfloat162float(__float2bfloat16(xb[h])) * rb[h];
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            if (!(q & 1) && c_ok && r < n) bin[(long long)(m0 + r) * ld_bin + bin_col0 + c] = __float2bfloat16(v / float(hc));
        }
    }
}

}  // namespace qw

using namespace qw;

QW_DCHECK_TU(hc)

QW_API int qwk_embed_rows(const int *tokens, const void *table, int ld_table, int col0, int SH, int hc, int vocab,
                          float *X, int M, cudaStream_t s) {
    if (((SH | col0 | ld_table) & 3) == 0 && aligned16(table, X))
        embed_rows_kernel<4><<<dim3(M, (SH + 1023) / 1024), 256, 0, s>>>(tokens, (const bf16 *)table, ld_table, col0, SH, hc, vocab, X);
    else
        embed_rows_kernel<1><<<dim3(M, (SH + 255) / 256), 256, 0, s>>>(tokens, (const bf16 *)table, ld_table, col0, SH, hc, vocab, X);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

QW_API int qwk_hc_pre(float *X, const float *pend, int ld_pend, const float *inj, int ld_inj, const float *w1, int SH,
                      int hc, void *y, float *ssq, int ld_ssq, int M, cudaStream_t s) {
    dim3 grid(M, hc);
    if ((SH & 3) == 0 && (!pend || (ld_pend & 3) == 0) && aligned16(X, pend, y ? w1 : nullptr, (bf16 *)y))
        hc_pre_kernel<4><<<grid, 256, 0, s>>>(X, pend, ld_pend, inj, ld_inj, w1, SH, hc, (bf16 *)y, ssq, ld_ssq);
    else
        hc_pre_kernel<1><<<grid, 256, 0, s>>>(X, pend, ld_pend, inj, ld_inj, w1, SH, hc, (bf16 *)y, ssq, ld_ssq);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// One-time (per device) opt-in to the kernels' dynamic shared memory.
static void hc_configure() {
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!attr_set[dev]) {
        cudaFuncSetAttribute(hc_down_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
        cudaFuncSetAttribute(hc_down_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
        cudaFuncSetAttribute(hc_down_mma_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(hc_up_mma_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
        cudaFuncSetAttribute(hc_up_mma_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
        cudaFuncSetAttribute(hc_down_mma_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        attr_set[dev] = true;
    }
}

QW_API int qwk_hc_up_mix(const float *red, int ld_red, const void *Wu, const float *X, const float *w1, int SH, int hc,
                         int R, int n_inj, int H, float eps, int M, float *inj, int ld_inj, void *bin, int ld_bin,
                         int bin_col0, cudaStream_t s) {
    if (hc != 4 || (R & 7) || R > 8 * 8 * UP_MAXI) return -1;
    const FuseIn fi = take_fi();
    const FuseOut fo = take_fo();
    if ((fi.active != 0) != (fo.mode != 0)) return -1;          // the fused mixer both receives and sends
    if (!fi.active && R + n_inj <= HM_THREADS) {
        hc_configure();
        const size_t smem = sizeof(bf16) * (3 * HM_ROWS + 4 * HU_COLS) * (((R + 31) & ~31) + HU_PAD);
        const int blocks = (SH + HU_COLS - 1) / HU_COLS;
        if (M < HU_CLUSTER_MIN)
            return launch_pdl(hc_up_mma_kernel<false>, dim3(blocks), dim3(HM_THREADS), smem, s, red, ld_red, (const bf16 *)Wu, X, w1, SH, R, R + n_inj,
                              1.f / float(H), eps, M, inj, ld_inj, (bf16 *)bin, ld_bin, bin_col0) == cudaSuccess ? 0 : -2;
        return launch_pdl_cluster(hc_up_mma_kernel<true>, HD_CL, dim3((blocks + HD_CL - 1) / HD_CL * HD_CL), dim3(HM_THREADS), smem, s, red, ld_red,
                                  (const bf16 *)Wu, X, w1, SH, R, R + n_inj, 1.f / float(H), eps, M, inj, ld_inj, (bf16 *)bin, ld_bin,
                                  bin_col0) == cudaSuccess ? 0 : -2;
    }
    dim3 grid((SH + 7) / 8, (M + UP_ROWS - 1) / UP_ROWS);
    const size_t smem = sizeof(float) * ((size_t)UP_ROWS * R + UP_ROWS * hc + (size_t)UP_ROWS * ld_red);
    if (smem > 48 * 1024) return -1;
    return launch_pdl(fi.active ? hc_up_mix_kernel<true, UP_ROWS> : hc_up_mix_kernel<false, UP_ROWS>, grid, dim3(256), smem, s, red, ld_red, (const bf16 *)Wu, X, w1, SH, hc, R, R + n_inj,
                      1.f / float(H), eps, M, inj, ld_inj, (bf16 *)bin, ld_bin, bin_col0, fi, fo) == cudaSuccess ? 0 : -2;
}

// Fused combine + sum of squares + down projection (see hc_down_kernel).  Xout == null keeps X in place.
QW_API int qwk_hc_down(const float *Xin, float *Xout, const float *pend, int ld_pend, const float *inj_prev,
                       const float *w1, const void *Wd, float *send, int ld_send, int SH, int hc, int down, int M,
                       cudaStream_t s) {
    if ((SH & 7) || (pend && !Xout)) return -1;
    HcDownArgs a;
    a.Xin = Xin; a.Xout = Xout; a.pend = pend; a.ld_pend = ld_pend; a.inj_prev = inj_prev; a.w1 = w1;
    a.Wd = (const bf16 *)Wd; a.send = send; a.ld_send = ld_send; a.SH = SH; a.hc = hc; a.down = down; a.M = M;
    a.fi = take_fi(); a.fo = take_fo();
    if (a.fi.active && !a.fo.mode) return -1;          // a fused down projection always sends its all-reduce
    hc_configure();
    // room for eight weight rows and eight rows of the step, whatever M is: a row's sums do not depend on the rows beside it
    if (!a.fo.mode && sizeof(bf16) * (HD_J + HD_ROWS) * (SH + HM_PAD) <= 200 * 1024) {
        const int tiles = (down + HD_J - 1) / HD_J;
        const size_t smem = sizeof(bf16) * (size_t)(HD_J + (M < HD_ROWS ? M : HD_ROWS)) * (SH + HM_PAD);
        if (M < HD_CLUSTER_MIN) return launch_pdl(hc_down_mma_kernel<false>, dim3(tiles, hc), dim3(HM_THREADS), smem, s, a) == cudaSuccess ? 0 : -2;
        return launch_pdl_cluster(hc_down_mma_kernel<true>, HD_CL, dim3((tiles + HD_CL - 1) / HD_CL * HD_CL, hc), dim3(HM_THREADS), smem, s, a) ==
                       cudaSuccess ? 0 : -2;
    }
    const long long rows = (long long)down * hc;
    a.wpr = rows >= NUM_SMS * 8 * 2 ? 1 : (rows >= NUM_SMS * 4 * 2 ? 2 : (rows >= NUM_SMS * 2 * 2 ? 4 : 8));
    if ((SH >> 3) < a.wpr * 32) {          // short rows: do not spread a row over more warps than it has pieces
        while (a.wpr > 1 && (SH >> 3) < a.wpr * 32) a.wpr >>= 1;
    }
    const int rpb = 8 / a.wpr;
    dim3 grid((down + rpb - 1) / rpb, hc, (M + 7) / 8);
    const size_t smem = (size_t)8 * SH * sizeof(bf16);
    return launch_pdl(a.fo.mode ? hc_down_kernel<true> : hc_down_kernel<false>, grid, dim3(256), smem, s, a) == cudaSuccess ? 0 : -2;
}
