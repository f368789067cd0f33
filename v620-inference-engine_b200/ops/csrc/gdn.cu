// Gated delta net kernels for row batches: causal depthwise conv + gating + per-head L2 norm,
// and the recurrent delta-rule update with the gated output norm fused in
// (roles of the reference's src/kernels/gdn.hip:174-309; math in docs/MODEL.md:108-133).
//
// Per-rank layout of the projection output row (fp32): [ q (KL heads) | k (KL heads) | v (VL heads) |
// z (VL heads x 128) | b (VL) | a (VL) ], head dim 128.
#include "common.cuh"

namespace qw {

constexpr int GD = 128;      // GDN head dim

struct GdnConvArgs {
    const float *proj;       // [M][ld_proj]
    int ld_proj;
    float *ring;             // [slots][GDN_RING][qkv_l] pre-conv rows of this layer
    const float *cw;         // [qkv_l][4] conv taps (oldest first)
    const float *A_log, *dt_bias;   // [VL]
    int KL, VL;
    Rows rows;
    float *qkv;              // [M][qkv_l] conv output: q (normed, scaled) | k (normed) | v
    float *decay, *beta;     // [M][VL]
    float eps;
};

// Pre-conv value of channel c at `back` rows before row m: from this batch while that row belongs to m's run, else from
// the slot's ring (positions before the run), else zero (before the sequence's start).
__device__ __forceinline__ float gdn_preconv(const GdnConvArgs &a, const float *ring, int qkv_l, int m, int rs, int pos,
                                             int back, int c) {
    if (m - back >= rs) return a.proj[(long long)(m - back) * a.ld_proj + c];
    const int q = pos - back;
    return q >= 0 ? ring[(q % GDN_RING) * qkv_l + c] : 0.f;
}

constexpr int CONV_ROWS = 8;     // rows of the batch per block

// grid (ceil(M / 8), 2*KL+VL), 128 threads: one head and eight consecutive rows per block.  The four-tap window slides
// down the rows in registers (one new load per row while the rows stay in one run).
__global__ void __launch_bounds__(128) gdn_conv_kernel(GdnConvArgs a) {
    __shared__ float scratch[32];
    const int m_first = blockIdx.x * CONV_ROWS, head = blockIdx.y, d = threadIdx.x;
    const int qkv_l = (2 * a.KL + a.VL) * GD;
    const int c = head * GD + d;
    float tap[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) tap[k] = a.cw[c * 4 + k];
    float w0 = 0.f, w1 = 0.f, w2 = 0.f;      // values 3, 2, 1 rows back
    int prev_rs = -1;
    for (int i = 0; i < CONV_ROWS; ++i) {
        const int m = m_first + i;
        if (m >= a.rows.M) break;                // uniform for the block
        const int slot = a.rows.slot[m], pos = a.rows.pos[m], rs = a.rows.run_start[m];
        const float *ring = a.ring + (long long)slot * GDN_RING * qkv_l;
        if (i == 0 || rs != prev_rs || m == rs) {
            w0 = gdn_preconv(a, ring, qkv_l, m, rs, pos, 3, c);
            w1 = gdn_preconv(a, ring, qkv_l, m, rs, pos, 2, c);
            w2 = gdn_preconv(a, ring, qkv_l, m, rs, pos, 1, c);
        }
        prev_rs = rs;
        const float cur = a.proj[(long long)m * a.ld_proj + c];
        const float acc = fmaf(tap[3], cur, fmaf(tap[2], w2, fmaf(tap[1], w1, tap[0] * w0)));
        w0 = w1; w1 = w2; w2 = cur;
        float v = siluf_(acc);
        if (head < 2 * a.KL) {
            const float ss = block_sum<128>(v * v, scratch);
            v = v / sqrtf(ss + a.eps);
            if (head < a.KL) v *= 0.08838834764831845f;    // 1/sqrt(128)
        }
        a.qkv[(long long)m * qkv_l + c] = v;
        if (head == 0 && d < a.VL) {
            const float *row = a.proj + (long long)m * a.ld_proj + qkv_l + a.VL * GD;
            const float bb = row[d], aa = row[a.VL + d];
            const float g = -__expf(a.A_log[d]) * softplusf_(aa + a.dt_bias[d]);
            a.decay[m * a.VL + d] = __expf(g);
            a.beta[m * a.VL + d] = sigmoidf_(bb);
        }
    }
}

// The same for a prefill chunk (more than MAX_ROWS rows; long runs, though nothing depends on it): a warp per head and 8 rows, four
// channels per lane, so a head's norm is five shuffles instead of two meetings of a block per row and four rows' loads are in
// flight.  4096 rows, 80 heads, ring included: 179 us with the kernel above, 84 here.  The last row of blocks forms decay
// and beta.  grid (ceil(M / 8), ceil((2 KL + VL) / 4) + 1), 128 threads.
constexpr int CONVP_ROWS = 8;
__global__ void __launch_bounds__(128) gdn_conv_prefill_kernel(GdnConvArgs a) {
    const int head = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * CONVP_ROWS, m1 = min(a.rows.M, m0 + CONVP_ROWS);
    const int qkv_l = (2 * a.KL + a.VL) * GD, c = head * GD + lane * 4;
    if (blockIdx.y == gridDim.y - 1) {
        for (int i = threadIdx.x; i < (m1 - m0) * a.VL; i += 128) {
            const int m = m0 + i / a.VL, d = i % a.VL;
            const float *row = a.proj + (long long)m * a.ld_proj + qkv_l + a.VL * GD;
            const float g = -__expf(a.A_log[d]) * softplusf_(row[a.VL + d] + a.dt_bias[d]);
            a.decay[m * a.VL + d] = __expf(g);
            a.beta[m * a.VL + d] = sigmoidf_(row[d]);
        }
        return;
    }
    if (head >= 2 * a.KL + a.VL) return;
    float tap[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float4 t = *reinterpret_cast<const float4 *>(a.cw + (c + j) * 4);
        tap[j][0] = t.x; tap[j][1] = t.y; tap[j][2] = t.z; tap[j][3] = t.w;
    }
    auto proj_at = [&](int m) { return *reinterpret_cast<const float4 *>(a.proj + (long long)m * a.ld_proj + c); };
    auto back_from = [&](int m, int back) {  // pre-conv row `back` rows before m: of m's run, before it the slot's ring, before the sequence zero
        if (m - back >= a.rows.run_start[m]) return proj_at(m - back);
        const int q = a.rows.pos[m] - back;
        return q >= 0 ? *reinterpret_cast<const float4 *>(a.ring + ((long long)a.rows.slot[m] * GDN_RING + q % GDN_RING) * qkv_l + c)
                      : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    float4 w0 = back_from(m0, 3), w1 = back_from(m0, 2), w2 = back_from(m0, 1);
    for (int mb = m0; mb < m1; mb += 4) {
        float4 cur[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) cur[k] = mb + k < m1 ? proj_at(mb + k) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int m = mb + k;
            if (m >= m1) break;
            if (m > m0 && a.rows.run_start[m] == m) {          // a run begins inside these rows
                w0 = back_from(m, 3); w1 = back_from(m, 2); w2 = back_from(m, 1);
            }
            float4 v;
            v.x = siluf_(fmaf(tap[0][3], cur[k].x, fmaf(tap[0][2], w2.x, fmaf(tap[0][1], w1.x, tap[0][0] * w0.x))));
            v.y = siluf_(fmaf(tap[1][3], cur[k].y, fmaf(tap[1][2], w2.y, fmaf(tap[1][1], w1.y, tap[1][0] * w0.y))));
            v.z = siluf_(fmaf(tap[2][3], cur[k].z, fmaf(tap[2][2], w2.z, fmaf(tap[2][1], w1.z, tap[2][0] * w0.z))));
            v.w = siluf_(fmaf(tap[3][3], cur[k].w, fmaf(tap[3][2], w2.w, fmaf(tap[3][1], w1.w, tap[3][0] * w0.w))));
            w0 = w1; w1 = w2; w2 = cur[k];
            if (head < 2 * a.KL) {
                const float ss = warp_sum(fmaf(v.x, v.x, v.y * v.y) + fmaf(v.z, v.z, v.w * v.w));
                const float r = (head < a.KL ? 0.08838834764831845f : 1.f) / sqrtf(ss + a.eps);      // queries: 1 / sqrt(128) as well
                v.x *= r; v.y *= r; v.z *= r; v.w *= r;
            }
            *reinterpret_cast<float4 *>(a.qkv + (long long)m * qkv_l + c) = v;
        }
    }
}

// Stores the pre-conv rows of runs longer than `min_run` into the ring (after the convolution has read the old entries).
// grid (M, ceil(qkv_l/256)).
__global__ void gdn_ring_kernel(const float *proj, int ld_proj, float *ring, int qkv_l, Rows rows, int m_first, int min_run) {
    pdl_wait();
    pdl_trigger();
    const int m = m_first + blockIdx.x;
    const int c = blockIdx.y * 256 + threadIdx.x;
    if (c >= qkv_l) return;
    const int slot = rows.slot[m], pos = rows.pos[m];
    // a run longer than the ring keeps only its last GDN_RING rows
    const int rs = rows.run_start[m], len = rows.run_len[rs];
    if (len <= min_run || m - rs < len - GDN_RING) return;
    ring[((long long)slot * GDN_RING + (pos % GDN_RING)) * qkv_l + c] = proj[(long long)m * ld_proj + c];
}

struct GdnScanArgs {
    const float *qkv;        // [M][qkv_l]
    const float *decay, *beta;   // [M][VL]
    const float *proj;       // for z: proj[m][qkv_l + h*128 + d]
    int ld_proj;
    float *S;                // [slots][VL][128 k][128 v] state of this layer
    float *save;             // optional [M][VL][128][128]: state after each row (speculative rollback)
    const float *norm_w;     // [128]
    int KL, VL;
    Rows rows;
    bf16 *o;                 // [M][VL*128] gated, normed output
    float eps;
};

// grid (M, VL), 512 threads.  Only the first row of a run does work; it walks the run's rows.
// Thread (kg = tid/128, c = tid%128) holds S[kg*32 .. +32][c].
__global__ void __launch_bounds__(512) gdn_scan_kernel(GdnScanArgs a) {
    __shared__ float kq[2][GD];        // k and q of the row
    __shared__ float red[4][GD];
    __shared__ float scratch[32];
    const int m0 = blockIdx.x, h = blockIdx.y;
    if (a.rows.run_start[m0] != m0) return;
    const int len = a.rows.run_len[m0], slot = a.rows.slot[m0];
    const int tid = threadIdx.x, c = tid & 127, kg = tid >> 7;
    const int qkv_l = (2 * a.KL + a.VL) * GD;
    const int kh = h / (a.VL / a.KL);
    float *Sg = a.S + ((long long)slot * a.VL + h) * GD * GD;
    float S[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) S[i] = Sg[(kg * 32 + i) * GD + c];
    for (int r = 0; r < len; ++r) {
        const int m = m0 + r;
        const float *row = a.qkv + (long long)m * qkv_l;
        __syncthreads();
        if (tid < GD) kq[0][tid] = row[(a.KL + kh) * GD + tid];
        else if (tid < 2 * GD) kq[1][tid - GD] = row[kh * GD + (tid - GD)];
        __syncthreads();
        const float dec = a.decay[m * a.VL + h], be = a.beta[m * a.VL + h];
        float p = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            S[i] *= dec;
            p = fmaf(S[i], kq[0][kg * 32 + i], p);
        }
        red[kg][c] = p;
        __syncthreads();
        const float stk = red[0][c] + red[1][c] + red[2][c] + red[3][c];
        const float u = (row[2 * a.KL * GD + h * GD + c] - stk) * be;
        float oq = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            S[i] = fmaf(kq[0][kg * 32 + i], u, S[i]);
            oq = fmaf(S[i], kq[1][kg * 32 + i], oq);
        }
        __syncthreads();
        red[kg][c] = oq;
        __syncthreads();
        if (a.save) {
            float *sv = a.save + ((long long)m * a.VL + h) * GD * GD;
#pragma unroll
            for (int i = 0; i < 32; ++i) sv[(kg * 32 + i) * GD + c] = S[i];
        }
        // gated rms norm over the head's 128 outputs
        float ov = 0.f;
        if (kg == 0) ov = red[0][c] + red[1][c] + red[2][c] + red[3][c];
        const float ss = block_sum<512>(ov * ov, scratch);
        if (kg == 0) {
            const float z = a.proj[(long long)m * a.ld_proj + qkv_l + h * GD + c];
            const float y = ov * rsqrtf(ss / float(GD) + a.eps) * a.norm_w[c] * sigmoidf_(z);
            a.o[(long long)m * a.VL * GD + h * GD + c] = __float2bfloat16(y);
        }
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) Sg[(kg * 32 + i) * GD + c] = S[i];
}

// ------------------------------------------------------------------------------------------
// Fused step: conv + gating + L2 norm + delta-rule update + gated norm in one kernel, and the ring store of runs of up to
// RUN_INLINE rows.  grid (M, VL), 512 threads; the block of (run start, head h) walks the run, FR rows at a time: what does not
// depend on the state - the loads, conv, norms and gates of all these rows - first, then the state's rows one behind the other with one
// meeting each, then their outputs' norms, a warp per row.  (With a row's loads, norms and seven meetings on the chain of every row 24
// rows of four runs took 70 us; they take 36, and one row 9.)  q/k of the head's key head are recomputed by each of the value heads that share it.
// The ring entries of a run's first 13 rows are not those that conv reads (three positions before the run); a longer run's are stored
// by gdn_ring_kernel behind this kernel, because the blocks of a run do not wait for one another.
// ------------------------------------------------------------------------------------------
struct GdnFusedArgs {
    const float *proj;
    int ld_proj;
    float *ring;
    const float *cw, *A_log, *dt_bias, *norm_w;
    int KL, VL;
    Rows rows;
    float *S, *save;
    bf16 *o;
    float eps;
};
constexpr int RUN_INLINE = GDN_RING - 4;

// FR rows at a time, BLOCKS on an SM.  <8, 2>, at 64 registers, where there may be many runs.  <4, 1>, whose rows have the registers to fetch their
// operands ahead, where runs are few: then an SM has one block anyway, and the chain of its rows is what is waited for.  <1, 1>: a step of one row,
// which has nothing to gather rows for.
template <int FR, int BLOCKS>
__global__ void __launch_bounds__(512, BLOCKS) gdn_fused_kernel(GdnFusedArgs a) {
    __shared__ __align__(16) float qkv[FR][3][GD];       // conv output: q (normed, scaled), k (normed), v
    __shared__ float red[2][4][GD];                      // S k, by quarter of the keys; row r in buffer r & 1
    __shared__ float part[FR][4][GD];                    // S q, the same
    __shared__ float ssq[FR][8];                         // sums of squares: warps 0-3 q, 4-7 k
    __shared__ float gate[FR][2];                        // decay, beta
    __shared__ float zs[FR][GD];                         // output gates
    const int m0 = blockIdx.x, h = blockIdx.y;
    const int tid = threadIdx.x, c = tid & 127, kg = tid >> 7, warp = tid >> 5, lane = tid & 31;
    const int qkv_l = (2 * a.KL + a.VL) * GD;
    const int rep = a.VL / a.KL, kh = h / rep;
    // conv taps of this thread's channel (weights: independent of the predecessor)
    int ch = -1;
    if (kg == 0) ch = kh * GD + c;                       // q
    else if (kg == 1) ch = (a.KL + kh) * GD + c;         // k
    else if (kg == 2) ch = (2 * a.KL + h) * GD + c;      // v
    float tap[4] = {0.f, 0.f, 0.f, 0.f};
    if (ch >= 0) {
#pragma unroll
        for (int k = 0; k < 4; ++k) tap[k] = a.cw[ch * 4 + k];
    }
    // The row table was written before the step began and the recurrent state only by this kernel in the previous step:
    // neither depends on the predecessor, so the state (64 KB per head, from HBM) is fetched before waiting for it.
    if (a.rows.run_start[m0] != m0) return;
    const int len = a.rows.run_len[m0], slot = a.rows.slot[m0], pos0 = a.rows.pos[m0];
    float *ring = a.ring + (long long)slot * GDN_RING * qkv_l;
    float *Sg = a.S + ((long long)slot * a.VL + h) * GD * GD;
    float S[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) S[i] = Sg[(kg * 32 + i) * GD + c];
    pdl_wait();
    pdl_trigger();
    const bool stores = ch >= 0 && len <= RUN_INLINE && (kg == 2 || h % rep == 0);      // v channels by every head, q/k by the group's first
    float w[3] = {0.f, 0.f, 0.f};                        // pre-conv values 3, 2, 1 rows back
    if (ch >= 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int q = pos0 - 3 + k;
            if (q >= 0) w[k] = ring[(q % GDN_RING) * qkv_l + ch];
        }
    }
    for (int r0 = 0; r0 < len; r0 += FR) {
        const int n = min(FR, len - r0);
        const float *prow = a.proj + (long long)(m0 + r0) * a.ld_proj;
        // ---- conv + silu, norms and gates of these rows
        float x[FR];
        if (ch >= 0) {
#pragma unroll
            for (int i = 0; i < FR; ++i) x[i] = i < n ? prow[(long long)i * a.ld_proj + ch] : 0.f;
        } else if (c < n) {
            const float *row = prow + (long long)c * a.ld_proj + qkv_l + a.VL * GD;
            const float g = -__expf(a.A_log[h]) * softplusf_(row[a.VL + h] + a.dt_bias[h]);
            gate[c][0] = __expf(g);
            gate[c][1] = sigmoidf_(row[h]);
        }
        if (ch >= 0) {
#pragma unroll
            for (int i = 0; i < FR; ++i) {
                const float cur = x[i];
                const float acc = fmaf(tap[3], cur, fmaf(tap[2], w[2], fmaf(tap[1], w[1], tap[0] * w[0])));
                if (i < n) {
                    if (stores) ring[((pos0 + r0 + i) % GDN_RING) * qkv_l + ch] = cur;
                    w[0] = w[1]; w[1] = w[2]; w[2] = cur;
                }
                x[i] = siluf_(acc);
            }
            if (kg < 2) {
#pragma unroll
                for (int i = 0; i < FR; ++i) {
                    if (i >= n) break;
                    const float s = warp_sum(x[i] * x[i]);
                    if (lane == 0) ssq[i][warp] = s;
                }
            }
        }
        __syncthreads();                                 // sums and gates; the rows before these are consumed
        for (int i = kg; i < n; i += 4) zs[i][c] = prow[(long long)i * a.ld_proj + qkv_l + h * GD + c];
        if (ch >= 0) {
#pragma unroll
            for (int i = 0; i < FR; ++i) {
                if (i >= n) break;
                float v = x[i];
                if (kg < 2) {
                    const float *s = ssq[i] + kg * 4;
                    v = v / sqrtf(s[0] + s[1] + s[2] + s[3] + a.eps);
                    if (kg == 0) v *= 0.08838834764831845f;
                }
                qkv[i][kg][c] = v;
            }
        }
        __syncthreads();
        // ---- the state's rows
        for (int i = 0; i < n; ++i) {
            const float dec = gate[i][0], be = gate[i][1];
            const float *kk = qkv[i][1] + kg * 32, *qq = qkv[i][0] + kg * 32;
            float p = 0.f;
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                const float4 k4 = *reinterpret_cast<const float4 *>(kk + j);
                S[j] *= dec; S[j + 1] *= dec; S[j + 2] *= dec; S[j + 3] *= dec;
                p = fmaf(S[j], k4.x, p); p = fmaf(S[j + 1], k4.y, p); p = fmaf(S[j + 2], k4.z, p); p = fmaf(S[j + 3], k4.w, p);
            }
            float (*rd)[GD] = red[i & 1];
            rd[kg][c] = p;
            __syncthreads();
            const float u = (qkv[i][2][c] - (rd[0][c] + rd[1][c] + rd[2][c] + rd[3][c])) * be;
            float oq = 0.f;
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                const float4 k4 = *reinterpret_cast<const float4 *>(kk + j), q4 = *reinterpret_cast<const float4 *>(qq + j);
                S[j] = fmaf(k4.x, u, S[j]); S[j + 1] = fmaf(k4.y, u, S[j + 1]); S[j + 2] = fmaf(k4.z, u, S[j + 2]); S[j + 3] = fmaf(k4.w, u, S[j + 3]);
                oq = fmaf(S[j], q4.x, oq); oq = fmaf(S[j + 1], q4.y, oq); oq = fmaf(S[j + 2], q4.z, oq); oq = fmaf(S[j + 3], q4.w, oq);
            }
            part[i][kg][c] = oq;
            if (a.save) {
                float *sv = a.save + ((long long)(m0 + r0 + i) * a.VL + h) * GD * GD;
#pragma unroll
                for (int j = 0; j < 32; ++j) sv[(kg * 32 + j) * GD + c] = S[j];
            }
        }
        __syncthreads();                                 // all partial outputs
        if (warp < n) {
            float v[4], ss = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int d = j * 32 + lane;
                v[j] = part[warp][0][d] + part[warp][1][d] + part[warp][2][d] + part[warp][3][d];
                ss += warp_sum(v[j] * v[j]);
            }
            const float r = rsqrtf(ss / float(GD) + a.eps);
            bf16 *o = a.o + (long long)(m0 + r0 + warp) * a.VL * GD + h * GD;
#pragma unroll
            for (int j = 0; j < 4; ++j) o[j * 32 + lane] = __float2bfloat16(v[j] * r * a.norm_w[j * 32 + lane] * sigmoidf_(zs[warp][j * 32 + lane]));
        }
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) Sg[(kg * 32 + i) * GD + c] = S[i];
}


// Speculative acceptance: for every (slot, row) pair and every GDN layer, the state saved after `row` of the last
// verification step becomes the slot's state.  grid (blocks, pairs, layers); S_ptrs[layer] = [slots][state] fp32,
// save = [layers][max_rows][state].  state % 4 == 0.  A thread's four loads are in flight together, and there are as many blocks as
// the state has pieces of 16 KB (eight blocks per pair and layer, one load a thread at a time: 50 us for four pairs and three layers of 3 MB, now 13).
constexpr int ACCEPT_VALUES = 4;
__global__ void __launch_bounds__(256) gdn_accept_kernel(float *const *S_ptrs, const float *save, int max_rows, long long state,
                                                         const int *pairs) {
    const int layer = blockIdx.z, slot = pairs[2 * blockIdx.y], row = pairs[2 * blockIdx.y + 1];
    if (row < 0) return;
    const float4 *src = reinterpret_cast<const float4 *>(save + ((long long)layer * max_rows + row) * state);
    float4 *dst = reinterpret_cast<float4 *>(S_ptrs[layer] + (long long)slot * state);
    const long long n = state >> 2, i0 = (long long)blockIdx.x * (ACCEPT_VALUES * 256) + threadIdx.x;
    float4 v[ACCEPT_VALUES];
#pragma unroll
    for (int k = 0; k < ACCEPT_VALUES; ++k)
        if (i0 + k * 256 < n) v[k] = __ldcs(src + i0 + k * 256);
#pragma unroll
    for (int k = 0; k < ACCEPT_VALUES; ++k)
        if (i0 + k * 256 < n) dst[i0 + k * 256] = v[k];
}

}  // namespace qw

using namespace qw;

QW_API int qwk_gdn_conv(const float *proj, int ld_proj, float *ring, const float *cw, const float *A_log,
                        const float *dt_bias, int KL, int VL, int M, const int *slot, const int *pos,
                        const int *run_start, const int *run_len, float *qkv, float *decay, float *beta, float eps,
                        cudaStream_t s) {
    GdnConvArgs a;
    a.proj = proj; a.ld_proj = ld_proj; a.ring = ring; a.cw = cw; a.A_log = A_log; a.dt_bias = dt_bias;
    a.KL = KL; a.VL = VL; a.rows = Rows{M, slot, pos, run_start, run_len};
    a.qkv = qkv; a.decay = decay; a.beta = beta; a.eps = eps;
    if (VL > 128) return -1;
    if (M > MAX_ROWS && (ld_proj & 3) == 0 && aligned16(proj, ring, cw, qkv)) {
        gdn_conv_prefill_kernel<<<dim3((M + CONVP_ROWS - 1) / CONVP_ROWS, (2 * KL + VL + 3) / 4 + 1), 128, 0, s>>>(a);
    } else {
        dim3 grid((M + CONV_ROWS - 1) / CONV_ROWS, 2 * KL + VL);
        gdn_conv_kernel<<<grid, 128, 0, s>>>(a);
    }
    const int qkv_l = (2 * KL + VL) * GD;
    // The ring counts on a batch of more than MAX_ROWS rows being one run of one slot (a prefill chunk): only its last GDN_RING rows stay.
    const int m_first = M > MAX_ROWS ? M - GDN_RING : 0;
    dim3 g2(M - m_first, (qkv_l + 255) / 256);
    launch_pdl(gdn_ring_kernel, g2, dim3(256), 0, s, proj, ld_proj, ring, qkv_l, a.rows, m_first, 0);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

QW_API int qwk_gdn_scan(const float *qkv, const float *decay, const float *beta, const float *proj, int ld_proj, float *S,
                        float *save, const float *norm_w, int KL, int VL, int M, const int *slot, const int *pos,
                        const int *run_start, const int *run_len, void *o, float eps, cudaStream_t s) {
    GdnScanArgs a;
    a.qkv = qkv; a.decay = decay; a.beta = beta; a.proj = proj; a.ld_proj = ld_proj; a.S = S; a.save = save;
    a.norm_w = norm_w; a.KL = KL; a.VL = VL; a.rows = Rows{M, slot, pos, run_start, run_len};
    a.o = (bf16 *)o; a.eps = eps;
    dim3 grid(M, VL);
    gdn_scan_kernel<<<grid, 512, 0, s>>>(a);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// One GDN step for M rows: the fused kernel, and the ring store of long runs where there can be any.
QW_API int qwk_gdn_step(const float *proj, int ld_proj, float *ring, const float *cw, const float *A_log,
                        const float *dt_bias, const float *norm_w, int KL, int VL, int M, const int *slot, const int *pos,
                        const int *run_start, const int *run_len, float *S, float *save, float *qkv, float *decay,
                        float *beta, void *o, float eps, cudaStream_t s) {
    (void)qkv; (void)decay; (void)beta;          // not read: null will do
    GdnFusedArgs a;
    a.proj = proj; a.ld_proj = ld_proj; a.ring = ring; a.cw = cw; a.A_log = A_log; a.dt_bias = dt_bias;
    a.norm_w = norm_w; a.KL = KL; a.VL = VL; a.rows = Rows{M, slot, pos, run_start, run_len};
    a.S = S; a.save = save; a.o = (bf16 *)o; a.eps = eps;
    // Up to three runs of 48 heads are one block an SM.  Which rows are runs is known on the device alone: up to three rows cannot be more, and the rows
    // of a verification step (they save their states) are long runs, so that up to RUN_INLINE of them are taken for few.  us, <8, 2> / <4, 1>, 48 heads:
    // 2 rows 7.3 / 5.8; saved, one run of 6 rows 25.3 / 15.4, two of 6 26.0 / 17.1, three of 3 16.3 / 12.4; but four of 2 13.6 / 16.5, four of 6 32.6 /
    // 40, and 8 rows of 8 streams 17.0 / 18.2.
    const auto kernel = M == 1 ? gdn_fused_kernel<1, 1> : M <= 3 || (save && M <= RUN_INLINE) ? gdn_fused_kernel<4, 1> : gdn_fused_kernel<8, 2>;
    if (launch_pdl(kernel, dim3(M, VL), dim3(512), 0, s, a) != cudaSuccess) return -2;
    if (M > RUN_INLINE) {
        const int qkv_l = (2 * KL + VL) * GD;
        if (launch_pdl(gdn_ring_kernel, dim3(M, (qkv_l + 255) / 256), dim3(256), 0, s, proj, ld_proj, ring, qkv_l, a.rows, 0, RUN_INLINE) != cudaSuccess)
            return -2;
    }
    return 0;
}


// S_ptrs: device array of n_layers state pointers; pairs: device [n_pairs][2] = {slot, saved row (-1: keep)}.
QW_API int qwk_gdn_accept(const void *S_ptrs, const float *save, int n_layers, int max_rows, long long state, const int *pairs,
                          int n_pairs, cudaStream_t s) {
    if (n_pairs <= 0 || n_layers <= 0) return 0;
    if (state & 3) return -1;
    gdn_accept_kernel<<<dim3((unsigned)((state / 4 + ACCEPT_VALUES * 256 - 1) / (ACCEPT_VALUES * 256)), n_pairs, n_layers), 256, 0, s>>>((float *const *)S_ptrs, save, max_rows, state, pairs);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
