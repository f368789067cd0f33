// Routed-expert products of the decode path on the tensor cores.
//
// The q4 expert matrices are read once per chosen expert; with one token per pair the products are
// matrix-vector shaped, and in scalar code the unpack + multiply-add of every 4-bit weight made both
// kernels instruction-issue bound (63 % issue utilisation at 10 % of DRAM bandwidth).  Here a warp owns a
// tile of 16 weight rows and feeds mma.sync.m16n8k16 (bf16 x bf16 -> fp32) with the unpacked weights as the
// 16 x 16 operand and the activation vector as column 0 of the 16 x 8 operand: about 1.5 instructions per
// weight instead of ~16.
//
// Operand trick.  A dot product does not care in which order k is walked, as long as both operands agree.
// Lane (r = lane / 4, q = lane % 4) loads whole 32-bit words (8 weights, k = 8 w .. 8 w + 7) of rows r and
// r + 8 at word index w = w0 + q; nibble pair j of such a word ((word >> 4 j) & 0x000F000F, biased into bf16
// and re-centred) is exactly one operand register: two consecutive k of one row.  Pairs 0 / 1 feed one MMA
// (k slots 2q, 2q+1 and 2q+8, 2q+9), pairs 2 / 3 the next.  The matching activation registers of that lane are
// then the four 32-bit words of x[8 w .. 8 w + 7] - one 16-byte shared-memory load in natural order.
// Every byte a lane loads is used, a quad reads 32 contiguous bytes of a row, and nothing is shuffled.
// bf16 rows (the shared expert) use the same scheme with 16-byte loads as the operand registers directly.
//
// Scales: one per 128 k; a group is 8 MMAs into a fresh accumulator, then acc += scale * group.
// (Role of the reference's src/kernels/moe.hip pair kernels; the scheme is this engine's own.)
#pragma once
#include "fuse.cuh"
#include "mma.cuh"

namespace qw {

// bf16 pair (exact integers -8..7) of nibble pair j of a q4 word in engine order
__device__ __forceinline__ uint32_t q4_frag(uint32_t w, int j) {
    uint32_t p;
    // one three-input operation: gate/up and down of 8 rows take 35 and 28 us with it, 41 and 31 with (w & mask) | magic written out
    asm("{\n\t.reg .b32 m;\n\tmov.b32 m, 0x000F000F;\n\tlop3.b32 %0, %1, m, 0x43004300, 0xEA;\n\t}" : "=r"(p) : "r"(w >> (4 * j)));
    bf162 v = *reinterpret_cast<bf162 *>(&p);
    const bf162 off = __floats2bfloat162_rn(136.f, 136.f);
    v = __hsub2(v, off);
    return *reinterpret_cast<uint32_t *>(&v);
}

// Two MMAs for one word of rows r (wr) and r + 8 (wr8) against the activation words xv of the same 8 k.
__device__ __forceinline__ void mma_q4_word(float (&c)[4], uint32_t wr, uint32_t wr8, const uint4 &xv) {
    mma_bf16(c, q4_frag(wr, 0), q4_frag(wr8, 0), q4_frag(wr, 1), q4_frag(wr8, 1), xv.x, xv.y);
    mma_bf16(c, q4_frag(wr, 2), q4_frag(wr8, 2), q4_frag(wr, 3), q4_frag(wr8, 3), xv.z, xv.w);
}
// The same for 8 bf16 weights of rows r and r + 8 (16-byte loads).
__device__ __forceinline__ void mma_bf16_chunk(float (&c)[4], const uint4 &wr, const uint4 &wr8, const uint4 &xv) {
    mma_bf16(c, wr.x, wr8.x, wr.y, wr8.y, xv.x, xv.y);
    mma_bf16(c, wr.z, wr8.z, wr.w, wr8.w, xv.z, xv.w);
}

// Shared expert's activation of row m: sh_h[m][f] = bf16(silu(gate_f) * up_f * sigmoid(shared gate logit)), by one block.
__device__ __forceinline__ void shared_act_row(const SharedAct &sa, int m) {
    const float *l = sa.rs + (long long)m * sa.ld_rs + sa.E;
    const float sg = sigmoidf_(__ldcg(l));
    bf16 *o = reinterpret_cast<bf16 *>(sa.sh_h) + (long long)m * sa.SF;
    for (int f0 = threadIdx.x; f0 < sa.SF; f0 += 4 * blockDim.x) {          // four independent loads of each kind in flight
        float g[4], u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int f = f0 + k * blockDim.x;
            g[k] = f < sa.SF ? __ldcg(l + 1 + f) : 0.f;
            u[k] = f < sa.SF ? __ldcg(l + 1 + sa.SF + f) : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int f = f0 + k * blockDim.x;
            if (f < sa.SF) o[f] = __float2bfloat16(siluf_(g[k]) * u[k] * sg);
        }
    }
}

constexpr int MM_WARPS = 4;          // warps per block (128 threads: three blocks per SM stay resident, so 400 tiles are one wave)
constexpr int GU_NG = 5;             // k groups of 128 per warp in the gate/up kernel: K <= 4 * 5 * 128
constexpr int DN_NI = 13;            // (expert, k group) items per warp in the down kernel: top_k * F / 128 <= 52
constexpr int DN_NS = 5;             // quad-steps of the shared expert per warp: SF <= 4 * 5 * 32

// h[p][f] = silu(gate_e[f] . x_m) * (up_e[f] . x_m) for pair p = (m, j).  grid (F / 16, pairs), 128 threads.
// Warp w takes the k groups g = w, w + 4, ...; every weight load of the block is issued before the first
// one is used, and the four partial tiles are added in warp order.
__global__ void __launch_bounds__(128) moe_gate_up_mma_kernel(const uint32_t *w13, const bf16 *s13, const bf16 *x, int ldx,
                                                              const int *pair_expert, int top_k, int F, int K, bf16 *h, SharedAct sa, int npairs) {
    extern __shared__ __align__(16) unsigned char mm_smem[];
    uint4 *xs = reinterpret_cast<uint4 *>(mm_smem);                       // [K / 8] activation words
    float *red = reinterpret_cast<float *>(mm_smem + (size_t)K * 2);     // [4 warps][2][16]
    pdl_wait();
    pdl_trigger();
    if ((int)blockIdx.y >= npairs) {          // the extra rows of the grid: the shared expert's activation
        if (blockIdx.x == 0) shared_act_row(sa, blockIdx.y - npairs);
        return;
    }
    const int p = blockIdx.y;
    const int e = pair_expert[p];
    if (e < 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = lane >> 2, q = lane & 3;
    const int f0 = blockIdx.x * 16;
    const int m = p / top_k;
    const int wpr = K >> 3, ks = K >> 7;                                   // words and scale groups per row
    const long long row_g = (long long)e * 2 * F + f0 + r, row_u = row_g + F;
    const uint32_t *pg = w13 + row_g * wpr, *pg8 = pg + 8LL * wpr, *pu = w13 + row_u * wpr, *pu8 = pu + 8LL * wpr;
    uint2 wg[GU_NG][2], wg8[GU_NG][2], wu[GU_NG][2], wu8[GU_NG][2];
    float sg[GU_NG], sg8[GU_NG], su[GU_NG], su8[GU_NG];
#pragma unroll
    for (int i = 0; i < GU_NG; ++i) {
        const int g = warp + MM_WARPS * i;
        if (g < ks) {
#pragma unroll
            for (int ds = 0; ds < 2; ++ds) {
                const int wi = g * 16 + ds * 8 + 2 * q;
                wg[i][ds] = ld_stream8(pg + wi);
                wg8[i][ds] = ld_stream8(pg8 + wi);
                wu[i][ds] = ld_stream8(pu + wi);
                wu8[i][ds] = ld_stream8(pu8 + wi);
            }
            sg[i] = __bfloat162float(s13[row_g * ks + g]);
            sg8[i] = __bfloat162float(s13[(row_g + 8) * ks + g]);
            su[i] = __bfloat162float(s13[row_u * ks + g]);
            su8[i] = __bfloat162float(s13[(row_u + 8) * ks + g]);
        }
    }
    const uint4 *xr = reinterpret_cast<const uint4 *>(x + (long long)m * ldx);
    for (int i = tid; i < wpr; i += 128) xs[i] = __ldcg(xr + i);
    __syncthreads();
    float ag = 0.f, ag8 = 0.f, au = 0.f, au8 = 0.f;
#pragma unroll
    for (int i = 0; i < GU_NG; ++i) {
        const int g = warp + MM_WARPS * i;
        if (g < ks) {
            float cg[4] = {0.f, 0.f, 0.f, 0.f}, cu[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ds = 0; ds < 2; ++ds) {
                const int wi = g * 16 + ds * 8 + 2 * q;
                uint4 x0 = make_uint4(0u, 0u, 0u, 0u), x1 = x0;
                if (r == 0) {                                               // column 0 of the narrow operand is the token
                    x0 = xs[wi];
                    x1 = xs[wi + 1];
                }
                mma_q4_word(cg, wg[i][ds].x, wg8[i][ds].x, x0);
                mma_q4_word(cg, wg[i][ds].y, wg8[i][ds].y, x1);
                mma_q4_word(cu, wu[i][ds].x, wu8[i][ds].x, x0);
                mma_q4_word(cu, wu[i][ds].y, wu8[i][ds].y, x1);
            }
            // column 0 of the result sits in the lanes with q == 0: c[0] is row r, c[2] row r + 8
            ag = fmaf(sg[i], cg[0], ag); ag8 = fmaf(sg8[i], cg[2], ag8);
            au = fmaf(su[i], cu[0], au); au8 = fmaf(su8[i], cu[2], au8);
        }
    }
    if (q == 0) {
        red[(warp * 2 + 0) * 16 + r] = ag; red[(warp * 2 + 0) * 16 + r + 8] = ag8;
        red[(warp * 2 + 1) * 16 + r] = au; red[(warp * 2 + 1) * 16 + r + 8] = au8;
    }
    __syncthreads();
    if (tid < 16) {
        float gs = 0.f, us = 0.f;
#pragma unroll
        for (int w = 0; w < MM_WARPS; ++w) { gs += red[(w * 2) * 16 + tid]; us += red[(w * 2 + 1) * 16 + tid]; }
        h[(long long)p * F + f0 + tid] = __float2bfloat16(siluf_(gs) * us);
    }
}

// out[m][c] = sum_j w_j * (down_{e_j}[c] . h[p_j]) + shared_down[c] . sh_h[m].  grid (H / 16, M), 128 threads.
// The (expert, k group) items and the shared expert's k are dealt round-robin to the four warps; every weight
// load of the block is issued before the first one is used.
template <bool FUSED>
__global__ void __launch_bounds__(128) moe_down_mma_kernel(const uint32_t *w2, const bf16 *s2, const bf16 *h, const int *pair_expert,
                                                           const float *pair_w, int top_k, int F, int H, const bf16 *shared_down,
                                                           int ld_sd, const bf16 *sh_h, int SF, float *out, int ldo, FuseOut fo) {
    extern __shared__ __align__(16) unsigned char mm_smem[];
    uint4 *hs = reinterpret_cast<uint4 *>(mm_smem);                                       // [top_k][F / 8]
    uint4 *ss = hs + (size_t)top_k * (F >> 3);                                            // [SF / 8]
    float *red = reinterpret_cast<float *>(ss + (SF >> 3));                               // [4][16]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = lane >> 2, q = lane & 3;
    const int m = blockIdx.y, c0 = blockIdx.x * 16;
    // the shared expert's rows do not depend on the routing: fetch them before waiting for the router
    const int sch = SF >> 3;                                   // 16-byte pieces per shared row
    const bf16 *sr = shared_down ? shared_down + (long long)(c0 + r) * ld_sd : nullptr;
    uint4 sw[DN_NS], sw8[DN_NS];
#pragma unroll
    for (int i = 0; i < DN_NS; ++i) {
        const int pc = (warp + MM_WARPS * i) * 4 + q;
        sw[i] = sw8[i] = make_uint4(0u, 0u, 0u, 0u);
        if (shared_down && pc < sch) {
            sw[i] = ld_stream(reinterpret_cast<const uint4 *>(sr) + pc);
            sw8[i] = ld_stream(reinterpret_cast<const uint4 *>(sr + 8LL * ld_sd) + pc);
        }
    }
    pdl_wait();
    pdl_trigger();
    const int wpr = F >> 3, ks = F >> 7;
    const int nitems = top_k * ks;
    uint2 wv[DN_NI][2], wv8[DN_NI][2];
    float sc[DN_NI], sc8[DN_NI];
#pragma unroll
    for (int i = 0; i < DN_NI; ++i) {
        const int it = warp + MM_WARPS * i;
        sc[i] = sc8[i] = 0.f;
        if (it < nitems) {
            const int j = it / ks, g = it - j * ks;
            const int p = m * top_k + j;
            const int e = pair_expert[p];
            if (e >= 0) {
                const float pw = pair_w[p];
                const long long row = (long long)e * H + c0 + r;
                const uint32_t *pr = w2 + row * wpr;
#pragma unroll
                for (int ds = 0; ds < 2; ++ds) {
                    const int wi = g * 16 + ds * 8 + 2 * q;
                    wv[i][ds] = ld_stream8(pr + wi);
                    wv8[i][ds] = ld_stream8(pr + 8LL * wpr + wi);
                }
                sc[i] = __bfloat162float(s2[row * ks + g]) * pw;
                sc8[i] = __bfloat162float(s2[(row + 8) * ks + g]) * pw;
            } else {
#pragma unroll
                for (int ds = 0; ds < 2; ++ds) wv[i][ds] = wv8[i][ds] = make_uint2(0x88888888u, 0x88888888u);      // zeros in q4
            }
        }
    }
    for (int i = tid; i < top_k * wpr; i += 128) hs[i] = __ldcg(reinterpret_cast<const uint4 *>(h + (long long)m * top_k * F) + i);
    if (shared_down)
        for (int i = tid; i < sch; i += 128) ss[i] = __ldcg(reinterpret_cast<const uint4 *>(sh_h + (long long)m * SF) + i);
    __syncthreads();
    float a0 = 0.f, a8 = 0.f;
#pragma unroll
    for (int i = 0; i < DN_NI; ++i) {
        const int it = warp + MM_WARPS * i;
        if (it < nitems) {
            const int j = it / ks, g = it - j * ks;
            const uint4 *xj = hs + (size_t)j * wpr;
            float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ds = 0; ds < 2; ++ds) {
                const int wi = g * 16 + ds * 8 + 2 * q;
                uint4 x0 = make_uint4(0u, 0u, 0u, 0u), x1 = x0;
                if (r == 0) {
                    x0 = xj[wi];
                    x1 = xj[wi + 1];
                }
                mma_q4_word(c, wv[i][ds].x, wv8[i][ds].x, x0);
                mma_q4_word(c, wv[i][ds].y, wv8[i][ds].y, x1);
            }
            a0 = fmaf(sc[i], c[0], a0);
            a8 = fmaf(sc8[i], c[2], a8);
        }
    }
    if (shared_down) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < DN_NS; ++i) {
            const int pc = (warp + MM_WARPS * i) * 4 + q;
            if ((warp + MM_WARPS * i) * 4 < sch) {          // warp-uniform: the MMA needs every lane
                const uint4 xv = (r == 0 && pc < sch) ? ss[pc] : make_uint4(0u, 0u, 0u, 0u);
                mma_bf16_chunk(c, sw[i], sw8[i], xv);
            }
        }
        a0 += c[0];
        a8 += c[2];
    }
    if (q == 0) {
        red[warp * 16 + r] = a0;
        red[warp * 16 + r + 8] = a8;
    }
    __syncthreads();
    if (tid < 16) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < MM_WARPS; ++w) v += red[w * 16 + tid];
        if (FUSED) fuse_put_col(fo, fuse_seq(fo), m, c0 + tid, __float_as_uint(v));      // fused reduce-scatter: to the column's owner
        else out[(long long)m * ldo + c0 + tid] = v;
    }
}

// ---------------------------------------------------------------------------------------------------------------
// The same two products with the weights brought to padded shared memory by cp.async (row stride 32 bytes more than the row: the
// eight rows of a request fall into disjoint bank groups).  A tile's 16 rows are one piece of memory, so a warp's copies are
// whole lines and need no register while in flight.  Direct 8-byte loads touch one 32-byte sector of sixteen rows per request,
// and bulk copies of single rows (1,280 and 320 bytes) were bound by their number.  In a chain of their own, us for gate/up and
// down with bulk copies and now: 1 row 10.4, 8.6 -> 8.4, 7.7; 8 rows 59, 38 -> 35, 28; 24 rows 172, 106 -> 96, 72.  What bounds
// them now: the conversion (shift, merge and subtraction for two weights, beside 7 idle columns of every MMA) and, with few rows,
// the chain routing -> weights -> sums.
// Every column of the narrow operand holds the token: the result's column 0 is read, the others cost nothing.
// ---------------------------------------------------------------------------------------------------------------
constexpr int TM_PAD = 32;                 // bytes added to a weight row in shared memory
constexpr int CP_WARPS = 8, CP_THREADS = CP_WARPS * 32;

// p / d for the small numbers of this file (p < 4096, d >= 1): a multiplication by 2^20 / d, rounded up.
__device__ __forceinline__ int div_inv(int d) { return (1 << 20) / d + 1; }
__device__ __forceinline__ int div_by(int p, int inv) { return (int)(((long long)p * inv) >> 20); }

// One k group of 128 of 16 weight rows (at `w`, row stride srow) against the token's k group: c[0] is row r = lane / 4, c[2] row r + 8.
__device__ __forceinline__ void q4_group(float (&c)[4], const unsigned char *w, int srow, const uint4 *x, int lane) {
    const int r = lane >> 2, q = lane & 3;
#pragma unroll
    for (int ds = 0; ds < 2; ++ds) {
        const int wi = ds * 8 + 2 * q;
        const uint2 a0 = *reinterpret_cast<const uint2 *>(w + r * srow + wi * 4), a8 = *reinterpret_cast<const uint2 *>(w + (r + 8) * srow + wi * 4);
        mma_q4_word(c, a0.x, a8.x, x[wi]);
        mma_q4_word(c, a0.y, a8.y, x[wi + 1]);
    }
}

// grid (F / 16, pairs [+ M extra rows for the shared activation]), 256 threads.
__global__ void __launch_bounds__(CP_THREADS, 4) moe_gate_up_cp_kernel(const uint32_t *w13, const bf16 *s13, const bf16 *x, int ldx,
                                                                       const int *pair_expert, int top_k, int F, int K, bf16 *h,
                                                                       SharedAct sa, int npairs) {
    extern __shared__ __align__(128) unsigned char tm_smem[];
    const int rowb = K >> 1, srow = rowb + TM_PAD, ks = K >> 7, wpr = K >> 3;
    unsigned char *wg = tm_smem, *wu = wg + 16 * srow;
    bf16 *sg = reinterpret_cast<bf16 *>(wu + 16 * srow), *su = sg + 16 * ks;
    uint4 *xs = reinterpret_cast<uint4 *>(su + 16 * ks);       // 64 ks bytes of scales: 16-byte aligned
    float *red = reinterpret_cast<float *>(xs + wpr);          // [8 warps][2][16]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_wait();
    pdl_trigger();
    if ((int)blockIdx.y >= npairs) {          // the extra rows of the grid: the shared expert's activation
        if (blockIdx.x == 0) shared_act_row(sa, blockIdx.y - npairs);
        return;
    }
    const int p = blockIdx.y;
    const int e = pair_expert[p];
    if (e < 0) return;
    const int f0 = blockIdx.x * 16, m = p / top_k;
    const long long row_g = (long long)e * 2 * F + f0, row_u = row_g + F;
    {
        // a matrix's 16 rows are one piece of memory: whole lines in thread order
        const int ppr = rowb >> 4, inv = div_inv(ppr);
        const unsigned char *g = reinterpret_cast<const unsigned char *>(w13 + row_g * wpr), *up = reinterpret_cast<const unsigned char *>(w13 + row_u * wpr);
#pragma unroll 5
        for (int i = tid; i < 16 * ppr; i += CP_THREADS) {
            const int at = i * 16 + div_by(i, inv) * TM_PAD;
            cp_async16(wg + at, g + i * 16);
            cp_async16(wu + at, up + i * 16);
        }
    }
    for (int i = tid; i < 4 * ks; i += CP_THREADS)             // 16 rows' scales: 2 ks pieces of 16 bytes each
        cp_async16(reinterpret_cast<unsigned char *>(sg) + i * 16,
                   reinterpret_cast<const unsigned char *>(s13 + (i < 2 * ks ? row_g : row_u) * ks) + (i < 2 * ks ? i : i - 2 * ks) * 16);
    for (int i = tid; i < wpr; i += CP_THREADS) cp_async16(xs + i, reinterpret_cast<const uint4 *>(x + (long long)m * ldx) + i);
    cp_async_wait();
    __syncthreads();
    const int r = lane >> 2, q = lane & 3;
    float ag = 0.f, ag8 = 0.f, au = 0.f, au8 = 0.f;
    for (int g = warp; g < ks; g += CP_WARPS) {
        float cg[4] = {0.f, 0.f, 0.f, 0.f}, cu[4] = {0.f, 0.f, 0.f, 0.f};
        q4_group(cg, wg + g * 64, srow, xs + g * 16, lane);
        q4_group(cu, wu + g * 64, srow, xs + g * 16, lane);
        if (q == 0) {
            ag = fmaf(__bfloat162float(sg[r * ks + g]), cg[0], ag);
            ag8 = fmaf(__bfloat162float(sg[(r + 8) * ks + g]), cg[2], ag8);
            au = fmaf(__bfloat162float(su[r * ks + g]), cu[0], au);
            au8 = fmaf(__bfloat162float(su[(r + 8) * ks + g]), cu[2], au8);
        }
    }
    if (q == 0) {
        red[(warp * 2 + 0) * 16 + r] = ag; red[(warp * 2 + 0) * 16 + r + 8] = ag8;
        red[(warp * 2 + 1) * 16 + r] = au; red[(warp * 2 + 1) * 16 + r + 8] = au8;
    }
    __syncthreads();
    if (tid < 32) {                           // lanes 0-15 gate, 16-31 up
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < CP_WARPS; ++w) v += red[w * 32 + tid];
        const float up = __shfl_down_sync(0xffffffffu, v, 16);
        if (tid < 16) h[(long long)p * F + f0 + tid] = __float2bfloat16(siluf_(v) * up);
    }
}

constexpr int DC_NS = 3;                   // quad-steps of the shared expert per warp that are fetched before the dependency wait
// grid (H / 16, M), 256 threads.  Shared memory: top_k expert tiles [16][F/2 + pad] | scales [top_k][16][F/128] | h vectors |
// shared activation | reduction scratch (64 KB at the model's shapes: three blocks per SM).
template <bool FUSED>
__global__ void __launch_bounds__(CP_THREADS, 3) moe_down_cp_kernel(const uint32_t *w2, const bf16 *s2, const bf16 *h, const int *pair_expert,
                                                                 const float *pair_w, int top_k, int F, int H, const bf16 *shared_down,
                                                                 int ld_sd, const bf16 *sh_h, int SF, float *out, int ldo, FuseOut fo) {
    extern __shared__ __align__(128) unsigned char tm_smem[];
    const int rowb = F >> 1, srow = rowb + TM_PAD, ks = F >> 7, wpr = F >> 3;
    const int sch = shared_down ? SF >> 3 : 0;                           // 16-byte pieces of a shared row
    unsigned char *we = tm_smem;                                         // [top_k][16][srow]
    bf16 *sc = reinterpret_cast<bf16 *>(we + (size_t)top_k * 16 * srow); // [top_k][16 * ks]: 32 ks bytes per expert
    uint4 *hs = reinterpret_cast<uint4 *>(sc + (size_t)top_k * 16 * ks); // [top_k][wpr]
    uint4 *ss = hs + (size_t)top_k * wpr;                                // [sch]
    float *red = reinterpret_cast<float *>(ss + sch);                    // [8 warps][16]
    int *s_e = reinterpret_cast<int *>(red + CP_WARPS * 16);             // [top_k]
    float *s_w = reinterpret_cast<float *>(s_e + 32);                    // [top_k]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m = blockIdx.y, c0 = blockIdx.x * 16;
    const int r = lane >> 2, q = lane & 3;
    // the shared expert's rows do not depend on the routing: fetched, as operand words, before the wait for the router
    const bf16 *sr = shared_down + (long long)(c0 + r) * ld_sd;
    auto shared_words = [&](int st, uint4 &w0, uint4 &w8) {
        const int pc = st * 4 + q;
        w0 = w8 = make_uint4(0u, 0u, 0u, 0u);
        if (pc >= sch) return;
        w0 = __ldg(reinterpret_cast<const uint4 *>(sr) + pc);
        w8 = __ldg(reinterpret_cast<const uint4 *>(sr + 8LL * ld_sd) + pc);
    };
    uint4 sw[DC_NS], sw8[DC_NS];
#pragma unroll
    for (int i = 0; i < DC_NS; ++i) shared_words(warp + CP_WARPS * i, sw[i], sw8[i]);
    pdl_wait();
    pdl_trigger();
    if (tid < top_k) {
        const int p = m * top_k + tid;
        s_e[tid] = pair_expert[p];
        s_w[tid] = pair_w[p];
    }
    for (int i = tid; i < top_k * wpr; i += CP_THREADS) cp_async16(hs + i, reinterpret_cast<const uint4 *>(h + (long long)m * top_k * F) + i);
    for (int i = tid; i < sch; i += CP_THREADS) cp_async16(ss + i, reinterpret_cast<const uint4 *>(sh_h + (long long)m * SF) + i);
    __syncthreads();
    // an expert's 16 rows are one piece of memory; a thread keeps its places in the tile for all experts
    const int ppr = rowb >> 4, inv_ppr = div_inv(ppr), inv_ks = div_inv(ks);
    for (int i = tid; i < 16 * ppr; i += CP_THREADS) {
        unsigned char *dst = we + i * 16 + div_by(i, inv_ppr) * TM_PAD;
        const unsigned char *src = reinterpret_cast<const unsigned char *>(w2 + (long long)c0 * wpr) + i * 16;
#pragma unroll 5
        for (int j = 0; j < top_k; ++j) {
            const int e = s_e[j];
            if (e >= 0) cp_async16(dst + j * 16 * srow, src + (long long)e * H * rowb);
        }
    }
    for (int i = tid; i < top_k * 2 * ks; i += CP_THREADS) {
        const int j = div_by(i >> 1, inv_ks), b = i - j * 2 * ks, e = s_e[j];
        if (e >= 0) cp_async16(reinterpret_cast<unsigned char *>(sc) + i * 16, reinterpret_cast<const unsigned char *>(s2 + ((long long)e * H + c0) * ks) + b * 16);
    }
    cp_async_wait();
    __syncthreads();
    float a0 = 0.f, a8 = 0.f;
    const int nitems = top_k * ks;
    for (int it = warp; it < nitems; it += CP_WARPS) {
        const int j = div_by(it, inv_ks), g = it - j * ks;
        if (s_e[j] < 0) continue;                       // warp-uniform
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        q4_group(c, we + (size_t)j * 16 * srow + g * 64, srow, hs + (size_t)j * wpr + g * 16, lane);
        if (q == 0) {
            const bf16 *sj = sc + (size_t)j * 16 * ks;
            a0 = fmaf(__bfloat162float(sj[r * ks + g]) * s_w[j], c[0], a0);
            a8 = fmaf(__bfloat162float(sj[(r + 8) * ks + g]) * s_w[j], c[2], a8);
        }
    }
    {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        auto shared_step = [&](int st, const uint4 &w0, const uint4 &w8) {
            if (st * 4 >= sch) return;                  // warp-uniform
            mma_bf16_chunk(c, w0, w8, st * 4 + q < sch ? ss[st * 4 + q] : make_uint4(0u, 0u, 0u, 0u));
        };
#pragma unroll
        for (int i = 0; i < DC_NS; ++i) shared_step(warp + CP_WARPS * i, sw[i], sw8[i]);
        for (int st = warp + CP_WARPS * DC_NS; st * 4 < sch; st += CP_WARPS) {
            uint4 w0, w8;
            shared_words(st, w0, w8);
            shared_step(st, w0, w8);
        }
        a0 += c[0];
        a8 += c[2];
    }
    if (q == 0) {
        red[warp * 16 + r] = a0;
        red[warp * 16 + r + 8] = a8;
    }
    __syncthreads();
    if (tid < 16) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < CP_WARPS; ++w) v += red[w * 16 + tid];
        if (FUSED) fuse_put_col(fo, fuse_seq(fo), m, c0 + tid, __float_as_uint(v));      // fused reduce-scatter: to the column's owner
        else out[(long long)m * ldo + c0 + tid] = v;
    }
}

}  // namespace qw
