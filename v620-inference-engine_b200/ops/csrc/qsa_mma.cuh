// Tensor-core QSA attention for token-major prefill (included by qsa.cu inside namespace qw).
//
// One block per (query row, local KV head): the query heads that share the KV head (<= 16; 12 in the full model at
// one rank) are the 16 rows of the MMA tile, so the gathered K and V rows of a token are fetched once for all of
// them.  The row's token list (every visible token below the budget, else the selected groups plus the open tail) is
// walked in tiles of 64 tokens: rows gathered into padded shared memory by one 512-byte bulk-async copy per row
// straight from the paged pool (device pages or the spill cache; rows that live in host pages are copied by their
// thread with plain loads), completing on an mbarrier per tile, S = Q K^T and O += P V on mma.sync m16n8k16 bf16 with
// fp32 accumulation, online softmax in fp32 with one running maximum per query head shared by the four warps.
// The copies of the next tile's K overlap P V of this tile and the copies of its V overlap the next S.  Every wait on
// a tile's mbarrier is bounded.
// Output: o = softmax(..) V * sigmoid(gate) in bf16, with no partial buffers and no merge kernel
// (role of the reference's qsa_attend_T + combine, src/kernels/qsa.hip:136-243).
#pragma once

constexpr int AT = 64;               // tokens per tile
constexpr int KV_LD = HD + 8;        // shared row stride (bf16): 528 bytes keeps the 8 rows of an ldmatrix in distinct banks
constexpr int P_LD = AT + 8;
constexpr int ATT_SMEM = (2 * AT * KV_LD + 16 * P_LD) * 2 + (4 * 16 * 2) * 4 + 16;

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3, uint32_t saddr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(saddr));
}

// Starts the copies of one tile of K rows (which = 0) or V rows (which = 1): thread r < 64 owns token r of the tile
// and arrives once on `bar` (64 arrivals complete a tile).  Device rows: one bulk-async copy of the head's 512 bytes.
// Rows in host pages: copied here with plain loads.  Tokens past the list's end: zero-filled.
__device__ __forceinline__ void att_issue(const QsaAttendArgs &a, bf16 *dst_tile, uint64_t *bar, int which, int tile,
                                          int count, int dense, const int *sel, int nb, int slot, int kvh, bool record) {
    const int r = threadIdx.x;
    if (r >= AT) return;
    bf16 *dst = dst_tile + r * KV_LD;
    const int t = tile * AT + r;
    if (t < count) {
        const int tok = list_token(t, dense, sel, a.ratio, a.topk, nb);
        bool host;
        const long long off = kv_off(a.kv, slot, tok, host);
        const bf16 *kp = a.kv.k_dev + off, *vp = a.kv.v_dev + off;
        bool from_host = false;
        if (host) {
            kv_rows_read(a.kv, a.sc, slot, tok, record && which == 0, kp, vp);
            from_host = kp == a.kv.k_host + off;           // not in the spill cache
        }
        const bf16 *src = (which ? vp : kp) + kvh * HD;
        if (!from_host) {
            mbar_expect_tx(bar, HD * 2);
            bulk_g2s(dst, src, HD * 2, bar);
            return;
        }
        const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
        uint4 *d4 = reinterpret_cast<uint4 *>(dst);
#pragma unroll 8
        for (int i = 0; i < HD * 2 / 16; ++i) d4[i] = s4[i];
    } else {
        uint4 *d4 = reinterpret_cast<uint4 *>(dst);
#pragma unroll 8
        for (int i = 0; i < HD * 2 / 16; ++i) d4[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    mbar_arrive(bar);
}

// ------------------------------------------------------------------------------------------------------------------
// Flash-decode over the token list for the rows of a step.  A block takes 64 entries of one row's list for all query heads of one KV head (<= 16,
// the 16 rows of the MMA tile) and leaves the partial softmax (maximum, sum, sums of V) that qsa_combine_kernel merges.  Operands keep what fp32
// holds: the queries and the weights go through the MMAs as three bf16 parts each (24 bits), keys and values are bf16 anyway.  Sums are rounded
// fp32 additions of what one MMA sums; with one running sum in the tensor core the error was three times the scalar form's.
// Error of the merged output before bf16 against 64 bits, queries of size 0.3 / 1 / 2 / 4: scalar form 0.95, 1.34, 2.41, 3.64e-7; here 0.62, 1.18,
// 2.36, 3.51e-7.
// In a scalar form (four heads a block, a warp per token) each token's rows were fetched once for every four heads and every score was five
// shuffles.  With the merge, at 4,096 tokens: 24 rows 197 us, now 57; 8 rows 67 / 21.6; one 17.2 / 11.1.
// grid (nsplit, M, KVL), 256 threads.
// ------------------------------------------------------------------------------------------------------------------
constexpr int AD_SMEM = (2 * AT * KV_LD + 3 * 16 * KV_LD + 3 * 16 * P_LD) * 2 + 2 * 8 * 16 * 4 + 16;

// x as three bf16 parts, two values at a time
__device__ __forceinline__ void split3(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const bf162 h = __floats2bfloat162_rn(x, y);
        p[i] = *reinterpret_cast<const uint32_t *>(&h);
        x -= bf16_lo(p[i]);
        y -= bf16_hi(p[i]);
    }
}

// Sum over first parts + sum over the others.  An infinity of K or V has its sign from the first part alone: the others may be zero or of the other sign, and
// their products with it would make the sum NaN.
__device__ __forceinline__ float split_sum(float first, float rest) { return fabsf(first) == INFINITY ? first : rest + first; }

__global__ void __launch_bounds__(256, 2) qsa_attend_split_kernel(QsaAttendArgs a, ErrorWord *g_err) {
    extern __shared__ __align__(16) unsigned char att_sm[];
    bf16 *Ks = reinterpret_cast<bf16 *>(att_sm);             // [64][KV_LD]
    bf16 *Vs = Ks + AT * KV_LD;                              // [64][KV_LD]
    bf16 *Qs = Vs + AT * KV_LD;                              // [3][16][KV_LD]
    bf16 *Ps = Qs + 3 * 16 * KV_LD;                          // [3][16][P_LD]
    float *s_max = reinterpret_cast<float *>(Ps + 3 * 16 * P_LD);    // [8][16]
    float *s_l = s_max + 128;                                // [8][16]
    uint64_t *kbar = reinterpret_cast<uint64_t *>(s_l + 128), *vbar = kbar + 1;
    const int sp = blockIdx.x, m = blockIdx.y, kvh = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const int per_kv = a.QL / a.KVL, h0 = kvh * per_kv;
    if (tid == 0) {
        mbar_init(kbar, AT);
        mbar_init(vbar, AT);
        mbar_fence_init();
    }
    const int slot = a.rows.slot[m], pos = a.rows.pos[m];    // the row table: written before the step began
    const int nb = (pos + 1) / a.ratio;
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const int dense = a.sel_n[m] < 0;
    const int count = dense ? pos + 1 : a.topk * a.ratio + (pos + 1 - nb * a.ratio);
    if (sp * AT >= count) {                                  // the list ends before this block: nothing that the merge reads
        if (tid < per_kv) a.pm[((long long)m * a.QL + h0 + tid) * a.nsplit + sp] = -INFINITY;
        return;
    }
    const int *sel = a.sel + (long long)m * a.topk;
    att_issue(a, Ks, kbar, 0, sp, count, dense, sel, nb, slot, kvh, kvh == 0);
    att_issue(a, Vs, vbar, 1, sp, count, dense, sel, nb, slot, kvh, false);
    for (int i = tid; i < 16 * (HD / 4); i += 256) {
        const int r = i / (HD / 4), c = (i % (HD / 4)) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < per_kv) v = *reinterpret_cast<const float4 *>(a.q + ((long long)m * a.QL + h0 + r) * HD + c);
        uint32_t p0[3], p1[3];
        split3(v.x, v.y, p0);
        split3(v.z, v.w, p1);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint2 *>(Qs + (k * 16 + r) * KV_LD + c) = make_uint2(p0[k], p1[k]);
    }
    __syncthreads();
    const uint32_t ks_base = (uint32_t)__cvta_generic_to_shared(Ks), vs_base = (uint32_t)__cvta_generic_to_shared(Vs);
    const uint32_t qs_base = (uint32_t)__cvta_generic_to_shared(Qs), ps_base = (uint32_t)__cvta_generic_to_shared(Ps);
    bool ok = mbar_wait_warp(kbar, 0u, g_err);               // bounded; after a time-out the meetings still take place
    // ---- S = Q K^T for this warp's 8 tokens.  Of the queries' first parts every 16 products are summed from zero and added with rounding, in four
    // chains (the tensor core's own running sum cuts off); the other two parts are 2^-8 and 2^-16 of them
    float s1[4][4] = {}, s2[4] = {};
    {
        const uint32_t brow = ks_base + (uint32_t)((w * 8 + (lane & 7)) * KV_LD * 2 + (lane >> 3) * 16);
#pragma unroll 4
        for (int ks = 0; ks < 16; ks += 2) {
            uint32_t b[4];
            ldmatrix_x4(b[0], b[1], b[2], b[3], brow + ks * 32);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                uint32_t q0, q1, q2, q3;
                float c[4] = {};
                ldmatrix_x4(q0, q1, q2, q3, a_tile_addr(qs_base, KV_LD * 2, (ks + j) * 16, lane));
                mma_bf16(c, q0, q1, q2, q3, b[2 * j], b[2 * j + 1]);
#pragma unroll
                for (int i = 0; i < 4; ++i) s1[(ks + j) & 3][i] += c[i];
#pragma unroll
                for (int k = 1; k < 3; ++k) {
                    ldmatrix_x4(q0, q1, q2, q3, a_tile_addr(qs_base + k * 16 * KV_LD * 2, KV_LD * 2, (ks + j) * 16, lane));
                    mma_bf16(s2, q0, q1, q2, q3, b[2 * j], b[2 * j + 1]);
                }
            }
        }
    }
    float s[4], tm[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float first = (s1[0][i] + s1[1][i]) + (s1[2][i] + s1[3][i]);
        s[i] = sp * AT + w * 8 + 2 * t4 + (i & 1) < count ? split_sum(first, s2[i]) * 0.0625f : -INFINITY;       // 1/sqrt(256)
        tm[i >> 1] = fmaxf(tm[i >> 1], s[i]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        tm[h] = fmaxf(tm[h], __shfl_xor_sync(0xffffffffu, tm[h], 1));
        tm[h] = fmaxf(tm[h], __shfl_xor_sync(0xffffffffu, tm[h], 2));
        if (t4 == 0) s_max[w * 16 + g + 8 * h] = tm[h];
    }
    __syncthreads();
    bool none[2];                                            // every score is -inf (keys that are infinite): the block adds nothing to this row
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float mx = s_max[g + 8 * h];
#pragma unroll
        for (int k = 1; k < 8; ++k) mx = fmaxf(mx, s_max[k * 16 + g + 8 * h]);
        none[h] = mx == -INFINITY;
        const float p0 = __expf(s[2 * h] - mx), p1 = __expf(s[2 * h + 1] - mx);
        uint32_t p[3];
        split3(p0, p1, p);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t *>(Ps + (k * 16 + g + 8 * h) * P_LD + w * 8 + 2 * t4) = p[k];
        float l = p0 + p1;
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        if (t4 == 0) s_l[w * 16 + g + 8 * h] = l;
    }
    __syncthreads();                                         // P and the sums visible
    if (tid < per_kv) {
        float mx = s_max[tid], l = 0.f;
#pragma unroll
        for (int k = 1; k < 8; ++k) mx = fmaxf(mx, s_max[k * 16 + tid]);
#pragma unroll
        for (int k = 0; k < 8; ++k) l += s_l[k * 16 + tid];
        const long long o = ((long long)m * a.QL + h0 + tid) * a.nsplit + sp;
        a.pm[o] = fmaxf(mx, -FLT_MAX);
        a.pl[o] = mx == -INFINITY ? 0.f : l;
    }
    ok = ok && mbar_wait_warp(vbar, 0u, g_err);
    // ---- P V for this warp's 32 output dims, summed as the scores are
    float acc[4][4] = {}, acc2[4][4] = {};
    {
        const int mid = lane >> 3;
        const uint32_t vrow = vs_base + (uint32_t)((((mid & 1) * 8 + (lane & 7)) * KV_LD + w * 32 + (mid >> 1) * 8) * 2);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            uint32_t b[2][4];
#pragma unroll
            for (int n = 0; n < 2; ++n) ldmatrix_x4_trans(b[n][0], b[n][1], b[n][2], b[n][3], vrow + (uint32_t)(ks * 16 * KV_LD * 2 + n * 32));
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                uint32_t p0, p1, p2, p3;
                ldmatrix_x4(p0, p1, p2, p3, a_tile_addr(ps_base + k * 16 * P_LD * 2, P_LD * 2, ks * 16, lane));
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    const uint32_t b0 = b[n >> 1][(n & 1) * 2], b1 = b[n >> 1][(n & 1) * 2 + 1];
                    if (k) {
                        mma_bf16(acc2[n], p0, p1, p2, p3, b0, b1);
                    } else {
                        float c[4] = {};
                        mma_bf16(c, p0, p1, p2, p3, b0, b1);
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[n][i] += c[i];
                    }
                }
            }
        }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = none[i >> 1] ? 0.f : split_sum(acc[n][i], acc2[n][i]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = g + 8 * h;
        if (r >= per_kv) continue;
        float *o = a.pacc + (((long long)m * a.QL + h0 + r) * a.nsplit + sp) * HD + w * 32 + 2 * t4;
#pragma unroll
        for (int n = 0; n < 4; ++n) *reinterpret_cast<float2 *>(o + n * 8) = make_float2(acc[n][2 * h], acc[n][2 * h + 1]);
    }
}

// grid (KVL, M), 128 threads.
__global__ void __launch_bounds__(128, 3) qsa_attend_mma_kernel(QsaAttendArgs a, const float *proj, int ld_proj, bf16 *o,
                                                                ErrorWord *g_err) {
    extern __shared__ __align__(16) unsigned char att_sm[];
    bf16 *Ks = reinterpret_cast<bf16 *>(att_sm);             // [64][KV_LD]   (first: the 16 query rows, staged once)
    bf16 *Vs = Ks + AT * KV_LD;                              // [64][KV_LD]
    bf16 *Ps = Vs + AT * KV_LD;                              // [16][P_LD]
    float *s_max = reinterpret_cast<float *>(Ps + 16 * P_LD);    // [4][16]
    float *s_l = s_max + 64;                                 // [4][16]
    uint64_t *kbar = reinterpret_cast<uint64_t *>(s_l + 64), *vbar = kbar + 1;     // one phase per tile
    const int kvh = blockIdx.x, m = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const int per_kv = a.QL / a.KVL, h0 = kvh * per_kv;
    const int slot = a.rows.slot[m], pos = a.rows.pos[m];
    const int nb = (pos + 1) / a.ratio;
    const int dense = a.sel_n[m] < 0;
    const int count = dense ? pos + 1 : a.topk * a.ratio + (pos + 1 - nb * a.ratio);
    const int ntiles = (count + AT - 1) / AT;
    const int *sel = a.sel + (long long)m * a.topk;
    const uint32_t ks_base = (uint32_t)__cvta_generic_to_shared(Ks), vs_base = (uint32_t)__cvta_generic_to_shared(Vs);
    if (tid == 0) {
        mbar_init(kbar, AT);
        mbar_init(vbar, AT);
        mbar_fence_init();
    }
    const uint32_t ps_base = (uint32_t)__cvta_generic_to_shared(Ps);
    // ---- the query rows -> bf16 in shared memory -> A fragments held in registers for the whole walk
    for (int i = tid; i < 16 * (HD / 2); i += 128) {
        const int r = i / (HD / 2), c = (i % (HD / 2)) * 2;
        float2 v = make_float2(0.f, 0.f);
        if (r < per_kv) v = *reinterpret_cast<const float2 *>(a.q + ((long long)m * a.QL + h0 + r) * HD + c);
        *reinterpret_cast<bf162 *>(Ks + r * KV_LD + c) = __floats2bfloat162_rn(v.x, v.y);
    }
    __syncthreads();
    uint32_t qf[16][4];
#pragma unroll
    for (int ks = 0; ks < 16; ++ks)
        ldmatrix_x4(qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3], a_tile_addr(ks_base, KV_LD * 2, ks * 16, lane));
    __syncthreads();
    att_issue(a, Ks, kbar, 0, 0, count, dense, sel, nb, slot, kvh, kvh == 0);
    att_issue(a, Vs, vbar, 1, 0, count, dense, sel, nb, slot, kvh, false);
    float acc[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
    float mx0 = -INFINITY, mx1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    for (int tile = 0; tile < ntiles; ++tile) {
        mbar_wait_warp(kbar, (unsigned)tile & 1u, g_err);        // this tile's K rows have landed (bounded; a time-out is recorded)
        // ---- S = Q K^T for this warp's 16 tokens
        float s[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) s[n][i] = 0.f;
        {
            const int mid = lane >> 3;
            const uint32_t brow = ks_base + (uint32_t)((w * 16 + (mid >> 1) * 8 + (lane & 7)) * KV_LD * 2 + (mid & 1) * 16);
#pragma unroll
            for (int ks = 0; ks < 16; ++ks) {
                uint32_t b0, b1, b2, b3;
                ldmatrix_x4(b0, b1, b2, b3, brow + ks * 32);
                mma_bf16(s[0], qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3], b0, b1);
                mma_bf16(s[1], qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3], b2, b3);
            }
        }
        float tm0 = -INFINITY, tm1 = -INFINITY;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = tile * AT + w * 16 + n * 8 + 2 * t4 + (i & 1);
                const float v = t < count ? s[n][i] * 0.0625f : -INFINITY;       // 1/sqrt(256)
                s[n][i] = v;
                if (i < 2) tm0 = fmaxf(tm0, v); else tm1 = fmaxf(tm1, v);
            }
        tm0 = fmaxf(tm0, __shfl_xor_sync(0xffffffffu, tm0, 1));
        tm0 = fmaxf(tm0, __shfl_xor_sync(0xffffffffu, tm0, 2));
        tm1 = fmaxf(tm1, __shfl_xor_sync(0xffffffffu, tm1, 1));
        tm1 = fmaxf(tm1, __shfl_xor_sync(0xffffffffu, tm1, 2));
        if (t4 == 0) { s_max[w * 16 + g] = tm0; s_max[w * 16 + g + 8] = tm1; }
        __syncthreads();         // every warp is past its reads of the K tile, too
        if (tile + 1 < ntiles) att_issue(a, Ks, kbar, 0, tile + 1, count, dense, sel, nb, slot, kvh, kvh == 0);
        const float n0 = fmaxf(fmaxf(fmaxf(s_max[g], s_max[16 + g]), fmaxf(s_max[32 + g], s_max[48 + g])), mx0);
        const float n1 = fmaxf(fmaxf(fmaxf(s_max[g + 8], s_max[24 + g]), fmaxf(s_max[40 + g], s_max[56 + g])), mx1);
        // the first tile always holds a visible token, so n0 / n1 are finite
        const float c0 = __expf(mx0 - n0), c1 = __expf(mx1 - n1);
        mx0 = n0; mx1 = n1;
        l0 *= c0; l1 *= c1;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const float p0 = __expf(s[n][0] - n0), p1 = __expf(s[n][1] - n0);
            const float p2 = __expf(s[n][2] - n1), p3 = __expf(s[n][3] - n1);
            l0 += p0 + p1;
            l1 += p2 + p3;
            const int c = w * 16 + n * 8 + 2 * t4;
            *reinterpret_cast<bf162 *>(Ps + g * P_LD + c) = __floats2bfloat162_rn(p0, p1);
            *reinterpret_cast<bf162 *>(Ps + (g + 8) * P_LD + c) = __floats2bfloat162_rn(p2, p3);
        }
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            acc[n][0] *= c0; acc[n][1] *= c0;
            acc[n][2] *= c1; acc[n][3] *= c1;
        }
        __syncthreads();         // P visible
        mbar_wait_warp(vbar, (unsigned)tile & 1u, g_err);        // this tile's V rows have landed
        // ---- O += P V for this warp's 64 output dims
        {
            const int mid = lane >> 3;
            const uint32_t vrow = vs_base + (uint32_t)((((mid & 1) * 8 + (lane & 7)) * KV_LD + w * 64 + (mid >> 1) * 8) * 2);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                uint32_t p0, p1, p2, p3;
                ldmatrix_x4(p0, p1, p2, p3, a_tile_addr(ps_base, P_LD * 2, ks * 16, lane));
#pragma unroll
                for (int n2 = 0; n2 < 4; ++n2) {
                    uint32_t b0, b1, b2, b3;
                    ldmatrix_x4_trans(b0, b1, b2, b3, vrow + (uint32_t)(ks * 16 * KV_LD * 2 + n2 * 32));
                    mma_bf16(acc[2 * n2], p0, p1, p2, p3, b0, b1);
                    mma_bf16(acc[2 * n2 + 1], p0, p1, p2, p3, b2, b3);
                }
            }
        }
        __syncthreads();         // V, P and the maxima are free again
        if (tile + 1 < ntiles) att_issue(a, Vs, vbar, 1, tile + 1, count, dense, sel, nb, slot, kvh, false);
    }
    // ---- normalise, gate, store
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
    l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
    if (t4 == 0) { s_l[w * 16 + g] = l0; s_l[w * 16 + g + 8] = l1; }
    __syncthreads();
    const float L0 = s_l[g] + s_l[16 + g] + s_l[32 + g] + s_l[48 + g];
    const float L1 = s_l[g + 8] + s_l[24 + g] + s_l[40 + g] + s_l[56 + g];
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        const int r = g + hh * 8;
        if (r >= per_kv) continue;
        const float inv = 1.f / (hh ? L1 : L0);
        const float *gate = proj + (long long)m * ld_proj + (long long)(h0 + r) * 2 * HD + HD;
        bf16 *orow = o + ((long long)m * a.QL + h0 + r) * HD;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const int d = w * 64 + n * 8 + 2 * t4;
            const float2 gt = *reinterpret_cast<const float2 *>(gate + d);
            const float y0 = acc[n][2 * hh] * inv * sigmoidf_(gt.x), y1 = acc[n][2 * hh + 1] * inv * sigmoidf_(gt.y);
            *reinterpret_cast<bf162 *>(orow + d) = __floats2bfloat162_rn(y0, y1);
        }
    }
}

// ------------------------------------------------------------------------------------------------------------------
// Indexer scores of a prefill chunk on the tensor cores: score[m][c] = sum_h relu(iq[m][h] . ck[c]) / sqrt(128) for the
// groups c visible to row m, for rows whose visible groups exceed the budget (the others attend densely).
// A block takes 16 consecutive rows of the chunk (one slot, ascending positions): the MMA rows of a warp are its 4
// query rows x 4 indexer heads, the fp32 queries split into a bf16 high and low part (two MMAs per step) so that the
// ranking keeps fp32-like resolution against the bf16 keys; key tiles of 64 groups go through shared memory and are
// shared by the four warps.  The sum over the heads is two lane shuffles on the accumulator fragment.
// grid (ceil(M / 16), SC_SPLIT), 128 threads; block y takes key tiles y, y + SC_SPLIT, ...   IH == 4.
// (Role of the reference's score GEMM + score_reduce, src/kernels/qsa.hip and docs/MODEL.md:150-160.)
// ------------------------------------------------------------------------------------------------------------------
constexpr int SC_SPLIT = 4;
constexpr int SC_LD = ID + 8;        // shared row stride of a key tile (bf16)

__global__ void __launch_bounds__(128) qsa_scores_mma_kernel(const float *iq, const bf16 *ck, int ck_cap, Rows rows, int ratio,
                                                             int topk_blocks, float *scores, int ld_scores) {
    __shared__ __align__(16) bf16 tile[64 * SC_LD];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const int m0 = blockIdx.x * 16;
    const int m_last = min(m0 + 15, rows.M - 1);
    const int nb_max = (rows.pos[m_last] + 1) / ratio;
    if (nb_max <= topk_blocks) return;                       // every row of the block attends densely (uniform)
    const int slot = rows.slot[m0];
    const bf16 *keys = ck + (long long)slot * ck_cap * ID;
    // ---- A fragments: MMA row i = 4 * (query row within the warp) + head; rows g and g + 8 of this lane
    uint32_t ahi[8][4], alo[8][4];
    int nb_row[2];
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        const int i = g + hh * 8, m = m0 + w * 4 + (i >> 2), h = i & 3;
        const bool ok = m < rows.M;
        nb_row[hh] = ok ? (rows.pos[m] + 1) / ratio : 0;
        const float *q = iq + ((long long)(ok ? m : m0) * 4 + h) * ID;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float2 v = *reinterpret_cast<const float2 *>(q + ks * 16 + half * 8 + 2 * t4);
                if (!ok) v = make_float2(0.f, 0.f);
                const bf162 hi = __floats2bfloat162_rn(v.x, v.y);
                const float2 hf = __bfloat1622float2(hi);
                const bf162 lo = __floats2bfloat162_rn(v.x - hf.x, v.y - hf.y);
                ahi[ks][hh + 2 * half] = *reinterpret_cast<const uint32_t *>(&hi);
                alo[ks][hh + 2 * half] = *reinterpret_cast<const uint32_t *>(&lo);
            }
    }
    const uint32_t tile_base = (uint32_t)__cvta_generic_to_shared(tile);
    const int ntiles = (nb_max + 63) / 64;
    for (int kt = blockIdx.y; kt < ntiles; kt += SC_SPLIT) {
        const int c0 = kt * 64;
        __syncthreads();                                     // the previous tile has been read
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int idx = tid + i * 128;                   // 16-byte piece: 64 groups x 16
            const int r = idx >> 4, p = idx & 15;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (c0 + r < nb_max) v = __ldg(reinterpret_cast<const uint4 *>(keys + (long long)(c0 + r) * ID) + p);
            *reinterpret_cast<uint4 *>(tile + r * SC_LD + p * 8) = v;
        }
        __syncthreads();
        float acc[8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
        const int mid = lane >> 3;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
#pragma unroll
            for (int n2 = 0; n2 < 4; ++n2) {
                uint32_t b0, b1, b2, b3;
                ldmatrix_x4(b0, b1, b2, b3, tile_base + (uint32_t)(((n2 * 16 + (mid >> 1) * 8 + (lane & 7)) * SC_LD + ks * 16 + (mid & 1) * 8) * 2));
                mma_bf16(acc[2 * n2], ahi[ks][0], ahi[ks][1], ahi[ks][2], ahi[ks][3], b0, b1);
                mma_bf16(acc[2 * n2], alo[ks][0], alo[ks][1], alo[ks][2], alo[ks][3], b0, b1);
                mma_bf16(acc[2 * n2 + 1], ahi[ks][0], ahi[ks][1], ahi[ks][2], ahi[ks][3], b2, b3);
                mma_bf16(acc[2 * n2 + 1], alo[ks][0], alo[ks][1], alo[ks][2], alo[ks][3], b2, b3);
            }
        // relu, sum over the 4 heads (lanes that differ in the low two bits of g), store
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            float s[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float v = fmaxf(acc[n][i], 0.f);
                v += __shfl_xor_sync(0xffffffffu, v, 4);
                v += __shfl_xor_sync(0xffffffffu, v, 8);
                s[i] = v * 0.08838834764831845f;
            }
            if ((g & 3) == 0) {
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int m = m0 + w * 4 + ((g + hh * 8) >> 2);
                    const int nb = nb_row[hh];
                    if (m < rows.M && nb > topk_blocks) {
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            const int c = c0 + n * 8 + 2 * t4 + j;
                            if (c < nb) scores[(long long)m * ld_scores + c] = s[hh * 2 + j];
                        }
                    }
                }
            }
        }
    }
}
