// QSA attention of a prefill chunk on the 5th-generation tensor cores: every key of the context against 256 query rows at a time, the
// keys a row does not attend to masked out.
//
// The rows of one KV head - queries of the chunk times the query heads that share it - are numbered query by query; a pair of CTAs
// (cta_group::2) takes 256 of them, 128 per CTA, and walks the context in tiles of 128 keys.  Per tile S = Q K^T and O += P V
// accumulate in tensor memory (columns 0-255: two S buffers, over which P is written as bf16; 256-511: O).  A CTA loads half of each
// tile: 64 of the keys for S, 128 of V's 256 columns for O.
//   warp 0       TMA: K and V tiles, 32 KB a stage and CTA, five stages, in the order in which the MMAs take them
//   warp 1       MMAs (leader CTA): S of the next tile, then O of this one
//   warps 4-11   softmax: two threads per row, 64 keys each; the maxima meet in shared memory, O is rescaled by 128 columns each
// A row's set of keys is one bit per group of four (qsa_mask_kernel); only tiles that reach past a row's position compare positions.
// The reference of the exponentials is the row's running maximum, as in the kernel that gathers.
// A masked key's weight is 0, and 0 times a value that is not finite is NaN: a row that such a key of other rows, or of a later position, has
// spoiled is formed again from its own keys (qt_row_alone).
//
// Why not gather: 2,051 rows per query are 4.2 MB out of L2 for every query, and that, at 6.8 TB/s, is what the gather costs
// (qsa_mma.cuh: 0.66 us per query, wherever it lies).  Here a tile is read once for 21 queries of 12 heads; the price is the keys nobody
// chose, so contexts that are long for their chunk stay with the gather (qwk_qsa_takes_tc).  24 query heads over 2, us a layer,
// gathered / here: 1,021 tokens 220 / 58, 4,096 tokens 1897 / 314, 2,048 tokens at position 16,384 1340 / 991.
#include "kernels.h"
#include "tc.cuh"

namespace qw {

constexpr int QT_D = 256;                        // head dim
constexpr int QT_ST = 5, QT_STAGE = 32768, QT_Q = 65536, QT_THREADS = 384;
constexpr float QT_SCALE = 1.4426950408889634f / 16.f;          // log2(e) / sqrt(256)
constexpr int QT_STG_LD = 36;                    // floats between the rows of an epilogue piece
constexpr int QT_SMEM = QT_Q + QT_ST * QT_STAGE + 1024 /*alignment*/ + 128 /*barriers*/ + 2 * 128 * 4 /*maxima, sums*/;

struct QsaTcArgs {
    const float *q;          // [M][QL][256]
    int QL, KVL, M, n_dev_pages, staged;
    const bf16 *k_dev, *v_dev;       // the pages that the first pair of maps covers
    const bf16 *k_host, *v_host;     // pages from n_dev_pages on; staged: copies of them in device memory, which the second pair of maps covers
    const int *slot, *pos;   // one run of one slot: pos[m] = pos[0] + m
    const int *page_table;
    int max_pages;
    const uint32_t *mask;    // [M][ld_mask]: bit g of word j: group 32 j + g
    int ld_mask;
    const float *proj;
    int ld_proj;
    bf16 *o;                 // [M][QL][256]
    ErrorWord *err;
};

__device__ __forceinline__ float ex2(float x) {          // 2^x, two ulp; below 2^-126 zero
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Bits of the groups that row m attends to.  grid M, 128 threads.
__global__ void __launch_bounds__(128) qsa_mask_kernel(const int *pos, const int *sel, const int *sel_n, int topk, uint32_t *mask, int ld_mask) {
    extern __shared__ uint32_t bits[];
    const int m = blockIdx.x, last = pos[m], words = (last >> 7) + 1;
    const bool dense = sel_n[m] < 0;
    for (int i = threadIdx.x; i < words; i += 128) bits[i] = dense ? 0xffffffffu : 0u;
    __syncthreads();
    if (!dense) {
        for (int i = threadIdx.x; i < topk; i += 128) {
            const int g = sel[(long long)m * topk + i];
            atomicOr(bits + (g >> 5), 1u << (g & 31));
        }
        if (threadIdx.x == 0 && (last + 1) & 3) atomicOr(bits + (last >> 7), 1u << ((last >> 2) & 31));      // the open group
    }
    __syncthreads();
    for (int i = threadIdx.x; i < words; i += 128) mask[(long long)m * ld_mask + i] = bits[i];
}

// A stage's wait by the warp that issues for both CTAs: rows that a producer copied itself were released to the cluster.
__device__ __forceinline__ bool qt_try_cluster(uint64_t *bar, unsigned parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(20000u)
        : "memory");
    return ok != 0;
}

// 64 rows of K (four panels of 64 columns) or 128 rows of V (two) from memory that TMA does not read, by the producer warp.
__device__ __forceinline__ void qt_copy(unsigned char *d, const bf16 *src, int row, bool is_v, int lane) {
    const int u = is_v ? lane & 15 : lane, sub = is_v ? lane >> 4 : 0, per = is_v ? 2 : 1;
    unsigned char *p = d + (u >> 3) * (is_v ? 16384 : 8192);
    for (int r0 = 0; r0 < 64; r0 += 8) {
        uint4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = *reinterpret_cast<const uint4 *>(src + (long long)((r0 + i) * per + sub) * row + u * 8);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = (r0 + i) * per + sub;
            *reinterpret_cast<uint4 *>(p + r * 128 + (((u & 7) ^ (r & 7)) << 4)) = v[i];
        }
    }
}

// Row (m, h) from the keys that it attends to and no others, by one warp: eight of the 256 dims a lane, a key at a time, with the roundings of the tiles.
__device__ __noinline__ void qt_row_alone(const QsaTcArgs &a, int m, int h, int lane) {
    const int pos = a.pos[0] + m, row = a.KVL * QT_D, col = h / (a.QL / a.KVL) * QT_D + lane * 8;
    const int *pages = a.page_table + (long long)a.slot[0] * a.max_pages;
    const uint32_t *mask = a.mask + (long long)m * a.ld_mask;
    const float *qr = a.q + ((long long)m * a.QL + h) * QT_D + lane * 8;
    float q[8], acc[8], ref = -1e30f, sum = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        q[i] = __bfloat162float(__float2bfloat16(qr[i]));
        acc[i] = 0.f;
    }
    for (int t = 0; t <= pos; ++t) {
        if (!(mask[t >> 7] >> ((t >> 2) & 31) & 1u)) {
            t |= 3;                              // none of the group's four
            continue;
        }
        const int page = pages[t / KV_PAGE];
        const bool host = page >= a.n_dev_pages;
        const long long at = ((long long)(host ? page - a.n_dev_pages : page) * KV_PAGE + t % KV_PAGE) * row + col;
        const uint4 k = *reinterpret_cast<const uint4 *>((host ? a.k_host : a.k_dev) + at), v = *reinterpret_cast<const uint4 *>((host ? a.v_host : a.v_dev) + at);
        const uint32_t kw[4] = {k.x, k.y, k.z, k.w}, vw[4] = {v.x, v.y, v.z, v.w};
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) s = fmaf(q[i], i & 1 ? bf16_hi(kw[i >> 1]) : bf16_lo(kw[i >> 1]), s);
        s = warp_sum(s) * QT_SCALE;
        const float nref = fmaxf(ref, s), f = ex2(ref - nref), x = ex2(s - nref), w = __bfloat162float(__float2bfloat16(x));
        ref = nref;
        sum = fmaf(sum, f, x);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = fmaf(acc[i], f, w * (i & 1 ? bf16_hi(vw[i >> 1]) : bf16_lo(vw[i >> 1])));
    }
    const float inv = 1.f / sum, *gate = a.proj + (long long)m * a.ld_proj + h * 2 * QT_D + QT_D + lane * 8;
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = pack_bf16(acc[2 * i] * inv * sigmoidf_(gate[2 * i]), acc[2 * i + 1] * inv * sigmoidf_(gate[2 * i + 1]));
    uint2 *out = reinterpret_cast<uint2 *>(a.o + ((long long)m * a.QL + h) * QT_D + lane * 8);
    out[0] = make_uint2(o[0], o[1]);
    out[1] = make_uint2(o[2], o[3]);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(QT_THREADS, 1) qsa_attend_tc_kernel(const __grid_constant__ CUtensorMap mapK,
                                                                                               const __grid_constant__ CUtensorMap mapV,
                                                                                               const __grid_constant__ CUtensorMap hostK,
                                                                                               const __grid_constant__ CUtensorMap hostV, const __grid_constant__ QsaTcArgs a) {
    extern __shared__ unsigned char raw[];
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    unsigned char *sq = smem, *st = smem + QT_Q;
    uint64_t *full = reinterpret_cast<uint64_t *>(st + QT_ST * QT_STAGE), *empty = full + QT_ST;
    uint64_t *s_full = empty + QT_ST, *p_full = s_full + 2, *o_done = p_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(o_done + 1);
    float *s_max = reinterpret_cast<float *>(st + QT_ST * QT_STAGE + 128);       // [2 halves][128]
    const int per_kv = a.QL / a.KVL, rows = a.M * per_kv;
    // the last rows see the most keys: their units come first
    const int unit = (int)(gridDim.x >> 1) - 1 - (int)(blockIdx.x >> 1);
    const int kvh = unit % a.KVL, R0 = unit / a.KVL * 256;
    const int slot = a.slot[0], pos0 = a.pos[0];
    const int last = pos0 + (min(R0 + 256, rows) - 1) / per_kv, tiles = (last >> 7) + 1;
    if (threadIdx.x == 0) {
        for (int s = 0; s < QT_ST; ++s) { mbar_init(full + s, 2); mbar_init(empty + s, 1); }      // full: the leader's, both producers
        for (int b = 0; b < 2; ++b) { mbar_init(s_full + b, 1); mbar_init(p_full + b, 16); }      // p_full: the leader's, eight warps of each CTA
        mbar_init(o_done, 1);
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    // this CTA's 128 query rows as bf16, four 128B-swizzled panels of 64 columns
    for (int r0 = warp; r0 < 128; r0 += 4 * (QT_THREADS / 32)) {
        float4 x[4], y[4];                   // a lane's eight columns of four rows, all on their way at once
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = r0 + k * (QT_THREADS / 32), R = R0 + (int)rank * 128 + r;
            x[k] = y[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < 128 && R < rows) {
                const int m = R / per_kv;
                const float4 *p = reinterpret_cast<const float4 *>(a.q + ((long long)m * a.QL + kvh * per_kv + R - m * per_kv) * QT_D + lane * 8);
                x[k] = p[0];
                y[k] = p[1];
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = r0 + k * (QT_THREADS / 32);
            if (r < 128)
                *reinterpret_cast<uint4 *>(sq + (lane >> 3) * 16384 + r * 128 + (((lane & 7) ^ (r & 7)) << 4)) =
                    make_uint4(pack_bf16(x[k].x, x[k].y), pack_bf16(x[k].z, x[k].w), pack_bf16(y[k].x, y[k].y), pack_bf16(y[k].z, y[k].w));
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();                      // both CTAs' barriers and queries are there
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    if (warp == 0) {
        const int *pages = a.page_table + (long long)slot * a.max_pages;
        const int kcol = kvh * QT_D, vcol = kcol + (int)rank * 128;
        bool ok = true;
        // stages: K0, then K(j + 1), V(j)
        for (int i = 0; i < 2 * tiles && ok; ++i) {
            const bool is_v = i != 0 && ((i & 1) == 0 || i == 2 * tiles - 1);
            const int j = i == 0 ? 0 : is_v ? (i == 2 * tiles - 1 ? tiles - 1 : i / 2 - 1) : (i + 1) / 2;
            const int s = i % QT_ST;
            if (i >= QT_ST && !mg_wait_warp(empty + s, (unsigned)(i / QT_ST - 1) & 1u, a.err)) { ok = false; break; }
            const int page = pages[j >> 1], half = (j & 1) * 128;
            const uint32_t bar = map_to_cta(smem_u32(full + s), 0);
            unsigned char *d = st + s * QT_STAGE;
            const bool host = page >= a.n_dev_pages;
            if (host && !a.staged) {
                const int ld = a.KVL * QT_D, first = (page - a.n_dev_pages) * KV_PAGE + half;
                if (is_v) qt_copy(d, a.v_host + (long long)first * ld + vcol, ld, true, lane);
                else qt_copy(d, a.k_host + (long long)(first + (int)rank * 64) * ld + kcol, ld, false, lane);
                asm volatile("fence.proxy.async;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(bar);
                continue;
            }
            const int row = (host ? page - a.n_dev_pages : page) * KV_PAGE + half;
            const CUtensorMap *mk = host ? &hostK : &mapK, *mv = host ? &hostV : &mapV;
            if (elect_one()) {
                if (rank == 0) mbar_expect_tx(full + s, 2 * QT_STAGE);
                else mbar_arrive_cluster(bar);
                if (is_v) {
                    tma_load_2d_pair(d, mv, vcol, row, bar);
                    tma_load_2d_pair(d + 16384, mv, vcol + 64, row, bar);
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c) tma_load_2d_pair(d + c * 8192, mk, kcol + c * 64, row + (int)rank * 64, bar);
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // D fp32, A/B bf16, M = 256 (the pair's rows).  S: N = 128, both K-major; O: N = 256, B MN-major
            const uint32_t is = (1u << 4) | (1u << 7) | (1u << 10) | (16u << 17) | (16u << 24);
            const uint32_t io = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | (32u << 17) | (16u << 24);
            int i = 0;                       // next stage
            bool ok = true;
            auto stage_wait = [&]() {
                uint64_t *b = full + i % QT_ST;
                const unsigned p = (unsigned)(i / QT_ST) & 1u;
                return __all_sync(0xffffffffu, qt_try_cluster(b, p) || (mg_wait_slow(b, p, a.err) && qt_try_cluster(b, p))) != 0;
            };
            auto issue_s = [&](int j) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t q = smem_u32(sq), k = smem_u32(st + (i % QT_ST) * QT_STAGE), d = tmem + (uint32_t)(j & 1) * 128u;
                if (elect_one()) {
#pragma unroll
                    for (int c = 0; c < 16; ++c)
                        umma_bf16_pair(d, make_sw128_desc(q + (c >> 2) * 16384 + (c & 3) * 32), make_sw128_desc(k + (c >> 2) * 8192 + (c & 3) * 32), is, c ? 1u : 0u);
                    umma_commit_pair(empty + i % QT_ST);
                    umma_commit_pair(s_full + (j & 1));
                }
                ++i;
            };
            ok = stage_wait();
            if (ok) issue_s(0);
            for (int j = 0; j < tiles && ok; ++j) {
                if (j + 1 < tiles) {
                    if (!stage_wait()) { ok = false; break; }
                    issue_s(j + 1);
                }
                if (!mg_wait_warp(p_full + (j & 1), (unsigned)(j >> 1) & 1u, a.err) || !stage_wait()) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t v = smem_u32(st + (i % QT_ST) * QT_STAGE), p = tmem + (uint32_t)(j & 1) * 128u;
                const int steps = min(8, ((last - j * 128) >> 4) + 1);        // behind the last key there may be anything
                if (elect_one()) {
                    for (int c = 0; c < steps; ++c) umma_bf16_ts_pair(tmem + 256u, p + c * 8, make_mn_desc(v + c * 2048, 16384), io, (j | c) ? 1u : 0u);
                    umma_commit_pair(empty + i % QT_ST);
                    umma_commit_pair(o_done);
                }
                ++i;
            }
        }
    } else if (warp >= 4) {
        const int q = warp & 3, half = (warp - 4) >> 2, r = q * 32 + lane, R = R0 + (int)rank * 128 + r;
        const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16), obase = lane_base + 256u + half * 128u;
        const uint32_t p_bar = map_to_cta(smem_u32(p_full), 0);
        const int m = R < rows ? R / per_kv : 0, pos = R < rows ? pos0 + m : -1;
        const uint32_t *mask = a.mask + (long long)m * a.ld_mask;
        constexpr float scale = QT_SCALE;
        float ref = -1e30f, sum = 0.f;
        bool ok = true;                      // after a wait that ran out: no further waits, but every meeting
        uint32_t next = pos >= 0 ? __ldg(mask) : 0u;
        for (int j = 0; j < tiles; ++j) {
            const uint32_t word = next >> (half * 16);
            next = (j + 1) * 128 <= pos ? __ldg(mask + j + 1) : 0u;          // rows past the chunk's end, and tiles past a row: no key
            const int left = pos - j * 128 - half * 64;              // keys 0 .. left of this thread's 64 exist for the row
            ok = ok && mg_wait_warp(s_full + (j & 1), (unsigned)(j >> 1) & 1u, a.err);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t sbase = lane_base + (uint32_t)(j & 1) * 128u;
            uint32_t s[2][32];
            tmem_ld32_nowait(sbase + half * 64, s[0]);
            tmem_ld32_nowait(sbase + half * 64 + 32, s[1]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (__any_sync(0xffffffffu, left < 63)) {
#pragma unroll
                for (int c = 0; c < 64; ++c)
                    if (c > left) s[c >> 5][c & 31] = 0xff800000u;           // -inf
            }
            if (__any_sync(0xffffffffu, (word & 0xffffu) != 0xffffu)) {
#pragma unroll
                for (int g = 0; g < 16; ++g) {
                    const bool on = word >> g & 1u;
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (!on) s[g >> 3][(g & 7) * 4 + c] = 0xff800000u;
                }
            }
            float m4[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) m4[c] = fmaxf(__uint_as_float(s[0][c]), __uint_as_float(s[1][c]));
#pragma unroll
            for (int c = 4; c < 32; ++c) m4[c & 3] = fmaxf(m4[c & 3], fmaxf(__uint_as_float(s[0][c]), __uint_as_float(s[1][c])));
            asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");        // the two warps of these rows: both have read the last maxima
            s_max[half * 128 + r] = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
            asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");        // and now their scores
            const float nref = fmaxf(ref, fmaxf(s_max[r], s_max[128 + r]) * scale);
            const float f = j ? ex2(ref - nref) : 1.f;
            const bool risen = __any_sync(0xffffffffu, f != 1.f) != 0;
            ref = nref;
            sum *= f;
            float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t p[16];
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    const float x0 = ex2(fmaf(__uint_as_float(s[h][2 * c]), scale, -ref)), x1 = ex2(fmaf(__uint_as_float(s[h][2 * c + 1]), scale, -ref));
                    sum4[c & 3] += x0 + x1;
                    p[c] = pack_bf16(x0, x1);
                }
                tmem_st16(sbase + half * 32 + h * 16, p);
            }
            sum += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
            // waited for in every tile, risen or not: a barrier's parity only tells one phase from the next
            if (j) ok = ok && mg_wait_warp(o_done, (unsigned)(j - 1) & 1u, a.err);
            if (risen) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int c = 0; c < 128; c += 64) {
                    uint32_t o[4][16];
#pragma unroll
                    for (int k = 0; k < 4; ++k) tmem_ld16(obase + c + k * 16, o[k]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[k][i] = __float_as_uint(__uint_as_float(o[k][i]) * f);
                        tmem_st16(obase + c + k * 16, o[k]);
                    }
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(p_bar + (uint32_t)(j & 1) * 8u);
        }
        // ---- normalise, gate, store: 32 x 32 pieces through shared memory (the stages are free), so that rows leave as whole lines.  A lane's
        // rows are the same in every piece; the gates of a piece are fetched a piece ahead, the first ones under the last products
        int go[8], oo[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int RR = R0 + (int)rank * 128 + q * 32 + k * 4 + (lane >> 3), mm = RR / per_kv, h = kvh * per_kv + RR - mm * per_kv;
            go[k] = RR < rows ? mm * a.ld_proj + h * 2 * QT_D + QT_D + half * 128 + (lane & 7) * 4 : -1;
            oo[k] = (mm * a.QL + h) * QT_D + half * 128 + (lane & 7) * 4;
        }
        float4 gate[8];
        auto fetch_gates = [&](int c0) {
#pragma unroll
            for (int k = 0; k < 8; ++k) gate[k] = go[k] >= 0 ? *reinterpret_cast<const float4 *>(a.proj + go[k] + c0) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        fetch_gates(0);
        ok = ok && mg_wait_warp(o_done, (unsigned)(tiles - 1) & 1u, a.err);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
        s_max[half * 128 + r] = sum;
        asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
        const float total = s_max[r] + s_max[128 + r];
        float z[4] = {0.f, 0.f, 0.f, 0.f};   // NaN behind a value that is not finite
        if (ok) {
            const float inv = 1.f / total;
            float *stg = reinterpret_cast<float *>(st) + (warp - 4) * 32 * QT_STG_LD;
#pragma unroll 1
            for (int c0 = 0; c0 < 128; c0 += 32) {
                uint32_t v[32];
                tmem_ld32(obase + c0, v);
#pragma unroll
                for (int c = 0; c < 32; ++c) z[c & 3] = fmaf(__uint_as_float(v[c]), 0.f, z[c & 3]);
#pragma unroll
                for (int c = 0; c < 32; c += 4)
                    *reinterpret_cast<float4 *>(stg + lane * QT_STG_LD + c) =
                        make_float4(__uint_as_float(v[c]) * inv, __uint_as_float(v[c + 1]) * inv, __uint_as_float(v[c + 2]) * inv, __uint_as_float(v[c + 3]) * inv);
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (go[k] < 0) continue;
                    const float4 y = *reinterpret_cast<const float4 *>(stg + (k * 4 + (lane >> 3)) * QT_STG_LD + (lane & 7) * 4), g = gate[k];
                    *reinterpret_cast<uint2 *>(a.o + oo[k] + c0) =
                        make_uint2(pack_bf16(y.x * sigmoidf_(g.x), y.y * sigmoidf_(g.y)), pack_bf16(y.z * sigmoidf_(g.z), y.w * sigmoidf_(g.w)));
                }
                if (c0 + 32 < 128) fetch_gates(c0 + 32);
                __syncwarp();
            }
        }
        // A row whose own scores are finite has a finite sum.  The two warps share what they found and take every other row of it
        const float zs = (z[0] + z[1]) + (z[2] + z[3]);
        const unsigned mine = __ballot_sync(0xffffffffu, zs != zs && total > 0.f && total < INFINITY);
        asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
        if (lane == 0) s_max[half * 128 + q * 32] = __uint_as_float(mine);
        asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
        for (unsigned left = (__float_as_uint(s_max[q * 32]) | __float_as_uint(s_max[128 + q * 32])) & (half ? 0xaaaaaaaau : 0x55555555u); left; left &= left - 1) {
            const int RR = R0 + (int)rank * 128 + q * 32 + __ffs(left) - 1, mm = RR / per_kv;
            qt_row_alone(a, mm, kvh * per_kv + RR - mm * per_kv, lane);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();                      // nothing is in flight towards either CTA any more
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

}  // namespace qw

using namespace qw;

// What qwk_qsa_attend_tc can take: groups of four, a mask that fits its buffer, offsets in 32 bits.
static bool qsa_tc_fits(int QL, int KVL, int M, int last_pos, int ratio, int ld_mask, int ld_proj) {
    return KVL >= 1 && QL >= KVL && QL % KVL == 0 && M >= 1 && ratio == 4 && last_pos >= M - 1 && (last_pos >> 7) < ld_mask && (ld_proj & 3) == 0 &&
           (long long)M * ld_proj < (1LL << 31) - 65536 && (long long)M * QL * QT_D < (1LL << 31);
}

// 1: the attention of a chunk (M rows of one run, the last at position last_pos, topk groups chosen of `ratio` tokens) goes through
// qwk_qsa_attend_tc.  Both kernels run in waves of equal blocks.  Here a pair of CTAs has 256 rows of a KV head and takes 2.3 us per
// tile of 128 keys; the kernel that gathers has three blocks of a query and KV head on each SM and takes a wave 20 us and 112 more when
// the lists are full.  us, gathered / here: 1 row at position 1,000 69 / 46, at 9,000 129 / 186; 300 rows at 0 50 / 34, at 9,000 267 / 190,
// at 16,384 269 / 320; 1,021 at 16,384 683 / 641, at 24,000 688 / 922; 2,048 at 16,384 1340 / 978, at 24,000 1344 / 1385; 100 at 0 27 / 31.
// Where the keys lie makes no difference to the line: over host pages that are not staged the dense tiles cost 4 to 35 times less still (each row
// crosses the host link once per pair of CTAs, not once per query), ms: 300 rows at 0 7.4 / 0.44, at 4,000 49 / 2.6; 1,021 at 0 51 / 3.3, at 9,000
// 184 / 18; 4,096 at 0 571 / 16.  (Only where the cache of host rows holds all that a small chunk chose would the gather be the faster one.)
QW_API int qwk_qsa_takes_tc(int QL, int KVL, int M, int last_pos, int topk, int ratio, int ld_mask, int ld_proj) {
    if (!qsa_tc_fits(QL, KVL, M, last_pos, ratio, ld_mask, ld_proj)) return 0;
    const long long pairs = NUM_SMS / 2, blocks = 3 * NUM_SMS, units = ((long long)M * (QL / KVL) + 255) / 256 * KVL;
    const long long here = (units + pairs - 1) / pairs, gathered = ((long long)M * KVL + blocks - 1) / blocks;
    const double full = (double)ratio * topk + ratio - 1, len = last_pos + 1 - 0.5 * (M - 1);          // a row's list: all before it, until it is full
    return 27 + 2.3 * ((last_pos >> 7) + 1) * here < gathered * (20 + 112 * (len < full ? len : full) / 2051);
}

// Attention of the rows of one run (slot[0], positions pos[0] + m, the last of them last_pos); what sel / sel_n name is what a row attends
// to (see qsa_select_kernel; groups of four).  Pages from n_dev_pages on lie at k_host / v_host (null: there are none), in device memory if
// `staged`.  mask: [M][ld_mask] words of scratch, one bit per group.  The pool's rows behind last_pos, up to the next multiple of 16, have to
// be finite (qwk_qsa_prep_run zeroes them): the products read V in steps of 16 keys, and they meet weights of zero there.  Where q or proj do not lie on
// 16 bytes, or o not on 8, the rows are gathered instead: that kernel's loads and stores are narrower.
QW_API int qwk_qsa_attend_tc(const float *q, int QL, int KVL, int M, int last_pos, const int *slot, const int *pos, void *k_dev, void *v_dev,
                             void *k_host, void *v_host, int staged, int n_dev_pages, const int *page_table, int max_pages, const int *sel,
                             const int *sel_n, int topk, void *mask, int ld_mask, const float *proj, int ld_proj, void *o, cudaStream_t s) {
    if (!qsa_tc_fits(QL, KVL, M, last_pos, 4, ld_mask, ld_proj) || !aligned16(k_dev, v_dev, k_host, v_host)) return -1;
    if (!aligned16(q, proj) || ((uintptr_t)o & 7))
        return (staged ? qwk_qsa_attend_mma_staged : qwk_qsa_attend_mma)(q, QL, KVL, M, slot, pos, k_dev, v_dev, k_host, v_host, n_dev_pages, page_table, max_pages, sel, sel_n, topk, 4, proj, ld_proj, o, s);
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!done[dev]) {
        if (cudaFuncSetAttribute(qsa_attend_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, QT_SMEM) != cudaSuccess) return -3;
        done[dev] = true;
    }
    const int row = KVL * QT_D;
    auto maps = [row](CUtensorMap *k, CUtensorMap *v, const void *kp, const void *vp, long long rows) {
        return make_map(k, kp, rows, row, row, 64) && make_map(v, vp, rows, row, row, 128);
    };
    // a pool that has no pages has no map: no page id leads to it
    CUtensorMap mK{}, mV{}, hK{}, hV{};
    if (n_dev_pages > 0 && !maps(&mK, &mV, k_dev, v_dev, (long long)n_dev_pages * KV_PAGE)) return -3;
    staged = staged && k_host;
    if (staged && !maps(&hK, &hV, k_host, v_host, 1LL << 30)) return -3;
    qsa_mask_kernel<<<M, 128, ((size_t)(last_pos >> 7) + 1) * 4, s>>>(pos, sel, sel_n, topk, (uint32_t *)mask, ld_mask);
    QsaTcArgs a{};
    a.q = q; a.QL = QL; a.KVL = KVL; a.M = M; a.slot = slot; a.pos = pos; a.page_table = page_table; a.max_pages = max_pages;
    a.k_dev = (const bf16 *)k_dev; a.v_dev = (const bf16 *)v_dev;
    a.n_dev_pages = k_host ? n_dev_pages : 0x7fffffff; a.staged = staged; a.k_host = (const bf16 *)k_host; a.v_host = (const bf16 *)v_host;
    a.mask = (const uint32_t *)mask; a.ld_mask = ld_mask; a.proj = proj; a.ld_proj = ld_proj; a.o = (bf16 *)o; a.err = g_err_ptr;
    const long long rows = (long long)M * (QL / KVL);
    const unsigned units = (unsigned)((rows + 255) / 256) * KVL;
    qsa_attend_tc_kernel<<<2 * units, QT_THREADS, QT_SMEM, s>>>(mK, mV, hK, hV, a);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
