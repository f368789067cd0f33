// Attention of the vision tower on the 5th-generation tensor cores: non-causal, one image or video slice, head dim 72.
// (Role of the reference's src/kernels/vision.hip attention.)
//
// A CTA takes 256 queries of one head as two tiles of 128 and walks the keys in tiles of 128.  Per tile S = Q K^T (128 x 128, fp32)
// and O += P V accumulate in tensor memory; a thread of the tile's warp group owns one query row: it reads its 128 scores, keeps
// the running reference maximum and sum in registers, and writes the probabilities back over the scores as bf16, where the second
// product reads them as its A operand.  While one tile's scores are turned into probabilities the tensor core works for the other.
//   warp 0       TMA: Q once per unit, K and V tiles of 128 rows, three stages each
//   warp 1       MMAs: S0, S1, then per key tile PV0, next S0, PV1, next S1
//   warps 4-11   softmax, one warp group per query tile
// The reference is the row's running maximum, so that its largest weight is exactly 1: left up to 8 (in log2 units) below it, O needs rescaling
// rarely and the kernel takes 111 us at 3520 patches, but the largest weights are rounded to bf16 as well, and the error against 64 bits
// is up to 25 % above that of the kernel this one replaces (scores of size 3; 3 % at size 1).  With the maximum it is the same.  O is rescaled
// behind the probabilities, all 80 columns in flight at once (in front of them, 16 at a time, 128 us).
// Head dim 72 = 64 + 8: a row's first 64 values are a 128B-swizzled panel, the last 8 a panel of 16-byte rows whose partner (the
// other 8 of an MMA's k = 16) is a zeroed block.  V is read as it lies (key-major): 64 + 64 columns, of which the second panel's
// first 8 count; the rest belongs to other heads and lands in columns of O that nobody reads.
// The units' key tiles are dealt to the CTAs in equal runs (VitSplit) where whole units would leave SMs idle: 3520 patches and 16 heads are 224
// units, one and a half for each of 148 SMs.  A run that does not hold all of a unit's keys leaves its O, reference and sum, and a second kernel
// merges them: 129 us whole, 108 + 12 dealt.
// What bounds it: the exponentials (128 x 128 per tile at 16 a cycle and SM: 1024 cycles; MMAs 780).  It replaces a flash kernel on mma.sync (16 queries a warp, each warp reading every K and V fragment
// from shared memory), which took 444 us there.
#include "tc.cuh"

namespace qw {

constexpr int VT_D = 72, VT_STAGES = 3, VT_THREADS = 384;
constexpr int VT_KA = 128 * 128, VT_KB = 128 * 16, VT_K = VT_KA + 2 * VT_KB;      // K (and Q) tile: wide panel, narrow panel, its zeros
constexpr int VT_V = 2 * 128 * 128;
constexpr int VT_SMEM = 2 * VT_K + VT_STAGES * (VT_K + VT_V) + 1024 + 512;

constexpr int VT_PART = 76;                      // floats of a row of a part: 72 of O, reference, sum

// The key tiles of all units one after another, dealt to `ctas` CTAs in equal runs; a run's piece of one unit is a segment.
struct VitSplit {
    int ktiles, units, ctas, whole;              // whole: runs begin and end with a unit
    __host__ __device__ long long first(int c) const {
        return whole ? (long long)units * c / ctas * ktiles : (long long)units * ktiles * c / ctas;
    }
};
struct VitSeg {
    int unit, k0, len;
    __device__ __forceinline__ VitSeg(const VitSplit &s, long long at, long long end) {
        unit = (int)(at / s.ktiles);
        k0 = (int)(at - (long long)unit * s.ktiles);
        len = (int)min((long long)(s.ktiles - k0), end - at);
    }
};

struct VitAttnArgs {
    int L, heads, qtiles;
    VitSplit split;
    float *parts;            // [CTA][first segment | last][256][VT_PART]
    bf16 *out;
    float scale;             // log2(e) / sqrt(72)
    ErrorWord *err;
};

// No-swizzle K-major operand: rows of 16 bytes, 8-row groups 128 bytes apart, the second k half `lbo` bytes further.
__device__ __forceinline__ uint64_t make_plain_desc(uint32_t saddr, uint32_t lbo) {
    return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) | ((uint64_t)1 << 46);
}
__global__ void __launch_bounds__(VT_THREADS, 1) vit_attn_tc_kernel(const __grid_constant__ CUtensorMap mapA,      // 64-column boxes of qkv
                                                                    const __grid_constant__ CUtensorMap mapB,      // 8-column boxes
                                                                    VitAttnArgs a) {
    extern __shared__ unsigned char raw[];
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    // V stages first, then the wide panels, then the narrow ones: every swizzled panel starts on a multiple of 1024 bytes
    unsigned char *sv = smem, *sq = sv + VT_STAGES * VT_V, *sk = sq + 2 * VT_K;
    uint64_t *q_full = reinterpret_cast<uint64_t *>(sk + VT_STAGES * VT_K), *q_empty = q_full + 1;
    uint64_t *k_full = q_empty + 1, *k_empty = k_full + VT_STAGES, *v_full = k_empty + VT_STAGES, *v_empty = v_full + VT_STAGES;
    uint64_t *s_full = v_empty + VT_STAGES, *p_full = s_full + 2, *o_full = p_full + 2, *o_empty = o_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(o_empty + 2);
    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        mbar_init(q_empty, 1);
        for (int s = 0; s < VT_STAGES; ++s) { mbar_init(k_full + s, 1); mbar_init(k_empty + s, 1); mbar_init(v_full + s, 1); mbar_init(v_empty + s, 1); }
        for (int t = 0; t < 2; ++t) { mbar_init(s_full + t, 1); mbar_init(p_full + t, 4); mbar_init(o_full + t, 1); mbar_init(o_empty + t, 4); }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // the zero partners of the narrow panels (never written again)
    for (int i = threadIdx.x; i < (2 + VT_STAGES) * (VT_KB / 16); i += VT_THREADS) {
        const int tile = i / (VT_KB / 16), at = i % (VT_KB / 16);
        *reinterpret_cast<uint4 *>(sq + tile * VT_K + VT_KA + VT_KB + at * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const int ktiles = a.split.ktiles, D = a.heads * VT_D;
    const long long from = a.split.first(blockIdx.x), to = a.split.first(blockIdx.x + 1);
    if (warp == 0) {
        unsigned it = 0, u = 0;
        bool ok = true;
        for (long long at = from; at < to && ok; ++u) {
            const VitSeg g(a.split, at, to);
            at += g.len;
            const int h = g.unit / a.qtiles, q0 = (g.unit % a.qtiles) * 256, col = h * VT_D;
            if (u && !mg_wait_warp(q_empty, (u - 1) & 1u, a.err)) break;
            if (elect_one()) {
                mbar_expect_tx(q_full, 2 * (VT_KA + VT_KB));
                for (int t = 0; t < 2; ++t) {
                    tma_load_2d(sq + t * VT_K, &mapA, col, q0 + t * 128, q_full);
                    tma_load_2d(sq + t * VT_K + VT_KA, &mapB, col + 64, q0 + t * 128, q_full);
                }
            }
            for (int j = g.k0; j < g.k0 + g.len; ++j, ++it) {
                const unsigned s = it % VT_STAGES, ph = (it / VT_STAGES - 1) & 1u;
                if (it >= VT_STAGES && !mg_wait_warp(k_empty + s, ph, a.err)) { ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(k_full + s, VT_KA + VT_KB);
                    tma_load_2d(sk + s * VT_K, &mapA, D + col, j * 128, k_full + s);
                    tma_load_2d(sk + s * VT_K + VT_KA, &mapB, D + col + 64, j * 128, k_full + s);
                }
                if (it >= VT_STAGES && !mg_wait_warp(v_empty + s, ph, a.err)) { ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(v_full + s, VT_V);
                    tma_load_2d(sv + s * VT_V, &mapA, 2 * D + col, j * 128, v_full + s);
                    tma_load_2d(sv + s * VT_V + VT_V / 2, &mapA, 2 * D + col + 64, j * 128, v_full + s);
                }
            }
        }
    } else if (warp == 1) {
        // instruction descriptors: D fp32, A/B bf16, M = 128; S: N = 128, both K-major; O: N = 80, B MN-major
        const uint32_t is = (1u << 4) | (1u << 7) | (1u << 10) | (16u << 17) | (8u << 24);
        const uint32_t io = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | (10u << 17) | (8u << 24);
        unsigned it = 0, u = 0;
        bool ok = true;
        auto issue_s = [&](int t, unsigned st) {
            const uint32_t q = smem_u32(sq + t * VT_K), k = smem_u32(sk + st * VT_K);
            if (elect_one()) {
#pragma unroll
                for (int i = 0; i < 4; ++i) umma_bf16(tmem + t * 128u, make_sw128_desc(q + i * 32), make_sw128_desc(k + i * 32), is, i ? 1u : 0u);
                umma_bf16(tmem + t * 128u, make_plain_desc(q + VT_KA, VT_KB), make_plain_desc(k + VT_KA, VT_KB), is, 1u);
                umma_commit(s_full + t);
                if (t) umma_commit(k_empty + st);
            }
        };
        for (long long at = from; at < to && ok; ++u) {
            const int len = VitSeg(a.split, at, to).len;
            at += len;
            if (!mg_wait_warp(q_full, u & 1u, a.err) || !mg_wait_warp(k_full + it % VT_STAGES, (it / VT_STAGES) & 1u, a.err)) break;
            // the scores of a new unit overwrite probabilities that the last products of the old one read: same pipe, in order
            issue_s(0, it % VT_STAGES);
            issue_s(1, it % VT_STAGES);
            if (len == 1 && elect_one()) umma_commit(q_empty);
            for (int j = 0; j < len && ok; ++j, ++it) {
                const unsigned s = it % VT_STAGES, sn = (it + 1) % VT_STAGES;
                const bool more = j + 1 < len;
                if (more && !mg_wait_warp(k_full + sn, ((it + 1) / VT_STAGES) & 1u, a.err)) { ok = false; break; }
                if (!mg_wait_warp(v_full + s, (it / VT_STAGES) & 1u, a.err)) { ok = false; break; }
                for (int t = 0; t < 2; ++t) {
                    if (j == 0 && u && !mg_wait_warp(o_empty + t, (u - 1) & 1u, a.err)) { ok = false; break; }
                    if (!mg_wait_warp(p_full + t, it & 1u, a.err)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t v = smem_u32(sv + s * VT_V);
                    if (elect_one()) {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            umma_bf16_ts(tmem + 256u + t * 80u, tmem + t * 128u + i * 8, make_mn_desc(v + i * 2048, VT_V / 2), io, (j | i) ? 1u : 0u);
                        if (t) umma_commit(v_empty + s);
                        if (!more) umma_commit(o_full + t);
                    }
                    if (more) issue_s(t, sn);
                }
                if (ok && j + 2 == len && elect_one()) umma_commit(q_empty);      // the last scores of this unit are under way
            }
        }
    } else if (warp >= 4) {
        const int t = (warp - 4) >> 2, q = warp & 3;
        const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
        const uint32_t sbase = lane_base + t * 128u, obase = lane_base + 256u + t * 80u;
        unsigned it = 0, u = 0;
        bool ok = true;
        for (long long at = from; at < to && ok; ++u) {
            const VitSeg g(a.split, at, to);
            const bool begins = at == from;
            at += g.len;
            const int h = g.unit / a.qtiles, r256 = t * 128 + q * 32 + lane, row = (g.unit % a.qtiles) * 256 + r256;
            float ref = 0.f, sum = 0.f;
            for (int j = 0; j < g.len; ++j, ++it) {
                if (!mg_wait_warp(s_full + t, it & 1u, a.err)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t s[4][32];
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_ld32_nowait(sbase + c * 32, s[c]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (g.k0 + j + 1 == ktiles) {
                    const int left = a.L - (g.k0 + j) * 128;
#pragma unroll
                    for (int c = 0; c < 128; ++c)
                        if (c >= left) s[c >> 5][c & 31] = 0xff800000u;      // -inf
                }
                float m4[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) m4[c] = __uint_as_float(s[c][0]);
#pragma unroll
                for (int i = 1; i < 32; ++i)
#pragma unroll
                    for (int c = 0; c < 4; ++c) m4[c] = fmaxf(m4[c], __uint_as_float(s[c][i]));
                const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * a.scale;
                // a row whose first scores are all -inf keeps a finite reference
                const float nref = j ? fmaxf(ref, mx) : fmaxf(mx, -1e30f), f = j ? exp2f(ref - nref) : 1.f;
                const bool risen = __any_sync(0xffffffffu, f != 1.f) != 0;
                ref = nref;
                sum *= f;
                float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t p[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float x0 = exp2f(fmaf(__uint_as_float(s[c][2 * i]), a.scale, -ref)), x1 = exp2f(fmaf(__uint_as_float(s[c][2 * i + 1]), a.scale, -ref));
                        sum4[i & 3] += x0 + x1;
                        p[i] = pack_bf16(x0, x1);
                    }
                    tmem_st16(sbase + c * 16, p);
                }
                sum += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
                if (risen) {
                    // every product issued before these scores is complete, this tile's last O among them.  Behind the probabilities the
                    // scores' registers are free: the whole row of O is on its way at once
                    uint32_t o[5][16];
#pragma unroll
                    for (int c = 0; c < 5; ++c) tmem_ld16(obase + c * 16, o[c]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int c = 0; c < 5; ++c) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[c][i] = __float_as_uint(__uint_as_float(o[c][i]) * f);
                        tmem_st16(obase + c * 16, o[c]);
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full + t);
            }
            if (!ok || !mg_wait_warp(o_full + t, u & 1u, a.err)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (g.len < ktiles) {                        // a part: as it is, with what the merge needs
                float *o = a.parts + ((long long)(blockIdx.x * 2 + (begins ? 0 : 1)) * 256 + r256) * VT_PART;
#pragma unroll
                for (int c = 0; c < 80; c += 16) {
                    uint32_t v[16];
                    tmem_ld16(obase + c, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 16; i += 4)
                        if (c + i < VT_D) *reinterpret_cast<uint4 *>(o + c + i) = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                }
                *reinterpret_cast<float4 *>(o + VT_D) = make_float4(ref, sum, 0.f, 0.f);
            } else {
                const float r = 1.f / sum;
                bf16 *o = a.out + (long long)row * D + h * VT_D;
    #pragma unroll
                for (int c = 0; c < 80; c += 16) {
                    uint32_t v[16];
                    tmem_ld16(obase + c, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    #pragma unroll
                    for (int i = 0; i < 16; i += 8) {
                        if (c + i >= VT_D || row >= a.L) continue;
                        uint4 pk;
                        pk.x = pack_bf16(__uint_as_float(v[i]) * r, __uint_as_float(v[i + 1]) * r);
                        pk.y = pack_bf16(__uint_as_float(v[i + 2]) * r, __uint_as_float(v[i + 3]) * r);
                        pk.z = pack_bf16(__uint_as_float(v[i + 4]) * r, __uint_as_float(v[i + 5]) * r);
                        pk.w = pack_bf16(__uint_as_float(v[i + 6]) * r, __uint_as_float(v[i + 7]) * r);
                        *reinterpret_cast<uint4 *>(o + c + i) = pk;
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(o_empty + t);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// Units whose keys lie in several CTAs' runs: O = sum of the parts' O, each relative to the largest reference, over the sum of their sums.
// grid (18, units), 256 threads: a thread per row and four columns.
__global__ void __launch_bounds__(256) vit_merge_kernel(VitAttnArgs a) {
    const int unit = blockIdx.y, i = blockIdx.x * 256 + threadIdx.x, r = i / (VT_D / 4), c = (i - r * (VT_D / 4)) * 4;
    // 32-bit arithmetic: the launcher checks that units x key tiles x CTAs fit
    const int kt = a.split.ktiles, G = a.split.ctas, total = a.split.units * kt, lo = unit * kt, hi = lo + kt;
    auto first = [&](int c) { return (int)((unsigned)total * (unsigned)c / (unsigned)G); };
    int c0 = (int)((unsigned)lo * (unsigned)G / (unsigned)total);                 // the run that holds the unit's first key tile
    while (first(c0 + 1) <= lo) ++c0;
    while (first(c0) > lo) --c0;
    int f0 = first(c0), f1 = first(c0 + 1);
    if (f1 >= hi) return;                                // one run holds them all: done
    const int h = unit / a.qtiles, row = (unit % a.qtiles) * 256 + r;
    if (row >= a.L) return;
    float m = -1e30f, sum = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = c0; f0 < hi; ++k, f0 = f1, f1 = first(k + 1)) {
        const float *p = a.parts + ((long long)(k * 2 + (f0 >= lo ? 0 : 1)) * 256 + r) * VT_PART;
        const float2 rs = *reinterpret_cast<const float2 *>(p + VT_D);
        const float4 v = *reinterpret_cast<const float4 *>(p + c);
        const float nm = fmaxf(m, rs.x), f = exp2f(m - nm), w = exp2f(rs.x - nm);
        m = nm;
        sum = sum * f + rs.y * w;
        o.x = o.x * f + v.x * w; o.y = o.y * f + v.y * w; o.z = o.z * f + v.z * w; o.w = o.w * f + v.w * w;
    }
    const float inv = 1.f / sum;
    *reinterpret_cast<uint2 *>(a.out + (long long)row * a.heads * VT_D + h * VT_D + c) =
        make_uint2(pack_bf16(o.x * inv, o.y * inv), pack_bf16(o.z * inv, o.w * inv));
}

}  // namespace qw

using namespace qw;

// How the key tiles are dealt: whole units where their waves fill the SMs to nine tenths, else equal runs of at least two tiles.  (The
// merge costs a tenth of 224 units: what two waves that are three quarters full lose is twice that.)
static VitSplit vit_split(int L, int heads, bool parts) {
    VitSplit s;
    s.ktiles = (L + 127) / 128;
    s.units = (L + 255) / 256 * heads;
    const int sms = (int)persistent_grid(1 << 30, 1), waves = (s.units + sms - 1) / sms;
    const long long runs = (long long)s.units * s.ktiles / 2;
    s.whole = !parts || (long long)s.units * s.ktiles * sms >= (1LL << 32) || 10LL * s.units >= 9LL * waves * sms || runs <= s.units;
    s.ctas = s.whole ? (s.units < sms ? s.units : sms) : (int)(runs < sms ? runs : sms);
    return s;
}

// Bytes of scratch that let qwk_vit_attention deal a slice's keys evenly (0: it deals whole units anyway).
QW_API int qwk_vit_attention_scratch(int L, int heads) {
    if (L <= 0 || heads <= 0) return 0;
    const VitSplit s = vit_split(L, heads, true);
    return s.whole ? 0 : s.ctas * 2 * 256 * VT_PART * 4;
}

// qkv [L][3 * heads * 72] bf16 (bias and rotary applied) -> out [L][heads * 72] bf16.  qkv, out and parts 16-byte aligned; parts: scratch of
// qwk_vit_attention_scratch bytes, or null.
QW_API int qwk_vit_attention_split(const void *qkv, int L, int heads, void *out, void *parts, cudaStream_t s) {
    if (L <= 0) return 0;
    if (((uintptr_t)qkv & 15) || ((uintptr_t)out & 15) || ((uintptr_t)parts & 15) || heads <= 0) return -1;
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!done[dev]) {
        if (cudaFuncSetAttribute(vit_attn_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, VT_SMEM) != cudaSuccess) return -3;
        done[dev] = true;
    }
    const long long ld = 3LL * heads * VT_D;
    CUtensorMap mA, mB;
    if (!make_map(&mA, qkv, L, ld, ld, 128) || !make_map(&mB, qkv, L, ld, ld, 128, MAP_BF16_X8)) return -3;
    VitAttnArgs a{};
    a.L = L; a.heads = heads; a.qtiles = (L + 255) / 256; a.out = (bf16 *)out; a.err = g_err_ptr;
    a.split = vit_split(L, heads, parts != nullptr);
    a.parts = (float *)parts;
    a.scale = 1.4426950408889634f / sqrtf((float)VT_D);
    vit_attn_tc_kernel<<<a.split.ctas, VT_THREADS, VT_SMEM, s>>>(mA, mB, a);
    if (!a.split.whole) vit_merge_kernel<<<dim3(VT_D / 4, a.split.units), 256, 0, s>>>(a);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Without scratch.
QW_API int qwk_vit_attention(const void *qkv, int L, int heads, void *out, cudaStream_t s) { return qwk_vit_attention_split(qkv, L, heads, out, nullptr, s); }
