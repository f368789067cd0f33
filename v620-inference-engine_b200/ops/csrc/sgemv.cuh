// Streaming skinny matrix product core: D[n][m] = sum_k W[n][k] x[m][k] for bf16 weights and up to
// 24 activation rows per pass (tiles of eight), with caller-supplied functors that build the activation rows in
// shared memory and consume each finished 16-row tile.
//
// One persistent block per SM: two groups of eight consumer warps and a producer warp.  The producer copies weight
// rows global -> shared memory with TMA (one box of 16 rows x 512-768 columns a stage, 64 columns at a time in 128B-swizzled rows, up
// to eight stages in flight), runs ahead of the consumers through full/empty mbarriers, and never waits for
// the predecessor kernel because weights do not depend on it (programmatic dependent launch lets it
// start during the predecessor's tail).  The consumer warps of a group split a stage's k range and feed the
// tensor core (ldmatrix + m16n8k16, fp32 accumulate) with the activation rows as the narrow operand,
// so eight activation rows cost the same instructions as one; the warps' partial sums are added in warp
// order, so a row's result does not depend on how many other rows share the step.
//
// What bounds it: the weights, and beside them the work per stage that does not shrink with the rows.  Boxes of 16 rows (single rows as bulk
// copies cost 85 cycles each), two groups that take every other tile (one converts its sums while the other multiplies) and up to
// 24 rows in one pass (x in parts of K where it has no room).  us, one group and 16 rows a pass / now: 248,320 x 2,560 at 1 row 215 / 187, at 8
// 216 / 195, at 16 226 / 217, at 24 422 / 268, at 32 (two passes) 447 / 430; 16,480 x 2,560 at 1 15.9 / 14.3, at 16 19.2 / 19.4, at 24 33 / 24;
// 2,560 x 6,144 at 1 10.7 / 9.8, at 16 28 / 17, at 24 41 / 18.7, at 32 54 / 30.
// Used by: the bf16 GEMV (projections, lm_head, PLE) and the MoE router (+ routing epilogue).
#pragma once
#include "fuse.cuh"
#include "mma.cuh"
#include "tc.cuh"

namespace qw {

struct SGemvArgs {
    const bf16 *W;      // [N][ldw] (+ split * w_split)
    const bf16 *x;      // [M][ldx]           (default activation fill)
    float *y;           // [M][ldy]           (default store)
    bf16 *y_bf16;       // optional bf16 copy of y
    int N, K, M;
    int ldw, ldx, ldy;
    int accumulate;
    int P, Kc;          // k parts per row tile and their size (a multiple of 128; the last may be shorter)
    int KH;             // the activation rows are in shared memory one KH-th of the parts at a time
    int box3;           // 1: the map's boxes are whole stages (K a multiple of 64); 0: they are 64 columns
    int nstage, groups; // stages; groups of warps that take tiles in turn (each has its share of the stages)
    ErrorWord *err;
    FuseIn fi = {};     // fused all-gather: the activation rows are built from the ranks' words
    FuseOut fo = {};    // fused reduce-scatter: y goes to the ranks that own its columns instead of memory
};

constexpr int SG_FIXED = 1024 + 128;     // alignment, mbarriers: full[8], empty[8]
constexpr int SG_GROUPS = 2, SG_CONSUMERS = SG_GROUPS * 256;
constexpr int SG_THREADS = SG_CONSUMERS + 32;      // + the producer warp
constexpr int SG_TILE = 16;              // weight rows per tile
constexpr int SG_PN = 20;                // floats between the activation rows of a partial tile (16 used): its stores hit 32 banks
constexpr int SG_STEPS = 6;              // k steps of a warp in a stage of 768 columns
constexpr int SG_STAGES = 6, SG_MIN_STAGES = 4;      // three for each group, or at least two
constexpr size_t SG_SMEM_MAX = 226 * 1024;

struct SGemvSmem {
    unsigned char *stages;      // [stage][64 columns][16 rows][128 bytes]
    float *part;        // [group][8 warps][8 NT rows][SG_PN] partial tiles
    unsigned char *xs;  // [(rows)+1][xrow] activation rows + one zero row
    unsigned xrow;      // bytes between activation rows
};

// Default activation fill: columns k0 .. k0 + n - 1 of rows m0.. of a.x as they are (bf16), plus the zero row.
struct XFillCopy {
    const SGemvArgs &a;
    __device__ __forceinline__ void operator()(int m0, int nm, int k0, int n, const SGemvSmem &sm, int tid) const {
        const int nchunk = n >> 3, total = (nm + 1) * nchunk;
        // four loads per thread in flight: the fill is on the kernel's critical path (one L2 round trip per batch)
        for (int i0 = tid; i0 < total; i0 += 4 * SG_CONSUMERS) {
            uint4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * SG_CONSUMERS;
                const int m = i / nchunk, c = i - m * nchunk;
                v[u] = make_uint4(0u, 0u, 0u, 0u);
                if (i < total && m < nm) v[u] = __ldcg(reinterpret_cast<const uint4 *>(a.x + (long long)(m0 + m) * a.ldx + k0) + c);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * SG_CONSUMERS;
                const int m = i / nchunk, c = i - m * nchunk;
                if (i < total) *reinterpret_cast<uint4 *>(sm.xs + (size_t)m * sm.xrow + (size_t)c * 16) = v[u];
            }
        }
    }
};

// Activation fill from a fused all-gather (KH = 1): column r * n + w of row m is word w of row m in rank r's slot (one bf16
// per word).  Block 0 also leaves the dense rows in a.x for later kernels that read them from memory.
struct XFillGather {
    const SGemvArgs &a;
    __device__ __forceinline__ void operator()(int m0, int nm, int, int, const SGemvSmem &sm, int tid) const {
        const unsigned int seq = fuse_seq(a.fi);
        const int n = a.fi.n;                              // columns per rank (a multiple of 8)
        const int nchunk = a.K >> 3;
        for (int i = tid; i < nm * nchunk; i += SG_CONSUMERS) {
            const int m = i / nchunk, c = (i - m * nchunk) * 8;
            const int r = c / n, w = c - r * n;
            const uint4 v = fuse_get8_u16(a.fi, seq, r, (long long)(m0 + m) * n + w);
            *reinterpret_cast<uint4 *>(sm.xs + (size_t)m * sm.xrow + (size_t)c * 2) = v;
            if (blockIdx.x == 0) *reinterpret_cast<uint4 *>(const_cast<bf16 *>(a.x) + (long long)(m0 + m) * a.ldx + c) = v;
        }
        for (int c = tid; c < (a.K >> 3); c += SG_CONSUMERS)
            *reinterpret_cast<uint4 *>(sm.xs + (size_t)nm * sm.xrow + (size_t)c * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
};

// Default epilogue: y[m][row] (+)= v.
template <bool FUSED = false>
struct EpiStore {
    const SGemvArgs &a;
    __device__ __forceinline__ void operator()(int m, int row, float v) const {
        if (FUSED && a.fo.mode) {          // fused reduce-scatter: straight to the owner of the column
            fuse_put_col(a.fo, fuse_seq(a.fo), m, row, __float_as_uint(v));
            return;
        }
        const long long o = (long long)m * a.ldy + row;
        if (a.accumulate) v += a.y[o];
        a.y[o] = v;
        if (a.y_bf16) a.y_bf16[o] = __float2bfloat16(v);
    }
};

__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 256;" ::"r"(2 + group) : "memory"); }

// NT = activation-row tiles of 8 handled per pass (1, 2 or 3).
template <int NT, class XFill, class Epi>
__device__ __forceinline__ void sgemv_core(const CUtensorMap &map, const SGemvArgs &a, unsigned char *raw, const XFill &xfill, const Epi &epi) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int Px = a.P / a.KH, Kx = Px * a.Kc;
    const unsigned stage_bytes = SG_TILE * a.Kc * 2u;
    constexpr int MT = 8 * NT, PART = MT * SG_PN;
    SGemvSmem sm;
    sm.stages = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *full = reinterpret_cast<uint64_t *>(sm.stages + (size_t)a.nstage * stage_bytes), *empty = full + 8;
    sm.part = reinterpret_cast<float *>(empty + 8);
    sm.xs = reinterpret_cast<unsigned char *>(sm.part + SG_GROUPS * 8 * PART);
    sm.xrow = (unsigned)min(a.K, Kx) * 2u + ROW_PAD;
    const int nitems = (a.N + SG_TILE - 1) / SG_TILE;
    const int cnt = (int)blockIdx.x < nitems ? (nitems - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int mtiles = (a.M + MT - 1) / MT;
    if (tid == 0) {
        for (int s = 0; s < a.nstage; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 8);          // one arrival per warp of the group whose tile it is
        }
        mbar_fence_init();
    }
    __syncthreads();
    // Each group has a ring of its own: a wait tells one round of a stage from the next only while it is at most one ahead, and in a
    // common ring a group could wait for a round before the other group's round of that stage has even landed.
    const int groups = cnt > 1 ? a.groups : 1, ring = a.nstage / groups;
    // a group's stages in their order: pass of rows, part of the activations, tile, k part
    if (tid >= SG_CONSUMERS) {
        int at0 = 0, at1 = 0;
        unsigned round0 = 0, round1 = 0;
        for (int t = 0; t < mtiles * a.KH; ++t)
            for (int i = 0; i < cnt; ++i) {
                const int row0 = ((int)blockIdx.x + i * (int)gridDim.x) * SG_TILE;
                const bool second = groups > 1 && (i & 1);
                for (int kp = 0; kp < Px; ++kp) {
                    const int s = second ? ring + at1 : at0;
                    const unsigned round = second ? round1 : round0;
                    if (round && !mbar_wait_warp(empty + s, (round - 1) & 1u, a.err)) return;
                    const int k0 = (t % a.KH) * Kx + kp * a.Kc;
                    unsigned char *dst = sm.stages + (size_t)s * stage_bytes;
                    if (a.box3) {
                        if (lane == 0) {
                            mbar_expect_tx(full + s, stage_bytes);
                            tma_load_3d(dst, &map, 0, row0, k0 >> 6, full + s);
                        }
                    } else {
                        const int chunks = (min(a.Kc, a.K - k0) + 63) >> 6;
                        if (lane == 0) mbar_expect_tx(full + s, (unsigned)chunks * 2048u);
                        __syncwarp();
                        if (lane < chunks) tma_load_2d(dst + lane * 2048, &map, k0 + lane * 64, row0, full + s);
                    }
                    __syncwarp();
                    if (second) { if (++at1 == ring) { at1 = 0; ++round1; } }
                    else if (++at0 == ring) { at0 = 0; ++round0; }
                }
            }
        return;
    }
    pdl_wait();
    pdl_trigger();
    const int group = tid >> 8, gt = tid & 255, warp = gt >> 5;
    const uint32_t xs_base = smem_u32(sm.xs);
    // a warp's k steps are every eighth: its place in the 64 columns of a swizzled row stays
    const uint32_t a_base = smem_u32(sm.stages) + (unsigned)(warp >> 2) * 2048u + (unsigned)(lane & 15) * 128u +
                            (unsigned)((((warp & 3) * 2 + (lane >> 4)) ^ (lane & 7)) << 4);
    float *part = sm.part + group * 8 * PART;
    bool ok = true;                          // after a wait that ran out: no further waits, but every meeting
    int at = 0;                              // next stage of the group's ring
    unsigned phase = 0;
    for (int tile = 0; tile < mtiles; ++tile) {
        const int m0 = tile * MT;
        const int nm = min(MT, a.M - m0);
        uint32_t b_base[(NT + 1) / 2];       // lanes 16-31 of a pair of tiles address the second one; rows past the last read the zero row
#pragma unroll
        for (int t = 0; t < (NT + 1) / 2; ++t) {
            const int r = min((2 * t + (lane >> 4)) * 8 + (lane & 7), nm);
            b_base[t] = xs_base + (unsigned)r * sm.xrow + (unsigned)(((lane >> 3) & 1) << 4) + (unsigned)warp * 32u;
        }
        float c[NT][4];
        for (int h = 0; h < a.KH; ++h) {
            if (tile || h) consumer_sync(SG_CONSUMERS);          // everyone is done reading the old rows
            xfill(m0, nm, h * Kx, min(Kx, a.K - h * Kx), sm, tid);
            consumer_sync(SG_CONSUMERS);
            for (int i = group < groups ? group : cnt; i < cnt; i += groups) {       // KH > 1: one tile per group at most
                if (h == 0) {
#pragma unroll
                    for (int t = 0; t < NT; ++t) c[t][0] = c[t][1] = c[t][2] = c[t][3] = 0.f;
                }
                for (int kp = 0; kp < Px; ++kp) {
                    const int s = group * ring + at;
                    if (ok) ok = mbar_wait_warp(full + s, phase, a.err);
                    if (++at == ring) { at = 0; phase ^= 1u; }
                    // this warp's pieces of the stage go to registers at once, so that it is free again while the products are formed
                    const uint32_t ab = a_base + (unsigned)s * stage_bytes;
                    const int steps = min(a.Kc, a.K - h * Kx - kp * a.Kc) >> 4;
                    uint32_t w[SG_STEPS][4];
#pragma unroll
                    for (int j = 0; j < SG_STEPS; ++j)
                        if (warp + 8 * j < steps) ldmatrix_x4(w[j][0], w[j][1], w[j][2], w[j][3], ab + j * 4096);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(empty + s);
                    const uint32_t bk = (unsigned)(kp * a.Kc) * 2u;
#pragma unroll
                    for (int j = 0; j < SG_STEPS; ++j) {
                        if (warp + 8 * j >= steps) break;
#pragma unroll
                        for (int t = 0; t < NT / 2; ++t) {
                            uint32_t b0, b1, b2, b3;
                            ldmatrix_x4(b0, b1, b2, b3, b_base[t] + bk + j * 256);
                            mma_bf16(c[2 * t], w[j][0], w[j][1], w[j][2], w[j][3], b0, b1);
                            mma_bf16(c[2 * t + 1], w[j][0], w[j][1], w[j][2], w[j][3], b2, b3);
                        }
                        if (NT & 1) {
                            uint32_t b0, b1;
                            ldmatrix_x2(b0, b1, b_base[NT / 2] + bk + j * 256);
                            mma_bf16(c[NT - 1], w[j][0], w[j][1], w[j][2], w[j][3], b0, b1);
                        }
                    }
                }
                if (h + 1 < a.KH) continue;
                group_sync(group);                   // the previous tile's sums have been formed
                float *pp = part + warp * PART + (lane & 3) * 2 * SG_PN + (lane >> 2);
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    pp[t * 8 * SG_PN] = c[t][0];
                    pp[(t * 8 + 1) * SG_PN] = c[t][1];
                    pp[t * 8 * SG_PN + 8] = c[t][2];
                    pp[(t * 8 + 1) * SG_PN + 8] = c[t][3];
                }
                group_sync(group);                   // partial sums of all warps visible
                const int row0 = ((int)blockIdx.x + i * (int)gridDim.x) * SG_TILE;
                for (int e = gt; e < nm * SG_TILE; e += 256) {
                    const int m = e >> 4, r = e & 15;
                    const float *ps = part + m * SG_PN + r;
                    float v = 0.f;
#pragma unroll
                    for (int w = 0; w < 8; ++w) v += ps[w * PART];      // warp order: fixed
                    if (row0 + r < a.N) epi(m0 + m, row0 + r, v);
                }
            }
        }
    }
}

// Picks the k partition and the pipeline depth; returns the dynamic shared memory size (0 = does not fit).
static inline size_t sgemv_plan(SGemvArgs &a, int NT, int &grid) {
    // Parts of a multiple of 128 give a warp the same k steps whatever their size, so it may depend on the room that the activations
    // leave; they can be taken in two or four passes over k.
    const int nitems = (a.N + SG_TILE - 1) / SG_TILE;
    grid = nitems < NUM_SMS ? nitems : NUM_SMS;
    const int xrows = (a.M < 8 * NT ? a.M : 8 * NT) + 1;
    const size_t fixed = SG_FIXED + sizeof(float) * SG_GROUPS * 8 * (8 * NT * SG_PN);
    // parts of less than 512 columns only where nothing else fits
    for (int least = 4; least >= 1; least -= 3)
        for (a.KH = 1; a.KH <= 4; a.KH *= 2) {
            // the sums wait in registers between the passes: at most one tile per group
            if (a.KH > 1 && (nitems > SG_GROUPS * grid || a.fi.active)) break;
            const int most = (a.K + 127) / 128;
            // Three stages for each group, where shorter parts make room for them, before two of longer parts: at 16 rows of 2,560 (four parts with two
            // stages / five with three) 16,480 weight rows take 20.7 / 19.5 us and 248,320 227 / 217.  In passes over k the longer parts are better (2,560 x
            // 6,144 at 24 rows 18.7 us, shorter 19.7).
            for (int stages = a.KH == 1 ? SG_STAGES : SG_MIN_STAGES; stages >= SG_MIN_STAGES; stages -= SG_GROUPS)
                for (int P = ((most + SG_STEPS - 1) / SG_STEPS + a.KH - 1) / a.KH * a.KH; P <= most; P += a.KH) {
                    const int Kc = (most + P - 1) / P * 128;
                    if ((a.K + Kc - 1) / Kc != P || (Kc < least * 128 && P > 1)) continue;
                    const size_t xbytes = (size_t)xrows * ((a.KH == 1 ? a.K : P / a.KH * Kc) * 2 + ROW_PAD), stage = (size_t)SG_TILE * Kc * 2;
                    if (fixed + xbytes + stages * stage > SG_SMEM_MAX) continue;
                    const long long ns = ((long long)SG_SMEM_MAX - (long long)(fixed + xbytes)) / (long long)stage;
                    a.P = P;
                    a.Kc = Kc;
                    a.box3 = a.K % 64 == 0;
                    a.nstage = (int)(ns > 8 ? 8 : ns);
                    a.groups = SG_GROUPS;
                    return fixed + xbytes + (size_t)a.nstage * stage;
                }
        }
    return 0;
}

// The weights as sgemv_core reads them: boxes of 16 rows x 64 columns, or a whole stage of such boxes.
static inline bool sgemv_map(CUtensorMap *m, const SGemvArgs &a) {
    if (!a.box3) return make_map(m, a.W, a.N, a.K, a.ldw, SG_TILE);
    return make_map(m, a.W, a.N, a.K, a.ldw, SG_TILE + (a.Kc << 8), MAP_BF16_3D);
}

// The plain GEMV body: default fill and store.
template <int NT, bool FUSED = false>
__device__ __forceinline__ void sgemv_body(const CUtensorMap &map, const SGemvArgs &a, unsigned char *smem) {
    if constexpr (FUSED) {
        if (a.fi.active) sgemv_core<NT>(map, a, smem, XFillGather{a}, EpiStore<true>{a});
        else sgemv_core<NT>(map, a, smem, XFillCopy{a}, EpiStore<true>{a});
    } else {
        sgemv_core<NT>(map, a, smem, XFillCopy{a}, EpiStore<>{a});
    }
}

}  // namespace qw
