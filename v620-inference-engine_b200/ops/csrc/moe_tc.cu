// Routed experts of token-major prefill on the 5th-generation tensor cores: grouped products over expert-sorted rows with the
// weights in q4 (group 128, bf16 scales).
// (Role of the reference's moe_gate_up_T / moe_down_T, src/kernels/moe_experts.hip:17-27.)
//
// The product is formed transposed: D[weight row][token] = W . X^T.  The weights are the A operand and live in tensor memory:
// a thread owns one of a tile's 128 weight rows, turns its nibbles into bf16 pairs in registers and stores them to its TMEM
// lane (tcgen05.st), so a converted tile crosses neither shared memory nor a proxy fence; the tokens are the B operand, so the
// MMA is as wide as the expert has rows (multiples of 16) and no work is done for padding to 128 rows.  A unit of work is two
// 128-row weight tiles against up to 128 rows of one expert - the gate and up rows of the same 128 hidden values (their lanes
// meet in the epilogue, which writes silu(gate) * up), or two neighbouring tiles of the down projection - so the tokens of a k
// block are fetched once for both.
//
//   warp 0       loads, 128 k values a stage: two 128-row x 64-byte TMA tiles of packed weights (64B swizzle) and ceil(rows / 16) x 2
//                boxes of 16 token rows x 64 k values.  down: both on one ring of four stages.  gate/up: weights only, on a ring of six that
//                the conversion alone sets free, and warp 2 brings the tokens on a ring of four: four times the k blocks, and weights that
//                wait for the MMAs' tokens left memory idle (us, one ring and two: 100 tokens 236, 218; 1,021 288, 263; 4,096 480, 455).
//                (For down, five k blocks a unit, two rings are slower: 154 and 159 us at 1,021 tokens, 239 and 255 at 4,096.)
//   warps 8-23   conversion: warp group (tile, parity) owns every other stage of one tile; four TMEM stages of 64 k values
//   warps 1, 3   issue the MMAs of one tile each (A in TMEM, B in shared memory, D in TMEM): with one warp for both, its waits and
//                issue were the longest chain
//   warps 4-7    epilogue
// TMEM: columns 0-255 hold D (two slots of 2 x 64 columns for experts of up to 64 rows, else one of 2 x 128), 256-511 the
// four converted stages of two tiles.  One CTA per SM walks the units round-robin.
//
// What bounds it: the conversion (without the MMAs a unit takes 93 % of its time), beside MMAs of at least 39 cycles each; above 64 rows also the epilogue, which then shares its one D slot.  One layer,
// 512 experts x (1280 x 2560 + 2560 x 640), random routing, us for gate/up with the activation and for down, before (W converted
// into swizzled shared memory by 8 warps, 128-row token tiles as A, activation in a kernel of its own) and now:
//   100 tokens  434 + 5, 245 -> 221, 118     1021  520 + 26, 290 -> 273, 143     4096  695 + 96, 447 -> 443, 217
#include "tc.cuh"

namespace qw {

template <bool SWIGLU> constexpr int mg_wst() { return SWIGLU ? 6 : 4; }
constexpr int MG_XST = 4, MG_AHEAD = 2;
constexpr int MG_W_TILE = 128 * 64, MG_X_PANEL = 128 * 128;
constexpr int MG_THREADS = 768, MG_CONV_WARP0 = 8, MG_EPI_WARP0 = 4;
template <bool SWIGLU>
constexpr int mg_smem() { return MG_XST * 2 * MG_X_PANEL + mg_wst<SWIGLU>() * 2 * MG_W_TILE + 1024 /*alignment*/ + 512 /*barriers*/; }

struct MoeTcArgs {
    const int4 *tiles;       // {first token row, rows (<= 128; 0 = unused), first weight row of the expert, -}
    int total, units_n;      // units of the launch; units per tile entry
    int K, Nw;               // Nw: outputs of a row (swiglu: F)
    int row_step, row_second;// weight rows from one unit to the next of an entry, and from a unit's first tile to its second
    long long w_rows;
    const bf16 *scale;       // [w_rows][K / 128]
    float *C32;              // one of the outputs: fp32 or bf16 [row][ldc]
    bf16 *C16;
    int ldc;
    ErrorWord *err;
    // 0x000F000F and 0x43004300.  As parameters gate/up and down of 100 tokens take 221 and 118 us, as literals 250 and 134
    uint32_t mask, magic;
};

// D (slots and columns) of the units in their order; every role that needs it keeps its own copy.
struct MgSlots {
    int next;                // slot of the next unit of up to 64 rows
    unsigned used[2], committed[2];
};

// Eight columns at a time: the packed pairs of two q4 words go out as they are formed, so no 32-register block is assembled.
// The caller has just voted on a wait: its warp is whole.
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};"
                 ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(taddr)
                 : "memory");
}

// The first used unit at or after `id` (steps of the grid); tl must hold the entry of `id` when id < total.
__device__ __forceinline__ void mg_skip(const MoeTcArgs &a, int &id, int4 &tl) {
    while (id < a.total && tl.y <= 0) {
        id += gridDim.x;
        if (id < a.total) tl = __ldg(a.tiles + id / a.units_n);
    }
}

// The units of this CTA, with the entry of the next one already loaded: it is looked at a whole unit after its load.
struct MgWalk {
    int id, id1;
    int4 tl, tl1;
    __device__ __forceinline__ explicit MgWalk(const MoeTcArgs &a) {
        id = blockIdx.x;
        if (id < a.total) tl = __ldg(a.tiles + id / a.units_n);
        mg_skip(a, id, tl);
        fetch(a);
    }
    __device__ __forceinline__ void fetch(const MoeTcArgs &a) {
        id1 = id + gridDim.x;
        if (id1 < a.total) tl1 = __ldg(a.tiles + id1 / a.units_n);
    }
    __device__ __forceinline__ bool valid(const MoeTcArgs &a) const { return id < a.total; }
    __device__ __forceinline__ void next(const MoeTcArgs &a) {
        mg_skip(a, id1, tl1);
        id = id1;
        tl = tl1;
        if (id < a.total) fetch(a);
    }
    // For the roles that issue as whole warps: one unit for all lanes, said to the compiler.
    __device__ __forceinline__ void uniform() {
        id = __shfl_sync(0xffffffffu, id, 0);
        tl.x = __shfl_sync(0xffffffffu, tl.x, 0);
        tl.y = __shfl_sync(0xffffffffu, tl.y, 0);
        tl.z = __shfl_sync(0xffffffffu, tl.z, 0);
    }
};

template <bool SWIGLU>
__global__ void __launch_bounds__(MG_THREADS, 1) moe_tc_kernel(const __grid_constant__ CUtensorMap mapX,
                                                               const __grid_constant__ CUtensorMap mapW, MoeTcArgs a) {
    constexpr int MG_WST = mg_wst<SWIGLU>();
    constexpr bool JOINT = !SWIGLU;          // weights and tokens of a k block share a stage
    extern __shared__ unsigned char raw[];
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    unsigned char *sx = smem, *sw = smem + MG_XST * 2 * MG_X_PANEL;
    uint64_t *w_full = reinterpret_cast<uint64_t *>(sw + MG_WST * 2 * MG_W_TILE), *w_empty = w_full + MG_WST;
    uint64_t *x_full = w_empty + MG_WST, *x_empty = x_full + MG_XST;
    uint64_t *a_full = x_empty + MG_XST;                        // [tile][parity]: a converted 128 x 128 block
    uint64_t *a_empty = a_full + 4, *done = a_empty + 8;         // [tile][parity][half]: its halves, free again
    uint64_t *acc_empty = done + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
    if (threadIdx.x == 0) {
        for (int s = 0; s < MG_WST; ++s) { mbar_init(w_full + s, 1); mbar_init(w_empty + s, JOINT ? 8 + 2 : 8); }      // 8 converting warps
        for (int s = 0; s < MG_XST; ++s) { mbar_init(x_full + s, 1); mbar_init(x_empty + s, 2); }                      // the MMAs of two tiles
        for (int s = 0; s < 4; ++s) mbar_init(a_full + s, 4);
        for (int s = 0; s < 8; ++s) mbar_init(a_empty + s, 1);
        for (int s = 0; s < 2; ++s) { mbar_init(done + s, 2); mbar_init(acc_empty + s, 4); }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const int kblocks = a.K >> 7;                    // 128 k values each: one scale group
    if (warp == 0 || (!JOINT && warp == 2)) {
        const bool weights = warp == 0, tokens = JOINT || warp == 2;
        const unsigned stages = weights ? MG_WST : MG_XST;
        uint64_t *const full = weights ? w_full : x_full, *const empty = weights ? w_empty : x_empty;
        unsigned s = 0, round = 0;
        bool ok = true;
        MgWalk w(a);
        for (w.uniform(); w.valid(a) && ok; w.next(a), w.uniform()) {
            const int row = w.tl.z + (w.id % a.units_n) * a.row_step;
            const int boxes = tokens ? (w.tl.y + 15) >> 4 : 0;
            for (int kb = 0; kb < kblocks; ++kb) {
                if (round && !mg_wait_warp(empty + s, (round - 1) & 1u, a.err)) { ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(full + s, (weights ? 2u * MG_W_TILE : 0u) + (unsigned)boxes * 4096u);
                    if (weights) {
                        unsigned char *st = sw + s * 2 * MG_W_TILE;
                        tma_load_2d(st, &mapW, kb * 64, row, full + s);
                        tma_load_2d(st + MG_W_TILE, &mapW, kb * 64, row + a.row_second, full + s);
                    }
                    unsigned char *st = sx + s * 2 * MG_X_PANEL;
                    for (int b = 0; b < boxes; ++b) {
                        tma_load_2d(st + b * 2048, &mapX, kb * 128, w.tl.x + b * 16, full + s);
                        tma_load_2d(st + MG_X_PANEL + b * 2048, &mapX, kb * 128 + 64, w.tl.x + b * 16, full + s);
                    }
                }
                if (++s == stages) { s = 0; ++round; }
            }
        }
    } else if (warp == 1 || warp == 3) {
        // one wait per 128 k values where the converting warps have seen the stage's loads complete, tokens included
        const int tile = warp >> 1;
        uint64_t *const a_full1 = a_full + tile * 2, *const a_empty1 = a_empty + tile * 4;
        unsigned it = 0;
        bool ok = true;
        MgSlots sl = {0, {0u, 0u}, {0u, 0u}};
        MgWalk w(a);
        for (w.uniform(); w.valid(a) && ok; w.next(a), w.uniform()) {
            const int N = (w.tl.y + 15) & ~15;
            const bool big = N > 64;
            const int s0 = big ? 0 : sl.next;
            // instruction descriptor: D fp32, A/B bf16, both K-major, N, M = 128
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | (8u << 24);
            for (int s = s0; s < (big ? 2 : s0 + 1) && ok; ++s) {
                if (sl.used[s] && !mg_wait_warp(acc_empty + s, (sl.used[s] - 1) & 1u, a.err)) ok = false;
                ++sl.used[s];
            }
            if (!ok) break;
            const uint32_t d = tmem + (uint32_t)(s0 * 128) + (tile ? (big ? 128u : 64u) : 0u);
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const unsigned odd = it & 1u;
                if (!JOINT && !mg_wait_warp(x_full + it % MG_XST, (it / MG_XST) & 1u, a.err)) { ok = false; break; }
                if (!mg_wait_warp(a_full1 + odd, (it >> 1) & 1u, a.err)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ta = tmem + 256u + odd * 128u + (uint32_t)(tile * 32);
                const uint32_t xb = smem_u32(sx + (it % MG_XST) * 2 * MG_X_PANEL);
                if (elect_one()) {
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_bf16_ts(d, ta + half * 64 + k * 8, make_sw128_desc(xb + half * MG_X_PANEL + k * 32), idesc, (kb | half | k) ? 1u : 0u);
                        umma_commit(a_empty1 + odd * 2 + half);
                    }
                    umma_commit((JOINT ? w_empty : x_empty) + it % MG_XST);
                }
            }
            if (ok && elect_one()) umma_commit(done + s0);
            if (!big) sl.next ^= 1;
        }
    } else if (warp >= MG_CONV_WARP0) {
        const int g = (warp - MG_CONV_WARP0) >> 2, tile = g & 1, odd = g >> 1, q = warp & 3, r = q * 32 + lane;
        const int spr = a.K >> 7;
        const unsigned short *scale = reinterpret_cast<const unsigned short *>(a.scale);
        const bf162 off2 = __floats2bfloat162_rn(136.f, 136.f);
        const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16) + 256u + (uint32_t)(odd * 128 + tile * 32);
        const unsigned char *row_base = sw + tile * MG_W_TILE + r * 64;
        const int swz = ((r >> 1) & 3) << 4;                     // row r's 64 bytes: 16-byte chunk c lies at chunk c ^ ((r >> 1) & 3)
        uint64_t *const a_full2 = a_full + tile * 2 + odd, *const a_empty2 = a_empty + tile * 4 + odd * 2;
        auto scale_row = [&](int id, int z) {
            const long long row = min((long long)z + (id % a.units_n) * a.row_step + tile * a.row_second + r, a.w_rows - 1);
            return scale + row * spr;
        };
        unsigned ws = (unsigned)odd, w_phase = 0;                // stage and phase of this group's next k block
        unsigned n = 0;                                          // k blocks that this group has converted
        bool ok = true;
        MgWalk w(a);
        const unsigned short *sp = nullptr;
        int kb = odd;                                            // first k block of the unit that is this group's
        unsigned short ring[MG_AHEAD], first[MG_AHEAD];          // scales of its coming k blocks, and of the next unit's first ones
#pragma unroll
        for (int i = 0; i < MG_AHEAD; ++i) ring[i] = first[i] = 0;
        if (w.valid(a)) {
            sp = scale_row(w.id, w.tl.z);
#pragma unroll
            for (int i = 0; i < MG_AHEAD; ++i)
                if (kb + 2 * i < kblocks) ring[i] = __ldg(sp + kb + 2 * i);
        }
        while (w.valid(a) && ok) {
            // the next unit's first scales travel while this one is converted (with an odd number of k blocks the groups swap)
            mg_skip(a, w.id1, w.tl1);
            const bool more = w.id1 < a.total;
            const unsigned short *sp1 = more ? scale_row(w.id1, w.tl1.z) : sp;
            const int kb_next = (kb + kblocks) & 1;
#pragma unroll
            for (int i = 0; i < MG_AHEAD; ++i)
                if (more && kb_next + 2 * i < kblocks) first[i] = __ldg(sp1 + kb_next + 2 * i);
            while (kb < kblocks && ok) {
#pragma unroll
                for (int i = 0; i < MG_AHEAD; ++i) {
                    if (kb >= kblocks) break;
                    const uint32_t sc_bits = (uint32_t)ring[i] * 0x10001u;
                    const bf162 sc2 = *reinterpret_cast<const bf162 *>(&sc_bits);
                    if (kb + 2 * MG_AHEAD < kblocks) ring[i] = __ldg(sp + kb + 2 * MG_AHEAD);
                    if (!mg_wait_warp(w_full + ws, w_phase, a.err)) { ok = false; break; }
                    uint32_t words[16];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint4 v = *reinterpret_cast<const uint4 *>(row_base + ws * 2 * MG_W_TILE + ((c << 4) ^ swz));
                        words[4 * c] = v.x; words[4 * c + 1] = v.y; words[4 * c + 2] = v.z; words[4 * c + 3] = v.w;
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(w_empty + ws);
                    ws += 2;
                    if (ws >= MG_WST) { ws -= MG_WST; w_phase ^= 1u; }
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        uint32_t o[4][8];            // converted before the stage is free: behind the wait only the stores remain
#pragma unroll
                        for (int c = 0; c < 4; ++c)
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                // (nibble - 8) is exact in bf16; its product with the bf16 scale is rounded once
                                uint32_t bits;
                                asm("lop3.b32 %0, %1, %2, %3, 0xEA;"
                                    : "=r"(bits)
                                    : "r"(words[half * 8 + c * 2 + (j >> 2)] >> (4 * (j & 3))), "r"(a.mask), "r"(a.magic));
                                const bf162 v = __hmul2(__hsub2(*reinterpret_cast<bf162 *>(&bits), off2), sc2);
                                o[c][j] = *reinterpret_cast<const uint32_t *>(&v);
                            }
                        if (n && !mg_wait_warp(a_empty2 + half, (n - 1) & 1u, a.err)) { ok = false; break; }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                        for (int c = 0; c < 4; ++c) tmem_st8(lane_base + half * 64 + c * 8, o[c]);
                    }
                    if (!ok) break;
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(a_full2);
                    ++n;
                    kb += 2;
                }
            }
            kb = kb_next;
            w.next(a);
            sp = sp1;
#pragma unroll
            for (int i = 0; i < MG_AHEAD; ++i) ring[i] = first[i];
        }
    } else if (warp >= MG_EPI_WARP0) {
        const int q = warp & 3, r = q * 32 + lane;
        bool ok = true;
        MgSlots sl = {0, {0u, 0u}, {0u, 0u}};
        for (MgWalk w(a); w.valid(a) && ok; w.next(a)) {
            const int rows = w.tl.y, N = (rows + 15) & ~15;
            const bool big = N > 64;
            const int s = big ? 0 : sl.next;
            if (!mg_wait_warp(done + s, sl.committed[s] & 1u, a.err)) { ok = false; break; }
            ++sl.committed[s];
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t d0 = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(s * 128), d1 = d0 + (big ? 128u : 64u);
            const int col = (w.id % a.units_n) * (SWIGLU ? 128 : 256) + r;
            for (int c0 = 0; c0 < N; c0 += 16) {
                uint32_t u[16], v[16];
                tmem_ld16(d0 + c0, u);
                tmem_ld16(d1 + c0, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                const int n = rows - c0;                 // rows of this piece that exist (16 or more: all)
                const long long at = (long long)(w.tl.x + c0) * a.ldc + col;
                if (SWIGLU) {
                    bf16 *p = a.C16 + at;
                    const int nc = col < a.Nw ? n : 0;
#pragma unroll
                    for (int j = 0; j < 16; ++j, p += a.ldc)
                        if (j < nc) *p = __float2bfloat16(siluf_(__uint_as_float(u[j])) * __uint_as_float(v[j]));
                } else if (a.C32 && n >= 16 && col + 128 < a.Nw) {
                    float *p = a.C32 + at;
#pragma unroll
                    for (int j = 0; j < 16; ++j, p += a.ldc) {
                        p[0] = __uint_as_float(u[j]);
                        p[128] = __uint_as_float(v[j]);
                    }
                } else {
                    const bool c1 = col < a.Nw, c2 = col + 128 < a.Nw;
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (j >= n) continue;
                        if (a.C32) {
                            if (c1) a.C32[at + (long long)j * a.ldc] = __uint_as_float(u[j]);
                            if (c2) a.C32[at + (long long)j * a.ldc + 128] = __uint_as_float(v[j]);
                        } else {
                            if (c1) a.C16[at + (long long)j * a.ldc] = __float2bfloat16(__uint_as_float(u[j]));
                            if (c2) a.C16[at + (long long)j * a.ldc + 128] = __float2bfloat16(__uint_as_float(v[j]));
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(acc_empty + s);
                if (big) mbar_arrive(acc_empty + 1);
            }
            if (!big) sl.next ^= 1;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

}  // namespace qw

using namespace qw;

template <bool SWIGLU>
static int moe_tc_launch(MoeTcArgs &a, const void *A, const void *Wq, int rows, int lda, int max_tiles, cudaStream_t s) {
    if ((a.K & 127) || (lda & 7) || ((uintptr_t)A & 15) || ((uintptr_t)Wq & 15)) return -1;
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!done[dev]) {
        if (cudaFuncSetAttribute(moe_tc_kernel<SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, mg_smem<SWIGLU>()) != cudaSuccess) return -3;
        done[dev] = true;
    }
    CUtensorMap mX, mW;
    if (!make_map(&mX, A, rows, a.K, lda, 16) || !make_map(&mW, Wq, a.w_rows, a.K / 2, a.K / 2, 128, MAP_BYTES64)) return -3;
    a.err = g_err_ptr;
    a.mask = 0x000F000Fu;
    a.magic = 0x43004300u;
    a.total = max_tiles * a.units_n;
    moe_tc_kernel<SWIGLU><<<persistent_grid(a.total, 1), MG_THREADS, mg_smem<SWIGLU>(), s>>>(mX, mW, a);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Expert-sorted rows against q4 weights: A bf16 [rows][lda] holds the rows of group after group, Wq uint32 [w_rows][K/8] (engine
// nibble order) and scale bf16 [w_rows][K/128] the groups' weight matrices one after another (Nw rows each), tiles (device, int4 x
// max_tiles) lists {first A row, valid rows (at most 128, 0 = unused entry), first W row of the group, 0}.
// C[row][0..Nw) = A[row] . W_group^T, fp32 (out_bf16 = 0) or bf16 [row][ldc].  K a multiple of 128.
QW_API int qwk_gemm_q4_tc_grouped(const void *A, const void *Wq, const void *scale, void *C, const void *tiles, int max_tiles,
                                  int rows, long long w_rows, int Nw, int K, int lda, int ldc, int out_bf16, cudaStream_t s) {
    if (rows <= 0 || max_tiles <= 0) return 0;
    MoeTcArgs a{};
    a.tiles = (const int4 *)tiles;
    a.units_n = (Nw + 255) / 256;
    a.K = K; a.Nw = Nw; a.row_step = 256; a.row_second = 128; a.w_rows = w_rows; a.scale = (const bf16 *)scale;
    a.C32 = out_bf16 ? nullptr : (float *)C;
    a.C16 = out_bf16 ? (bf16 *)C : nullptr;
    a.ldc = ldc;
    return moe_tc_launch<false>(a, A, Wq, rows, lda, max_tiles, s);
}

// The same with the activation: a group's weights are F gate rows, then F up rows; C bf16 [row][ldc >= F] = silu(gate) * up,
// formed from the fp32 sums.
QW_API int qwk_gemm_q4_tc_swiglu(const void *A, const void *Wq, const void *scale, void *C, const void *tiles, int max_tiles,
                                 int rows, long long w_rows, int F, int K, int lda, int ldc, cudaStream_t s) {
    if (rows <= 0 || max_tiles <= 0) return 0;
    MoeTcArgs a{};
    a.tiles = (const int4 *)tiles;
    a.units_n = (F + 127) / 128;
    a.K = K; a.Nw = F; a.row_step = 128; a.row_second = F; a.w_rows = w_rows; a.scale = (const bf16 *)scale;
    a.C16 = (bf16 *)C;
    a.ldc = ldc;
    return moe_tc_launch<true>(a, A, Wq, rows, lda, max_tiles, s);
}
