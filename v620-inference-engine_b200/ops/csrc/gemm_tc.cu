// Dense bf16 GEMM on the 5th-generation tensor cores: C[T][N] = A[T][K] . W[N][K]^T, fp32 accumulate in
// tensor memory, fp32 or bf16 output (prefill path: projections, mixers, router with fp32 output,
// lm_head; role of the reference's rocBLAS call sites, src/kernels/gemm.hip:10-18).
//
// Persistent CTAs (two per SM) walk the 128 x 128 output tiles round-robin.  Warp roles:
//   warp 0   : TMA producer - one elected lane issues cp.async.bulk.tensor loads (no multicast) of the
//              128 x 64 A tile and the 128 x 64 W tile of each k block into a 3-stage ring of
//              128B-swizzled shared-memory tiles, completing on the stage's "full" mbarrier;
//   warp 1   : allocates 256 TMEM columns (two accumulators), and issues tcgen05.mma (one elected lane; M=128, N=128, K=16,
//              four per k block) reading both operands straight from shared memory through matrix descriptors;
//              tcgen05.commit releases a stage ("empty" mbarrier) and, after a tile's last k block, signals that
//              tile's accumulator ("done" mbarrier of the buffer);
//   warps 2-9: epilogue - tcgen05.ld the accumulator (each warp its 32 TMEM lanes = 32 output rows; warps 2-5 the
//              first 64 columns, warps 6-9 the other 64), convert and store, then hand the buffer back
//              ("acc_empty" mbarrier, one arrival per warp).
// The ring and the barriers' phases run on across tiles, so the loads and MMAs of the next tile start while the
// epilogue of this one drains the other accumulator; barrier set-up, the TMEM allocation and the tensor-map fetch are
// paid once per CTA, not once per tile (what weighed on the products with 5-10 k blocks per tile).  Two CTAs share
// an SM: 3 stages x 32 KB and 256 of the 512 TMEM columns each.
// Every mbarrier wait is bounded; a wait that runs out records an error, the roles leave their loops and the
// TMEM allocation is released before the kernel returns.
#include "tc.cuh"
#include "tp.cuh"

#include <cooperative_groups.h>

namespace qw {

constexpr int TC_BM = 128, TC_BN = 128, TC_BK = 64, TC_STAGES = 3;
constexpr int TC_A_BYTES = TC_BM * TC_BK * 2, TC_B_BYTES = TC_BN * TC_BK * 2;     // 16 KB each
constexpr int TC_STAGE_BYTES = TC_A_BYTES + TC_B_BYTES;
constexpr int TC_SMEM = TC_STAGES * TC_STAGE_BYTES + 1024 /*alignment*/ + 256 /*barriers*/;
constexpr int TC_TMEM_COLS = 2 * TC_BN;          // two accumulators
// The wide form of the dense kernel: 128 x 256 tiles (the widest MMA: per k block 48 KB of operands feed twice the
// math of a 128 x 128 tile's 32 KB), four stages, one CTA per SM holding all 512 TMEM columns for its two accumulators.
constexpr int TC_WIDE_BN = 256, TC_WIDE_STAGES = 4;
template <int BN>
constexpr int tc_stage_bytes() { return TC_A_BYTES + BN * TC_BK * 2; }
// Staged epilogue (the tensor-parallel forms): 4 KB per epilogue warp behind the barriers, where a 32 x 32 fp32 piece is
// turned from "a thread owns a row" into "eight lanes own 128 contiguous bytes of a row" before it leaves for a peer.
constexpr int TC_EPI_WARPS = 8, TC_STG_BYTES = 4096;
constexpr int TC_STG_STAGES = 5;                 // k-block ring of the staged 128-wide form (one CTA per SM)
template <int BN, int ST, bool STG = false>
constexpr int tc_smem_bytes() {
    return ST * tc_stage_bytes<BN>() + 1024 /*alignment*/ + 256 /*barriers*/ + (STG ? TC_EPI_WARPS * TC_STG_BYTES : 0);
}

struct GemmTcArgs {
    float *C32;          // one of the two outputs
    bf16 *C16;
    int T, N, K, ldc;
    ErrorWord *err;
    // grouped mode (expert-sorted rows): tiles[entry] = {first A row, valid rows, first W row of the group, -}
    const int4 *tiles;
    int total, tiles_t, tiles_n;     // linear tile ids 0..total-1; plain: id = (split * tiles_n + n) * tiles_t + t; grouped: id = entry * tiles_n + n
    // split-K (plain mode, fp32 output): split s covers k blocks [s * kb_per, (s + 1) * kb_per) and writes its partial sums
    // to C + s * c_split (the consumer adds the splits in order); ksplit == 1: the whole K, c_split unused
    int ksplit, kb_per;
    long long c_split;
    // tensor-parallel prefill (tp.cuh): the producer thread waits for a gathered A operand before its first load; the
    // epilogue sends fp32 tiles to other ranks' receive buffers instead of (mode != 0) storing them to C
    TpWait wait;
    TpEpilogue epi;
    // mixer form: output columns 4 c + s are the gate logits of stream s of column c; the epilogue turns them into the block
    // input C16[row][c] = mean over s of sigmoid(logit) * mix_xn[row][s][c] (rows of 4 * mix_cols) and no logit is stored
    const bf16 *mix_xn;
    int mix_cols;
    bool vec;            // every row and part of C starts on 16 bytes: whole pieces leave as 16-byte stores
};

struct TileAt {
    int t0, rows_valid, n0, w0;
    int kb0, kbn;                    // first k block and number of k blocks of this tile's share of K
    long long c_off;                 // element offset of its output within C
};
// Tile `id` of the launch; false for an unused entry of the tile table (every role skips it alike).
template <int BN = TC_BN>
__device__ __forceinline__ bool tile_at(const GemmTcArgs &a, int id, TileAt &t) {
    const int kblocks = (a.K + TC_BK - 1) / TC_BK;
    t.kb0 = 0;
    t.kbn = kblocks;
    t.c_off = 0;
    if (a.tiles) {
        const int4 tl = __ldg(a.tiles + id / a.tiles_n);
        t.n0 = (id % a.tiles_n) * BN;
        t.t0 = tl.x;
        t.rows_valid = tl.y;
        t.w0 = tl.z + t.n0;
        return tl.y > 0;
    }
    // plain: the row tiles of one column panel are neighbours, so the CTAs in flight share a W panel and the (smaller)
    // activation matrix stays in L2 while W streams through once
    if (a.ksplit > 1) {
        const int per = a.tiles_t * a.tiles_n, sp = id / per;
        id -= sp * per;
        t.kb0 = sp * a.kb_per;
        t.kbn = min(a.kb_per, kblocks - t.kb0);
        t.c_off = sp * a.c_split;
    }
    t.n0 = (id / a.tiles_t) * BN;
    t.t0 = (id % a.tiles_t) * TC_BM;
    t.rows_valid = TC_BM;
    t.w0 = t.n0;
    return true;
}

// One 32-column piece of an accumulator row -> C.
__device__ __forceinline__ void store_piece(const GemmTcArgs &a, long long c_off, int row, int col0, const uint32_t (&v)[32]) {
    const int nmax = a.N - col0;
    if (a.epi.mode) {
        // fp32 pieces to the receive buffers: every rank's (parts of an all-reduce) or the column owner's (reduce-scatter)
        const int owner = a.epi.mode == 2 ? col0 / a.epi.cols_per_rank : 0;
        const long long off = (long long)row * a.epi.ld + (col0 - owner * a.epi.cols_per_rank * (a.epi.mode == 2));
        const bool vec = nmax >= 32 && ((a.epi.ld | col0) & 3) == 0;
#pragma unroll
        for (int d = 0; d < TP_MAX_RANKS; ++d) {
            if (d >= a.epi.ranks || (a.epi.mode == 2 && d != owner)) continue;
            float *o = a.epi.dst[d] + off;
            if (vec) {
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    *reinterpret_cast<float4 *>(o + j) = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                                     __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
            } else {
                for (int j = 0; j < 32 && j < nmax; ++j) o[j] = __uint_as_float(v[j]);
            }
        }
        return;
    }
    if (a.C32) {
        float *o = a.C32 + c_off + (long long)row * a.ldc + col0;
        if (nmax >= 32 && a.vec) {
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<float4 *>(o + j) = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                                 __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
        } else {
            for (int j = 0; j < 32 && j < nmax; ++j) o[j] = __uint_as_float(v[j]);
        }
    } else {
        bf16 *o = a.C16 + (long long)row * a.ldc + col0;
        if (nmax >= 32 && a.vec) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
                uint4 pk;
                pk.x = pack_bf16(__uint_as_float(v[j]), __uint_as_float(v[j + 1]));
                pk.y = pack_bf16(__uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                pk.z = pack_bf16(__uint_as_float(v[j + 4]), __uint_as_float(v[j + 5]));
                pk.w = pack_bf16(__uint_as_float(v[j + 6]), __uint_as_float(v[j + 7]));
                *reinterpret_cast<uint4 *>(o + j) = pk;
            }
        } else {
            for (int j = 0; j < 32 && j < nmax; ++j) o[j] = __float2bfloat16(__uint_as_float(v[j]));
        }
    }
}

// The same piece on its way to other ranks, through the warp's staging buffer: lane r writes its row as eight 16-byte
// chunks (chunk k at position k ^ (r & 7): no bank conflicts either way), then lanes 8i..8i+7 read row 4j + i back and
// store its 128 bytes as one contiguous line - a peer store of whole 128-byte lines instead of 32 scattered 16-byte ones,
// which is what NVLink carries at full rate.  `row0` is the output row of lane 0, `rows_ok` how many of the 32 rows exist.
template <bool LOCAL = false>
__device__ __forceinline__ void send_piece(const GemmTcArgs &a, float *stg, int lane, int row0, int rows_ok, int col0,
                                           const uint32_t (&v)[32], long long c_off = 0) {
    float4 *s4 = reinterpret_cast<float4 *>(stg);
#pragma unroll
    for (int k = 0; k < 8; ++k)
        s4[lane * 8 + (k ^ (lane & 7))] = make_float4(__uint_as_float(v[4 * k]), __uint_as_float(v[4 * k + 1]),
                                                      __uint_as_float(v[4 * k + 2]), __uint_as_float(v[4 * k + 3]));
    __syncwarp();
    const int ch = lane & 7, rsub = lane >> 3;
    const int col = col0 + ch * 4;                                   // first of this lane's four columns
    if constexpr (LOCAL) {
        // the same transposition for this GPU's own fp32 output: whole lines instead of 16-byte pieces of 32 rows
        const bool vec = a.vec && col + 4 <= a.N;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = 4 * i + rsub;
            const float4 val = s4[r * 8 + (ch ^ (r & 7))];
            if (r >= rows_ok || col >= a.N) continue;
            float *o = a.C32 + c_off + (long long)(row0 + r) * a.ldc + col;
            if (vec) {
                *reinterpret_cast<float4 *>(o) = val;
            } else {
                const float e[4] = {val.x, val.y, val.z, val.w};
                for (int j = 0; j < 4 && col + j < a.N; ++j) o[j] = e[j];
            }
        }
        __syncwarp();
        return;
    }
    // the lane's eight float4 (rows rsub, rsub + 4, ...) come out of shared memory once; the destination is chosen once
    // per piece (reduce-scatter: the owner of these columns) or per rank (all-reduce), not once per store
    float4 val[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = 4 * i + rsub;
        val[i] = s4[r * 8 + (ch ^ (r & 7))];
    }
    __syncwarp();
    if (col >= a.N) return;
    const bool rs = a.epi.mode == 2;
    const int owner = rs ? col0 / a.epi.cols_per_rank : 0;
    const int ccol = col - (rs ? owner * a.epi.cols_per_rank : 0);
    const bool vec = ((a.epi.ld | col0) & 3) == 0 && col + 4 <= a.N;
    const long long off0 = (long long)(row0 + rsub) * a.epi.ld + ccol, step = 4ll * a.epi.ld;
    const int d0 = rs ? owner : 0, d1 = rs ? owner + 1 : a.epi.ranks;
    for (int d = d0; d < d1; ++d) {
        float *o = tp_pick(a.epi.dst, d) + off0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (4 * i + rsub >= rows_ok) break;
            if (vec) {
                *reinterpret_cast<float4 *>(o + i * step) = val[i];
            } else {
                const float e[4] = {val[i].x, val[i].y, val[i].z, val[i].w};
                for (int j = 0; j < 4 && col + j < a.N; ++j) o[i * step + j] = e[j];
            }
        }
    }
}

// The epilogue role of both kernels: warps `first_warp` .. `first_warp + n_warps - 1` (n_warps = 4: all 128 columns per warp;
// 8: half of them), for every tile of this CTA in order.
template <int BN = TC_BN, bool STG = false>
__device__ __forceinline__ void epilogue_role(const GemmTcArgs &a, uint32_t tmem, uint64_t *done, uint64_t *acc_empty,
                                              int warp, int lane, int first_warp, int n_warps, float *stg = nullptr) {
    const int q = warp & 3;
    const int cbeg = (n_warps == 8 && warp >= first_warp + 4) ? BN / 2 : 0;
    const int cend = n_warps == 8 ? cbeg + BN / 2 : BN;
    int j = 0;
    for (int id = blockIdx.x; id < a.total; id += gridDim.x) {
        TileAt t;
        if (!tile_at<BN>(a, id, t)) continue;
        const int b = j & 1;
        if (!mbar_wait_warp(done + b, (unsigned)(j >> 1) & 1u, a.err)) return;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int row = t.t0 + q * 32 + lane;
        const bool row_ok = row < a.T && q * 32 + lane < t.rows_valid;
#pragma unroll 1
        for (int c0 = cbeg; c0 < cend; c0 += 32) {
            uint32_t v[32];
            tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN + c0), v);
            if constexpr (STG) {
                const int r0 = t.t0 + q * 32, rows_ok = min(32, min(a.T - r0, t.rows_valid - q * 32));
                if (a.epi.mode) {
                    send_piece(a, stg, lane, r0, rows_ok, t.n0 + c0, v);
                    continue;
                }
                if (a.C32) {
                    send_piece<true>(a, stg, lane, r0, rows_ok, t.n0 + c0, v, t.c_off);
                    continue;
                }
            }
            if (row_ok) store_piece(a, t.c_off, row, t.n0 + c0, v);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty + b);
        ++j;
    }
}

// 32 logits of a row (8 columns of 4 streams) and the streams' values -> 8 means of gated values.
__device__ __forceinline__ void mix_piece(const uint32_t (&v)[32], const uint4 &x0, const uint4 &x1, const uint4 &x2, const uint4 &x3, uint32_t (&o)[4]) {
    const uint32_t x[4][4] = {{x0.x, x0.y, x0.z, x0.w}, {x1.x, x1.y, x1.z, x1.w}, {x2.x, x2.y, x2.z, x2.w}, {x3.x, x3.y, x3.z, x3.w}};
#pragma unroll
    for (int k = 0; k < 4; ++k) {                           // columns 2 k, 2 k + 1 of the piece
        float lo = 0.f, hi = 0.f;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            lo = fmaf(sigmoidf_(__uint_as_float(v[8 * k + s])), bf16_lo(x[s][k]), lo);
            hi = fmaf(sigmoidf_(__uint_as_float(v[8 * k + 4 + s])), bf16_hi(x[s][k]), hi);
        }
        o[k] = pack_bf16(lo * 0.25f, hi * 0.25f);
    }
}

// The mixer form's epilogue: logits to gates, times the streams' values, their mean.  A warp's half of a tile is 32 rows of two pieces of 8
// columns (of 4 streams).  The values of a piece of the next tile are on their way as soon as this tile's are used: fetched when they were needed,
// every tile waited for memory twice.  4,096 rows x 10,240 x 320: 112 us, then 90.
__device__ __forceinline__ void mix_role(const GemmTcArgs &a, uint32_t tmem, uint64_t *done, uint64_t *acc_empty, int warp, int lane) {
    const int q = warp & 3, cbeg = warp >= 6 ? TC_BN / 2 : 0;
    uint4 xv[2][4];
    auto fetch = [&](const TileAt &t, int p) {
        const int row = t.t0 + q * 32 + lane, col = t.n0 + cbeg + p * 32;
        const bf16 *x = a.mix_xn + (long long)row * 4 * a.mix_cols + (col >> 2);
#pragma unroll
        for (int s = 0; s < 4; ++s)
            xv[p][s] = row < a.T && col < a.N ? __ldg(reinterpret_cast<const uint4 *>(x + (long long)s * a.mix_cols)) : make_uint4(0u, 0u, 0u, 0u);
    };
    TileAt t;
    int j = 0;
    if ((int)blockIdx.x < a.total && tile_at<TC_BN>(a, blockIdx.x, t)) {
        fetch(t, 0);
        fetch(t, 1);
    }
    for (int id = blockIdx.x; id < a.total; id += gridDim.x, ++j) {          // every tile of a plain product exists
        const int b = j & 1, row = t.t0 + q * 32 + lane, n0 = t.n0 + cbeg;
        const bool more = id + (int)gridDim.x < a.total;
        if (more) tile_at<TC_BN>(a, id + gridDim.x, t);
        if (!mbar_wait_warp(done + b, (unsigned)(j >> 1) & 1u, a.err)) return;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            uint32_t v[32], o[4];
            tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * TC_BN + cbeg + p * 32), v);
            mix_piece(v, xv[p][0], xv[p][1], xv[p][2], xv[p][3], o);
            if (more) fetch(t, p);
            // mix_cols is a multiple of 8: pieces are whole
            if (row < a.T && n0 + p * 32 < a.N) *reinterpret_cast<uint4 *>(a.C16 + (long long)row * a.ldc + ((n0 + p * 32) >> 2)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty + b);
    }
}

// The MMA role of both kernels (one warp).
template <int BN = TC_BN, int ST = TC_STAGES>
__device__ __forceinline__ void mma_role(const GemmTcArgs &a, unsigned char *smem, uint32_t tmem, uint64_t *full, uint64_t *empty,
                                         uint64_t *done, uint64_t *acc_empty, int kblocks) {
    // instruction descriptor: D fp32, A/B bf16, both K-major, N and M of the tile
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
    int j = 0;
    unsigned it = 0;
    for (int id = blockIdx.x; id < a.total; id += gridDim.x) {
        TileAt t;
        if (!tile_at<BN>(a, id, t)) continue;
        const int b = j & 1;
        if (j >= 2 && !mbar_wait_warp(acc_empty + b, (unsigned)((j >> 1) - 1) & 1u, a.err)) return;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int kb = 0; kb < t.kbn; ++kb, ++it) {
            const unsigned s = it % ST;
            if (!mbar_wait_warp(full + s, (it / ST) & 1u, a.err)) return;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t sa = smem_u32(smem + s * tc_stage_bytes<BN>()), sb = sa + TC_A_BYTES;
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < TC_BK / 16; ++k) {
                    const uint64_t da = make_sw128_desc(sa + k * 32), db = make_sw128_desc(sb + k * 32);
                    umma_bf16(tmem + (uint32_t)(b * BN), da, db, idesc, (kb | k) ? 1u : 0u);
                }
                umma_commit(empty + s);          // the stage is free once these MMAs have read it
            }
        }
        if (elect_one()) umma_commit(done + b);               // this tile's accumulator is complete
        ++j;
    }
}

// Shared set-up of both kernels: barriers, TMEM allocation (warp 1), and the pointers into shared memory.
struct TcShared {
    unsigned char *smem;
    uint64_t *full, *empty, *done, *acc_empty;
    uint32_t tmem;
};
template <int BN = TC_BN, int ST = TC_STAGES>
__device__ __forceinline__ TcShared tc_setup(unsigned char *raw, int warp, unsigned full_count, unsigned acc_empty_count) {
    TcShared t;
    t.smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    t.full = reinterpret_cast<uint64_t *>(t.smem + ST * tc_stage_bytes<BN>());
    t.empty = t.full + ST;
    t.done = t.empty + ST;
    t.acc_empty = t.done + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(t.acc_empty + 2);
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(t.full + s, full_count);
            mbar_init(t.empty + s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(t.done + b, 1);
            mbar_init(t.acc_empty + b, acc_empty_count);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    t.tmem = *tmem_slot;
    return t;
}
template <int BN = TC_BN>
__device__ __forceinline__ void tc_teardown(const TcShared &t, int warp) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(t.tmem), "r"(2 * BN) : "memory");
    }
}

// grid: min(tiles, CTAs per SM x SMs) CTAs of 320 threads (two per SM with 128-wide tiles, one with 256-wide tiles).
template <int BN, int ST, bool STG = false>
__global__ void __launch_bounds__(320, (BN == TC_BN && !STG) ? 2 : 1) gemm_tc_kernel(const __grid_constant__ CUtensorMap mapA,
                                                         const __grid_constant__ CUtensorMap mapW, GemmTcArgs a) {
    extern __shared__ unsigned char raw[];
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const TcShared sh = tc_setup<BN, ST>(raw, warp, 1, 8);
    const int kblocks = (a.K + TC_BK - 1) / TC_BK;
    if (warp == 0) {
        unsigned it = 0;
        bool ok = __all_sync(0xffffffffu, tp_wait_thread(a.wait)) != 0;
        for (int id = blockIdx.x; id < a.total && ok; id += gridDim.x) {
            TileAt t;
            if (!tile_at<BN>(a, id, t)) continue;
            for (int kb = 0; kb < t.kbn; ++kb, ++it) {
                const unsigned s = it % ST;
                if (it >= ST && !mbar_wait_warp(sh.empty + s, (it / ST - 1) & 1u, a.err)) { ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(sh.full + s, tc_stage_bytes<BN>());
                    unsigned char *st = sh.smem + s * tc_stage_bytes<BN>();
                    tma_load_2d(st, &mapA, (t.kb0 + kb) * TC_BK, t.t0, sh.full + s);
                    tma_load_2d(st + TC_A_BYTES, &mapW, (t.kb0 + kb) * TC_BK, t.w0, sh.full + s);
                }
            }
        }
    } else if (warp == 1) {
        mma_role<BN, ST>(a, sh.smem, sh.tmem, sh.full, sh.empty, sh.done, sh.acc_empty, kblocks);
    } else {
        float *stg = nullptr;
        if constexpr (STG)
            stg = reinterpret_cast<float *>(sh.smem + ST * tc_stage_bytes<BN>() + 256 + (warp - 2) * TC_STG_BYTES);
        bool mixes = false;
        if constexpr (BN == TC_BN && !STG) mixes = a.mix_xn != nullptr;
        if (mixes) mix_role(a, sh.tmem, sh.done, sh.acc_empty, warp, lane);
        else epilogue_role<BN, STG>(a, sh.tmem, sh.done, sh.acc_empty, warp, lane, 2, TC_EPI_WARPS, stg);
    }
    tc_teardown<BN>(sh, warp);
    tp_signal(a.epi.sig);
}

// ------------------------------------------------------------------------------------------------------------------
// The split form, for products with few output tiles: a cluster of KS CTAs shares one 128 x 128 tile, each over its part of the k
// blocks.  A k block takes a CTA 0.3 us however few CTAs run, so 20 tiles of 96 k blocks took 29 us on 20 SMs.  When all
// accumulators are complete, CTA c owns the columns [c * 128 / KS, ...): the others write theirs into its (now free) pipeline
// stages, and it adds the parts in rank order - the sum does not depend on timing - and stores.
// grid KS x tiles, 320 threads: warp 0 TMA, warp 1 MMA, warps 2-9 epilogue.
// ------------------------------------------------------------------------------------------------------------------
constexpr int TC_KS_STAGES = 5;
template <int KS>
__global__ void __launch_bounds__(320, 1) gemm_tc_ksplit_kernel(const __grid_constant__ CUtensorMap mapA,
                                                                const __grid_constant__ CUtensorMap mapW, GemmTcArgs a) {
    namespace cg = cooperative_groups;
    constexpr int QC = TC_BN / KS;                                    // columns of a CTA's share of the tile
    constexpr int PART = TC_BM * QC * 4, CH = QC / 4;                 // one part in shared memory; 16-byte chunks of its row
    static_assert((KS - 1) * PART <= TC_KS_STAGES * TC_STAGE_BYTES, "the parts fit into the stages");
    extern __shared__ unsigned char raw[];
    const cg::cluster_group cl = cg::this_cluster();
    const int warp = uniform_warp(), lane = threadIdx.x & 31, rank = blockIdx.x % KS;
    const TcShared sh = tc_setup<TC_BN, TC_KS_STAGES>(raw, warp, 1, 8);
    TileAt t;
    tile_at(a, blockIdx.x / KS, t);
    const int per = (t.kbn + KS - 1) / KS, k0 = min(t.kbn, rank * per), k1 = min(t.kbn, k0 + per);
    if (warp == 0) {
        for (int kb = k0; kb < k1; ++kb) {
            const unsigned it = (unsigned)(kb - k0), s = it % TC_KS_STAGES;
            if (it >= TC_KS_STAGES && !mbar_wait_warp(sh.empty + s, (it / TC_KS_STAGES - 1) & 1u, a.err)) break;
            if (elect_one()) {
                mbar_expect_tx(sh.full + s, TC_STAGE_BYTES);
                unsigned char *st = sh.smem + s * TC_STAGE_BYTES;
                tma_load_2d(st, &mapA, (t.kb0 + kb) * TC_BK, t.t0, sh.full + s);
                tma_load_2d(st + TC_A_BYTES, &mapW, (t.kb0 + kb) * TC_BK, t.w0, sh.full + s);
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TC_BN >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
        bool ok = true;
        for (int kb = k0; kb < k1; ++kb) {
            const unsigned it = (unsigned)(kb - k0), s = it % TC_KS_STAGES;
            if (!mbar_wait_warp(sh.full + s, (it / TC_KS_STAGES) & 1u, a.err)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t sa = smem_u32(sh.smem + s * TC_STAGE_BYTES), sb = sa + TC_A_BYTES;
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < TC_BK / 16; ++k)
                    umma_bf16(sh.tmem, make_sw128_desc(sa + k * 32), make_sw128_desc(sb + k * 32), idesc, (it | k) ? 1u : 0u);
                umma_commit(sh.empty + s);
            }
        }
        if (ok && k1 > k0 && elect_one()) umma_commit(sh.done);
    } else if (k1 > k0) {
        mbar_wait_warp(sh.done, 0u, a.err);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    __syncwarp();
    cl.sync();                                                        // every accumulator is complete, every stage free
    const int q = warp & 3, hf = warp >= 6 ? 1 : 0;                   // epilogue warps: 32 rows, every other share
    if (warp >= 2 && k1 > k0) {
        for (int c = hf; c < KS; c += 2) {
            if (c == rank) continue;
            unsigned char *dst = cl.map_shared_rank(sh.smem, c) + (rank < c ? rank : rank - 1) * PART + (q * 32 + lane) * QC * 4;
#pragma unroll
            for (int x = 0; x < QC; x += 16) {
                uint32_t v[16];
                tmem_ld16(sh.tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(c * QC + x), v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 4; ++j)                           // chunk k of a row at chunk k ^ (row & (CH - 1)): no bank conflicts
                    *reinterpret_cast<uint4 *>(dst + (((x / 4 + j) ^ (lane & (CH - 1))) << 4)) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            }
        }
    }
    cl.sync();
    if (warp >= 2) {
        const int parts = (t.kbn + per - 1) / per;                    // ranks past these had no k blocks
        const int row = t.t0 + q * 32 + lane;
#pragma unroll
        for (int x = hf * 16; x < QC; x += 32) {
            uint32_t own[16];
            tmem_ld16(sh.tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(rank * QC + x), own);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            float sum[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[j] = 0.f;
            for (int r = 0; r < parts; ++r) {
                const unsigned char *src = sh.smem + (r < rank ? r : r - 1) * PART + (q * 32 + lane) * QC * 4;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float4 v;
                    if (r == rank) v = make_float4(__uint_as_float(own[4 * j]), __uint_as_float(own[4 * j + 1]), __uint_as_float(own[4 * j + 2]), __uint_as_float(own[4 * j + 3]));
                    else v = *reinterpret_cast<const float4 *>(src + (((x / 4 + j) ^ (lane & (CH - 1))) << 4));
                    sum[4 * j] += v.x; sum[4 * j + 1] += v.y; sum[4 * j + 2] += v.z; sum[4 * j + 3] += v.w;
                }
            }
            const int col = t.n0 + rank * QC + x;
            if (row >= a.T || col >= a.N) continue;
            const long long at = t.c_off + (long long)row * a.ldc + col;
            if (a.C32 && col + 16 <= a.N && a.vec) {
#pragma unroll
                for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4 *>(a.C32 + at + j) = make_float4(sum[j], sum[j + 1], sum[j + 2], sum[j + 3]);
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (col + j >= a.N) break;
                    if (a.C32) a.C32[at + j] = sum[j];
                    else a.C16[at + j] = __float2bfloat16(sum[j]);
                }
            }
        }
    }
    tc_teardown(sh, warp);
}

// ------------------------------------------------------------------------------------------------------------------
// The pair form of the dense kernel: two CTAs of a cluster (two neighbouring SMs) compute one 256 x 256 output tile with
// tcgen05.mma.cta_group::2.  Each CTA loads its own 128 rows of A and ONE HALF of the tile's W rows (128 of 256) per k
// block - 32 KB for 128 x 256 x 64 multiply-adds per SM, where the single-CTA forms need 48 KB (128 x 256 tile) or 64 KB
// (two 128 x 128 tiles) for the same math: those stop at what an SM can pull out of L2 (~64 bytes per cycle), this one
// does not.  The tensor cores of both SMs read both CTAs' shared memory; each SM accumulates its 128 rows x 256 columns
// in its own tensor memory (two accumulators = all 512 columns).
//   producer (warp 0, one elected lane, both CTAs): waits for its own "empty" barrier of the stage, loads its A tile and its W
//       half with cp.async.bulk.tensor.cta_group::2 (no multicast), both completing on the LEADER's "full" barrier, on
//       which the leader's producer has announced the 64 KB of the pair;
//   MMA (warp 1, one elected lane, leader CTA only): four cta_group::2 MMAs per k block; tcgen05.commit (to both CTAs of the
//       pair) frees the stage in both CTAs and, after a tile's last k block, publishes the accumulator to both CTAs'
//       epilogue warps;
//   epilogue (warps 2-9, both CTAs): as in the single-CTA kernel, on the CTA's own 128 rows; hands the accumulator back
//       by arriving on the leader's "acc_empty" barrier (16 arrivals: 8 warps of 2 CTAs).
// Barriers are initialised before a cluster-wide barrier and nobody leaves before another one, so no signal is ever
// sent to a CTA that is not there; every wait is bounded as elsewhere.
// ------------------------------------------------------------------------------------------------------------------
constexpr int TC_PAIR_BN = 256, TC_PAIR_BM = 256, TC_PAIR_STAGES = 6, TC_PAIR_STG_STAGES = 5;
constexpr int TC_PAIR_STAGE_BYTES = TC_A_BYTES + TC_B_BYTES;          // per CTA: 128 x 64 of A and 128 x 64 of W
template <int ST, bool STG>
constexpr int tc_pair_smem_bytes() { return ST * TC_PAIR_STAGE_BYTES + 1024 + 256 + (STG ? TC_EPI_WARPS * TC_STG_BYTES : 0); }

struct PairTile {
    int t0, n0, w0, rows_valid;          // this CTA's first A row / the tile's first column / this CTA's first W row
};
__device__ __forceinline__ PairTile pair_tile_at(const GemmTcArgs &a, int id, uint32_t rank) {
    PairTile t;
    // the row tiles of one column panel are neighbours (W streams once, A stays in L2)
    t.n0 = (id / a.tiles_t) * TC_PAIR_BN;
    t.t0 = (id % a.tiles_t) * TC_PAIR_BM + (int)rank * TC_BM;
    t.w0 = t.n0 + (int)rank * (TC_PAIR_BN / 2);
    t.rows_valid = TC_BM;
    return t;
}

// grid: 2 x min(pair tiles, SMs / 2) CTAs of 320 threads in clusters of two.  a.tiles_t / a.total count 256 x 256 tiles.
template <int ST, bool STG>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(320, 1) gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap mapA,
                                                                                        const __grid_constant__ CUtensorMap mapW,
                                                                                        GemmTcArgs a) {
    extern __shared__ unsigned char raw[];
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + ST * TC_PAIR_STAGE_BYTES);
    uint64_t *empty = full + ST, *done = empty + ST, *acc_empty = done + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(full + s, 1);          // the leader's: one arrival (its producer's expect_tx) + the pair's bytes
            mbar_init(empty + s, 1);         // one commit arrival
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(done + b, 1);
            mbar_init(acc_empty + b, 2 * TC_EPI_WARPS);          // the leader's: the epilogue warps of both CTAs
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();                      // both CTAs' barriers exist before anything is sent to them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const int kblocks = (a.K + TC_BK - 1) / TC_BK;
    if (warp == 0) {
        unsigned it = 0;
        bool ok = __all_sync(0xffffffffu, tp_wait_thread(a.wait)) != 0;
        for (int id = cluster_id; id < a.total && ok; id += n_clusters) {
            const PairTile t = pair_tile_at(a, id, rank);
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const unsigned s = it % ST;
                if (it >= ST && !mbar_wait_warp(empty + s, (it / ST - 1) & 1u, a.err)) { ok = false; break; }
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(full + s, 2 * TC_PAIR_STAGE_BYTES);
                    const uint32_t bar = map_to_cta(smem_u32(full + s), 0);
                    unsigned char *st = smem + s * TC_PAIR_STAGE_BYTES;
                    tma_load_2d_pair(st, &mapA, kb * TC_BK, t.t0, bar);
                    tma_load_2d_pair(st + TC_A_BYTES, &mapW, kb * TC_BK, t.w0, bar);
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // instruction descriptor: D fp32, A/B bf16, both K-major, N = 256, M = 256 (the pair's rows)
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TC_PAIR_BN >> 3) << 17) | ((uint32_t)(TC_PAIR_BM >> 4) << 24);
            int j = 0;
            unsigned it = 0;
            bool ok = true;
            for (int id = cluster_id; id < a.total && ok; id += n_clusters) {
                const int b = j & 1;
                if (j >= 2 && !mbar_wait_warp(acc_empty + b, (unsigned)((j >> 1) - 1) & 1u, a.err)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const unsigned s = it % ST;
                    if (!mbar_wait_warp(full + s, (it / ST) & 1u, a.err)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t sa = smem_u32(smem + s * TC_PAIR_STAGE_BYTES), sb = sa + TC_A_BYTES;
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < TC_BK / 16; ++k)
                            umma_bf16_pair(tmem + (uint32_t)(b * TC_PAIR_BN), make_sw128_desc(sa + k * 32), make_sw128_desc(sb + k * 32), idesc,
                                           (kb | k) ? 1u : 0u);
                        umma_commit_pair(empty + s);
                    }
                }
                if (ok && elect_one()) umma_commit_pair(done + b);
                ++j;
            }
        }
    } else {
        float *stg = nullptr;
        if constexpr (STG) stg = reinterpret_cast<float *>(smem + ST * TC_PAIR_STAGE_BYTES + 256 + (warp - 2) * TC_STG_BYTES);
        const int q = warp & 3;
        const int cbeg = warp >= 6 ? TC_PAIR_BN / 2 : 0, cend = cbeg + TC_PAIR_BN / 2;
        const uint32_t acc_bar = map_to_cta(smem_u32(acc_empty), 0);
        int j = 0;
        for (int id = cluster_id; id < a.total; id += n_clusters) {
            const PairTile t = pair_tile_at(a, id, rank);
            const int b = j & 1;
            if (!mbar_wait_warp(done + b, (unsigned)(j >> 1) & 1u, a.err)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int row = t.t0 + q * 32 + lane;
            const bool row_ok = row < a.T;
#pragma unroll 1
            for (int c0 = cbeg; c0 < cend; c0 += 32) {
                uint32_t v[32];
                tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * TC_PAIR_BN + c0), v);
                if (t.n0 + c0 >= a.N) continue;
                if constexpr (STG) {
                    const int r0 = t.t0 + q * 32;
                    if (a.epi.mode) {
                        send_piece(a, stg, lane, r0, min(32, a.T - r0), t.n0 + c0, v);
                        continue;
                    }
                    if (a.C32) {
                        send_piece<true>(a, stg, lane, r0, min(32, a.T - r0), t.n0 + c0, v);
                        continue;
                    }
                }
                if (row_ok) store_piece(a, 0, row, t.n0 + c0, v);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(acc_bar + (uint32_t)(b * 8));
            ++j;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();                      // nothing is in flight towards either CTA any more
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
    tp_signal(a.epi.sig);
}

// The mixer form of chunks: a CTA keeps 256 weight rows whole (K <= 320: 160 KB) and takes a run of row tiles, column panel by
// column panel, so that a tile brings 80 KB of activations and nothing else.  (As 128 x 128 tiles, two CTAs an SM, each brought 160 KB for a
// quarter of that: 420 MB out of L2 at 4,096 rows.)  Sixteen epilogue warps of 64 columns, whose 32 bytes of each stream's row are whole sectors.
// 4,096 x 10,240 x 320: 85 us, now 70; 2,048 rows 43, 39; 1,021 rows 27 either way.
//   warp 0 TMA, warp 1 MMA, warps 2-17 epilogue; columns 0-255 and 256-511 of tensor memory: two accumulators
constexpr int MX_KB = 5, MX_ST = 4, MX_EPI = 16, MX_THREADS = 64 + MX_EPI * 32, MX_W_BYTES = 256 * TC_BK * 2;
constexpr int MX_SMEM = MX_KB * MX_W_BYTES + MX_ST * TC_A_BYTES + 1024 /*alignment*/ + 256 /*barriers*/;

__global__ void __launch_bounds__(MX_THREADS, 1) gemm_mix_tc_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapW,
                                                                    GemmTcArgs a) {
    extern __shared__ unsigned char raw[];
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    unsigned char *sw = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023), *sa = sw + MX_KB * MX_W_BYTES;
    uint64_t *w_full = reinterpret_cast<uint64_t *>(sa + MX_ST * TC_A_BYTES), *w_empty = w_full + MX_KB, *full = w_empty + 1, *empty = full + MX_ST,
             *done = empty + MX_ST, *acc_empty = done + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
    if (threadIdx.x == 0) {
        for (int k = 0; k < MX_KB; ++k) mbar_init(w_full + k, 1);
        mbar_init(w_empty, 1);
        for (int k = 0; k < MX_ST; ++k) { mbar_init(full + k, 1); mbar_init(empty + k, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(done + b, 1); mbar_init(acc_empty + b, MX_EPI); }
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
    const int kblocks = (a.K + TC_BK - 1) / TC_BK;
    const int from = (int)((long long)a.total * blockIdx.x / gridDim.x), to = (int)((long long)a.total * (blockIdx.x + 1) / gridDim.x);
    if (warp == 0) {
        unsigned it = 0, panels = 0;
        int at = -1;
        bool ok = true;
        for (int id = from; id < to && ok; ++id) {
            const int n = id / a.tiles_t, t0 = (id - n * a.tiles_t) * TC_BM;
            if (n != at) {                               // the next panel, once the last one's products have read theirs
                if (panels && !mbar_wait_warp(w_empty, (panels - 1) & 1u, a.err)) break;
                if (elect_one())
                    for (int kb = 0; kb < kblocks; ++kb) {
                        mbar_expect_tx(w_full + kb, MX_W_BYTES);
                        tma_load_2d(sw + kb * MX_W_BYTES, &mapW, kb * TC_BK, n * 256, w_full + kb);
                    }
                at = n;
                ++panels;
            }
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const unsigned st = it % MX_ST;
                if (it >= MX_ST && !mbar_wait_warp(empty + st, (it / MX_ST - 1) & 1u, a.err)) { ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(full + st, TC_A_BYTES);
                    tma_load_2d(sa + st * TC_A_BYTES, &mapA, kb * TC_BK, t0, full + st);
                }
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(256 >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
        unsigned it = 0, panels = 0;
        int at = -1;
        bool ok = true;
        for (int id = from, j = 0; id < to && ok; ++id, ++j) {
            const int n = id / a.tiles_t, b = j & 1;
            const bool fresh = n != at;
            if (fresh) { at = n; ++panels; }
            if (j >= 2 && !mbar_wait_warp(acc_empty + b, (unsigned)((j >> 1) - 1) & 1u, a.err)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const unsigned st = it % MX_ST;
                if ((fresh && !mbar_wait_warp(w_full + kb, (panels - 1) & 1u, a.err)) || !mbar_wait_warp(full + st, (it / MX_ST) & 1u, a.err)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t pa = smem_u32(sa + st * TC_A_BYTES), pb = smem_u32(sw + kb * MX_W_BYTES);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < TC_BK / 16; ++k)
                        umma_bf16(tmem + (uint32_t)(b * 256), make_sw128_desc(pa + k * 32), make_sw128_desc(pb + k * 32), idesc, (kb | k) ? 1u : 0u);
                    umma_commit(empty + st);
                }
            }
            if (ok && elect_one()) {
                umma_commit(done + b);
                if (id + 1 < to && (id + 1) / a.tiles_t != n) umma_commit(w_empty);
            }
        }
    } else {
        const int q = warp & 3, c0 = ((warp - 2) >> 2) * 64;             // this warp's 32 rows and 64 columns of a tile
        uint4 xv[4][2];
        auto fetch = [&](int id) {                       // both halves of a sector at once (a half behind each piece: 70 us -> 87)
            const int n = id / a.tiles_t, row = (id - n * a.tiles_t) * TC_BM + q * 32 + lane, col = n * 256 + c0;
            const bf16 *x = a.mix_xn + (long long)row * 4 * a.mix_cols + (col >> 2);
#pragma unroll
            for (int s = 0; s < 4; ++s)
#pragma unroll
                for (int p = 0; p < 2; ++p)
                    xv[s][p] = row < a.T && col + p * 32 < a.N ? __ldg(reinterpret_cast<const uint4 *>(x + (long long)s * a.mix_cols) + p) : make_uint4(0u, 0u, 0u, 0u);
        };
        if (from < to) fetch(from);
        for (int id = from, j = 0; id < to; ++id, ++j) {
            const int n = id / a.tiles_t, row = (id - n * a.tiles_t) * TC_BM + q * 32 + lane, col = n * 256 + c0, b = j & 1;
            if (!mbar_wait_warp(done + b, (unsigned)(j >> 1) & 1u, a.err)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t o[2][4];
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                uint32_t v[32];
                tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * 256 + c0 + p * 32), v);
                if (p == 1) {                            // the accumulator is read
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_empty + b);
                }
                mix_piece(v, xv[0][p], xv[1][p], xv[2][p], xv[3][p], o[p]);
            }
            if (id + 1 < to) fetch(id + 1);
            // mix_cols is a multiple of 8: pieces are whole
#pragma unroll
            for (int p = 0; p < 2; ++p)
                if (row < a.T && col + p * 32 < a.N)
                    *reinterpret_cast<uint4 *>(a.C16 + (long long)row * a.ldc + ((col + p * 32) >> 2)) = make_uint4(o[p][0], o[p][1], o[p][2], o[p][3]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// The pair form with the operands' roles exchanged: the pair's 256 rows are weight rows and the tokens the columns, so that a
// tile is as wide as the tokens want - any multiple of 16 up to 256 - and a prompt whose length is no multiple of 256 is not padded to one.  A
// lane of the accumulator is an output column: the epilogue's stores are whole 128-byte lines without a staging buffer.  us,
// roles kept / exchanged: 777 x 16,480 x 2,560 78 / 61, 1,021 x 2,560 x 6,144 45 / 35, 4,096 x 16,480 x 2,560 260 / 235, 4,096 x 2,560 x 6,144
// 124 / 99, 300 x 2,560 x 6,144 47 / 31.
// grid as above; a.tiles_t / a.total count tiles of nt tokens x 256 columns.
template <bool BF16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(320, 1) gemm_tc_exchange_kernel(const __grid_constant__ CUtensorMap mapX,
                                                                                        const __grid_constant__ CUtensorMap mapW, GemmTcArgs a, int nt) {
    constexpr int ST = TC_PAIR_STAGES;
    extern __shared__ unsigned char raw[];
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + ST * TC_PAIR_STAGE_BYTES);
    uint64_t *empty = full + ST, *done = empty + ST, *acc_empty = done + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(done + b, 1); mbar_init(acc_empty + b, 2 * TC_EPI_WARPS); }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();                      // both CTAs' barriers exist before anything is sent to them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const int kblocks = (a.K + TC_BK - 1) / TC_BK;
    if (warp == 0) {
        unsigned it = 0;
        bool ok = true;
        for (int id = cluster_id; id < a.total && ok; id += n_clusters) {
            const int t0 = id % a.tiles_t * nt + (int)rank * (nt >> 1), n0 = id / a.tiles_t * 256 + (int)rank * 128;
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const unsigned s = it % ST;
                if (it >= ST && !mbar_wait_warp(empty + s, (it / ST - 1) & 1u, a.err)) { ok = false; break; }
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(full + s, 2u * (16384u + (unsigned)nt * 64u));
                    const uint32_t bar = map_to_cta(smem_u32(full + s), 0);
                    unsigned char *st = smem + s * TC_PAIR_STAGE_BYTES;
                    tma_load_2d_pair(st, &mapW, kb * TC_BK, n0, bar);
                    tma_load_2d_pair(st + 16384, &mapX, kb * TC_BK, t0, bar);
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // instruction descriptor: D fp32, A/B bf16, both K-major, N = nt, M = 256 (the pair's rows)
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nt >> 3) << 17) | (16u << 24);
            int j = 0;
            unsigned it = 0;
            bool ok = true;
            for (int id = cluster_id; id < a.total && ok; id += n_clusters) {
                const int b = j & 1;
                if (j >= 2 && !mbar_wait_warp(acc_empty + b, (unsigned)((j >> 1) - 1) & 1u, a.err)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const unsigned s = it % ST;
                    if (!mbar_wait_warp(full + s, (it / ST) & 1u, a.err)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t sw = smem_u32(smem + s * TC_PAIR_STAGE_BYTES), sx = sw + 16384;
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < TC_BK / 16; ++k)
                            umma_bf16_pair(tmem + (uint32_t)(b * 256), make_sw128_desc(sw + k * 32), make_sw128_desc(sx + k * 32), idesc, (kb | k) ? 1u : 0u);
                        umma_commit_pair(empty + s);
                    }
                }
                if (ok && elect_one()) umma_commit_pair(done + b);
                ++j;
            }
        }
    } else {
        const int q = warp & 3;
        const uint32_t acc_bar = map_to_cta(smem_u32(acc_empty), 0);
        int j = 0;
        for (int id = cluster_id; id < a.total; id += n_clusters) {
            const int t0 = id % a.tiles_t * nt, n = id / a.tiles_t * 256 + (int)rank * 128 + q * 32 + lane, b = j & 1;
            if (!mbar_wait_warp(done + b, (unsigned)(j >> 1) & 1u, a.err)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * 256);
#pragma unroll 1
            for (int c0 = warp >= 6 ? 32 : 0; c0 < nt && t0 + c0 < a.T; c0 += 64) {
                uint32_t v[2][16];
                tmem_ld16(acc + c0, v[0]);
                if (c0 + 16 < nt) tmem_ld16(acc + c0 + 16, v[1]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                const int rows = min(min(32, nt - c0), a.T - t0 - c0);
                const long long at = (long long)(t0 + c0) * a.ldc;
                if (BF16 && a.vec) {
                    // a lane and its neighbour exchange a token each, so that each writes two columns of one of them
                    const bool odd = lane & 1, ok = (n | 1) < a.N;
                    bf16 *o = a.C16 + at + (n & ~1) + (odd ? a.ldc : 0);
#pragma unroll
                    for (int i = 0; i < 32; i += 2, o += 2 * a.ldc) {
                        const uint32_t x = v[i >> 4][i & 15], y = v[i >> 4][(i & 15) + 1], r = __shfl_xor_sync(0xffffffffu, odd ? x : y, 1);
                        if (i + (odd ? 1 : 0) >= rows) continue;
                        if (ok) *reinterpret_cast<uint32_t *>(o) = odd ? pack_bf16(__uint_as_float(r), __uint_as_float(y)) : pack_bf16(__uint_as_float(x), __uint_as_float(r));
                        else if ((n & ~1) < a.N) *o = __float2bfloat16(__uint_as_float(odd ? r : x));
                    }
                } else if (n < a.N) {
                    float *o = a.C32 + at + n;
                    bf16 *h = a.C16 + at + n;
                    if (!BF16 && rows == 32) {
#pragma unroll
                        for (int i = 0; i < 32; ++i, o += a.ldc) *o = __uint_as_float(v[i >> 4][i & 15]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            if (i >= rows) break;
                            if (BF16) h[(long long)i * a.ldc] = __float2bfloat16(__uint_as_float(v[i >> 4][i & 15]));
                            else o[(long long)i * a.ldc] = __uint_as_float(v[i >> 4][i & 15]);
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(acc_bar + (uint32_t)(b * 8));
            ++j;
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

// One-time (per device) opt-in to the kernels' dynamic shared memory.
static bool configure_once(int which) {          // 0 dense 128-wide, 2 dense 256-wide, 3 / 4 the two with a staged epilogue, 5 / 6 the pair form, 7 / 8 exchanged
    static bool done[10][64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!done[which][dev]) {
        cudaError_t e;
        if (which == 0) e = cudaFuncSetAttribute(gemm_tc_kernel<TC_BN, TC_STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM);
        else if (which == 2) e = cudaFuncSetAttribute(gemm_tc_kernel<TC_WIDE_BN, TC_WIDE_STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      tc_smem_bytes<TC_WIDE_BN, TC_WIDE_STAGES>());
        else if (which == 3) e = cudaFuncSetAttribute(gemm_tc_kernel<TC_BN, TC_STG_STAGES, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      tc_smem_bytes<TC_BN, TC_STG_STAGES, true>());
        else if (which == 4) e = cudaFuncSetAttribute(gemm_tc_kernel<TC_WIDE_BN, TC_WIDE_STAGES, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      tc_smem_bytes<TC_WIDE_BN, TC_WIDE_STAGES, true>());
        else if (which == 5) e = cudaFuncSetAttribute(gemm_tc_pair_kernel<TC_PAIR_STAGES, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      tc_pair_smem_bytes<TC_PAIR_STAGES, false>());
        else if (which == 9) e = cudaFuncSetAttribute(gemm_mix_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MX_SMEM);
        else if (which >= 7) e = cudaFuncSetAttribute(which == 7 ? gemm_tc_exchange_kernel<false> : gemm_tc_exchange_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_pair_smem_bytes<TC_PAIR_STAGES, false>());
        else e = cudaFuncSetAttribute(gemm_tc_pair_kernel<TC_PAIR_STG_STAGES, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      tc_pair_smem_bytes<TC_PAIR_STG_STAGES, true>());
        if (e != cudaSuccess) return false;
        done[which][dev] = true;
    }
    return true;
}

// C [T][ldc] in fp32 or bf16; parts of a split-K product `c_split` elements apart.
static void set_output(GemmTcArgs &a, void *C, int out_bf16, int ldc, long long c_split = 0) {
    a.C32 = out_bf16 ? nullptr : (float *)C;
    a.C16 = out_bf16 ? (bf16 *)C : nullptr;
    a.ldc = ldc;
    a.c_split = c_split;
    const int n = out_bf16 ? 8 : 4;
    a.vec = aligned16((char *)C) && ldc % n == 0 && c_split % n == 0;
}

static int g_wide_min_n = 1024;          // products at least this wide may use the 128 x 256 tile form (0: never)
constexpr int TC_PAIR_MIN_N = 1024;
static int g_pair_min_n = TC_PAIR_MIN_N;          // products at least this wide and of more than 128 rows may use CTA pairs (0: never, negative: always)
static int g_stage_local = 1;            // 1: fp32 output of the wide and pair forms also leaves through the staging buffers

// How many CTAs share a tile: of products of up to 256 rows, whose `tiles` tiles per 128 rows leave most SMs idle (1: none; every
// CTA keeps at least four k blocks).  What that does to a row's bits: the number does not depend on the rows below that line, so
// that a short chunk and its halves give the same rows, and above it every form adds k in one chain, so that they do there as well; the two
// sides differ by the rounding of the sum (a few 1e-6 of the result's size; the split sum is the nearer one to 64 bits).
constexpr int TC_KS_ROWS = 256;
static int ksplit_of(int T, long long tiles, int kblocks) {
    int ks = 1;
    while (T <= TC_KS_ROWS && ks < 8 && tiles * ks * 2 <= NUM_SMS && kblocks >= 8 * ks) ks *= 2;
    return ks;
}
template <int KS>
static int launch_ksplit_of(const CUtensorMap &mA, const CUtensorMap &mW, GemmTcArgs &a, cudaStream_t s) {
    constexpr int smem = tc_smem_bytes<TC_BN, TC_KS_STAGES>();
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!done[dev]) {
        if (cudaFuncSetAttribute(gemm_tc_ksplit_kernel<KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -3;
        done[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(a.total * KS));
    cfg.blockDim = dim3(320);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = KS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, gemm_tc_ksplit_kernel<KS>, mA, mW, a) == cudaSuccess ? 0 : -2;
}
static int launch_ksplit(int ks, const CUtensorMap &mA, const CUtensorMap &mW, GemmTcArgs &a, cudaStream_t s) {
    if (ks == 2) return launch_ksplit_of<2>(mA, mW, a, s);
    if (ks == 4) return launch_ksplit_of<4>(mA, mW, a, s);
    return launch_ksplit_of<8>(mA, mW, a, s);
}

// The form of a plain product.  Few tiles are split over clusters (ksplit_of).  Otherwise the form with the least time by what its tiles
// cost per 64 k values, measured in us: a 256 x 256 tile of a pair of SMs 0.45 (waves over 74 pairs), a 128 x 256 tile of an SM 0.55, a
// 128 x 128 tile 0.31 (bound by the 32 KB it loads; two share an SM and take twice that).  777 x 16480 x 2560: single CTAs 86 us,
// pairs (a quarter of their tiles' area padding) 76; 520 x 12800 x 2560: wide 49, pairs 57 (a third wave for 2 of 150 tiles).  A last
// column tile that is mostly padding rules the wide form out.
enum TcForm { FORM_ONE = 0, FORM_WIDE = 1, FORM_PAIR = 2, FORM_SPLIT = 3 };
static double form_cost(TcForm form, int T, int N) {          // per 64 k values
    auto tiles = [&](int bm, int bn) { return (long long)((T + bm - 1) / bm) * ((N + bn - 1) / bn); };
    auto waves = [](long long n, int at_once) { return (double)((n + at_once - 1) / at_once); };
    if (form == FORM_PAIR) return 0.45 * waves(tiles(TC_PAIR_BM, TC_PAIR_BN), NUM_SMS / 2);
    if (form == FORM_WIDE) return 0.55 * waves(tiles(TC_BM, TC_WIDE_BN), NUM_SMS);
    return 0.31 * waves(tiles(TC_BM, TC_BN), NUM_SMS);
}
static TcForm form_of(int T, int N, int K, bool peers) {
    if (!peers && ksplit_of(T, (N + TC_BN - 1) / TC_BN, (K + TC_BK - 1) / TC_BK) > 1) return FORM_SPLIT;
    const long long n_wide = (long long)((T + TC_BM - 1) / TC_BM) * ((N + TC_WIDE_BN - 1) / TC_WIDE_BN);
    const double c_one = form_cost(FORM_ONE, T, N), c_wide = form_cost(FORM_WIDE, T, N), c_pair = form_cost(FORM_PAIR, T, N);
    const bool wide_ok = g_wide_min_n > 0 && N >= g_wide_min_n && (N % TC_WIDE_BN == 0 || N % TC_WIDE_BN > TC_BN);
    const bool pair_ok = g_pair_min_n && N >= abs(g_pair_min_n) && T > TC_BM;
    if (pair_ok && (g_pair_min_n < 0 || (c_pair < c_one && (!wide_ok || c_pair < c_wide)))) return FORM_PAIR;
    return wide_ok && n_wide >= NUM_SMS / 2 && c_wide < c_one ? FORM_WIDE : FORM_ONE;
}

// Tokens of a tile of the pair form with the operands exchanged, or 0 where that form does not pay (or cannot be: peers' products keep their
// roles).  What a tile of nt tokens costs, by the same measure: 0.07 + 0.00127 nt us, at least 0.21 (256 tokens 0.395, 208 0.33, 160 0.26, 96
// 0.21; 4,096 x 16,480 x 2,560 in tiles of 96 to 256 tokens: 315, 266 (128), 242 (160), 235 (208), 237 us (256), and 260 with the roles kept).  The
// widest of equally cheap tiles is taken: it reads the least.  A caller that moves the line of the pairs measures the forms that keep the roles.
// By these figures an exchanged tile of 256 tokens costs less than a pair's tile that keeps the roles, so that form is left to products between ranks.
static int g_exchange_nt = 0;            // 0: by cost; > 0: that many; < 0: never (measurements and tests)
static int exchanged_tile(int T, int N, int K) {
    if (g_exchange_nt < 0 || g_pair_min_n != TC_PAIR_MIN_N) return 0;
    const TcForm form = form_of(T, N, K, false);
    if (form == FORM_SPLIT) return 0;
    if (g_exchange_nt > 0) return g_exchange_nt;
    auto cost = [&](int nt) {
        const long long n = (long long)((T + nt - 1) / nt) * ((N + 255) / 256), pairs = NUM_SMS / 2;
        return (double)((n + pairs - 1) / pairs) * fmax(0.207, 0.07 + 0.00127 * nt);
    };
    int best = 256;
    for (int nt = 240; nt >= 32; nt -= 16)
        if (cost(nt) < cost(best)) best = nt;
    return cost(best) < form_cost(form, T, N) ? best : 0;
}

static int gemm_plain(GemmTcArgs &a, const void *A, const void *W, void *C, int T, int N, int K, int lda, int ldw, int ldc,
                      int out_bf16, cudaStream_t s) {
    if ((K & 7) || (lda & 7) || (ldw & 7) || ((uintptr_t)A & 15) || ((uintptr_t)W & 15)) return -1;
    const int tiles_t = (T + TC_BM - 1) / TC_BM;
    const TcForm form = a.mix_xn ? FORM_ONE : form_of(T, N, K, a.epi.mode != 0 || a.wait.flags);
    const bool wide = form == FORM_WIDE;
    if (form == FORM_SPLIT) {
        const int ks = ksplit_of(T, (N + TC_BN - 1) / TC_BN, (K + TC_BK - 1) / TC_BK);
        CUtensorMap mA, mW;
        if (!make_map(&mA, A, T, K, lda, TC_BM) || !make_map(&mW, W, N, K, ldw, TC_BN)) return -3;
        set_output(a, C, out_bf16, ldc);
        a.T = T; a.N = N; a.K = K; a.err = g_err_ptr; a.tiles = nullptr;
        a.tiles_t = tiles_t; a.tiles_n = (N + TC_BN - 1) / TC_BN; a.total = a.tiles_t * a.tiles_n;
        a.ksplit = 1; a.kb_per = 0;
        return launch_ksplit(ks, mA, mW, a, s);
    }
    if (const int nt = a.mix_xn || a.epi.mode || a.wait.flags ? 0 : exchanged_tile(T, N, K)) {
        CUtensorMap mX, mW;
        if (!make_map(&mX, A, T, K, lda, nt / 2) || !make_map(&mW, W, N, K, ldw, 128)) return -3;
        set_output(a, C, out_bf16, ldc);
        a.T = T; a.N = N; a.K = K; a.err = g_err_ptr; a.tiles = nullptr;
        a.tiles_t = (T + nt - 1) / nt; a.tiles_n = (N + 255) / 256; a.total = a.tiles_t * a.tiles_n;
        a.ksplit = 1; a.kb_per = 0;
        if (!configure_once(out_bf16 ? 8 : 7)) return -3;
        const unsigned sm_pairs = persistent_grid(1 << 30, 1) / 2, clusters = (unsigned)a.total < sm_pairs ? (unsigned)a.total : sm_pairs;
        constexpr int smem = tc_pair_smem_bytes<TC_PAIR_STAGES, false>();
        if (out_bf16) gemm_tc_exchange_kernel<true><<<2 * clusters, 320, smem, s>>>(mX, mW, a, nt);
        else gemm_tc_exchange_kernel<false><<<2 * clusters, 320, smem, s>>>(mX, mW, a, nt);
        return cudaGetLastError() == cudaSuccess ? 0 : -2;
    }
    if (form == FORM_PAIR) {
        CUtensorMap mA, mW;
        if (!make_map(&mA, A, T, K, lda, TC_BM) || !make_map(&mW, W, N, K, ldw, TC_PAIR_BN / 2)) return -3;
        set_output(a, C, out_bf16, ldc);
        a.T = T; a.N = N; a.K = K; a.err = g_err_ptr; a.tiles = nullptr;
        a.tiles_t = (T + TC_PAIR_BM - 1) / TC_PAIR_BM; a.tiles_n = (N + TC_PAIR_BN - 1) / TC_PAIR_BN; a.total = a.tiles_t * a.tiles_n;
        a.ksplit = 1; a.kb_per = 0;
        const bool staged = a.epi.mode != 0 || (g_stage_local && !out_bf16);
        if (!configure_once(staged ? 6 : 5)) return -3;
        const unsigned sm_pairs = persistent_grid(1 << 30, 1) / 2;          // SMs / 2
        const unsigned clusters = (unsigned)a.total < sm_pairs ? (unsigned)a.total : sm_pairs;
        const unsigned ctas = 2 * clusters;
        if (a.epi.sig.ticket) a.epi.sig.nblocks = ctas;
        if (staged) gemm_tc_pair_kernel<TC_PAIR_STG_STAGES, true><<<ctas, 320, tc_pair_smem_bytes<TC_PAIR_STG_STAGES, true>(), s>>>(mA, mW, a);
        else gemm_tc_pair_kernel<TC_PAIR_STAGES, false><<<ctas, 320, tc_pair_smem_bytes<TC_PAIR_STAGES, false>(), s>>>(mA, mW, a);
        return cudaGetLastError() == cudaSuccess ? 0 : -2;
    }
    const int BN = wide ? TC_WIDE_BN : TC_BN;
    CUtensorMap mA, mW;
    if (!make_map(&mA, A, T, K, lda, TC_BM) || !make_map(&mW, W, N, K, ldw, BN)) return -3;
    set_output(a, C, out_bf16, ldc);
    a.T = T; a.N = N; a.K = K; a.err = g_err_ptr; a.tiles = nullptr;
    a.tiles_t = tiles_t; a.tiles_n = (N + BN - 1) / BN; a.total = a.tiles_t * a.tiles_n;
    a.ksplit = 1; a.kb_per = 0;
    // tiles that leave for other ranks go out as whole 128-byte lines (optionally this GPU's own fp32 tiles of the wide form too)
    const bool staged = a.epi.mode != 0 || (g_stage_local && wide && !out_bf16);
    if (!configure_once(staged ? (wide ? 4 : 3) : (wide ? 2 : 0))) return -3;
    const unsigned grid = persistent_grid(a.total, (wide || staged) ? 1 : 2);
    if (a.epi.sig.ticket) a.epi.sig.nblocks = grid;
    if (staged && wide)
        gemm_tc_kernel<TC_WIDE_BN, TC_WIDE_STAGES, true><<<grid, 320, tc_smem_bytes<TC_WIDE_BN, TC_WIDE_STAGES, true>(), s>>>(mA, mW, a);
    else if (staged)
        gemm_tc_kernel<TC_BN, TC_STG_STAGES, true><<<grid, 320, tc_smem_bytes<TC_BN, TC_STG_STAGES, true>(), s>>>(mA, mW, a);
    else if (wide) gemm_tc_kernel<TC_WIDE_BN, TC_WIDE_STAGES><<<grid, 320, tc_smem_bytes<TC_WIDE_BN, TC_WIDE_STAGES>(), s>>>(mA, mW, a);
    else gemm_tc_kernel<TC_BN, TC_STAGES><<<grid, 320, TC_SMEM, s>>>(mA, mW, a);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Products at least `min_n` columns wide may use the 128 x 256 tile form (0 switches it off; measurements and tests).
QW_API int qwk_gemm_tc_wide_min_n(int min_n) {
    const int old = g_wide_min_n;
    g_wide_min_n = min_n;
    return old;
}

// 1: the wide and pair forms write fp32 output through the staging buffers as well (whole lines per store instruction).
QW_API int qwk_gemm_tc_stage_local(int on) {
    const int old = g_stage_local;
    g_stage_local = on;
    return old;
}

// Products at least `min_n` columns wide and of more than 128 rows may use the CTA-pair form (0 switches it off; a negative number makes
// all of them that are at least -min_n wide and not split use it, whatever it costs: measurements and tests).
QW_API int qwk_gemm_tc_pair_min_n(int min_n) {
    const int old = g_pair_min_n;
    g_pair_min_n = min_n;
    return old;
}

// Tokens of an exchanged tile, a multiple of 16 up to 256 (0: by cost; negative: the form is not used; measurements and tests).  Any other number leaves
// the setting as it is: a wider tile would not fit its stage nor its accumulator, and there is no such shape between the multiples.
QW_API int qwk_gemm_tc_exchange_nt(int nt) {
    const int old = g_exchange_nt;
    if (nt <= 0 || (nt <= 256 && nt % 16 == 0)) g_exchange_nt = nt;
    return old;
}
// Tokens per tile where qwk_gemm_bf16_tc exchanges the operands, 0 where it keeps their roles.
QW_API int qwk_gemm_tc_exchanged(int T, int N, int K) { return exchanged_tile(T, N, K); }

// The form of a product whose operands keep their roles: 0 128 x 128 tiles, 1 128 x 256, 2 CTA pairs, 3 tiles split over a cluster.
QW_API int qwk_gemm_tc_form(int T, int N, int K) { return form_of(T, N, K, false); }

// C = A . W^T.  A bf16 [T][lda], W bf16 [N][ldw], C fp32 (out_bf16 = 0) or bf16 [T][ldc].
// Base addresses 16-byte aligned, lda/ldw multiples of 8 elements, K a multiple of 8.
QW_API int qwk_gemm_bf16_tc(const void *A, const void *W, void *C, int T, int N, int K, int lda, int ldw, int ldc,
                            int out_bf16, cudaStream_t s) {
    if (T <= 0 || N <= 0) return 0;
    GemmTcArgs a{};
    return gemm_plain(a, A, W, C, T, N, K, lda, ldw, ldc, out_bf16, s);
}

// Tensor-parallel forms of the same product (tp.cuh); `tp` is the rank's QwTp channel.
//   wait_kind >= 0 : A lies in the receive buffer of that all-gather kind; the kernel waits for the kind's latest
//                    collective before its first load of A.
//   epi_mode 0     : C as above.
//   epi_mode 1     : the fp32 result goes to every rank's receive buffer of kind `epi_kind` as this rank's part of an
//                    all-reduce (rows of ld_epi floats); C is not written.
//   epi_mode 2     : N = ranks * cols_per_rank; columns go to the rank that owns them, as this rank's part of a
//                    reduce-scatter (rows of cols_per_rank floats, cols_per_rank a multiple of 32); C is not written.
// In modes 1 and 2 the kernel publishes the collective when its last CTA has stored its tiles.
QW_API int qwk_gemm_bf16_tc_tp(void *tp_, const void *A, const void *W, void *C, int T, int N, int K, int lda, int ldw, int ldc,
                               int out_bf16, int wait_kind, int epi_mode, int epi_kind, int ld_epi, cudaStream_t s) {
    if (T <= 0 || N <= 0) return 0;
    QwTp *tp = (QwTp *)tp_;
    GemmTcArgs a{};
    if (!tp || tp->ranks < 1 || tp->ranks > TP_MAX_RANKS) return -1;
    if (wait_kind >= 0) {
        if (wait_kind >= TP_KINDS) return -1;
        a.wait = tp_make_wait(tp, wait_kind);
    }
    if (epi_mode) {
        if (epi_kind < 0 || epi_kind >= TP_KINDS || out_bf16) return -1;
        a.epi.mode = epi_mode;
        a.epi.ranks = tp->ranks;
        if (epi_mode == 2) {
            if (N % tp->ranks) return -1;
            a.epi.cols_per_rank = N / tp->ranks;
            if (a.epi.cols_per_rank & 31) return -1;
            a.epi.ld = a.epi.cols_per_rank;
        } else {
            a.epi.cols_per_rank = 0;
            a.epi.ld = ld_epi;
            if (ld_epi < N) return -1;
        }
        if ((long long)T * a.epi.ld * 4 > tp->part_bytes[epi_kind]) return -1;
        for (int d = 0; d < tp->ranks; ++d) a.epi.dst[d] = (float *)tp_part_on(tp, epi_kind, d);
        a.epi.sig = tp_make_signal(tp, epi_kind, 1);
    }
    return gemm_plain(a, A, W, C, T, N, K, lda, ldw, ldc, out_bf16, s);
}

// From here on the form that keeps its weights: 777 rows 22.6 / 20.5 us, but 400 to 600 18.5 / 20.5 and 1,021 26.7 / 26.6 (a CTA's tiles are few and
// the last ones lonely); 1,500 34.8 / 32.8, 2,048 43 / 39.
constexpr int MX_MIN_T = 1200;
// The mixer's up projection with the block input formed in the epilogue: A bf16 [T][lda] (the activated low-rank vector), W bf16
// [4 SH][ldw] (row 4 c + s: gate of stream s, column c), xn bf16 [T][4][SH]; out bf16 [T][ld_out]: mean over the streams of
// sigmoid(A . W^T) * xn.  The logits (fp32, 4 SH a row) are never stored: as a product and a kernel that read them back
// 118 us at 4096 x 2560 and 41 at 1021, here 70 and 27.  Below MX_MIN_T 128 x 128 tiles: two CTAs on an SM have the warps that
// the epilogue wants (with 128 x 256 tiles 8 to 10 % more from 300 rows on).  SH a multiple of 8.
QW_API int qwk_gemm_mix_tc(const void *A, const void *W, const void *xn, int SH, void *out, int ld_out, int T, int K, int lda, int ldw,
                           cudaStream_t s) {
    if (T <= 0) return 0;
    if ((SH & 7) || (ld_out & 7) || ((uintptr_t)xn & 15) || ((uintptr_t)out & 15)) return -1;
    GemmTcArgs a{};
    a.mix_xn = (const bf16 *)xn;
    a.mix_cols = SH;
    if (K <= MX_KB * TC_BK && T >= MX_MIN_T) {
        if ((K & 7) || (lda & 7) || (ldw & 7) || ((uintptr_t)A & 15) || ((uintptr_t)W & 15)) return -1;
        CUtensorMap mA, mW;
        if (!make_map(&mA, A, T, K, lda, TC_BM) || !make_map(&mW, W, 4 * SH, K, ldw, 256)) return -3;
        set_output(a, out, 1, ld_out);
        a.T = T; a.N = 4 * SH; a.K = K; a.err = g_err_ptr;
        a.tiles_t = (T + TC_BM - 1) / TC_BM; a.tiles_n = (4 * SH + 255) / 256; a.total = a.tiles_t * a.tiles_n;
        if (!configure_once(9)) return -3;
        gemm_mix_tc_kernel<<<persistent_grid(a.total, 1), MX_THREADS, MX_SMEM, s>>>(mA, mW, a);
        return cudaGetLastError() == cudaSuccess ? 0 : -2;
    }
    return gemm_plain(a, A, W, out, T, 4 * SH, K, lda, ldw, ld_out, 1, s);
}

// Grouped form for expert-sorted rows: A bf16 [rows][lda] holds the rows of group after group, W bf16
// [w_rows][ldw] the groups' weight matrices one after another (Nw rows each), tiles (device, int4 x max_tiles)
// lists {first A row, valid rows (0 = unused entry), first W row of the group, 0} per 128-row tile.
// C[row][0..Nw) = A[row] . W_group^T.
QW_API int qwk_gemm_bf16_tc_grouped(const void *A, const void *W, void *C, const void *tiles, int max_tiles, int rows,
                                    long long w_rows, int Nw, int K, int lda, int ldw, int ldc, int out_bf16,
                                    cudaStream_t s) {
    if (rows <= 0 || max_tiles <= 0) return 0;
    if ((K & 7) || (lda & 7) || (ldw & 7) || ((uintptr_t)A & 15) || ((uintptr_t)W & 15)) return -1;
    CUtensorMap mA, mW;
    if (!make_map(&mA, A, rows, K, lda, TC_BM) || !make_map(&mW, W, w_rows, K, ldw, TC_BN)) return -3;
    GemmTcArgs a{};
    set_output(a, C, out_bf16, ldc);
    a.T = rows; a.N = Nw; a.K = K; a.err = g_err_ptr; a.tiles = (const int4 *)tiles;
    a.tiles_t = max_tiles; a.tiles_n = (Nw + TC_BN - 1) / TC_BN; a.total = a.tiles_t * a.tiles_n;
    a.ksplit = 1; a.kb_per = 0;
    if (!configure_once(0)) return -3;
    gemm_tc_kernel<TC_BN, TC_STAGES><<<persistent_grid(a.total), 320, TC_SMEM, s>>>(mA, mW, a);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Split-K form for products with few output tiles and a long K (the mixers' down projection): C_s = A[:, K_s] . W[:, K_s]^T
// for ksplit shares of K, partial s written as fp32 to C + s * c_split (elements); the consumer adds the partials in
// order, so the sum does not depend on timing.  ksplit <= number of k blocks.
QW_API int qwk_gemm_bf16_tc_splitk(const void *A, const void *W, float *C, int T, int N, int K, int lda, int ldw, int ldc,
                                   int ksplit, long long c_split, cudaStream_t s) {
    if (T <= 0 || N <= 0) return 0;
    const int kblocks = (K + TC_BK - 1) / TC_BK;
    if ((K & 7) || (lda & 7) || (ldw & 7) || ((uintptr_t)A & 15) || ((uintptr_t)W & 15) || ksplit < 1 || ksplit > kblocks) return -1;
    CUtensorMap mA, mW;
    if (!make_map(&mA, A, T, K, lda, TC_BM) || !make_map(&mW, W, N, K, ldw, TC_BN)) return -3;
    GemmTcArgs a{};
    set_output(a, C, 0, ldc, c_split);
    a.T = T; a.N = N; a.K = K; a.err = g_err_ptr; a.tiles = nullptr;
    a.tiles_t = (T + TC_BM - 1) / TC_BM; a.tiles_n = (N + TC_BN - 1) / TC_BN;
    a.kb_per = (kblocks + ksplit - 1) / ksplit;
    a.ksplit = (kblocks + a.kb_per - 1) / a.kb_per;          // every share holds at least one k block
    if (a.ksplit != ksplit) return -1;
    a.total = a.tiles_t * a.tiles_n * a.ksplit;
    const int ks = ksplit_of(T, (long long)a.tiles_n * a.ksplit, a.kb_per);
    if (ks > 1) return launch_ksplit(ks, mA, mW, a, s);
    if (!configure_once(0)) return -3;
    gemm_tc_kernel<TC_BN, TC_STAGES><<<persistent_grid(a.total), 320, TC_SMEM, s>>>(mA, mW, a);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
