// Chunked (WY) gated delta rule for token-major prefill: the recurrent scan of a run of M tokens done as
// dense 64-token chunk products on the tensor cores, with the state in fp32.
//
// The reference only has the token-by-token scan (gdn_scan_T, src/kernels/gdn.hip:229-309) and lists the
// chunked form as future work (its design document under docs/, line 512).  Math (per value head, state S [128 k][128 v], chunk of
// C = 64 rows, entry state S0, g_t = sum_{s<=t} log decay_s):
//
//     A[t,s] = beta_t exp(g_t - g_s) (k_t . k_s)       s <  t
//     (I + A) Wv = diag(beta) V      (I + A) Wk = diag(beta exp(g)) K
//     P[t,s] = exp(g_t - g_s) (q_t . k_s)              s <= t
//     U  = Wv - Wk S0
//     O  = diag(exp(g)) Q S0 + P U
//     S1 = exp(g_C) S0 + (diag(exp(g_C - g)) K)^T U
//
// Three launches per layer:
//   1. gdn_chunk_prep_kernel   grid (chunks, VL): everything that does not depend on the state (A, Wv, Wk, P, g),
//      all chunks in parallel.  K K^T and Q K^T on mma.sync tf32; the two triangular solves by forward substitution in
//      fp32, a column of each per thread.
//   2. gdn_chunk_apply_kernel  grid (2, VL): walks the chunks in order with the state of one head's 64 value
//      columns in registers; three tf32 products per chunk.  The value columns of a head are independent in
//      every state-dependent product, so a head is split over two blocks.
//   3. gdn_chunk_norm_kernel   grid (M, VL): gated RMS norm over the head's 128 outputs -> bf16.
//
// The run must be one slot's: rows 0..M-1 of the batch are consecutive positions of slot[0].  Rows past M in
// the last chunk are masked (beta = 0, decay = 1, q = k = 0), which leaves the state untouched.
#include "common.cuh"

namespace qw {

constexpr int CD = 128;          // head dim (keys and values)
constexpr int CC = 64;           // rows per chunk
// Row strides of shared tiles: 4 mod 32 words, so that the eight 16-byte rows of an ldmatrix lie in different banks ...
constexpr int LDA = CD + 4;      // [.][128]
constexpr int LDP = CC + 4;      // [.][64]
constexpr int LDT = CD + 8;      // ... and 8 mod 32 for the tile that is read down its columns

__device__ __forceinline__ uint32_t tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const float *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm2(uint32_t &r0, uint32_t &r1, const float *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
// A 32-bit element is two of ldmatrix's: an 8 x 8 matrix is 8 rows x 4 values, and lane (g = lane / 4, t = lane % 4) gets row g's value t.
// This lane's row address of a 16 x 8 operand-A tile: the four matrices are (rows 0-7 | 8-15) x (k 0-3, then 4-7) ...
__device__ __forceinline__ const float *a_row(const float *m, int ld, int r0, int lane) {
    return m + (r0 + (lane & 7) + (lane & 8)) * ld + (lane >> 4) * 4;
}
// ... and of two operand-B tiles whose columns are the matrix's rows n0 .. n0 + 15: (n 0-7: k 0-3, k 4-7), (n 8-15: k 0-3, k 4-7).
__device__ __forceinline__ const float *b_row(const float *m, int ld, int n0, int lane) {
    return m + (n0 + (lane & 7) + (lane >> 4) * 8) * ld + ((lane >> 3) & 1) * 4;
}
__device__ __forceinline__ void round4(uint32_t (&r)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = tf32(__uint_as_float(r[i]));
}

struct GdnChunkArgs {
    const float *qkv;            // [M][qkv_l]  q (KL heads) | k (KL heads) | v (VL heads), after conv / norm
    const float *decay, *beta;   // [M][VL]
    const float *proj;           // z gate: proj[m][qkv_l + h*128 + d]
    int ld_proj;
    float *S;                    // [slots][VL][128 k][128 v]
    const float *norm_w;         // [128]
    int KL, VL, M;
    const int *slot;             // slot[0] = the run's slot
    float *Wk, *Wv;              // scratch [chunks][VL][64][128]; Wk rounded to tf32
    float *P;                    // scratch [chunks][VL][64][64], rounded to tf32
    float *G;                    // scratch [chunks][VL][64]   cumulative log decay
    float *Oraw;                 // scratch [M][VL*128]
    bf16 *o;                     // [M][VL*128]
    float eps;
};

// 16-byte asynchronous copy global -> shared; `ok` false: the destination is zero-filled (rows past the run's end).
__device__ __forceinline__ void cp_async16(float *dst, const float *src, bool ok) {
    const unsigned int d = (unsigned int)__cvta_generic_to_shared(dst);
    const int n = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Rows [m0, m0+64) x 128 floats at column offset col of the qkv rows -> shared tile of stride ld, asynchronously; rows
// >= M become zero.  256 threads.
template <int TH = 256>
__device__ __forceinline__ void load_tile_async(float *dst, int ld, const float *qkv, int qkv_l, int col, int m0, int M, int tid) {
#pragma unroll
    for (int i = 0; i < 2048 / TH; ++i) {
        const int idx = tid + i * TH;           // float4 index: 64 rows x 32
        const int r = idx >> 5, c4 = idx & 31;
        const bool ok = m0 + r < M;
        cp_async16(dst + r * ld + c4 * 4, qkv + (long long)(ok ? m0 + r : 0) * qkv_l + col + c4 * 4, ok);
    }
}

// ------------------------------------------------------------------------------------------------
// 1. state-independent part of every chunk
// ------------------------------------------------------------------------------------------------
// Forward substitution in fp32, a column of Wv and a column of Wk per thread: a 16-byte shared load (four cycles, although its lanes share it) serves
// eight multiply-adds.  As products with T = (I + A)^-1 in two tf32 parts Wv was 3.3 times as far from 64 bits as by substitution, for the
// tensor core's sums cut off.  The whole scan, 48 heads, one column a thread / those products / now: 4,096 tokens 840 / 605 / 591 us, 1,021
// 235 / 171 / 165, 100 77 / 40 / 44.
constexpr int PREP_THREADS = 128, HC_ = CC / 2;
constexpr int PREP_SMEM = (2 * CC * LDA + 3 * CC) * 4;      // 68 KB: three blocks per SM

__global__ void __launch_bounds__(PREP_THREADS, 3) gdn_chunk_prep_kernel(GdnChunkArgs a) {
    extern __shared__ __align__(16) float sm[];
    float *Ks = sm;                      // [64][LDA]
    float *Qs = Ks + CC * LDA;           // [64][LDA]
    float *As = Qs;                      // [64][LDP]  takes Q's place once Q K^T is done
    float *gs = Qs + CC * LDA;           // [64] cumulative log decay
    float *bs = gs + CC;                 // [64] beta
    float *be = bs + CC;                 // [64] beta exp(g)
    const int ch = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int qkv_l = (2 * a.KL + a.VL) * CD;
    const int kh = h / (a.VL / a.KL);
    const int m0 = ch * CC;
    load_tile_async<PREP_THREADS>(Ks, LDA, a.qkv, qkv_l, (a.KL + kh) * CD, m0, a.M, tid);
    load_tile_async<PREP_THREADS>(Qs, LDA, a.qkv, qkv_l, kh * CD, m0, a.M, tid);
    cp_async_commit();
    if (w == 0) {
        const int r0 = 2 * lane, r1 = r0 + 1;
        float x0 = 0.f, x1 = 0.f, b0 = 0.f, b1 = 0.f;
        if (m0 + r0 < a.M) {
            x0 = fmaxf(__logf(a.decay[(long long)(m0 + r0) * a.VL + h]), -87.f);
            b0 = a.beta[(long long)(m0 + r0) * a.VL + h];
        }
        if (m0 + r1 < a.M) {
            x1 = fmaxf(__logf(a.decay[(long long)(m0 + r1) * a.VL + h]), -87.f);
            b1 = a.beta[(long long)(m0 + r1) * a.VL + h];
        }
        float s = x0 + x1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float n = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += n;
        }
        gs[r0] = s - x1;
        gs[r1] = s;
        bs[r0] = b0;
        bs[r1] = b1;
        be[r0] = b0 * __expf(s - x1);
        be[r1] = b1 * __expf(s);
    }
    cp_async_wait<0>();
    __syncthreads();
    // K K^T and Q K^T: 16 rows per warp; tiles above the diagonal stay zero
    const int r0 = w * 16;
    float akk[8][4], aqk[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) akk[n][i] = aqk[n][i] = 0.f;
    {
        const float *ka = a_row(Ks, LDA, r0, lane), *qa = a_row(Qs, LDA, r0, lane), *kb = b_row(Ks, LDA, 0, lane);
#pragma unroll 2
        for (int k0 = 0; k0 < CD; k0 += 8) {
            uint32_t fk[4], fq[4];
            ldsm4(fk, ka + k0); ldsm4(fq, qa + k0);
            round4(fk); round4(fq);
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                if (n > w) break;
                uint32_t b[4];
                ldsm4(b, kb + n * 16 * LDA + k0);
                round4(b);
                mma_tf32(akk[2 * n], fk, b[0], b[1]); mma_tf32(akk[2 * n + 1], fk, b[2], b[3]);
                mma_tf32(aqk[2 * n], fq, b[0], b[1]); mma_tf32(aqk[2 * n + 1], fq, b[2], b[3]);
            }
        }
    }
    // column tid of V, the first half of its rows: on their way under what follows
    const float *v = a.qkv + (long long)m0 * qkv_l + (2 * a.KL + h) * CD + tid;
    float wv[HC_], wk[HC_], nv[HC_];
    auto fetch_v = [&](int o) {
#pragma unroll
        for (int r = 0; r < HC_; ++r) nv[r] = m0 + o + r < a.M ? v[(long long)(o + r) * qkv_l] : 0.f;
    };
    fetch_v(0);
    __syncthreads();                     // every warp is done reading Q before A overwrites it
    float *Pg = a.P + ((long long)ch * a.VL + h) * CC * CC;
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
            const int r = r0 + g + (i >> 1) * 8, c = n * 8 + 2 * t;
            const float d0 = c <= r ? __expf(gs[r] - gs[c]) : 0.f, d1 = c + 1 <= r ? __expf(gs[r] - gs[c + 1]) : 0.f;
            *reinterpret_cast<float2 *>(As + r * LDP + c) = make_float2(c < r ? bs[r] * d0 * akk[n][i] : 0.f, c + 1 < r ? bs[r] * d1 * akk[n][i + 1] : 0.f);
            *reinterpret_cast<float2 *>(Pg + r * CC + c) =
                make_float2(__uint_as_float(tf32(c <= r ? d0 * aqk[n][i] : 0.f)), __uint_as_float(tf32(c + 1 <= r ? d1 * aqk[n][i + 1] : 0.f)));
        }
    if (tid < CC) a.G[((long long)ch * a.VL + h) * CC + tid] = gs[tid];
    __syncthreads();
    // The rows in two halves by the same code (all 64 unrolled are 80 KB of instructions, which a short run waits for: the scan of 100 tokens 62 us, so 44).
    // What the first half's rows add to the second's sums waits in this thread's own columns of shared memory.
    float *sv = Ks + tid, *sk = As + CC * LDP + tid;       // [32][LDA]: K's first rows are consumed by then; [32][128]: the rest of Q's place
#pragma unroll 1
    for (int o = 0; o < CC; o += HC_) {
        const float *A = As + o * LDP + o;
#pragma unroll
        for (int r = 0; r < HC_; ++r) {
            wv[r] = bs[o + r] * nv[r];
            wk[r] = be[o + r] * Ks[(o + r) * LDA + tid];
        }
#pragma unroll
        for (int r = 0; r < HC_; ++r) {
            // four chains each: a row's sum is r / 4 dependent multiply-adds deep
            float av[4] = {o ? sv[r * LDA] : 0.f, 0.f, 0.f, 0.f}, ak[4] = {o ? sk[r * CD] : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int s4 = 0; s4 < r; s4 += 4) {
                const float4 f = *reinterpret_cast<const float4 *>(A + r * LDP + s4);
                const float x[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (s4 + e < r) {
                        av[e] = fmaf(x[e], wv[s4 + e], av[e]);
                        ak[e] = fmaf(x[e], wk[s4 + e], ak[e]);
                    }
            }
            wv[r] -= (av[0] + av[1]) + (av[2] + av[3]);
            wk[r] -= (ak[0] + ak[1]) + (ak[2] + ak[3]);
        }
        const long long at = (((long long)ch * a.VL + h) * CC + o) * CD + tid;
#pragma unroll
        for (int r = 0; r < HC_; ++r) {
            a.Wv[at + r * CD] = wv[r];
            a.Wk[at + r * CD] = __uint_as_float(tf32(wk[r]));
        }
        if (o) break;
        fetch_v(HC_);
#pragma unroll 2
        for (int r = 0; r < HC_; ++r) {
            float av[4] = {0.f, 0.f, 0.f, 0.f}, ak[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int s4 = 0; s4 < HC_; s4 += 4) {
                const float4 f = *reinterpret_cast<const float4 *>(As + (HC_ + r) * LDP + s4);
                const float x[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    av[e] = fmaf(x[e], wv[s4 + e], av[e]);
                    ak[e] = fmaf(x[e], wk[s4 + e], ak[e]);
                }
            }
            sv[r * LDA] = (av[0] + av[1]) + (av[2] + av[3]);
            sk[r * CD] = (ak[0] + ak[1]) + (ak[2] + ak[3]);
        }
    }
}

// ------------------------------------------------------------------------------------------------
// 2. state-dependent part: one block per (half of the value columns, head) walks the chunks
// ------------------------------------------------------------------------------------------------
// NC = value columns of the state per block (64, 32 or 16): the value columns of a head are independent in every
// state-dependent product, so a head is split over 128 / NC blocks; with few heads per rank (tensor parallel) a finer
// split keeps the number of blocks up.  Every output element's sum runs over k in the same order whatever NC is.
template <int NC>
constexpr int apply_smem() {
    return (NC * LDA + 2 * CC * LDA + 2 * CC * LDT + 2 * CC * LDP + NC * LDP + 3 * CC) * 4;
}

// The kernel walks the chunks in order; what a chunk needs from global memory (Wk, Q, P, K and the cumulative log decays) is fetched with
// cp.async under the second and third product of the chunk before it.  The chain of 64 chunk steps of a 4,096-token run is what bounds the
// kernel (it does not shorten with fewer heads per rank), so nothing on it waits for a global load, and a step has two meetings.
// The state stays in fp32 in the accumulators of the product that updates it, transposed (value columns x keys): a warp owns
// 8 or 16 keys.  What other warps read of it, and of U, lies rounded to tf32 in shared memory with k along the rows, so that ldmatrix
// brings an operand in one instruction where single loads and conversions took ten.
// 4,096 tokens, 48 heads: 400 us, now 343 (1,021: 106, 89; with 16 warps 420).
template <int NC>
constexpr int apply_threads() { return 256; }
template <int NC>
__global__ void __launch_bounds__(apply_threads<NC>()) gdn_chunk_apply_kernel(GdnChunkArgs a) {
    constexpr int TH = apply_threads<NC>(), NW = TH / 32;
    constexpr int NT = NC / 2 / NW;      // 8-column tiles of a warp in the row-tiled products (NW / 4 warps beside each other)
    constexpr int MT = NC / 16, KN = 16 / NW;      // 16-row and 8-column tiles of a warp's part of the state
    extern __shared__ __align__(16) float sm[];
    float *St = sm;                      // [NC][LDA]      state, this block's value columns x keys
    float *Wks = St + NC * LDA;          // [64][LDA]
    float *Qs = Wks + CC * LDA;          // [64][LDA]
    float *Ks = Qs + CC * LDA;           // [2][64][LDT]   chunk c in buffer c & 1
    float *Ps = Ks + 2 * CC * LDT;       // [2][64][LDP]
    float *Ut = Ps + 2 * CC * LDP;       // [NC][LDP]      U, value columns x rows of the chunk
    float *gb = Ut + NC * LDP;           // [2][64]        cumulative log decay g_t of the chunk
    float *ek = gb + 2 * CC;             // [64]           exp(g_C - g_t)
    const int vh = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int qkv_l = (2 * a.KL + a.VL) * CD;
    const int kh = h / (a.VL / a.KL);
    const int slot = a.slot[0];
    float *Sg = a.S + ((long long)slot * a.VL + h) * CD * CD + vh * NC;
    const int nch = (a.M + CC - 1) / CC;
    auto fetch = [&](int ch) {
        const long long cb = (long long)ch * a.VL + h;
        const int m0 = ch * CC;
        load_tile_async<TH>(Qs, LDA, a.qkv, qkv_l, kh * CD, m0, a.M, tid);
        load_tile_async<TH>(Wks, LDA, a.Wk + cb * CC * CD, CD, 0, 0, CC, tid);
        load_tile_async<TH>(Ks + (ch & 1) * CC * LDT, LDT, a.qkv, qkv_l, (a.KL + kh) * CD, m0, a.M, tid);
        const float *Pg = a.P + cb * CC * CC;
        float *Pd = Ps + (ch & 1) * CC * LDP;
#pragma unroll
        for (int i = 0; i < 1024 / TH; ++i) {
            const int idx = tid + i * TH;       // float4 index: 64 rows x 16
            const int r = idx >> 4, c4 = idx & 15;
            cp_async16(Pd + r * LDP + c4 * 4, Pg + r * CC + c4 * 4, true);
        }
        if (tid < CC / 4) cp_async16(gb + (ch & 1) * CC + tid * 4, a.G + cb * CC + tid * 4, true);
        cp_async_commit();
    };
    fetch(0);
    // accS[i][n]: value columns 16 i + g, + 8; keys k0w + 8 n + 2 t, + 1
    float accS[MT][KN][4];
    const int k0w = w * 8 * KN;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int n = 0; n < KN; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) accS[i][n][e] = Sg[(long long)(k0w + n * 8 + 2 * t + (e & 1)) * CD + i * 16 + g + (e >> 1) * 8];
    auto publish = [&]() {               // the state as the next chunk's operand
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int n = 0; n < KN; ++n)
#pragma unroll
                for (int e = 0; e < 4; e += 2)
                    *reinterpret_cast<float2 *>(St + (i * 16 + g + e * 4) * LDA + k0w + n * 8 + 2 * t) =
                        make_float2(__uint_as_float(tf32(accS[i][n][e])), __uint_as_float(tf32(accS[i][n][e + 1])));
    };
    publish();
    const int r0 = (w & 3) * 16, c0 = (w >> 2) * (8 * NT);
    const float *wa = a_row(Wks, LDA, r0, lane), *qa = a_row(Qs, LDA, r0, lane), *sb = b_row(St, LDA, c0, lane), *ub = b_row(Ut, LDP, c0, lane);
    for (int ch = 0; ch < nch; ++ch) {
        const int m0 = ch * CC;
        const long long cb = (long long)ch * a.VL + h;
        const float *gc = gb + (ch & 1) * CC;
        // Wv of this thread's U elements: issued now, used after the first product
        const float *Wvg = a.Wv + cb * CC * CD + vh * NC;
        float2 wv0[NT], wv1[NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const int c = c0 + n * 8 + 2 * t;
            wv0[n] = *reinterpret_cast<const float2 *>(Wvg + (r0 + g) * CD + c);
            wv1[n] = *reinterpret_cast<const float2 *>(Wvg + (r0 + g + 8) * CD + c);
        }
        cp_async_wait<0>();
        __syncthreads();                 // this chunk's tiles and the state are there
        // U = Wv - Wk S0 and Q S0: warp tile 16 rows x NC / 2 value columns
        float accW[NT][4], accO[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) accW[n][i] = accO[n][i] = 0.f;
#pragma unroll 4
        for (int k0 = 0; k0 < CD; k0 += 8) {
            uint32_t fw[4], fq[4];
            ldsm4(fw, wa + k0);
            ldsm4(fq, qa + k0);
            round4(fq);
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                uint32_t b[4];
                if (NT > 1) ldsm4(b, sb + n * 8 * LDA + k0);
                else ldsm2(b[0], b[1], sb + k0);
                mma_tf32(accW[n], fw, b[0], b[1]);
                mma_tf32(accO[n], fq, b[0], b[1]);
                if (NT > 1) {
                    mma_tf32(accW[n + 1 < NT ? n + 1 : n], fw, b[2], b[3]);
                    mma_tf32(accO[n + 1 < NT ? n + 1 : n], fq, b[2], b[3]);
                }
            }
        }
        const float gC = gc[CC - 1];
        {
            if (tid < CC) ek[tid] = __expf(gC - gc[tid]);
            const float e0 = __expf(gc[r0 + g]), e1 = __expf(gc[r0 + g + 8]);
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                float *u = Ut + (c0 + n * 8 + 2 * t) * LDP + r0 + g;
                u[0] = __uint_as_float(tf32(wv0[n].x - accW[n][0]));
                u[LDP] = __uint_as_float(tf32(wv0[n].y - accW[n][1]));
                u[8] = __uint_as_float(tf32(wv1[n].x - accW[n][2]));
                u[LDP + 8] = __uint_as_float(tf32(wv1[n].y - accW[n][3]));
                accO[n][0] *= e0; accO[n][1] *= e0;
                accO[n][2] *= e1; accO[n][3] *= e1;
            }
        }
        __syncthreads();                 // U is complete; the Q and Wk tiles and the state's copy are free
        if (ch + 1 < nch) fetch(ch + 1);
        // O += P U (P is zero above the diagonal: k tiles past the warp's rows are skipped)
        {
            const float *pa = a_row(Ps + (ch & 1) * CC * LDP, LDP, r0, lane);
#pragma unroll 2
            for (int k0 = 0; k0 < r0 + 16; k0 += 8) {
                uint32_t fp[4];
                ldsm4(fp, pa + k0);
#pragma unroll
                for (int n = 0; n < NT; n += 2) {
                    uint32_t b[4];
                    if (NT > 1) ldsm4(b, ub + n * 8 * LDP + k0);
                    else ldsm2(b[0], b[1], ub + k0);
                    mma_tf32(accO[n], fp, b[0], b[1]);
                    if (NT > 1) mma_tf32(accO[n + 1 < NT ? n + 1 : n], fp, b[2], b[3]);
                }
            }
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int c = h * CD + vh * NC + c0 + n * 8 + 2 * t;
                const int ra = m0 + r0 + g, rb = ra + 8;
                if (ra < a.M) *reinterpret_cast<float2 *>(a.Oraw + (long long)ra * a.VL * CD + c) = make_float2(accO[n][0], accO[n][1]);
                if (rb < a.M) *reinterpret_cast<float2 *>(a.Oraw + (long long)rb * a.VL * CD + c) = make_float2(accO[n][2], accO[n][3]);
            }
        }
        // S1^T = exp(g_C) S0^T + U^T diag(ek) K
        {
            const float eC = __expf(gC);
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int n = 0; n < KN; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) accS[i][n][e] *= eC;
            const float *kp = Ks + (ch & 1) * CC * LDT + t * LDT + k0w + g;
            const float *ua = a_row(Ut, LDP, 0, lane);
#pragma unroll 2
            for (int s0 = 0; s0 < CC; s0 += 8) {
                const float ea = ek[s0 + t], eb = ek[s0 + t + 4];
                uint32_t b[KN][2];
#pragma unroll
                for (int n = 0; n < KN; ++n) {
                    b[n][0] = tf32(kp[s0 * LDT + n * 8] * ea);
                    b[n][1] = tf32(kp[(s0 + 4) * LDT + n * 8] * eb);
                }
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    uint32_t fu[4];
                    ldsm4(fu, ua + i * 16 * LDP + s0);
#pragma unroll
                    for (int n = 0; n < KN; ++n) mma_tf32(accS[i][n], fu, b[n][0], b[n][1]);
                }
            }
        }
        publish();
    }
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int n = 0; n < KN; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) Sg[(long long)(k0w + n * 8 + 2 * t + (e & 1)) * CD + i * 16 + g + (e >> 1) * 8] = accS[i][n][e];
}

// ------------------------------------------------------------------------------------------------
// 3. gated RMS norm over each head's 128 outputs
// ------------------------------------------------------------------------------------------------
// A warp per (row, head), four values per lane (a block of 128 with two meetings per head and row took 121 us at 4096 x 48, this 44).
template <bool VEC>
__global__ void __launch_bounds__(256) gdn_chunk_norm_kernel(GdnChunkArgs a) {
    const long long i = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= (long long)a.M * a.VL) return;
    const int m = (int)(i / a.VL), h = (int)(i - (long long)m * a.VL), c = (threadIdx.x & 31) * 4;
    const int qkv_l = (2 * a.KL + a.VL) * CD;
    const float4 o = *reinterpret_cast<const float4 *>(a.Oraw + i * CD + c);
    const float *wp = a.norm_w + c, *zp = a.proj + (long long)m * a.ld_proj + qkv_l + h * CD + c;
    float4 w, z;
    if (VEC) {
        w = *reinterpret_cast<const float4 *>(wp);
        z = *reinterpret_cast<const float4 *>(zp);
    } else {                                                     // rows of the projection that do not start on 16 bytes
        w = make_float4(wp[0], wp[1], wp[2], wp[3]);
        z = make_float4(zp[0], zp[1], zp[2], zp[3]);
    }
    const float r = rsqrtf(warp_sum(fmaf(o.x, o.x, o.y * o.y) + fmaf(o.z, o.z, o.w * o.w)) / float(CD) + a.eps);
    *reinterpret_cast<uint2 *>(a.o + i * CD + c) =
        make_uint2(pack_bf16(o.x * r * w.x * sigmoidf_(z.x), o.y * r * w.y * sigmoidf_(z.y)), pack_bf16(o.z * r * w.z * sigmoidf_(z.z), o.w * r * w.w * sigmoidf_(z.w)));
}

}  // namespace qw

using namespace qw;

// The scan of one slot's run of M rows (rows 0..M-1 consecutive positions of slot[0]): same inputs and outputs
// as qwk_gdn_scan without the per-row state saves.  `scratch` holds
// 4 * (ceil(M / 64) * VL * (2 * 64 * 128 + 64 * 64 + 64) + M * VL * 128) bytes.
QW_API int qwk_gdn_scan_chunked(const float *qkv, const float *decay, const float *beta, const float *proj, int ld_proj,
                                float *S, const float *norm_w, int KL, int VL, int M, const int *slot, float *scratch,
                                void *o, float eps, cudaStream_t s) {
    if (M < 1 || KL < 1 || VL % KL != 0) return -1;
    static bool attr_done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!attr_done[dev]) {
        if (cudaFuncSetAttribute(gdn_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PREP_SMEM) != cudaSuccess ||
            cudaFuncSetAttribute(gdn_chunk_apply_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, apply_smem<64>()) != cudaSuccess ||
            cudaFuncSetAttribute(gdn_chunk_apply_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, apply_smem<32>()) != cudaSuccess ||
            cudaFuncSetAttribute(gdn_chunk_apply_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, apply_smem<16>()) != cudaSuccess)
            return -3;
        attr_done[dev] = true;
    }
    const long long nch = (M + CC - 1) / CC;
    GdnChunkArgs a;
    a.qkv = qkv; a.decay = decay; a.beta = beta; a.proj = proj; a.ld_proj = ld_proj; a.S = S; a.norm_w = norm_w;
    a.KL = KL; a.VL = VL; a.M = M; a.slot = slot; a.eps = eps; a.o = (bf16 *)o;
    a.Wk = scratch;
    a.Wv = a.Wk + nch * VL * CC * CD;
    a.P = a.Wv + nch * VL * CC * CD;
    a.G = a.P + nch * VL * CC * CC;
    a.Oraw = a.G + nch * VL * CC;
    gdn_chunk_prep_kernel<<<dim3((unsigned)nch, VL), PREP_THREADS, PREP_SMEM, s>>>(a);
    // blocks of the sequential walk: 128 / NC per head, NC chosen so that about a hundred blocks run
    if (VL >= 32) gdn_chunk_apply_kernel<64><<<dim3(2, VL), apply_threads<64>(), apply_smem<64>(), s>>>(a);
    else if (VL >= 16) gdn_chunk_apply_kernel<32><<<dim3(4, VL), 256, apply_smem<32>(), s>>>(a);
    else gdn_chunk_apply_kernel<16><<<dim3(8, VL), 256, apply_smem<16>(), s>>>(a);
    const unsigned blocks = (unsigned)(((long long)M * VL + 7) / 8);
    if ((ld_proj & 3) == 0 && aligned16(proj, norm_w)) gdn_chunk_norm_kernel<true><<<blocks, 256, 0, s>>>(a);
    else gdn_chunk_norm_kernel<false><<<blocks, 256, 0, s>>>(a);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
