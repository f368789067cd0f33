// Shared device helpers for the sm_100a kernels: warp/block reductions, bf16 packing, the
// exact q4 -> bf16 pair conversion, activation functions, bounded waits and the row tables
// that batched-decode kernels take.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define QW_API extern "C" __attribute__((visibility("default")))

namespace qw {

typedef __nv_bfloat16 bf16;
typedef __nv_bfloat162 bf162;

constexpr int MAX_ROWS = 32;       // rows of one batched decode step
constexpr int KV_PAGE = 256;       // tokens per KV page (also the prefix-cache block size)
constexpr int RAW_RING = 16;       // raw indexer keys kept per slot and layer
constexpr int GDN_RING = 16;       // pre-conv rows kept per slot and layer
constexpr int PLE_RING = 32;       // normalised conv inputs kept per slot
constexpr int LIST_CAP = 2048 + 8; // attended tokens per query: 512 groups x 4 + open tail

// Error word shared by every kernel that can give up (bounded waits, bounds checks).  Kernels
// never trap: they record a code here (first writer wins) and return.
struct ErrorWord {
    unsigned int code;      // 0 = ok
    unsigned int detail;
};
enum ErrCode : unsigned int {
    ERR_NONE = 0,
    ERR_WAIT_TIMEOUT = 1,   // a flag / mbarrier wait ran out
    ERR_BOUNDS = 2,         // a data-derived index was out of range (checked builds)
    ERR_CAPACITY = 3,       // a table or list was too small
};
__device__ __forceinline__ void report(ErrorWord *e, unsigned int code, unsigned int detail) {
    if (e && atomicCAS(&e->code, 0u, code) == 0u) e->detail = detail;
}
// Checked builds (-DQW_DEVICE_CHECKS, the library libqw_kernels_checked.so): indices that come from data - token ids,
// positions, page numbers - are validated where they are used.  A violation records ERR_BOUNDS with `detail` in the
// error word and the kernel skips the access and returns; nothing traps, so the context stays usable and the host reads
// the word like any other kernel failure.  Without the flag the checks compile to nothing.  A translation unit that uses
// QW_DCHECK registers itself with QW_DCHECK_TU(name); qwk_set_error_word then hands the word's address to every one of
// them (each unit keeps its own copy: the library is built without relocatable device code).
// (Role of the reference's QW_DCHECK, src/kernels/common.cuh:13-24, which traps instead.)
#ifdef QW_DEVICE_CHECKS
static __device__ __attribute__((unused)) ErrorWord *s_dcheck_word = nullptr;
#define QW_DCHECK(cond, detail)                                             \
    do {                                                                    \
        if (!(cond)) {                                                      \
            report(s_dcheck_word, ERR_BOUNDS, (unsigned int)(detail));      \
            return;                                                         \
        }                                                                   \
    } while (0)
#define QW_DCHECK_TU(name)                                                                                  \
    extern "C" __attribute__((visibility("default"))) int qw_dcheck_set_##name(void *p) {                   \
        return cudaMemcpyToSymbol(qw::s_dcheck_word, &p, sizeof(p)) == cudaSuccess ? 0 : -2;                \
    }
#else
#define QW_DCHECK(cond, detail) \
    do {                        \
    } while (0)
#define QW_DCHECK_TU(name)
#endif

// Device address of the error word every launcher hands to its kernel (set once by the host through
// qwk_set_error_word; null until then, in which case kernels only give up silently).
extern ErrorWord *g_err_ptr;
// host side: asks the next expert gate/up launch to also form the shared expert's activation from the router's outputs
// (a few extra blocks of that launch, in parallel with the routed experts) instead of the router's last block doing it
// in its serial tail.  rs == null: nothing extra.
struct SharedAct {
    const float *rs;     // [M][ld_rs]: router logits (E) | shared gate logit | shared gate rows (SF) | shared up rows (SF)
    int ld_rs, E, SF;
    void *sh_h;          // out: [M][SF] bf16
};
extern SharedAct g_shared_act;
inline SharedAct take_shared_act() {
    SharedAct r = g_shared_act;
    g_shared_act = SharedAct{nullptr, 0, 0, 0, nullptr};
    return r;
}
extern int *g_moe_stats;     // host side: where the next routing launch adds its count of local pairs (null = nowhere)

// Row tables of a batched step.  Row i appends one token to slot[i] at position pos[i]; rows of
// one slot are consecutive and run_start[i] is the first row of that slot's run.
struct Rows {
    int M;
    const int *slot;        // [M]
    const int *pos;         // [M]
    const int *run_start;   // [M]
    const int *run_len;     // [M] (valid at the first row of a run)
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sum over a block of NT threads (NT a multiple of 32, <= 1024); every thread gets the result.
// Fixed order: lanes by xor-shuffle, then warps 0..n-1 serially.
template <int NT>
__device__ __forceinline__ float block_sum(float v, float *scratch /* >= 32 floats */) {
    v = warp_sum(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) scratch[w] = v;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NT / 32; ++i) s += scratch[i];
    return s;
}

// 1 / (1 + e^-x): the hardware's reciprocal and one step of Newton's method.  (As a division the compiler adds a branch per value, which no
// other value's instructions fill: the mixer's up projection at 100 rows 15.4 us, so 12.3; the experts' gate/up product at 4,096 tokens 458, so
// 396.)  Error against 64 bits: the division's, to every digit of its largest and its mean (|x| up to 1, 4, 10, 30, 80).  Below x = -87.2, where the
// reciprocal leaves the normal numbers, it is taken of 2^-32 of the sum: the division keeps those results too.  (The mixer's up projection at 4,096 rows
// 68.0 us without that, 69.0 with it.)
__device__ __forceinline__ float sigmoidf_(float x) {
    float e, y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -1.4426950408889634f));
    const float d = 1.f + e;
    const bool usual = d < 8.5e37f;          // not: infinity and NaN, either; the step has nothing to correct there
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d * (usual ? 1.f : 0x1p-32f)));
    return usual ? fmaf(y, fmaf(-d, y, 1.f), y) : y * 0x1p-32f;
}
__device__ __forceinline__ float siluf_(float x) { return x * sigmoidf_(x); }
__device__ __forceinline__ float softplusf_(float x) { return x > 20.f ? x : log1pf(__expf(x)); }

__device__ __forceinline__ float bf16_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    bf162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&h);
}

// V neighbouring columns of a row: V = 4 as one access (16-byte aligned floats, 8-byte aligned bf16), V = 1 for any width and address.
template <int V>
__device__ __forceinline__ void ld_cols(const float *p, float (&v)[V]) {
    if constexpr (V == 4) {
        const float4 t = *reinterpret_cast<const float4 *>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
        v[0] = *p;
    }
}
template <int V>
__device__ __forceinline__ void ld_cols(const bf16 *p, float (&v)[V]) {
    if constexpr (V == 4) {
        const uint2 t = *reinterpret_cast<const uint2 *>(p);
        v[0] = bf16_lo(t.x); v[1] = bf16_hi(t.x); v[2] = bf16_lo(t.y); v[3] = bf16_hi(t.y);
    } else {
        v[0] = __bfloat162float(*p);
    }
}
template <int V>
__device__ __forceinline__ void st_cols(float *p, const float (&v)[V]) {
    if constexpr (V == 4) *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else *p = v[0];
}
template <int V>
__device__ __forceinline__ void st_cols(bf16 *p, const float (&v)[V]) {
    if constexpr (V == 4) *reinterpret_cast<uint2 *>(p) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
    else *p = __float2bfloat16(v[0]);
}
// host side: do all of these start on 16 bytes (null does)
template <typename... P>
inline bool aligned16(const P *...p) { return ((reinterpret_cast<uintptr_t>(p) | ...) & 15) == 0; }

// Streaming 16-byte load that does not allocate in L1 (weights are read once).
__device__ __forceinline__ uint4 ld_stream(const void *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ld_stream8(const void *p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

// q4 engine order: elements 2j and 2j+1 of a word sit at bits 4j and 16+4j.  (w >> 4j) & 0x000F000F
// OR 0x43004300 is the bf16 pair (128+n_even, 128+n_odd); subtracting 136 gives the exact values.
__device__ __forceinline__ void q4_pair(uint32_t w, int j, float &e0, float &e1) {
    uint32_t p = ((w >> (4 * j)) & 0x000F000Fu) | 0x43004300u;
    e0 = bf16_lo(p) - 136.f;
    e1 = bf16_hi(p) - 136.f;
}
// Same as a packed bf16 pair (exact: the integers -8..7 are representable).
__device__ __forceinline__ uint32_t q4_pair_bf16(uint32_t w, int j) {
    uint32_t p = ((w >> (4 * j)) & 0x000F000Fu) | 0x43004300u;
    bf162 v = *reinterpret_cast<bf162 *>(&p);
    bf162 off = __floats2bfloat162_rn(136.f, 136.f);
    bf162 r = __hsub2(v, off);
    return *reinterpret_cast<uint32_t *>(&r);
}

// dot of 8 bf16 weights (uint4) with 8 bf16 activations (uint4), fp32 accumulate, fixed order
__device__ __forceinline__ float dot8(const uint4 &w, const uint4 &x, float acc) {
    acc = fmaf(bf16_lo(w.x), bf16_lo(x.x), acc);
    acc = fmaf(bf16_hi(w.x), bf16_hi(x.x), acc);
    acc = fmaf(bf16_lo(w.y), bf16_lo(x.y), acc);
    acc = fmaf(bf16_hi(w.y), bf16_hi(x.y), acc);
    acc = fmaf(bf16_lo(w.z), bf16_lo(x.z), acc);
    acc = fmaf(bf16_hi(w.z), bf16_hi(x.z), acc);
    acc = fmaf(bf16_lo(w.w), bf16_lo(x.w), acc);
    acc = fmaf(bf16_hi(w.w), bf16_hi(x.w), acc);
    return acc;
}

// ---- programmatic dependent launch (PDL) -------------------------------------------------
// Every kernel of the decode step is launched with the programmatic-stream-serialization
// attribute.  A kernel first lets its successor start (pdl_trigger), prefetches weights — which
// no kernel writes — and only then waits for its predecessor to finish and flush (pdl_wait)
// before it touches activations.  Every block must reach pdl_wait before it exits: a grid that
// completes without waiting would let its successor run ahead of the grid before it.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

// The same with clusters of `cl` CTAs along x.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl_cluster(void (*kernel)(KArgs...), int cl, dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)cl;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

constexpr int NUM_SMS = 148;

// NeoX rotation angle tables: cos/sin for (pos, i) computed in double like the oracle.
__device__ __forceinline__ void rope_cs(int pos, int i, int rope_dim, double theta, float &c, float &s) {
    double inv = pow(theta, -2.0 * double(i) / double(rope_dim));
    double a = double(pos) * inv;
    double sd, cd;
    sincos(a, &sd, &cd);
    c = float(cd);
    s = float(sd);
}

}  // namespace qw
