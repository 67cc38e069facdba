// Shared declarations of the htree_b200 kernels: parameter blocks, storage-type helpers, block primitives.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <mutex>

#include "../../include/htree_b200.h"

namespace htree {

constexpr float kNegInf = -1.0e10f;      // HTREE_SCORE_NEG_INF of the reference (src/parallel.py:75)
constexpr float kHasMass = 1.0e-10f;     // "has contribution" guard of the level merge (src/parallel.py:289-314)
constexpr float kForcedImportance = 1.0e6f;  // importance given to the right-most candidate (src/parallel.py:745)

// Everything the attention kernels need, passed by value as a __grid_constant__ block.
struct AttnParams {
    const void* q;
    const void* lk[HTREE_MAX_LEVELS];
    const void* lv[HTREE_MAX_LEVELS];
    const void* lkr[HTREE_MAX_LEVELS];   // keys pre-rotated by their child index (16-bit storage types only), or NULL
    const void* lvb[HTREE_MAX_LEVELS];   // values re-laid-out per parent block for the P.V fragments (tree.cu), or NULL
    const void* lkb[HTREE_MAX_LEVELS];   // pre-rotated keys per parent block in fragment-major order (tree.cu), or NULL
    const void* blk[HTREE_MAX_LEVELS];   // operand blocks of the transposed kernels (tform.cuh), or NULL
    const void* vkblk[HTREE_MAX_LEVELS]; // their backward part, or NULL
    const void* tab;                     // rotary table of the transposed kernels, rows [cos | sin]: IEEE half times scale, or fp32 (split-half)
    float* ktop;                         // rotated keys of the top level (select_top.cu), or NULL
    int32_t first_level;                 // fwd_generic_kernel: where it starts, the lists of that level given; 0 = the top
    const void* tab32;                   // fp32 rows [cos | sin] for the selection kernel
    int32_t sel_maxc;                    // most candidates of a group on a level that selects (set by the selection's launch)
    int32_t ln[HTREE_MAX_LEVELS];   // N_l
    int64_t lpow[HTREE_MAX_LEVELS]; // CR^l
    const float* cosc;
    const float* sinc;
    const __half* cosh;   // optional: cos * scale and sin * scale as IEEE half, same shape as cosc/sinc
    const __half* sinh;
    int32_t* parents[HTREE_MAX_LEVELS];  // may be all NULL in the forward
    int32_t* status;
    // forward outputs
    void* out;
    float* gmax;
    float* gsum;
    float* tr_max;
    float* tr_sum;
    float* tr_out;
    // backward inputs / outputs
    const void* dO;
    float* dq;          // fp32 dq (the reference's contract), or NULL when dq_typed is set
    void* dq_typed;     // dq in the storage type of q, or NULL
    float* dk[HTREE_MAX_LEVELS];
    float* dv[HTREE_MAX_LEVELS];
    int32_t B, T, H, Hkv, K, V, CR, TK, L, G, n_pos;
    // single-level mode of the generic forward (per-kernel compatibility surface): only level `level_index` runs, its
    // parent lists come from parents_in and the kept nodes go to next_out; the per-level state goes to tr_* slot 0
    const int32_t* parents_in;
    int32_t* next_out;
    int32_t level_mode, level_index;
    int32_t Tq, t0;   // query window: rows 0..Tq-1 of q/out are sequence positions t0..t0+Tq-1
    float scale;
    uint32_t flags;
};

// The fp32 arithmetic that decides selections outside the tensor cores, one rounding each: a pair of a key or of a query rotated by
// (cos, sin), and a term of a score.  Kernels that have to select alike use these, not expressions: which of two products is contracted
// with their sum is up to the compiler, and it took another one for keys than for queries (kept here: the bits of earlier builds).
__device__ __forceinline__ void rotate_key_f32(float lo, float hi, float cs, float sn, float& x, float& y) {
    x = __fmaf_rn(lo, cs, -__fmul_rn(hi, sn));
    y = __fmaf_rn(lo, sn, __fmul_rn(hi, cs));
}
__device__ __forceinline__ void rotate_query_f32(float lo, float hi, float cs, float sn, float& x, float& y) {
    x = __fmaf_rn(lo, cs, -__fmul_rn(hi, sn));
    y = __fmaf_rn(hi, cs, __fmul_rn(lo, sn));
}
__device__ __forceinline__ float score_term(float q, float k, float sum) { return __fmaf_rn(q, k, sum); }

template <typename T> __device__ __forceinline__ float to_f(T x);
template <> __device__ __forceinline__ float to_f<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <> __device__ __forceinline__ float to_f<__half>(__half x) { return __half2float(x); }

template <typename T> __device__ __forceinline__ T from_f(float x);
template <> __device__ __forceinline__ float from_f<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ __half from_f<__half>(float x) { return __float2half_rn(x); }

// Four consecutive elements as floats with one vector load (pointer must be aligned to 4 elements).
template <typename T> __device__ __forceinline__ void load4(const T* p, float (&o)[4]);
template <> __device__ __forceinline__ void load4<float>(const float* p, float (&o)[4]) {
    float4 x = __ldg(reinterpret_cast<const float4*>(p));
    o[0] = x.x; o[1] = x.y; o[2] = x.z; o[3] = x.w;
}
template <> __device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, float (&o)[4]) {
    uint2 x = __ldg(reinterpret_cast<const uint2*>(p));
    o[0] = __uint_as_float(x.x << 16); o[1] = __uint_as_float(x.x & 0xffff0000u);
    o[2] = __uint_as_float(x.y << 16); o[3] = __uint_as_float(x.y & 0xffff0000u);
}
template <> __device__ __forceinline__ void load4<__half>(const __half* p, float (&o)[4]) {
    uint2 x = __ldg(reinterpret_cast<const uint2*>(p));
    float2 a = __half22float2(*reinterpret_cast<__half2*>(&x.x));
    float2 b = __half22float2(*reinterpret_cast<__half2*>(&x.y));
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Exclusive scan of one flag per thread over the block, in thread order.  `wtot` is shared scratch of NT/32 ints.
// Returns the number of set flags in lower threads; *total receives the block total.  Two barriers.
template <int NT>
__device__ __forceinline__ int block_scan_flag(bool f, int* wtot, int* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned m = __ballot_sync(0xffffffffu, f);
    if (lane == 0) wtot[w] = __popc(m);
    __syncthreads();
    int before = 0, tot = 0;
#pragma unroll
    for (int i = 0; i < NT / 32; ++i) {
        int c = wtot[i];
        if (i < w) before += c;
        tot += c;
    }
    __syncthreads();
    *total = tot;
    return before + __popc(m & ((1u << lane) - 1u));
}

void note_launch(int n = 1);   // diagnostic launch counter (api.cu)

// The operator's launches depend on one another in a chain, and the small ones are as long as the gap between two of them.  A chained
// launch is set up while its predecessor ends (programmatic dependent launch): its first act is to wait until that one's writes are
// visible, and everything behind chain_enter() is ordered as by the stream.  Predecessors do not let it begin sooner: blocks that waited
// early took their places wherever the predecessor had left room, and launches of less than a chip's worth of blocks then ran several to
// an SM beside empty ones (123 -> 153 us for a dq of 2020 queries; 110 drawn calls of all sizes: 6% on the geometric mean).
// A decode call 76 -> 69 us, a forward of 2048 positions 117 -> 106.
__device__ __forceinline__ void chain_enter() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
template <typename... P>
int launch_chained_clusters(void (*kernel)(P...), int cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t st, const P&... args) {
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster; at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cfg.attrs = at; cfg.numAttrs = cluster > 1 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e == cudaSuccess) note_launch(); else cudaGetLastError();     // (returned; not left behind for an unrelated call to report)
    return (int)e;
}
// ... of `CL` blocks a cluster along x, or, where the device has no room for such a cluster, of one
template <typename... P>
int launch_clusters(void (*kernel)(P...), int CL, dim3 grid, dim3 block, size_t smem, cudaStream_t st, const P&... args) {
    const int rc = launch_chained_clusters(kernel, CL, dim3(grid.x * CL, grid.y), block, smem, st, args...);
    if (rc == 0 || CL == 1) return rc;
    return launch_chained_clusters(kernel, 1, grid, block, smem, st, args...);
}
template <typename... P>
int launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const P&... args) {
    return launch_chained_clusters(kernel, 1, grid, block, smem, st, args...);
}

// Blocks of a cluster (along x) that work on one query: rank, barrier and the other blocks' shared memory.
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t x; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(x)); return x; }
__device__ __forceinline__ uint32_t cluster_blocks() { uint32_t x; asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(x)); return x; }
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {         // p, in this block's shared memory, of block `rank`
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ float ld_cluster(uint32_t a) { float x; asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(a) : "memory"); return x; }
__device__ __forceinline__ float2 ld_cluster2(uint32_t a) {
    float2 x;
    asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];" : "=f"(x.x), "=f"(x.y) : "r"(a) : "memory");
    return x;
}
__device__ __forceinline__ void st_cluster(uint32_t a, uint32_t x) { asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(a), "r"(x) : "memory"); }

// Exact Top-K over non-negative floats, whose bit patterns order like the values: search for the TK-th largest key by counting the keys at
// or above a probe, in the bracket [lo, hi) that the smallest and the largest key span (one forced key above hi left out of it).  The next
// probe is where the logit of the count, interpolated over the bit patterns, reaches TK, every fourth one the middle: 5 to 8 counts where
// bisecting the 31 bits takes 13 to 21.
struct TopKBound {
    uint32_t tau;      // keys above are kept
    int need;          // and this many of those equal to it, the smallest positions
    bool exact;        // none equal to it is
};
template <typename Count>
__device__ __forceinline__ TopKBound topk_search(Count count, uint32_t lo, uint32_t hi, int nc, int TK) {
    int c_lo = nc, c_hi = 1;
    if (TK == 1) { hi = 0x7f800000u; c_hi = 0; }       // only the forced candidate is kept
    bool exact = false;
    auto logit = [&](int c) { return __log2f(__fdividef((float)c - 0.25f, (float)(nc - c) + 0.75f)); };
    const float want = logit(TK);
    float f_lo = logit(c_lo), f_hi = logit(c_hi < 1 ? 1 : c_hi);
    for (int it = 0; hi - lo > 1u; ++it) {
        uint32_t x = lo + ((hi - lo) >> 1);
        if ((it & 3) != 3) {
            const float f = fminf(fmaxf(__fdividef(f_lo - want, f_lo - f_hi), 0.f), 1.f);
            x = lo + (uint32_t)(f * (float)(hi - lo));
            x = x <= lo ? lo + 1u : x >= hi ? hi - 1u : x;
        }
        const int c = count(x);
        if (c == TK) { lo = x - 1u; c_hi = TK; exact = true; break; }    // the kept keys are those at or above x
        if (c > TK) { lo = x; f_lo = logit(c); } else { hi = x; c_hi = c; f_hi = logit(c < 1 ? 1 : c); }
    }
    return TopKBound{lo, TK - c_hi, exact};
}

// Parent lists: int32 with -1 for "none" (the reference's layout), or uint16 with 0xFFFF under HTREE_PARENTS_U16.
__device__ __forceinline__ int load_parent(const AttnParams& p, int l, int64_t idx) {
    if (p.flags & HTREE_PARENTS_U16) {
        const uint16_t v = reinterpret_cast<const uint16_t*>(p.parents[l])[idx];
        return v == 0xFFFFu ? -1 : (int)v;
    }
    return p.parents[l][idx];
}
__device__ __forceinline__ void store_parent(const AttnParams& p, int l, int64_t idx, int v) {
    if (p.flags & HTREE_PARENTS_U16) reinterpret_cast<uint16_t*>(p.parents[l])[idx] = v < 0 ? (uint16_t)0xFFFFu : (uint16_t)v;
    else p.parents[l][idx] = v;
}

// A kernel's dynamic shared-memory limit per device, raised when a launch needs more than any before it (setting the attribute
// on every launch costs as much as a third of the launch).  One object per kernel.
class SmemLimit {
    std::mutex m_;
    std::atomic<size_t> have_[64] = {};

  public:
    cudaError_t raise(const void* kernel, size_t bytes) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        if (dev < 64 && have_[dev].load(std::memory_order_acquire) >= bytes) return cudaSuccess;
        std::lock_guard<std::mutex> lock(m_);
        if (dev < 64 && have_[dev].load(std::memory_order_relaxed) >= bytes) return cudaSuccess;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e == cudaSuccess && dev < 64) have_[dev].store(bytes, std::memory_order_release);
        if (e != cudaSuccess) cudaGetLastError();
        return e;
    }
};

constexpr uint32_t kFlagSplitOk = 1u << 30;   // internal: a forward whose selections are not kept for a backward

// transposed tensor-core kernels (operands.cu, acc_mma.cu)
bool pack_supported(int dtype, int K, int V, int CR);
bool pack_split(int dtype, int D);                       // split-half operands?
size_t pack_block_bytes(int D, bool x3, int CR);         // bytes of one forward block
int launch_pack_listed(const HtreeShape& s, int Tq, const void* k, const void* v, void* blk, const void* parents, bool narrow,
                       const float* cosc, const float* sinc, cudaStream_t st);
int launch_pack_blocks(const HtreeShape& s, int first, int L, const int32_t* ln, void* const* lk, void* const* lv, void* const* blk,
                       void* const* vkblk, bool pool, const float* cosc, const float* sinc, cudaStream_t st);
int64_t top_keys_bytes(const HtreeShape& s, int L, const int32_t* ln);       // select_top.cu
int launch_select_top(const AttnParams& p, int dtype, bool sums, cudaStream_t st);
bool fwd_generic_tiled(const AttnParams& p);             // does fwd_generic_kernel take its tiled form?
bool select_blk_supported(const AttnParams& p, int dtype);
int launch_select_blk(const AttnParams& p, int dtype, cudaStream_t st);
bool select_mma_supported(const AttnParams& p, int dtype);
bool acc_mma_supported(const AttnParams& p, int dtype);
int launch_acc_mma(const AttnParams& p, int dtype, cudaStream_t st);

// launchers implemented in the .cu files (return cudaError_t as int)
int launch_tree_build(const HtreeShape& s, int L, const int32_t* ln, void* const* lk, void* const* lv, cudaStream_t st);
// typed_dk / typed_dv: NULL, or buffers of the storage type that receive the finished leaf gradients (the cast is fused
// into the last streaming pass; the fp32 level-0 buffers then only hold the accumulators)
int launch_tree_backward(const HtreeShape& s, int L, const int32_t* ln, float* const* dk, float* const* dv, cudaStream_t st,
                         void* typed_dk = nullptr, void* typed_dv = nullptr);
int launch_rotate_keys(const HtreeShape& s, int L, const int32_t* ln, void* const* lk, void* const* lkr, const float* cosc,
                       const float* sinc, cudaStream_t st);
int launch_fwd_generic(const AttnParams& p, int dtype, cudaStream_t st);
int launch_merge_to_global(const float* lmax, const float* lsum, const float* lout, float* gmax, float* gsum, float* gout,
                           int64_t rows, int V, cudaStream_t st);
int launch_final_normalize(const float* gout, const float* gsum, void* out, int dtype, int64_t rows, int V, cudaStream_t st);
int launch_block_values(const HtreeShape& s, int L, const int32_t* ln, void* const* lv, void* const* lvb, cudaStream_t st);
int launch_block_keys(const HtreeShape& s, int L, const int32_t* ln, void* const* lkr, void* const* lkb, cudaStream_t st);

// Element order inside a block of the blocked values: fragment-major ([16-byte piece][lane]) for 128-wide heads with 16
// children per parent and a 16-bit storage type (read through shared memory by the pipelined forward), lane-major
// (each lane's pieces consecutive) otherwise.
template <int D, int CR, bool SPLIT>
constexpr bool kFragmentMajor = (D == 128 && CR == 16 && !SPLIT);
bool fwd_mma_supported(const AttnParams& p, int dtype);
int launch_fwd_mma(const AttnParams& p, int dtype, cudaStream_t st);
bool bwd_mma_supported(const AttnParams& p, int dtype);
int launch_bwd_mma(const AttnParams& p, int dtype, cudaStream_t st);
bool bwd_generic_supported(const AttnParams& p, int dtype);
int launch_bwd_generic(const AttnParams& p, int dtype, cudaStream_t st);

}  // namespace htree
