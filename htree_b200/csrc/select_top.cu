// Selection of the top pooled level in fp32 arithmetic, for the shapes whose selections are made that way (32-wide heads, fp32 storage
// with 128-wide heads).  Every query's candidates are the level's nodes in their order, so a key's position is its index: the keys are
// rotated once (rotate_top_keys_kernel) and the scores are a dense product, eight queries against 128 nodes at a time.  Levels below
// take their lists from here (fwd_generic.cu).
//
// The selections are fwd_generic_kernel's: rotate_key_f32, rotate_query_f32 and score_term in the same order of dimensions (ffma2: two
// heads' terms, each half rounded like the scalar one), its importance sums in both their forms, an exact Top-K.  The forms: a maximum
// and a sum per candidate (kPerNode, where a level's scores exceed that kernel's shared memory), or sums relative to the level's maximum, which is known behind
// the last score: the scores are computed twice (kTwice; keeping them in shared memory left 8 of 24 warps an SM: 161 -> 183 us).
//
// One warp per query: 4 nodes a lane, all heads; keys from a tile in shared memory that the block's warps share.  Bound by the
// shared-memory reads: 2 GP + 8 wavefronts for the 4 GP packed multiply-adds of a pair of dimensions, 12 cycles an SM for a node and a
// group of 8 heads of 128 where one thread per node, reading its row and its table row from memory, took 140.  4096 positions, 2 groups
// of 8 heads of 128: 537 -> 161 us; 12000 positions, 4 groups of 4 heads of 32, 750 nodes: 1390 -> 214 us.
#include "mma_common.cuh"

namespace htree {

constexpr int kTopTile = 128, kTopPairs = 16;          // nodes and pairs of dimensions of a tile in shared memory
enum TopForm { kPerNode, kTwice };

struct TopKeysArgs {
    const void* k;             // [B, N, Hkv, D]
    float* out;                // [B, Hkv][tile][pair][lo, hi][128 nodes]
    const float* cosc;
    const float* sinc;
    int32_t N, Hkv, units;
};
template <typename T, int D>
__global__ void __launch_bounds__(128) rotate_top_keys_kernel(const __grid_constant__ TopKeysArgs a) {
    chain_enter();
    constexpr int HALF = D / 2;
    const int tile = blockIdx.x, unit = blockIdx.y, node = tile * kTopTile + threadIdx.x, d0 = blockIdx.z * 8;
    float* out = a.out + ((int64_t)unit * gridDim.x + tile) * (D * kTopTile) + threadIdx.x;
    const int64_t row = ((int64_t)(unit / a.Hkv) * a.N + node) * a.Hkv + unit % a.Hkv;
#pragma unroll
    for (int d = d0; d < d0 + 8; d += 4) {
        float lo[4] = {0.f, 0.f, 0.f, 0.f}, hi[4] = {0.f, 0.f, 0.f, 0.f}, cs[4] = {0.f, 0.f, 0.f, 0.f}, sn[4] = {0.f, 0.f, 0.f, 0.f};
        if (node < a.N) {
            load4<T>(reinterpret_cast<const T*>(a.k) + row * D + d, lo);
            load4<T>(reinterpret_cast<const T*>(a.k) + row * D + d + HALF, hi);
            load4<float>(a.cosc + (int64_t)node * HALF + d, cs);
            load4<float>(a.sinc + (int64_t)node * HALF + d, sn);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            float x, y;
            rotate_key_f32(lo[u], hi[u], cs[u], sn[u], x, y);
            out[(2 * (d + u)) * kTopTile] = x;
            out[(2 * (d + u) + 1) * kTopTile] = y;
        }
    }
}

// shared memory: two tiles of keys; per warp the rotated query, importances and (kPerNode) maxima of its nodes
__host__ __device__ inline size_t top_warp_bytes(int D, int GP, int nodes, TopForm form) {
    return (size_t)D * GP * 4 + (size_t)nodes * (form == kPerNode ? 8 : 4);
}
constexpr size_t kTopKeyBytes = 2 * (size_t)kTopPairs * 2 * kTopTile * 4;

template <typename T, int D, int GP, TopForm FORM>
__global__ void __launch_bounds__(256) select_top_kernel(const __grid_constant__ AttnParams p) {
    chain_enter();
    constexpr int HALF = D / 2, CHUNKS = HALF / kTopPairs;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, QW = blockDim.x >> 5;
    const int l = p.L - 1, N = p.ln[l], nodes = (N + kTopTile - 1) / kTopTile * kTopTile, TK = p.TK, G = p.G;
    const int b = blockIdx.y / p.Hkv, hk = blockIdx.y % p.Hkv;
    const int t0 = (int)(gridDim.x - 1 - blockIdx.x) * QW, tl = t0 + warp;               // (the longest first)
    const bool on = tl < p.Tq;
    const int last = min(t0 + QW, p.Tq) - 1;
    const int nc = on ? (int)((int64_t)(p.t0 + tl) / p.lpow[l]) + 1 : 0, rp = nc - 1;       // nodes 0..rp: a query's candidates
    const int most = (int)((int64_t)(p.t0 + last) / p.lpow[l]) + 1;                         // of the block's queries
    float* keys = reinterpret_cast<float*>(smem_raw);
    float* qT = reinterpret_cast<float*>(smem_raw + kTopKeyBytes + warp * top_warp_bytes(D, GP, nodes, FORM));   // [pair][lo, hi][GP]
    uint32_t* key = reinterpret_cast<uint32_t*>(qT + D * GP);
    float* mj = reinterpret_cast<float*>(key + nodes);                       // kPerNode
    const int64_t hbase = ((int64_t)b * p.Tq + tl) * p.H + (int64_t)hk * G, qidx = ((int64_t)b * p.Tq + tl) * p.Hkv + hk;

    if (on) {
        for (int i = lane; i < GP * HALF; i += 32) {
            const int g = i / HALF, d = i - g * HALF;
            float a = 0.f, c = 0.f;
            if (g < G) {
                const T* q = reinterpret_cast<const T*>(p.q) + (hbase + g) * D;
                const float lo = to_f(q[d]), hi = to_f(q[d + HALF]);
                const float cs = __ldg(p.cosc + (int64_t)rp * HALF + d), sn = __ldg(p.sinc + (int64_t)rp * HALF + d);
                rotate_query_f32(lo, hi, cs, sn, a, c);
                a *= p.scale; c *= p.scale;
            }
            qT[2 * d * GP + g] = a;
            qT[(2 * d + 1) * GP + g] = c;
        }
        const int np = rp / p.CR + 1;                  // virtual parents of the top level (src/parallel.py:1026-1038)
        for (int i = lane; i < TK; i += 32) store_parent(p, l, qidx * TK + i, i < np ? i : -1);
    }
    if (most <= TK) {                                  // every candidate of every query is kept
        if (on) for (int i = lane; i < TK; i += 32) store_parent(p, l - 1, qidx * TK + i, i < nc ? i : -1);
        return;
    }

    const float* src = p.ktop + (int64_t)blockIdx.y * nodes * D;
    const int total = (most + kTopTile - 1) / kTopTile * CHUNKS;                            // pieces of 16 pairs, tile by tile
    auto fetch = [&](int i, int buf) {
        constexpr int BYTES = kTopPairs * 2 * kTopTile * 4;
        const unsigned char* s = reinterpret_cast<const unsigned char*>(src) + (int64_t)i * BYTES;
        const uint32_t dst = smem_u32(keys) + buf * BYTES;
        for (int o = threadIdx.x * 16; o < BYTES; o += blockDim.x * 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + o), "l"(s + o) : "memory");
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    float M = -INFINITY;
    for (int pass = 0; pass < (FORM == kTwice ? 2 : 1); ++pass) {
        float tmax = -INFINITY;
        float2 acc[GP / 2][4];
        __syncthreads();
        fetch(0, 0);
#pragma unroll 1
        for (int i = 0; i < total; ++i) {
            if (i % CHUNKS == 0) {
#pragma unroll
                for (int g = 0; g < GP / 2; ++g)
#pragma unroll
                    for (int u = 0; u < 4; ++u) acc[g][u] = make_float2(0.f, 0.f);
            }
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            __syncthreads();                           // this piece is there, and everybody is done with the one before
            if (i + 1 < total) fetch(i + 1, (i + 1) & 1);
            const int j0 = i / CHUNKS * kTopTile + 4 * lane;
            if (i / CHUNKS * kTopTile >= nc) continue;
            const float* kp = keys + (i & 1) * (kTopPairs * 2 * kTopTile) + 4 * lane;
            const float* qp = qT + (i % CHUNKS) * (kTopPairs * 2 * GP);
#pragma unroll 4
            for (int d = 0; d < 2 * kTopPairs; ++d) {  // lo and hi dimension of a pair, one after the other
                const float4 k4 = *reinterpret_cast<const float4*>(kp + d * kTopTile);
                const float kk[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
                for (int g = 0; g < GP; g += 4) {
                    const float4 q4 = *reinterpret_cast<const float4*>(qp + d * GP + g);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        acc[g / 2][u] = ffma2(make_float2(q4.x, q4.y), make_float2(kk[u], kk[u]), acc[g / 2][u]);
                        acc[g / 2 + 1][u] = ffma2(make_float2(q4.z, q4.w), make_float2(kk[u], kk[u]), acc[g / 2 + 1][u]);
                    }
                }
            }
            if (i % CHUNKS != CHUNKS - 1) continue;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + u;
                if (j >= nc) continue;
                auto S = [&](int g) { return g & 1 ? acc[g / 2][u].y : acc[g / 2][u].x; };
                if (FORM != kTwice || pass == 0) {
                    float m = -INFINITY;
#pragma unroll
                    for (int g = 0; g < GP; ++g) if (g < G) m = fmaxf(m, S(g));
                    tmax = fmaxf(tmax, m);
                    if constexpr (FORM == kPerNode) {
                        float e = 0.f;
#pragma unroll
                        for (int g = 0; g < GP; ++g) if (g < G) e += expf(S(g) - m);
                        mj[j] = m; key[j] = __float_as_uint(e);
                    }
                } else {
                    float s = 0.f;
#pragma unroll
                    for (int g = 0; g < GP; ++g) if (g < G) s += expf(S(g) - M);
                    key[j] = __float_as_uint(j == rp ? kForcedImportance : s);
                }
            }
        }
        if (pass == 0) M = warp_max(tmax);
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    if (!on) return;
    __syncwarp();
    if (nc <= TK) {
        for (int i = lane; i < TK; i += 32) store_parent(p, l - 1, qidx * TK + i, i < nc ? i : -1);
        return;
    }
    uint32_t lo = 0xffffffffu, hi = 0u;
    for (int j = lane; j < nc; j += 32) {
        uint32_t k = key[j];
        if constexpr (FORM == kPerNode) {
            const float s = __uint_as_float(k) * expf(mj[j] - M);
            key[j] = k = __float_as_uint(j == rp ? kForcedImportance : s);
        }
        if (j != rp) { lo = min(lo, k); hi = max(hi, k); }
    }
    __syncwarp();
    auto count = [&](uint32_t x) {
        int c = 0;
        for (int j = lane; j < nc; j += 32) c += key[j] >= x;
        return (int)__reduce_add_sync(0xffffffffu, c);
    };
    const TopKBound bound = topk_search(count, __reduce_min_sync(0xffffffffu, lo), __reduce_max_sync(0xffffffffu, hi) + 1u, nc, TK);
    int base_eq = 0, base_out = 0;
    const uint32_t below = (1u << lane) - 1u;
    for (int j0 = 0; j0 < nc; j0 += 32) {
        const int j = j0 + lane;
        const uint32_t k = j < nc ? key[j] : 0u;
        const bool eq = !bound.exact && j < nc && k == bound.tau;
        const uint32_t meq = __ballot_sync(0xffffffffu, eq);
        const bool keep = (j < nc && k > bound.tau) || (eq && base_eq + __popc(meq & below) < bound.need);
        const uint32_t mk = __ballot_sync(0xffffffffu, keep);
        if (keep) store_parent(p, l - 1, qidx * TK + base_out + __popc(mk & below), j);
        base_eq += __popc(meq); base_out += __popc(mk);
    }
    for (int i = base_out + lane; i < TK; i += 32) store_parent(p, l - 1, qidx * TK + i, -1);
}

// Bytes of the rotated top keys, 0 where the top level is not selected here.
int64_t top_keys_bytes(const HtreeShape& s, int L, const int32_t* ln) {
    if (L < 2 || s.K != s.V || !(s.K == 32 || (s.K == 128 && s.dtype == HTREE_F32)) || s.H / s.H_kv > 16) return 0;
    return (int64_t)s.B * s.H_kv * ((ln[L - 1] + kTopTile - 1) / kTopTile * kTopTile) * s.K * 4;
}

template <typename T, int D>
static int launch_rotate(const AttnParams& p, cudaStream_t st) {
    const int l = p.L - 1;
    const TopKeysArgs a{p.lk[l], p.ktop, p.cosc, p.sinc, p.ln[l], p.Hkv, p.B * p.Hkv};
    return launch_chained(rotate_top_keys_kernel<T, D>, dim3((p.ln[l] + kTopTile - 1) / kTopTile, p.B * p.Hkv, D / 16), dim3(kTopTile), 0, st, a);
}
template <typename T, int D, int GP, TopForm FORM>
static int launch_top(const AttnParams& p, cudaStream_t st) {
    const int nodes = (p.ln[p.L - 1] + kTopTile - 1) / kTopTile * kTopTile;
    const size_t per_warp = top_warp_bytes(D, GP, nodes, FORM), limit = 227 * 1024;
    int QW = 8;
    while (QW > 1 && kTopKeyBytes + QW * per_warp > limit / 2) QW /= 2;       // two blocks per SM
    const size_t smem = kTopKeyBytes + QW * per_warp;
    // Two warps an SM (a level of more than 5376 nodes, with more than 8 heads 5120) are too few with 32-wide heads, whose tiles are as large as
    // those of 128 for a quarter of the products: 2400 queries, 2 x 8 heads, 6000 nodes 4.51 ms against 3.77 of a block per query; 5300 nodes,
    // three warps, 3.22 against 3.48; 4096 nodes, four, 2.43 against 2.93.  128-wide heads: 6000 nodes 12.2 against 16.9, 7500 14.5 against 20.4.
    if (D < 128 && 228 * 1024 / (smem + 1024) * QW < 3) return HTREE_E_UNSUPPORTED;
    if (smem > limit) return HTREE_E_UNSUPPORTED;
    auto* k = select_top_kernel<T, D, GP, FORM>;
    static SmemLimit shared;
    const cudaError_t e = shared.raise((const void*)k, smem);
    if (e != cudaSuccess) return (int)e;
    const int rc = launch_rotate<T, D>(p, st);
    return rc ? rc : launch_chained(k, dim3((p.Tq + QW - 1) / QW, p.B * p.Hkv), dim3(QW * 32), smem, st, p);
}
template <typename T, int D, int GP>
static int launch_top_form(const AttnParams& p, bool sums, cudaStream_t st) {
    return sums ? launch_top<T, D, GP, kTwice>(p, st) : launch_top<T, D, GP, kPerNode>(p, st);
}
template <typename T, int D>
static int launch_top_g(const AttnParams& p, bool sums, cudaStream_t st) {
    return p.G <= 4 ? launch_top_form<T, D, 4>(p, sums, st) : p.G <= 8 ? launch_top_form<T, D, 8>(p, sums, st) : launch_top_form<T, D, 16>(p, sums, st);
}

// Lists of the levels L - 1 and L - 2.  `sums`: which of the two importance sums the levels' other kernel would take.  Calls of few
// groups stay with that kernel, which has a block for each (a warp's walk over the nodes would be longer than its).
int launch_select_top(const AttnParams& p, int dtype, bool sums, cudaStream_t st) {
    if (!p.ktop || p.L < 2 || (int64_t)p.Tq * p.B * p.Hkv < 4 * 148) return HTREE_E_UNSUPPORTED;
    if (p.K == 128) return dtype == HTREE_F32 ? launch_top_g<float, 128>(p, sums, st) : HTREE_E_UNSUPPORTED;
    switch (dtype) {
        case HTREE_F32: return launch_top_g<float, 32>(p, sums, st);
        case HTREE_BF16: return launch_top_g<__nv_bfloat16, 32>(p, sums, st);
        default: return launch_top_g<__half, 32>(p, sums, st);
    }
}

}  // namespace htree
