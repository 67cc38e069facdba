// Parent-stationary pass of the backward (bwd_tform.cuh): the counting sort of the visits by parent, dK and dV, and the
// mean-pool gradient.  Replaces htree_bwd_dkv_bottom/upper_kernel and htree_bwd_tree_backward_kernel (src/backward.py:443-841).
#include "bwd_tform.cuh"

namespace htree {

// 16-bit storage: what bounds dS (ds_scale), the largest |dO|_1 of a row and the largest value of every unit, of those that are
// finite.  Streams dO (the first `of_dO` blocks) and the leaves' values (`of_v` blocks a unit; pooled values are means of them) once, and
// clears the accumulators on the way (a launch of their own cost 2 of the 121 us of a step of 1000 positions).  18 us at 2 x 16384
// positions, 16 heads of 64; 27 us at 2 x 7777, 32 heads of 128 (5 TB/s).
struct RangeArgs {
    const uint4* dO;
    const uint4* v;              // blocks [b][parent][KV head] of `piece` 16-byte pieces
    int64_t n_dO;
    uint4* zero;                 // the accumulators to clear, or n_zero = 0
    int64_t n_zero;
    int32_t of_dO, of_v, NBLK, Hkv, piece;
    uint32_t* range;
};
template <typename T, int D>
__global__ void __launch_bounds__(256) bwd_range_kernel(const __grid_constant__ RangeArgs a) {
    chain_enter();
    constexpr int LPR = D / 8, U = 4;              // lanes per row; 16-byte pieces in flight
    using F = Frag<T>;
    __shared__ float part[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < a.n_zero; i += (int64_t)gridDim.x * 256) a.zero[i] = make_uint4(0u, 0u, 0u, 0u);
    const bool values = (int)blockIdx.x >= a.of_dO;
    const int at = values ? ((int)blockIdx.x - a.of_dO) % a.of_v : (int)blockIdx.x, unit = values ? ((int)blockIdx.x - a.of_dO) / a.of_v : 0;
    const int64_t n = values ? (int64_t)a.NBLK * a.piece : a.n_dO, step = (int64_t)(values ? a.of_v : a.of_dO) * 8 * 32 * U;
    const uint4* src = values ? a.v + ((int64_t)(unit / a.Hkv) * a.NBLK * a.Hkv + unit % a.Hkv) * a.piece : a.dO;
    float most = 0.f;
    for (int64_t i0 = ((int64_t)at * 8 + warp) * 32 * U; i0 < n; i0 += step) {
        uint4 x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t i = i0 + 32 * u + lane;
            const uint32_t row = (uint32_t)i / (uint32_t)a.piece;      // (a unit's values are below 2^32 pieces)
            x[u] = i < n ? __ldg(src + (values ? i + (int64_t)row * a.piece * (a.Hkv - 1) : i)) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t w[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
            float s = 0.f, m = 0.f;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 f = F::unpack(w[k]);
                s += fabsf(f.x) + fabsf(f.y);
                if (fabsf(f.x) < INFINITY) m = fmaxf(m, fabsf(f.x));
                if (fabsf(f.y) < INFINITY) m = fmaxf(m, fabsf(f.y));
            }
#pragma unroll
            for (int o = 1; o < LPR; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (values) s = m;
            if (s < INFINITY) most = fmaxf(most, s);
        }
    }
    most = redux_max_f32(most, 0xffffffffu);
    if (lane == 0) part[warp] = most;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) most = fmaxf(most, part[w]);
        atomicMax(a.range + (values ? 1 + unit : 0), __float_as_uint(most));
    }
}

// Exclusive prefix sums over a window's parents of their visits and of their work items (pieces of at most `seg` visits of one parent), by
// the NTH threads of a block; returns the number of items.
template <int NTH>
__device__ __forceinline__ int scan_parents(const int32_t* cnt, int2* base, int NK, int seg) {
    __shared__ int2 wsum[NTH / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per = (NK + NTH - 1) / NTH, k0 = tid * per, k1 = min(NK, k0 + per);
    int2 s = make_int2(0, 0);
    for (int k = k0; k < k1; ++k) { const int c = cnt[k]; s.x += c; s.y += (c + seg - 1) / seg; }
    int2 inc = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, inc.x, o), y = __shfl_up_sync(0xffffffffu, inc.y, o);
        if (lane >= o) { inc.x += x; inc.y += y; }
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    int2 before = make_int2(inc.x - s.x, inc.y - s.y);
    int total = 0;
    for (int w = 0; w < NTH / 32; ++w) {
        if (w < warp) { before.x += wsum[w].x; before.y += wsum[w].y; }
        total += wsum[w].y;
    }
    for (int k = k0; k < k1; ++k) {
        const int c = cnt[k];
        base[k] = before;
        before.x += c; before.y += (c + seg - 1) / seg;
    }
    return total;
}
// One block per window.  The items themselves are written by the next kernel: one block that wrote them all took 80 us where
// parents have thousands of visits (12000 positions, 512 nodes per layer).
__global__ void __launch_bounds__(1024) bwd_scan_kernel(const __grid_constant__ BwdParams bp) {
    chain_enter();
    const int sub = blockIdx.x;
    const int total = scan_parents<1024>(bp.cnt + (int64_t)sub * bp.NK, bp.base + (int64_t)sub * bp.NK, bp.NK, bp.seg);
    if (threadIdx.x == 0) bp.nitems[sub] = total;
}
// Few parents and few blocks that need their sums: every block of the fill kernel makes them for itself, a launch less.
constexpr int kOwnScan = 1024;
template <bool OWN>
__device__ __forceinline__ const int2* window_base(const BwdParams& bp) {
    if constexpr (!OWN) return bp.base + (int64_t)blockIdx.y * bp.NK;
    __shared__ int2 own[kOwnScan];
    const int total = scan_parents<256>(bp.cnt + (int64_t)blockIdx.y * bp.NK, own, bp.NK, bp.seg);
    if (blockIdx.x == 0 && threadIdx.x == 0) bp.nitems[blockIdx.y] = total;
    __syncthreads();
    return own;
}

// One warp per group: every visit's entry goes to its place in its parent's list; the first visit of an item writes the item.
template <bool OWN>
__global__ void __launch_bounds__(256) bwd_fill_kernel(const __grid_constant__ BwdParams bp) {
    chain_enter();
    const int2* sums = window_base<OWN>(bp);
    const AttnParams& p = bp.a;
    const int lane = threadIdx.x & 31, qi = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int sub = bp.sub0 + blockIdx.y, unit = sub / bp.nw;
    const int tl = (sub % bp.nw) * bp.subq + qi;
    if (qi >= bp.subq || tl >= p.Tq) return;
    const int b = unit / p.Hkv, hk = unit % p.Hkv, TK = p.TK, CR = p.CR;
    const int64_t grp = (int64_t)blockIdx.y * bp.subq + qi;
    const int64_t qidx = ((int64_t)b * p.Tq + tl) * p.Hkv + hk;
    const int t = p.t0 + tl;
    const int64_t entry0 = (int64_t)blockIdx.y * bp.subq * bp.MV;
    BwdItem* items = bp.items + (int64_t)blockIdx.y * bp.cap;
    for (int l = p.L - 1; l >= 0; --l) {
        if (bp.voff[l] < 0) continue;
        const int nblk = (p.ln[l] + CR - 1) / CR;
        int np = 0;                                // the parents, counted and bounded as ParentList::load does for the first pass
        for (int i = lane; i < min(TK, nblk); i += 32) np += load_parent(p, l, qidx * TK + i) >= 0;
        np = __reduce_add_sync(0xffffffffu, np);
        const int rp = (np - 1) * CR + (int)(((int64_t)t / p.lpow[l]) % CR);
        if (np <= 0 || (l > 0 && rp + 1 <= TK)) continue;
        const int2* base = sums + bp.koff[l];
        const int32_t* cnt = bp.cnt + (int64_t)blockIdx.y * bp.NK + bp.koff[l];
        for (int i = lane; i < np; i += 32) {
            int x = load_parent(p, l, qidx * TK + i);
            if ((unsigned)x >= (unsigned)nblk) x = 0;
            const int64_t v = grp * bp.MV + bp.voff[l] + i;
            const int2 at = base[x];
            const int rank = bp.rank[v];
            const uint32_t where = (uint32_t)grp | ((uint32_t)(rp - CR * i) << 15);
            if (bp.fac) {
                const float2 f = bp.fac[grp * p.L + l];
                reinterpret_cast<BwdEntry<true, 1>*>(bp.entries)[entry0 + at.x + rank] = BwdEntry<true, 1>{(uint32_t)v, where, {f}};
            } else {
                reinterpret_cast<BwdEntry<false, 1>*>(bp.entries)[entry0 + at.x + rank] = BwdEntry<false, 1>{(uint32_t)v, where};
            }
            if (rank % bp.seg == 0) items[at.y + rank / bp.seg] = BwdItem{bp.koff[l] + x, at.x + rank, min(bp.seg, cnt[x] - rank), 0};
        }
    }
}

// The same for groups of several queries, whose visits the first pass has listed.
template <bool OWN>
__global__ void __launch_bounds__(256) bwd_fill_many_kernel(const __grid_constant__ BwdParams bp) {
    chain_enter();
    const int2* sums = window_base<OWN>(bp);
    const AttnParams& p = bp.a;
    const int lane = threadIdx.x & 31, gi = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (gi >= bp.ng || ((bp.sub0 + (int)blockIdx.y) % bp.nw) * bp.subq + gi * bp.PK >= p.Tq) return;
    const int64_t grp = (int64_t)blockIdx.y * bp.ng + gi, entry0 = (int64_t)blockIdx.y * bp.ng * bp.MV;
    BwdItem* items = bp.items + (int64_t)blockIdx.y * bp.cap;
    for (int l = p.L - 1; l >= 0; --l) {
        if (bp.voff[l] < 0) continue;
        const int n = bp.nvis[grp * p.L + l];
        const int2* base = sums + bp.koff[l];
        const int32_t* cnt = bp.cnt + (int64_t)blockIdx.y * bp.NK + bp.koff[l];
        for (int i = lane; i < n; i += 32) {
            const int64_t v = grp * bp.MV + bp.voff[l] + i;
            const uint4 x = bp.vis[v];
            const uint32_t parent = x.x & 0xffffu;
            const int2 at = base[parent];
            const int rank = (int)x.y;
            uint4* entry = reinterpret_cast<uint4*>(static_cast<unsigned char*>(bp.entries) + (entry0 + at.x + rank) * entry_bytes(bp.fac != nullptr, bp.PK));
            entry[0] = make_uint4((uint32_t)v, (uint32_t)grp | (x.x & ~0xffffu), x.z, x.w);
            if (bp.fac) {
                const uint4* f = reinterpret_cast<const uint4*>(bp.fac + (grp * p.L + l) * bp.PK);
                entry[1] = f[0];
                if (bp.PK > 2) entry[2] = f[1];
            }
            if (rank % bp.seg == 0) items[at.y + rank / bp.seg] = BwdItem{bp.koff[l] + (int)parent, at.x + rank, min(bp.seg, cnt[parent] - rank), 0};
        }
    }
}

// Is a factor (a power of two, or 0) near enough to the largest one of its product, that the operand can take the ratio?
__device__ __forceinline__ bool near_factor(float f, float top) { return top >= 0x1p-122f ? 16.f * f >= top : f == top; }

// dK' (KEYS) or dV of one item: dX^T[dims x children] += A[dims x heads] B[heads x children] over its visits, 16 rows (heads) a
// step: one visit of up to 16 heads, or two visits of up to 8.  A = the blocked queries rotated by the visit's distance, or the
// blocked output gradients; B = dS or P as the first pass left them.  One warp per item, operands through the warp's ring.
// A warp makes one of the two gradients: it gathers from one blocked tensor only (a window of it stays in L2) and its accumulator is 64
// registers, which leaves room for 12 and more warps per SM.  dK's items come first, split-half in a launch of their own, 16-bit in one
// launch with dV's.  Bound by that gather: 16.3 TB/s of a measured 20 with 16 heads of 128.
// Ring depth: three slots; two where that lets more blocks share an SM and they are the faster choice: split-half, and the keys of
// groups of 9 to 16 heads of 128 (65536 positions, 64 heads: 13.2 -> 12.4 ms; with 8 heads a group three slots keep a lead of 1%).
template <int D, bool X3, int NH, bool KEYS>
constexpr int dkv_stages() { return X3 || (KEYS && D == 128 && NH == 2) ? 2 : 3; }
// Blocks per SM that the registers have to allow: six for the smallest split-half dV accumulators (80 registers; the compiler's 83 and
// 86 left five), five for the smallest dK (96; 99 left four).
template <int D, bool X3, int CR, bool KEYS>
constexpr int dkv_min_blocks() { return X3 ? (D == 128 ? 2 : !KEYS && (D == 32 || CR == 8) ? 6 : D == 32 ? 5 : 3) : D == 128 ? 3 : 4; }

template <typename T, int D, bool X3, int NH, int CR, bool KEYS, int PK>
__device__ __forceinline__ void dkv_item(const BwdParams& bp) {
    using BF = BForm<D, X3, NH, CR>;
    using C = TForm<D, X3, CR>;
    using FT = typename std::conditional<X3 || KEYS, __half, T>::type;      // operand type of the products
    using F = Frag<FT>;
    constexpr int KS = BF::KS, NT = BF::NT, QB = BF::QB, SB = BF::SB, PPT = C::PPT, HALF = C::HALF;
    constexpr int TAB = KEYS ? C::TAB : 0;
    constexpr int SLOT = 2 * QB + 2 * SB + 2 * PK * TAB, NSTG = dkv_stages<D, X3, NH, KEYS>();
    const uint32_t tab_of_pair = PK == 1 ? 0 : Cols<PK>::of_pair(threadIdx.x & 3) * TAB;
    constexpr int PLANE = NT * 128;                                         // bytes from the hi to the lo words of a record
    using Ring = WarpRing<NSTG, SLOT>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const AttnParams& p = bp.a;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2;
    const int it = blockIdx.x * (blockDim.x >> 5) + warp, ls = blockIdx.y;
    if (it >= bp.nitems[ls]) return;
    const BwdItem item = bp.items[(int64_t)ls * bp.cap + it];
    Ring ring;
    ring.init(smem_raw + (size_t)warp * Ring::kBytes);
    using Entry = BwdEntry<X3, PK>;
    const Entry* entries = reinterpret_cast<const Entry*>(bp.entries) + (int64_t)ls * bp.ng * bp.MV + item.start;
    const unsigned char* qsrc = KEYS ? bp.qb : bp.dob;
    const unsigned char* ssrc = KEYS ? bp.sts : bp.stp;
    const unsigned char* tab = X3 ? reinterpret_cast<const unsigned char*>(p.tab) : bp.xtab;
    constexpr int VPS = NH == 2 ? 1 : 2;                                    // visits per step
    const int len = item.len, steps = (len + VPS - 1) / VPS;

    float acc[KS][NT][4];
#pragma unroll
    for (int i = 0; i < KS; ++i)
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[i][n][0] = acc[i][n][1] = acc[i][n][2] = acc[i][n][3] = 0.f;

    Entry cur = entries[min(lane, len - 1)], nxt = entries[min(32 + lane, len - 1)];
    static_assert(!X3 || NSTG == 2, "a step's factors are taken when the next one is fetched");
    // Split-half: the factors of the visits fetched last (of this lane's columns' query), and the largest of the step's.  Most steps have one
    // factor, `usual`; `odd` has a bit for every entry of `cur` with another one, `far` for those that are not within 2^4 of their step's largest.
    float fa = 0.f, fb = 0.f, ft = 0.f, usual = 0.f, largest = 0.f;
    uint32_t odd = 0u, far = 0u;
    int kind = 0;                                  // of the step fetched last: 1 if a visit is odd, 3 if one is far
    auto factor = [&](int j) { if constexpr (X3) return KEYS ? cur.f[j].x : cur.f[j].y; else return 1.f; };
    auto compare = [&]() {
        if constexpr (X3) {
            usual = __shfl_sync(0xffffffffu, factor(0), 0);
            const uint32_t others = __ballot_sync(0xffffffffu, factor(0) != usual);
            if (__popc(others) > 16) usual = __shfl_sync(0xffffffffu, factor(0), __ffs(others) - 1);
            bool off = false, out = false;
            largest = factor(0);
#pragma unroll
            for (int j = 0; j < PK; ++j) { off |= factor(j) != usual; largest = fmaxf(largest, factor(j)); }
            odd = __ballot_sync(0xffffffffu, off);
            if constexpr (VPS == 2) {
                largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, 1));
#pragma unroll
                for (int j = 0; j < PK; ++j) out |= !near_factor(factor(j), largest);
                far = __ballot_sync(0xffffffffu, out);
            }
        }
    };
    auto factor_of = [&](int e) {                  // of entry e
        float f = __shfl_sync(0xffffffffu, factor(0), e);
#pragma unroll
        for (int j = 1; j < PK; ++j) {
            const float x = __shfl_sync(0xffffffffu, factor(j), e);
            if (Cols<PK>::of_pair(lane & 3) == j) f = x;
        }
        return f;
    };
    compare();
    uint32_t skips = 0u;                           // PK > 1: per step on its way a byte, the queries of its two visits whose columns are left out
    auto fill = [&](int s, int ahead) {            // operand, record and table row of the step's one or two visits
        const int e0 = s * VPS;
        if (e0 && (e0 & 31) == 0) {
            cur = nxt; nxt = entries[min(e0 + 32 + lane, len - 1)];
            compare();
        }
        if constexpr (X3) {
            constexpr uint32_t BITS = VPS == 2 ? 3u : 1u;
            kind = (odd >> (e0 & 31) & BITS) != 0u;
            fa = fb = ft = usual;
            if (kind) {
                fa = factor_of(e0 & 31);
                if constexpr (VPS == 2) {
                    fb = factor_of((e0 + 1) & 31);                          // (past the end: the last entry again)
                    ft = __shfl_sync(0xffffffffu, largest, e0 & 31);
                    if (far >> (e0 & 31) & BITS) kind = 3;
                }
            }
        }
        const uint32_t ax = __shfl_sync(0xffffffffu, cur.visit, e0 & 31), ay = __shfl_sync(0xffffffffu, cur.where, e0 & 31);
        auto tab_rows = [&](int e, uint32_t off) {                     // of entry e, a row per query
            if constexpr (KEYS && PK > 1) {
                uint32_t w = __shfl_sync(0xffffffffu, cur.rows[0], e & 31);
                if constexpr (PK > 2) { const uint32_t w1 = __shfl_sync(0xffffffffu, cur.rows[1], e & 31); if (lane & 2) w = w1; }
                copy_tab_rows<PK, C::TAB>(ring, off, tab, (int)(lane & 1 ? w >> 16 : w & 0xffffu), lane);
            }
        };
        ring.template copy<NH * QB>(0, qsrc + (int64_t)(ay & 0x7fffu) * (NH * QB), lane);
        ring.template copy<NH * SB>(2 * QB, ssrc + (int64_t)ax * (NH * SB), lane);
        if constexpr (KEYS && PK == 1) ring.template copy<TAB>(2 * QB + 2 * SB, tab + (int64_t)(ay >> 15) * C::TAB, lane);
        tab_rows(e0, 2 * QB + 2 * SB);
        if (PK > 1 && ay >> 16) skips |= ay >> 16 << (8 * ahead);
        if constexpr (VPS == 2) {
            const int e1 = min(e0 + 1, len - 1);
            const uint32_t bx = __shfl_sync(0xffffffffu, cur.visit, e1 & 31), by = __shfl_sync(0xffffffffu, cur.where, e1 & 31);
            ring.template copy<QB>(QB, qsrc + (int64_t)(by & 0x7fffu) * QB, lane);
            ring.template copy<SB>(2 * QB + SB, ssrc + (int64_t)bx * SB, lane);
            if constexpr (KEYS && PK == 1) ring.template copy<TAB>(2 * QB + 2 * SB + TAB, tab + (int64_t)(by >> 15) * C::TAB, lane);
            tab_rows(e1, 2 * QB + 2 * SB + PK * TAB);
            if (PK > 1 && by >> 16) skips |= by >> 16 << (8 * ahead + 4);
        }
    };
    int next = 0;
#pragma unroll 1
    for (; next < NSTG - 1; ++next) {
        if (next < steps) fill(next, next);
        ring.commit();
    }
#pragma unroll 1
    for (int s = 0; s < steps; ++s) {
        __syncwarp();
        const float f0 = fa, f1 = fb, f01 = ft;    // of this step's visits
        const int mixed = kind;
        if (next < steps) fill(next, NSTG - 1);
        ring.commit();
        ++next;
        uint32_t slot = ring.wait();
        if (PK > 1 && skips) {
            const uint32_t skip = skips & 0xffu;
            skips >>= 8;
            constexpr int LB = KEYS && X3 ? 16 : 8;    // a lane's bytes at a time, which it alone reads
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                if (!(skip >> (4 * v + Cols<PK>::of_pair(lane & 3)) & 1)) continue;
#pragma unroll
                for (int i = 0; i < QB / 256; ++i)
                    asm volatile("st.shared.v2.b32 [%0], {%1,%1};\n" ::"r"(slot + v * QB + i / (LB / 8) * (32 * LB) + lane * LB + i % (LB / 8) * 8), "r"(0u) : "memory");
            }
            asm volatile("" : "+r"(slot)::"memory");   // (what orders the reads behind these writes)
        }
        const bool lone = VPS == 2 && 2 * s + 1 >= len;
        uint32_t bw[NT][2], bl[X3 ? NT : 1][2];
        auto lds32 = [](uint32_t a) { uint32_t x; asm("ld.shared.b32 %0, [%1];" : "=r"(x) : "r"(a)); return x; };
        auto lds64 = [](uint32_t a, uint32_t& x, uint32_t& y) { asm("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(x), "=r"(y) : "r"(a)); };
        auto load_records = [&]() {
            const uint32_t ra = slot + 2 * QB, rb = ra + SB;
#pragma unroll
            for (int pl = 0; pl < (X3 ? 2 : 1); ++pl) {
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    const uint32_t o = pl * PLANE + lane * (4 * NT) + 4 * n;
                    const uint32_t x = lds32(ra + o), y = lone ? 0u : lds32(rb + o);
                    if (pl == 0) { bw[n][0] = x; bw[n][1] = y; } else { bl[X3 ? n : 0][0] = x; bl[X3 ? n : 0][1] = y; }
                }
            }
        };
        load_records();
        if constexpr (KEYS && !X3) {
            const uint32_t ta = slot + 2 * QB + 2 * SB + 2 * KS * (4 * (g & 1) + (g >> 1)) + tab_of_pair;
            uint32_t ca[KS / 2], sa[KS / 2], cb[KS / 2], sb[KS / 2];
            lds_x<D>(ta, ca, sa);
            if constexpr (VPS == 2) lds_x<D>(ta + PK * TAB, cb, sb);
#pragma unroll
            for (int i = 0; i < KS; ++i) {
                uint32_t la, ha, lb, hb, a[4];
                lds64(slot + i * 256 + lane * 8, la, ha);
                lds64(slot + QB + i * 256 + lane * 8, lb, hb);
                const __half2 c0 = half_of(ca[i / 2], i & 1), s0 = half_of(sa[i / 2], i & 1);
                rotate_x<false>(la, ha, c0, s0, a[0], a[1]);
                if constexpr (VPS == 2) rotate_x<false>(lb, hb, half_of(cb[i / 2], i & 1), half_of(sb[i / 2], i & 1), a[2], a[3]);
                else rotate_x<false>(lb, hb, c0, s0, a[2], a[3]);
#pragma unroll
                for (int n = 0; n < NT; ++n) mma_acc<FT>(acc[i][n], a, bw[n][0], bw[n][1]);
            }
        } else if constexpr (!X3) {
#pragma unroll
            for (int i = 0; i < KS; ++i) {
                uint32_t a[4];
                lds64(slot + i * 256 + lane * 8, a[0], a[1]);
                lds64(slot + QB + i * 256 + lane * 8, a[2], a[3]);
#pragma unroll
                for (int n = 0; n < NT; ++n) mma_acc<FT>(acc[i][n], a, bw[n][0], bw[n][1]);
            }
        } else {
            auto products = [&](float vfac) {      // vfac: what brings them back
#pragma unroll
                for (int i = 0; i < KS; ++i) {
                    uint32_t ah[4], al[4];
                    if constexpr (KEYS) {
#pragma unroll
                        for (int v = 0; v < 2; ++v) {
                            const uint4 x = lds_u4(slot + v * QB + i * 512 + lane * 16);
                            const uint32_t t4 = slot + 2 * QB + 2 * SB + (VPS == 2 ? v : 0) * PK * TAB + tab_of_pair + 4 * (PPT * (g >> 1) + 2 * i + (g & 1));
                            const float cs = __uint_as_float(lds32(t4)), sn = __uint_as_float(lds32(t4 + 4 * HALF));
                            float2 u, w;
                            rotate_pairs_f32(make_float2(__uint_as_float(x.x), __uint_as_float(x.y)), make_float2(__uint_as_float(x.z), __uint_as_float(x.w)),
                                             make_float2(cs, cs), make_float2(sn, sn), make_float2(-sn, -sn), u, w);
                            split_half2(u.x, u.y, ah[2 * v], al[2 * v]);
                            split_half2(w.x, w.y, ah[2 * v + 1], al[2 * v + 1]);
                        }
                    } else {
#pragma unroll
                        for (int v = 0; v < 2; ++v) {
                            lds64(slot + v * QB + i * 256 + lane * 8, ah[2 * v], ah[2 * v + 1]);
                            lds64(slot + v * QB + D * 16 + i * 256 + lane * 8, al[2 * v], al[2 * v + 1]);
                        }
                    }
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        float t[4];
                        mma_zero<__half>(t, al, bw[n][0], bw[n][1]);
                        mma_acc<FT>(t, ah, bl[X3 ? n : 0][0], bl[X3 ? n : 0][1]);
                        mma_acc<FT>(t, ah, bw[n][0], bw[n][1]);
#pragma unroll
                        for (int u = 0; u < 4; ++u) acc[i][n][u] = fmaf(t[u], vfac, acc[i][n][u]);
                    }
                }
            };
            if constexpr (VPS == 1) {
                products(f0);
            } else {
                // Columns of several queries in one product.  Those whose factors are within a step (2^4) of the largest go into it, times
                // the ratio, and the others have products of their own: a half pair ends at 2^-25, so that with all of them brought to one
                // factor a query whose gradient (or q) is 2^-20 of its neighbour's lost 3.6e-4 of a P of 1/512, and 2^-30 all of it.
                float w0 = f0, w1 = f1, top = f01;
#pragma unroll 1
                for (;;) {
                    if (mixed) {
                        auto take = [&](float& w) {            // a column's ratio, 0: not in this product
                            const bool in = near_factor(w, top);
                            const float x = in ? __int_as_float(__float_as_int(1.f) + __float_as_int(w) - __float_as_int(top)) : 0.f;      // powers of two
                            if (in) w = 0.f;
                            return __float2half2_rn(x);
                        };
                        const __half2 r0 = take(w0), r1 = take(w1);
#pragma unroll
                        for (int n = 0; n < NT; ++n) {
                            bw[n][0] = as_u32(__hmul2(as_h2(bw[n][0]), r0)); bw[n][1] = as_u32(__hmul2(as_h2(bw[n][1]), r1));
                            bl[X3 ? n : 0][0] = as_u32(__hmul2(as_h2(bl[X3 ? n : 0][0]), r0)); bl[X3 ? n : 0][1] = as_u32(__hmul2(as_h2(bl[X3 ? n : 0][1]), r1));
                        }
                    }
                    products(top);
                    if (mixed < 3) break;
                    top = redux_max_f32(fmaxf(w0, w1), 0xffffffffu);
                    if (top == 0.f) break;
                    asm volatile("" : "+r"(slot));     // (what the products read again is not to be kept from the first of them)
                    load_records();
                }
            }
        }
#pragma unroll
        for (int i = 0; i < KS; ++i)
#pragma unroll
            for (int n = 0; n < NT; ++n) consumed(acc[i][n]);
    }

    int l = 0;
    while (l + 1 < p.L && (bp.voff[l] < 0 || item.key < bp.koff[l] || item.key >= bp.koff[l] + (p.ln[l] + CR - 1) / CR)) ++l;
    const int unit = (bp.sub0 + ls) / bp.nw, b = unit / p.Hkv, hk = unit % p.Hkv;
    const int nblk = (p.ln[l] + CR - 1) / CR;
    const float post = KEYS && !X3 ? pow2_inverse(ds_scale(__ldg(bp.range), __ldg(bp.range + 1 + unit))) : 1.f;
    float* dst = (KEYS ? bp.acck[l] : bp.accv[l]) + (((int64_t)b * nblk + (item.key - bp.koff[l])) * p.Hkv + hk) * BF::ACC + 4 * lane;
#pragma unroll
    for (int i = 0; i < KS; ++i)
#pragma unroll
        for (int n = 0; n < NT; ++n) red_add_v4(dst + (i * NT + n) * 128, acc[i][n][0] * post, acc[i][n][1] * post, acc[i][n][2] * post, acc[i][n][3] * post);
}

template <typename T, int D, bool X3, int NH, int CR, bool KEYS, int PK>
__global__ void __launch_bounds__(128, dkv_min_blocks<D, X3, CR, KEYS>()) bwd_dkv_kernel(const __grid_constant__ BwdParams bp) {
    chain_enter();
    dkv_item<T, D, X3, NH, CR, KEYS, PK>(bp);
}
// dK, then dV, of the 16-bit types in one launch: the same warps fit an SM for either, and the one's last blocks run beside the other's first.
template <typename T, int D, int NH, int CR, int PK>
__global__ void __launch_bounds__(128, dkv_min_blocks<D, false, CR, true>()) bwd_dkv_both_kernel(const __grid_constant__ BwdParams bp) {
    chain_enter();
    if (blockIdx.z == 0) dkv_item<T, D, false, NH, CR, true, PK>(bp);
    else dkv_item<T, D, false, NH, CR, false, PK>(bp);
}

// Accumulators to the leaves' gradients: dK' rotated back by the child index, plus the mean-pool shares of the ancestors' gradients
// (src/backward.py:787-841), which every block of leaves sums up for itself from the top: a row of D per level, where a launch per
// level would wait for the one before.  blockIdx.y: 0 = dK, 1 = dV; one warp per block of leaves.
struct FoldArgs {
    const float* acc[2][HTREE_MAX_LEVELS];
    void* out[2];            // leaf rows: fp32, or the storage type (typed)
    const float* cosc;
    const float* sinc;
    int64_t total;           // blocks of leaves
    int32_t N[HTREE_MAX_LEVELS];
    int32_t L, Hkv, typed;
};
template <typename TO, int D, int CR>
__global__ void __launch_bounds__(128) bwd_fold_kernel(const __grid_constant__ FoldArgs f) {
    chain_enter();
    constexpr int KS = D / 16, NT = CR / 8, HALF = D / 2, PPT = HALF / 4;
    __shared__ float sm[4][CR][D + 4];
    const int which = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, r = lane & 3;
    const int64_t blk = (int64_t)blockIdx.x * 4 + warp;
    if (blk >= f.total) return;
    const int nblk = (f.N[0] + CR - 1) / CR;
    const int h = (int)(blk % f.Hkv), pb = (int)((blk / f.Hkv) % nblk);
    const int64_t b = blk / ((int64_t)f.Hkv * nblk);

    // ---- the gradient of the block's own pooled row: lane x holds the pairs x + 32 u (dims x + 32 u and + D/2) ----
    constexpr int U = HALF > 32 ? HALF / 32 : 1;
    float ulo[U], uhi[U];
#pragma unroll
    for (int u = 0; u < U; ++u) ulo[u] = uhi[u] = 0.f;
    for (int m = f.L - 1; m > 0; --m) {
        int n = pb;
        for (int i = 1; i < m; ++i) n /= CR;
        const int c = n % CR, cnt = min(CR, f.N[m] - (n - c)), nb = (f.N[m] + CR - 1) / CR;
        const float* a = f.acc[which][m] + ((b * nb + n / CR) * f.Hkv + h) * (int64_t)(D * CR);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int x = lane + 32 * u;
            if (HALF < 32 && x >= HALF) break;
            // where the accumulators keep child c, dims x and x + D/2 (see BwdParams)
            const float* at = a + ((((x % PPT) >> 1) * NT + (c >> 3)) * 32 + 4 * (2 * (x / PPT) + (x & 1)) + ((c & 7) >> 1)) * 4 + (c & 1);
            float lo = at[0], hi = at[2];
            if (which == 0) {
                const float cs = __ldg(f.cosc + c * HALF + x), sn = __ldg(f.sinc + c * HALF + x), y = lo;
                lo = y * cs + hi * sn;
                hi = hi * cs - y * sn;
            }
            if (m + 1 < f.L) { const float k = (float)cnt; lo += ulo[u] / k; hi += uhi[u] / k; }
            ulo[u] = lo; uhi[u] = hi;
        }
    }

    const float4* a = reinterpret_cast<const float4*>(f.acc[which][0]) + blk * (D * CR / 4);
#pragma unroll
    for (int i = 0; i < KS; ++i) {
        const int x = PPT * (g >> 1) + 2 * i + (g & 1);
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const float4 v = __ldcs(a + (i * NT + n) * 32 + lane);
            const int c = 8 * n + 2 * r;
            float lo[2] = {v.x, v.y}, hi[2] = {v.z, v.w};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float u = lo[e], w = hi[e];
                if (which == 0) {
                    const float cs = __ldg(f.cosc + (c + e) * HALF + x), sn = __ldg(f.sinc + (c + e) * HALF + x);
                    u = lo[e] * cs + hi[e] * sn;
                    w = hi[e] * cs - lo[e] * sn;
                }
                sm[warp][c + e][x] = u;
                sm[warp][c + e][x + HALF] = w;
            }
        }
    }
    __syncwarp();
    const int cnt = min(CR, f.N[0] - pb * CR);
    if (f.L > 1) {
        const float n = (float)cnt;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int x = lane + 32 * u;
            if (HALF < 32 && x >= HALF) break;
            const float lo = ulo[u] / n, hi = uhi[u] / n;
            for (int c = 0; c < cnt; ++c) { sm[warp][c][x] += lo; sm[warp][c][x + HALF] += hi; }
        }
        __syncwarp();
    }
    constexpr int V4 = D / 4;
    for (int i = lane; i < cnt * V4; i += 32) {
        const int c = i / V4, col = i % V4;
        const float4 x = *reinterpret_cast<const float4*>(&sm[warp][c][4 * col]);
        const int64_t row = ((b * f.N[0] + pb * CR + c) * f.Hkv + h) * (int64_t)D + 4 * col;
        if (!f.typed || sizeof(TO) == 4) {
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(f.out[which]) + row) = x;
        } else {
            TO o[4] = {from_f<TO>(x.x), from_f<TO>(x.y), from_f<TO>(x.z), from_f<TO>(x.w)};
            *reinterpret_cast<uint2*>(reinterpret_cast<TO*>(f.out[which]) + row) = *reinterpret_cast<const uint2*>(o);
        }
    }
}

template <int D, bool X3, int NH, int CR, bool KEYS, int PK>
constexpr size_t dkv_smem() {
    using BF = BForm<D, X3, NH, CR>;
    return 4 * WarpRing<dkv_stages<D, X3, NH, KEYS>(), 2 * BF::QB + 2 * BF::SB + (KEYS ? 2 * PK * TForm<D, X3, CR>::TAB : 0)>::kBytes;
}
template <typename T, int D, bool X3, int NH, int CR, bool KEYS, int PK>
static int launch_dkv_one(const BwdParams& bp, cudaStream_t st) {
    constexpr size_t smem = dkv_smem<D, X3, NH, CR, KEYS, PK>();
    auto* k = bwd_dkv_kernel<T, D, X3, NH, CR, KEYS, PK>;
    static SmemLimit shared;
    const cudaError_t e = shared.raise((const void*)k, smem);
    if (e != cudaSuccess) return (int)e;
    return launch_chained(k, dim3((bp.cap + 3) / 4, bp.nsub), dim3(128), smem, st, bp);
}
template <typename T, int D, bool X3, int NH, int CR, int PK>
static int launch_dkv_pk(const BwdParams& bp, cudaStream_t st) {
    if constexpr (X3) {
        const int rc = launch_dkv_one<T, D, X3, NH, CR, true, PK>(bp, st);
        return rc ? rc : launch_dkv_one<T, D, X3, NH, CR, false, PK>(bp, st);
    } else {
        constexpr size_t k = dkv_smem<D, X3, NH, CR, true, PK>(), v = dkv_smem<D, X3, NH, CR, false, PK>(), smem = k > v ? k : v;
        auto* kernel = bwd_dkv_both_kernel<T, D, NH, CR, PK>;
        static SmemLimit shared;
        const cudaError_t e = shared.raise((const void*)kernel, smem);
        if (e != cudaSuccess) return (int)e;
        return launch_chained(kernel, dim3((bp.cap + 3) / 4, bp.nsub, 2), dim3(128), smem, st, bp);
    }
}
template <typename T, int D, bool X3, int NH, int CR>
static int launch_dkv_cr(const BwdParams& bp, cudaStream_t st) {
    if constexpr (NH == 1 && CR == 16) {
        if (bp.PK == 2) return launch_dkv_pk<T, D, X3, NH, CR, 2>(bp, st);
        if (bp.PK == 4) return launch_dkv_pk<T, D, X3, NH, CR, 4>(bp, st);
    }
    return launch_dkv_pk<T, D, X3, NH, CR, 1>(bp, st);
}
template <typename T, int D, bool X3>
static int launch_dkv_t(const BwdParams& bp, cudaStream_t st) {
    if (bp.a.CR == 16) return bp.a.G <= 8 ? launch_dkv_cr<T, D, X3, 1, 16>(bp, st) : launch_dkv_cr<T, D, X3, 2, 16>(bp, st);
    return bp.a.G <= 8 ? launch_dkv_cr<T, D, X3, 1, 8>(bp, st) : launch_dkv_cr<T, D, X3, 2, 8>(bp, st);
}
template <typename T>
static int launch_dkv_d(const BwdParams& bp, cudaStream_t st) {
    constexpr bool F32 = std::is_same<T, float>::value;
    return bp.a.K == 128 ? launch_dkv_t<T, 128, F32>(bp, st) : bp.a.K == 64 ? launch_dkv_t<T, 64, F32>(bp, st) : launch_dkv_t<T, 32, true>(bp, st);
}

template <typename T>
static int launch_range_t(const BwdParams& bp, void* zero, int64_t zero_bytes, cudaStream_t st) {
    const AttnParams& p = bp.a;
    RangeArgs a;
    a.dO = static_cast<const uint4*>(p.dO); a.v = static_cast<const uint4*>(p.vkblk[0]);
    a.n_dO = (int64_t)p.B * p.Tq * p.H * p.K / 8; a.piece = p.CR * p.K / 8;
    a.NBLK = (p.ln[0] + p.CR - 1) / p.CR; a.Hkv = p.Hkv; a.range = bp.range;
    a.zero = static_cast<uint4*>(zero); a.n_zero = zero_bytes / 16;
    // 16 KB a block and more; dO fills the chip and the units share it once more
    auto blocks = [](int64_t pieces, int most) { const int64_t b = (pieces + 1023) / 1024; return (int)(b < most ? b : most); };
    const int units = p.B * p.Hkv;
    a.of_dO = blocks(a.n_dO, 148 * 8); a.of_v = blocks((int64_t)a.NBLK * a.piece, units < 148 ? 148 * 8 / units : 8);
    const unsigned grid = (unsigned)(a.of_dO + units * a.of_v);
    return launch_chained(p.K == 128 ? bwd_range_kernel<T, 128> : bwd_range_kernel<T, 64>, dim3(grid), dim3(256), 0, st, a);
}
// Zeros, `n` 16-byte pieces (a memset node in the chain would have to end and be waited for like any launch that is not chained), and the
// rotary rows in lane order.
template <int D>
__global__ void __launch_bounds__(256) bwd_clear_kernel(uint4* p, int64_t n, const __half* tab, uint4* xtab, int rows) {
    chain_enter();
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) p[i] = make_uint4(0u, 0u, 0u, 0u);
    constexpr int PER = D / 8;                     // pieces of 8 halves per row
    for (int i = blockIdx.x * 256 + threadIdx.x; i < rows * PER; i += gridDim.x * 256) {
        const int row = i / PER, at = i % PER * 8, part = at / (D / 2);      // cosines, sines
        const __half* src = tab + (int64_t)row * D + part * (D / 2);
        alignas(16) __half x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = src[x_index<D>(at % (D / 2) + u)];
        xtab[i] = *reinterpret_cast<const uint4*>(x);
    }
}
// clears whole 16-byte pieces: `bytes` rounded up; rows of the table where `xtab` is given
int launch_bwd_clear(void* p, int64_t bytes, const void* tab, void* xtab, int rows, int D, cudaStream_t st) {
    const int64_t n = (bytes + 15) / 16, most = xtab && (int64_t)rows * (D / 8) > n ? (int64_t)rows * (D / 8) : n, blocks = (most + 1023) / 1024;
    return launch_chained(D == 128 ? bwd_clear_kernel<128> : bwd_clear_kernel<64>, dim3((unsigned)(blocks < 148 * 8 ? blocks : 148 * 8)), dim3(256), 0, st,
                          static_cast<uint4*>(p), n, static_cast<const __half*>(tab), static_cast<uint4*>(xtab), xtab ? rows : 0);
}
// Ahead of the first pass, bp.range being zero: clears `zero_bytes` of accumulators (a multiple of 256, or none) and finds the range of
// 16-bit operands (split ones have factors per group).
int launch_bwd_begin(const BwdParams& bp, int dtype, void* zero, int64_t zero_bytes, cudaStream_t st) {
    if (pack_split(dtype, bp.a.K)) return zero_bytes ? launch_bwd_clear(zero, zero_bytes, nullptr, nullptr, 0, bp.a.K, st) : 0;
    return dtype == HTREE_BF16 ? launch_range_t<__nv_bfloat16>(bp, zero, zero_bytes, st) : launch_range_t<__half>(bp, zero, zero_bytes, st);
}

int launch_bwd_dkv(const BwdParams& bp, int dtype, cudaStream_t st) {
    const dim3 grid((bp.ng + 7) / 8, bp.nsub);
    const bool own = bp.NK <= kOwnScan && (int64_t)grid.x * grid.y <= 148 * 4;
    int rc = own ? 0 : launch_chained(bwd_scan_kernel, dim3(bp.nsub), dim3(1024), 0, st, bp);
    if (rc == 0) rc = launch_chained(bp.PK > 1 ? (own ? bwd_fill_many_kernel<true> : bwd_fill_many_kernel<false>) : own ? bwd_fill_kernel<true> : bwd_fill_kernel<false>,
                                     grid, dim3(256), 0, st, bp);
    if (rc) return rc;
    switch (dtype) {
        case HTREE_F32: return launch_dkv_d<float>(bp, st);
        case HTREE_BF16: return launch_dkv_d<__nv_bfloat16>(bp, st);
        default: return launch_dkv_d<__half>(bp, st);
    }
}

template <typename TO, int CR>
static int launch_fold_t(const FoldArgs& f, int D, cudaStream_t st) {
    return launch_chained(D == 128 ? bwd_fold_kernel<TO, 128, CR> : D == 64 ? bwd_fold_kernel<TO, 64, CR> : bwd_fold_kernel<TO, 32, CR>,
                          dim3((unsigned)((f.total + 3) / 4), 2), dim3(128), 0, st, f);
}

// dk, dv in fp32 or, typed, the storage type.
int launch_bwd_fold(const BwdParams& bp, int dtype, void* dk, void* dv, bool typed, cudaStream_t st) {
    const AttnParams& p = bp.a;
    FoldArgs f;
    for (int l = 0; l < p.L; ++l) { f.acc[0][l] = bp.acck[l]; f.acc[1][l] = bp.accv[l]; f.N[l] = p.ln[l]; }
    f.out[0] = dk; f.out[1] = dv;
    f.cosc = p.cosc; f.sinc = p.sinc;
    f.L = p.L; f.Hkv = p.Hkv; f.typed = typed;
    f.total = (int64_t)p.B * ((p.ln[0] + p.CR - 1) / p.CR) * p.Hkv;
    if (dtype == HTREE_BF16) return p.CR == 16 ? launch_fold_t<__nv_bfloat16, 16>(f, p.K, st) : launch_fold_t<__nv_bfloat16, 8>(f, p.K, st);
    if (dtype == HTREE_F16) return p.CR == 16 ? launch_fold_t<__half, 16>(f, p.K, st) : launch_fold_t<__half, 8>(f, p.K, st);
    return p.CR == 16 ? launch_fold_t<float, 16>(f, p.K, st) : launch_fold_t<float, 8>(f, p.K, st);
}

}  // namespace htree
