// Forward accumulation: softmax(S) V over everything the selections leave to accumulate, all tree levels in one launch, one
// warp per (batch, query position, KV head) group.  Replaces the accumulation halves of htree_select_accumulate_gqa_kernel and
// htree_bottom_accumulate_gqa_kernel together with htree_merge_to_global_kernel and htree_final_normalize_kernel
// (src/parallel.py:248-867); reads the parent lists that a selection launch wrote.
//
// Products, operand blocks and chunk numbering: tform.cuh.  Per chunk of 16 positions a warp copies the operand block(s) and
// one rotary-table row into its ring in shared memory (asynchronously, NSTG - 1 chunks ahead), forms
// S^T = K' q^ (one query rotation per chunk), P^T, and O^T += V^T P^T.
//
// Bound by the L2 gather of the blocks (14.6 to 17.1 of a measured 20 TB/s) and the shared-memory read pipe (61% busy with 16 heads a
// group, 82% with 8): without its copies it would take about 80% of its time.  Measured against the kernel that gathers rows with heads on the matrix
// rows: 4 x 65536 positions, 64 heads of 128: 95 -> 77 ms.  Groups of at most 4 heads leave half of the 8 columns empty: where queries
// select many of the same parents two or four of them share a warp (tform.cuh): 12000 positions, 16 heads of 32, top_k 512: 5.06 -> 3.32 ms.
#include "tform.cuh"

namespace htree {

// Registers and rings: 168 per thread (12 warps per SM) hold a group of 16 heads of 128; those of up to 8 heads fit 16 warps, but
// two slots of 8448 bytes per warp do not.  There a warp has one slot for keys and one for values: the next keys are fetched as soon as
// the scores are formed, the next values behind the chunk's products, each with half a chunk (of 16 warps) to arrive.
// One slot against two (us, whole launch): 8 heads of 128, 65536 positions 14790 -> 14510 and 7777 positions 1356 -> 1307; 8 children
// 1140 -> 1081; fp32 storage, 128-wide heads 386 -> 357 and with 16 heads a group 1031 -> 866; fp32, 64-wide, 8 children 2696 -> 2534.
// Where the warps are as many either way it costs 1 to 10% (waits and barriers twice per chunk): 16 heads of 128, 64-wide 16-bit
// heads, 32-wide heads (634 -> 689), fp32 64-wide heads with 16 children (84.5 -> 88.9).
template <int D, bool X3, int NH, int CR>
constexpr bool acc_single() { return (D == 128 && (NH == 1 || X3)) || (X3 && D == 64 && NH == 1 && CR == 8); }
// Groups of up to 8 heads of 64 in 16 bits fit 20 warps, with two slots of 4 KB each: 20000 positions of 4 groups 2045 -> 1947 us, eight
// children 2513 -> 2470 (32-wide heads, two queries a warp: no change, 385 and 387).
template <int D, bool X3, int NH, int CR>
constexpr bool acc_twenty() { return D == 64 && !X3 && NH == 1; }
template <int D, bool X3, int NH, int CR>
constexpr int acc_stages() { return acc_single<D, X3, NH, CR>() ? 1 : D * (X3 ? 2 : 1) >= 128 || acc_twenty<D, X3, NH, CR>() ? 2 : 3; }     // slots of 8 KB: warps matter more than depth
constexpr int kAccWarps = 4, kAccSplitWarps = 8;
template <int D, bool X3, int NH, int CR>
constexpr int acc_min_blocks() { return (X3 && D == 128) ? 2 : D == 128 ? (NH == 1 ? 4 : 3) : (X3 && D == 64 && NH == 2) ? 3 : acc_twenty<D, X3, NH, CR>() ? 5 : 4; }
// Slots of the warps that share a query: two of 8 KB, three of less, so that two blocks of 64- and 32-wide heads still share an SM (a third
// slot of 8 KB gave nothing: 28.4 against 29.2 us).
template <int D, bool X3>
constexpr int acc_split_stages() { return D * (X3 ? 2 : 1) >= 256 ? 1 : D * (X3 ? 2 : 1) >= 128 ? 2 : 3; }
// A warp's rings: keys with their table rows, and values.
template <int D, bool X3, int NH, int CR, int PK = 1, bool SPLIT = false>
struct AccRings {
    // (lists of several queries beside three slots would cost warps: 12000 positions, 512 nodes per layer 3.60 -> 3.32 ms with two)
    static constexpr int NSTG = SPLIT ? acc_split_stages<D, X3>() : PK > 1 && acc_stages<D, X3, NH, CR>() > 2 ? 2 : acc_stages<D, X3, NH, CR>();
    using C = TForm<D, X3, CR, PK>;
    using Keys = WarpRing<NSTG, C::KSLOT + (NSTG > 1 ? C::VSLOT : 0)>;      // (of several stages: with the values)
    using Values = WarpRing<1, C::VSLOT>;
    static constexpr size_t kBytes = Keys::kBytes + (NSTG > 1 ? 0 : Values::kBytes);
};

template <typename T, int D, bool X3, int NH, int CR, bool SPLIT, int PK>
__global__ void __launch_bounds__((SPLIT ? kAccSplitWarps : kAccWarps) * 32, SPLIT ? 1 : acc_min_blocks<D, X3, NH, CR>())
acc_mma_kernel(const __grid_constant__ AttnParams p) {
    chain_enter();
    static_assert(PK == 1 || (NH == 1 && CR == 16 && !SPLIT), "several queries share a warp's 8 columns");
    using C = TForm<D, X3, CR, PK>;
    using QC = Cols<PK>;
    using FT = typename std::conditional<X3, __half, T>::type;        // type of the values and probabilities
    using F = Frag<FT>;
    constexpr int MT = C::MT, PPC = C::PPC;
    using Ring = AccRings<D, X3, NH, CR, PK, SPLIT>;
    constexpr int NSTG = Ring::NSTG, GP = QC::GP;
    extern __shared__ __align__(128) unsigned char smem_raw[];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, r = lane & 3;
    const int W = SPLIT ? kAccSplitWarps : blockDim.x >> 5;
    const int CL = SPLIT ? (int)cluster_blocks() : 1, rank = SPLIT ? (int)cluster_rank() : 0;       // the blocks that share a query
    const int from_end = SPLIT ? (int)blockIdx.x / CL : (int)(blockIdx.x * W + warp);
    const int npack = PK == 1 ? p.Tq : (p.Tq + PK - 1) / PK;
    if (!SPLIT && from_end >= npack) return;
    const int tl = (npack - 1 - from_end) * PK;                       // the longest walks first: they would be the tail of a short call
    const int b = blockIdx.y / p.Hkv, hk = blockIdx.y % p.Hkv;
    const int G = p.G, TK = p.TK, L = p.L;
    const int first = SPLIT ? rank * W + warp : 0, step = SPLIT ? CL * W : 1;      // this warp's chunks of every level

    // per warp: ring, parent list, kept-candidate bits
    const WalkLayout lay = walk_layout(p, CR);
    const size_t per_warp = SPLIT ? Ring::kBytes : walk_warp_bytes<Ring, PK>(lay);       // (SPLIT: one list for all)
    unsigned char* wbase = smem_raw + warp * per_warp;
    unsigned char* lists = SPLIT ? smem_raw + W * per_warp : wbase + Ring::kBytes;
    typename Ring::Keys kring;
    typename Ring::Values vring;
    kring.init(wbase);
    vring.init(wbase + Ring::Keys::kBytes);
    auto list_of = [&](int j) { return ParentList{lists + j * lay.list, lay.narrow}; };        // query tl + j
    auto bits_of = [&](int j) { return reinterpret_cast<uint32_t*>(lists + PK * lay.list + j * lay.bits); };
    const ParentList par = list_of(0);
    uint32_t* selw = bits_of(0);
    float* exchange = reinterpret_cast<float*>(lists + walk_lists_bytes(lay));                  // SPLIT: [W][3][16]
    uint32_t* votes = reinterpret_cast<uint32_t*>(exchange + 48 * kAccSplitWarps);              // SPLIT: [2][blocks], of even and odd rounds
    int round = 0;
    if (CL > 1) cluster_sync();                                       // every block has started: its shared memory may be written

    const int64_t hbase = ((int64_t)b * p.Tq + tl) * p.H + (int64_t)hk * G;
    const int64_t qidx = ((int64_t)b * p.Tq + tl) * p.Hkv + hk;

    QueryRegs<T, D, X3, NH> q;
    load_query<T, D, X3, NH, PK>([&](int h) -> const T* {
        const int j = QC::of_lane(g), head = PK == 1 ? 8 * h + g : g % GP;
        return head < G && (PK == 1 || tl + j < p.Tq) ? reinterpret_cast<const T*>(p.q) + (hbase + (int64_t)j * p.H + head) * D : nullptr;
    }, r, p.scale, q);
    const uint32_t tab_of_lane = PK == 1 ? 0 : QC::of_lane(g) * C::TAB;

    // Several queries of 16 bits: a block that only a neighbour selected may hold values that are not finite, and 0 times one of them is NaN.
    // If a sum is NaN at the end, the queries are walked once more one by one, as each would be in a warp of its own.
    constexpr bool kAlone = PK > 1 && !X3;                            // (split-half values are clamped as they are packed)
    int alone = -1;                                                   // the only query that is walked, or -1: all
    float O[NH][MT][4];
walk_again:
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
        for (int i = 0; i < MT; ++i) O[h][i][0] = O[h][i][1] = O[h][i][2] = O[h][i][3] = 0.f;
    // Online softmax with a lazily moved reference: probabilities are taken relative to m_run, which moves (and the
    // accumulators are rescaled) only when a score exceeds it by more than kLazyMax.  m_run is common to the lanes that share
    // a head; m_true (the maximum that goes to gmax) and s_run are per lane until the end.
    // With SPLIT a chunk's reference is the one that a single warp walking all chunks would have there: P is rounded to the storage type
    // relative to it, and with references of their own a query's row differed by 3e-3 (bf16) between calls of few and of many
    // queries.  The warps take their chunks in rounds; a vote says whether any of the round moves the reference, and only then (the
    // first round, and as often as scores grow by 8) they exchange their maxima and follow the moves in order.
    constexpr float kLazyMax = 8.f;
    constexpr float kNone = -1.0e30f;
    float m_run[NH][2], m_true[NH][2], s_run[NH][2], m_run2[NH][2];
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e) { m_run[h][e] = m_true[h][e] = kNone; m_run2[h][e] = kNone * kLog2e; s_run[h][e] = 0.f; }

    auto group_sync = [&]() { if constexpr (SPLIT) __syncthreads(); else __syncwarp(); };       // of the threads that share a list
    for (int l = L - 1; l >= 0; --l) {
        const int Nl = p.ln[l];
        group_sync();
        const int nblk = (Nl + CR - 1) / CR;
        int np, rp, nchunk = 0;
        UnionWalk<PK> walk;
        if constexpr (PK == 1) {
            np = par.load(p, l, qidx * TK, nblk, 4, lane);
            const int nc = (np - 1) * CR + (int)(((int64_t)(p.t0 + tl) / p.lpow[l]) % CR) + 1;
            rp = nc - 1;
            if (l > 0 && nc <= TK) continue;                          // every candidate is kept: nothing to accumulate
            if (np <= 0) continue;
            nchunk = (np + PPC - 1) / PPC;
            group_sync();                                             // (SPLIT: every warp has written the same list)
        } else {
            np = rp = 0;                                              // of query lane mod PK
            for (int j = 0; j < PK; ++j) {
                if (tl + j >= p.Tq) break;
                int n = list_of(j).load(p, l, (qidx + (int64_t)j * p.Hkv) * TK, nblk, 4, lane);
                const int right = (n - 1) * CR + (int)(((int64_t)(p.t0 + tl + j) / p.lpow[l]) % CR);
                if (l > 0 && right < TK) n = 0;                       // every candidate is kept: nothing to accumulate
                if (kAlone && alone >= 0 && j != alone) n = 0;
                if (l > 0 && n > 0) {
                    uint32_t* bits = bits_of(j);
                    for (int i = lane; i < (right + 32) / 32; i += 32) bits[i] = 0u;
                    __syncwarp();
                    mark_kept<32>(p, l, (qidx + (int64_t)j * p.Hkv) * TK, list_of(j), n, CR, bits, lane);
                }
                if (lane % PK == j) { np = n; rp = right; }
            }
            __syncwarp();
            walk.start(list_of(lane % PK), l > 0 ? bits_of(lane % PK) : nullptr, np, rp);
        }

        const uint32_t bstride = (uint32_t)p.Hkv * C::BLOCK;                // (a grid has at most 65535 KV heads)
        const unsigned char* blk = reinterpret_cast<const unsigned char*>(p.blk[l]) + ((int64_t)b * nblk * p.Hkv + hk) * C::BLOCK;
        const unsigned char* tab = reinterpret_cast<const unsigned char*>(p.tab);
        int n0 = 0, n1 = 0;                                           // the parents of the chunk whose keys were fetched last
        auto fill_keys = [&](int c) {                                 // chunk c of this level (several queries: of n0, c being this lane's row)
            if constexpr (PK == 1) n0 = par[c * PPC];
            kring.template copy<C::PB>(0, blk + (uint64_t)(uint32_t)n0 * bstride, lane);
            if constexpr (X3) kring.template copy<16>(C::DATA, blk + (uint64_t)(uint32_t)n0 * bstride + C::FACS_OFF, lane);
            if constexpr (CR == 8) {
                n1 = c * PPC + 1 < np ? par[c * PPC + 1] : n0;        // past the end of the list: masked, any finite block
                kring.template copy<C::PB>(C::PB, blk + (uint64_t)(uint32_t)n1 * bstride + 2 * C::ODD, lane);
                if constexpr (X3) kring.template copy<16>(C::DATA + 16, blk + (uint64_t)(uint32_t)n1 * bstride + C::FACS_OFF, lane);
            }
            if constexpr (PK > 1) { copy_tab_rows<PK, C::TAB>(kring, C::TAB_OFF, tab, c, lane); return; }
            const unsigned char* row = tab + (uint32_t)(rp - 16 * c) * C::TAB;
            kring.template copy<C::TAB>(C::TAB_OFF, row, lane);
            if constexpr (C::DUAL) kring.template copy<C::TAB>(C::TAB_OFF + C::TAB, rp - 16 * c >= 8 ? row - 8 * C::TAB : row, lane);
        };
        auto fill_values = [&]() {                                    // of the same chunk
            const uint32_t at = NSTG > 1 ? kring.fill + C::KSLOT : vring.fill;
            kring.template copy_to<C::PB>(at, blk + (uint64_t)(uint32_t)n0 * bstride + C::PB, lane);
            if constexpr (CR == 8) kring.template copy_to<C::PB>(at + C::PB, blk + (uint64_t)(uint32_t)n1 * bstride + C::PB, lane);
        };
        kring.start();
        vring.start();
        // several queries: the masks (of this lane's query) of the chunks that are on their way, and whether the chunk behind them exists
        constexpr int AHEAD = NSTG == 1 ? 1 : NSTG - 1;
        uint32_t masks[AHEAD];
        int pending = 0;
        bool more = true;
        int next = first;
        auto fetch_keys = [&](int slot) {
            if constexpr (PK == 1) {
                more = next < nchunk;
                if (more) fill_keys(next);
            } else {
                n0 = more ? walk.step() : -1;
                more = n0 >= 0;
                masks[slot] = more ? walk.mask() : 0u;
                if (more) { fill_keys(walk.row()); ++pending; }
            }
        };
#pragma unroll
        for (int s = 0; s < AHEAD; ++s, next += step) {
            fetch_keys(s);
            if constexpr (NSTG == 1) kring.commit();
            if (more) fill_values();
            if constexpr (NSTG == 1) vring.commit(); else kring.commit();
        }
        if (PK == 1 && l > 0) {                                       // found while the first blocks are on their way
            constexpr int NT = SPLIT ? kAccSplitWarps * 32 : 32;
            const int me = SPLIT ? (int)threadIdx.x : lane;
            for (int i = me; i < (rp + 32) / 32; i += NT) selw[i] = 0u;
            group_sync();
            mark_kept<NT>(p, l, qidx * TK, par, np, CR, selw, me);
            if constexpr (SPLIT) __syncthreads();
        }
        auto chunk_mask = [&](int c) {                                // the chunk's candidates that accumulate
            uint32_t mask = 0xffffu;
            if (l > 0) mask &= ~(selw[c >> 1] >> ((16 * c) & 31));
            if (16 * c + 15 > rp) mask &= (2u << (rp - 16 * c)) - 1u;
            return mask;
        };
        float2 fac[2] = {make_float2(1.f, 1.f), make_float2(1.f, 1.f)};
        auto scores = [&](uint32_t slot, uint32_t mask, const LaneBase<D, X3, CR>& lb, float (&S)[NH][4]) {
            chunk_factors<D, X3, CR>(slot, fac);
            score_t<T, D, X3, NH, CR>(lb, slot, r, q, S, tab_of_lane);
            if constexpr (X3) {
                const float f0 = fac[0].x * q.inv, f1 = fac[1].x * q.inv;
#pragma unroll
                for (int h = 0; h < NH; ++h) { S[h][0] *= f0; S[h][1] *= f0; S[h][2] *= f1; S[h][3] *= f1; }
            }
            if (mask != 0xffffu) {
                const bool c0 = (mask >> g) & 1, c1 = (mask >> (g + 8)) & 1;
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    S[h][0] = c0 ? S[h][0] : -INFINITY; S[h][1] = c0 ? S[h][1] : -INFINITY;
                    S[h][2] = c1 ? S[h][2] : -INFINITY; S[h][3] = c1 ? S[h][3] : -INFINITY;
                }
            }
        };
        auto head_max = [&](float a, float b) {                       // over the lanes of a head
            float m = fmaxf(a, b);
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
            return fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
        };
        auto rescale = [&](int h, int e, float n) {                   // the accumulators of a head to another reference
            const float f = X3 ? __expf(m_run[h][e] - n) : ex2_approx(m_run2[h][e] - n * kLog2e);
            m_run[h][e] = n; m_run2[h][e] = n * kLog2e;
            s_run[h][e] *= f;
#pragma unroll
            for (int i = 0; i < MT; ++i) { O[h][i][e] *= f; O[h][i][2 + e] *= f; }
        };
#pragma unroll 1
        for (int c = first; PK > 1 ? pending > 0 : c < (SPLIT ? nchunk + first : nchunk); c += step) {      // SPLIT: rounds of W chunks, some of the last missing
            uint32_t mask;                                            // the chunk's candidates that accumulate
            bool any;
            if constexpr (PK > 1) {
                any = __any_sync(0xffffffffu, masks[0] != 0u);
                mask = __shfl_sync(0xffffffffu, masks[0], QC::of_pair(r));        // those of the lane's columns
                --pending;
#pragma unroll
                for (int s = 0; s + 1 < AHEAD; ++s) masks[s] = masks[s + 1];
            }
            if constexpr (NSTG > 1) {
                __syncwarp();                                         // everybody is done with the slots that are refilled now
                fetch_keys(AHEAD - 1);
                if (more) fill_values();
                kring.commit();
                next += step;
            }
            if constexpr (PK == 1) {
                mask = SPLIT && c >= nchunk ? 0u : chunk_mask(c);
                any = mask != 0u;
            }
            const uint32_t keys = kring.template wait<NSTG == 1 ? 1 : NSTG - 1>();
            const LaneBase<D, X3, CR> lb(keys, keys, lane);
            float S[NH][4];
            if (any) {
                scores(keys, mask, lb, S);
            } else {                                                  // nothing to accumulate
#pragma unroll
                for (int h = 0; h < NH; ++h) S[h][0] = S[h][1] = S[h][2] = S[h][3] = -INFINITY;
            }
            if constexpr (NSTG == 1) {
#pragma unroll
                for (int h = 0; h < NH; ++h) consumed(S[h]);
                if constexpr (X3) asm volatile("" ::"f"(fac[0].x), "f"(fac[0].y), "f"(fac[1].x), "f"(fac[1].y) : "memory");
                __syncwarp();                                         // everybody is done with the keys
                fetch_keys(0);
                kring.commit();
            }
            auto wait_values = [&]() {                                // (of a chunk fetched as one they are here already)
                if constexpr (NSTG == 1) return vring.template wait<1>(); else return keys + C::KSLOT;
            };
            auto values_done = [&]() {                                // and with the values: the next chunk's follow
                if constexpr (NSTG == 1) {
                    __syncwarp();
                    if (more) fill_values();
                    vring.commit();
                    next += step;
                }
            };
            if (!SPLIT && !any) {
                wait_values();
                values_done();
                continue;
            }
            // exponents relative to the reference; fp32 storage keeps the plain difference (an exponent re-based by log2 e rounds
            // at 1e-6 relative)
            float ex[NH][4];
            auto exponents = [&]() {
#pragma unroll
                for (int h = 0; h < NH; ++h)
#pragma unroll
                    for (int i = 0; i < 4; ++i) ex[h][i] = X3 ? S[h][i] - m_run[h][i & 1] : fmaf(S[h][i], kLog2e, -m_run2[h][i & 1]);
            };
            exponents();
            float top = ex[0][0];
#pragma unroll
            for (int h = 0; h < NH; ++h)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    top = fmaxf(top, fmaxf(ex[h][e], ex[h][2 + e]));
                    m_true[h][e] = fmaxf(m_true[h][e], fmaxf(S[h][e], S[h][2 + e]));
                }
            constexpr float kMove = X3 ? kLazyMax : kLazyMax * kLog2e;
            float after[SPLIT ? NH : 1][2];                           // the reference behind the round's last chunk
            bool moved;
            if constexpr (SPLIT) {
                moved = __syncthreads_or(top > kMove);
                if (CL > 1) {
                    uint32_t* v = votes + 8 * (round & 1);
                    if ((int)threadIdx.x < CL) st_cluster(cluster_addr(v + rank, threadIdx.x), moved);
                    cluster_sync();
                    moved = false;
                    for (int i = 0; i < CL; ++i) moved |= v[i] != 0u;
                    ++round;
                }
                if (moved) {
                    float* st = exchange;
#pragma unroll
                    for (int h = 0; h < NH; ++h)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float m = head_max(S[h][e], S[h][2 + e]);
                            if (g == 0) st[warp * 48 + 8 * h + 2 * r + e] = m;
                            after[h][e] = m_run[h][e];
                        }
                    if (CL > 1) cluster_sync(); else __syncthreads();   // (the vote of the next round orders these reads before its writes)
                    float mine[NH][2];
                    for (int blk = 0; blk < CL; ++blk) {
                        const uint32_t from = cluster_addr(st + 2 * r, blk);
                        float m[kAccSplitWarps][NH][2];
#pragma unroll
                        for (int w = 0; w < kAccSplitWarps; ++w)
#pragma unroll
                            for (int h = 0; h < NH; ++h) {
                                const float2 x = ld_cluster2(from + 4 * (w * 48 + 8 * h));
                                m[w][h][0] = x.x; m[w][h][1] = x.y;
                            }
#pragma unroll
                        for (int w = 0; w < kAccSplitWarps; ++w) {
                            float t = -INFINITY;
#pragma unroll
                            for (int h = 0; h < NH; ++h)
#pragma unroll
                                for (int e = 0; e < 2; ++e)
                                    t = fmaxf(t, X3 ? m[w][h][e] - after[h][e] : fmaf(m[w][h][e], kLog2e, -(after[h][e] * kLog2e)));
                            const bool move = __any_sync(0xffffffffu, t > kMove);
#pragma unroll
                            for (int h = 0; h < NH; ++h)
#pragma unroll
                                for (int e = 0; e < 2; ++e) {
                                    if (move) after[h][e] = fmaxf(after[h][e], m[w][h][e]);
                                    if (w == warp && blk == rank) mine[h][e] = after[h][e];
                                }
                        }
                    }
                    bool later = false;                               // does a later chunk of the round move it again?
#pragma unroll
                    for (int h = 0; h < NH; ++h)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float n = any ? mine[h][e] : after[h][e];
                            later |= n != after[h][e];
                            rescale(h, e, n);
                        }
                    moved = __any_sync(0xffffffffu, later);
                    exponents();
                }
                if (!any) {
                    wait_values();
                    values_done();
                    continue;
                }
            } else {
                const uint32_t over = __ballot_sync(0xffffffffu, top > kMove);
                moved = over != 0u;
                if (moved) {
                    const bool mine = PK == 1 || (over & QC::lanes_of_pair(r)) != 0u;      // a query's reference follows its own scores
#pragma unroll
                    for (int h = 0; h < NH; ++h)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float m = head_max(S[h][e], S[h][2 + e]);
                            rescale(h, e, mine ? fmaxf(m_run[h][e], m) : m_run[h][e]);
                        }
                    exponents();
                }
            }
            uint32_t pb[NH][2], pl[X3 ? NH : 1][2];
            float ratio[2], vfac = fac[0].y;                          // split-half: what brings the block's values back
            if constexpr (X3 && CR == 8) vfac = common_factor(fac[0].y, fac[1].y, ratio);
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                float P[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) P[i] = X3 ? __expf(ex[h][i]) : ex2_approx(ex[h][i]);
                s_run[h][0] += P[0] + P[2];
                s_run[h][1] += P[1] + P[3];
                if constexpr (X3) {
                    uint32_t h0, l0, h1, l1;
                    if constexpr (CR == 8) { P[0] *= ratio[0]; P[1] *= ratio[0]; P[2] *= ratio[1]; P[3] *= ratio[1]; }
                    split_half2(P[0], P[1], h0, l0); split_half2(P[2], P[3], h1, l1);
                    pb[h][0] = movm(h0); pb[h][1] = movm(h1);
                    pl[X3 ? h : 0][0] = movm(l0); pl[X3 ? h : 0][1] = movm(l1);
                } else {
                    pb[h][0] = movm(F::pack(P[0], P[1])); pb[h][1] = movm(F::pack(P[2], P[3]));
                }
            }
            const uint32_t values = wait_values();
            const LaneBase<D, X3, CR> lv(values, values, lane);
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                uint32_t va[4];
                value_frag<D, X3, CR>(lv, 0, i, va);
                if constexpr (X3) {
                    // summed from zero and then added with a round-to-nearest fp32 add: the tensor core's own accumulation
                    // truncates, and over the ~10^3 chunks of a query that bias would reach 1e-4 relative
                    uint32_t vl[4];
                    value_frag<D, X3, CR>(lv, 1, i, vl);
#pragma unroll
                    for (int h = 0; h < NH; ++h) {
                        float acc[4];
                        mma_zero<__half>(acc, va, pl[X3 ? h : 0][0], pl[X3 ? h : 0][1]);
                        mma_acc<FT>(acc, vl, pb[h][0], pb[h][1]);
                        mma_acc<FT>(acc, va, pb[h][0], pb[h][1]);
#pragma unroll
                        for (int u = 0; u < 4; ++u) O[h][i][u] = fmaf(acc[u], vfac, O[h][i][u]);
                    }
                } else {
#pragma unroll
                    for (int h = 0; h < NH; ++h) mma_acc<FT>(O[h][i], va, pb[h][0], pb[h][1]);
                }
            }
            if constexpr (SPLIT) {
                if (moved) {
#pragma unroll
                    for (int h = 0; h < NH; ++h)
#pragma unroll
                        for (int e = 0; e < 2; ++e) rescale(h, e, after[h][e]);
                }
            }
#pragma unroll
            for (int h = 0; h < NH; ++h)
#pragma unroll
                for (int i = 0; i < MT; ++i) consumed(O[h][i]);
            values_done();
        }
    }

    // ---- totals over the lanes of a head ----
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                s_run[h][e] += __shfl_xor_sync(0xffffffffu, s_run[h][e], o);
                m_true[h][e] = fmaxf(m_true[h][e], __shfl_xor_sync(0xffffffffu, m_true[h][e], o));
            }
    if constexpr (SPLIT) {
        // Merge the warps' partial states (few queries: a group's chunks are spread over the warps of a block or of several).  All
        // followed the same references: their sums add up as they are.
        kring.idle();
        if (CL > 1) cluster_sync(); else __syncthreads();             // all rings are idle: their memory is free, and so is the exchange
        float* st = exchange;                                         // [W][3][16]: m_run, m_true, s; the block's in [0]
        float* po = reinterpret_cast<float*>(wbase);                  // this warp's O, [16 heads][D]; the block's in the first warp's
        float* bo = reinterpret_cast<float*>(smem_raw);
        if (g == 0) {
#pragma unroll
            for (int h = 0; h < NH; ++h)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int head = 8 * h + 2 * r + e;
                    st[(warp * 3 + 0) * 16 + head] = m_run[h][e]; st[(warp * 3 + 1) * 16 + head] = m_true[h][e]; st[(warp * 3 + 2) * 16 + head] = s_run[h][e];
                }
        }
#pragma unroll
        for (int h = 0; h < NH; ++h)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int head = 8 * h + 2 * r + e;
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    po[head * D + C::VB * g + 2 * i] = O[h][i][e];
                    po[head * D + C::VB * g + 2 * i + 1] = O[h][i][2 + e];
                }
            }
        __syncthreads();
        for (int i = threadIdx.x; i < G * D; i += blockDim.x) {
            float o = bo[i];
#pragma unroll
            for (int w = 1; w < kAccSplitWarps; ++w) o += reinterpret_cast<const float*>(smem_raw + w * per_warp)[i];
            bo[i] = o;
        }
        if (threadIdx.x < 8 * NH) {
            float mt = st[16 + threadIdx.x], s = st[32 + threadIdx.x];
            for (int w = 1; w < W; ++w) { mt = fmaxf(mt, st[w * 48 + 16 + threadIdx.x]); s += st[w * 48 + 32 + threadIdx.x]; }
            st[16 + threadIdx.x] = mt; st[32 + threadIdx.x] = s;
        }
        if (CL > 1) cluster_sync(); else __syncthreads();
        const int part = (G * D + CL - 1) / CL;                       // this block's share of the results
        for (int i = rank * part + (int)threadIdx.x; i < min(G * D, (rank + 1) * part); i += blockDim.x) {
            const int head = i / D;
            float o = 0.f, s = 0.f, mt = kNone;
            for (int c = 0; c < CL; ++c) {
                o += ld_cluster(cluster_addr(bo + i, c));
                s += ld_cluster(cluster_addr(st + 32 + head, c));
                mt = fmaxf(mt, ld_cluster(cluster_addr(st + 16 + head, c)));
            }
            reinterpret_cast<T*>(p.out)[hbase * D + i] = from_f<T>(o / s);
            if (i % D == 0) { p.gmax[hbase + head] = mt; p.gsum[hbase + head] = s * __expf(st[head] - mt); }
        }
        if (CL > 1) cluster_sync();                                   // nobody leaves while others read from it
    } else {
    if constexpr (kAlone) {
        bool nan = false;
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int u = 0; u < 4; ++u) nan |= O[0][i][u] != O[0][i][u];
        if (alone < 0 && __any_sync(0xffffffffu, nan)) { alone = 0; goto walk_again; }
    }
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int j = QC::of_pair(r), head = PK == 1 ? 8 * h + 2 * r + e : (2 * r + e) % GP;
            if (head >= G || (PK > 1 && tl + j >= p.Tq) || (kAlone && alone >= 0 && j != alone)) continue;
            const int64_t at = hbase + (int64_t)j * p.H + head;
            const float inv = 1.f / s_run[h][e];
            T* orow = reinterpret_cast<T*>(p.out) + at * D + C::VB * g;
            if constexpr (sizeof(T) == 4) {
#pragma unroll
                for (int i = 0; i < MT / 2; ++i)
                    reinterpret_cast<float4*>(orow)[i] = make_float4(O[h][2 * i][e] * inv, O[h][2 * i][2 + e] * inv, O[h][2 * i + 1][e] * inv, O[h][2 * i + 1][2 + e] * inv);
            } else {
                uint32_t w[MT];
#pragma unroll
                for (int i = 0; i < MT; ++i) w[i] = Frag<typename std::conditional<sizeof(T) == 4, __half, T>::type>::pack(O[h][i][e] * inv, O[h][i][2 + e] * inv);
                if constexpr (MT >= 4) {
#pragma unroll
                    for (int i = 0; i < MT / 4; ++i) reinterpret_cast<uint4*>(orow)[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
                } else {
                    *reinterpret_cast<uint2*>(orow) = make_uint2(w[0], w[1]);
                }
            }
            if (g == 0) { p.gmax[at] = m_true[h][e]; p.gsum[at] = s_run[h][e] * __expf(m_run[h][e] - m_true[h][e]); }
        }
    if (kAlone && alone >= 0 && ++alone < PK) goto walk_again;
    }
}

// One warp per group, or per PK queries.
template <typename T, int D, bool X3, int NH, int CR, int PK>
static int launch_acc_warps(const AttnParams& p, cudaStream_t st) {
    const size_t per_warp = walk_warp_bytes<AccRings<D, X3, NH, CR, PK>, PK>(walk_layout(p, CR));
    // warps per block: as many resident warps as registers allow, fewer where long parent lists leave no room for the rings
    const int max_warps = kAccWarps * acc_min_blocks<D, X3, NH, CR>();
    int W = 1, best = 0;
    for (int w = kAccWarps; w >= 1; --w) {
        if (w == 3) continue;
        int blocks = (int)(228 * 1024 / (w * per_warp + 1024));
        if (blocks * w > max_warps) blocks = max_warps / w;
        if (blocks > 0 && blocks * w > best) { best = blocks * w; W = w; }
    }
    if (best == 0 || W * per_warp > 227 * 1024) return HTREE_E_UNSUPPORTED;
    auto* k = acc_mma_kernel<T, D, X3, NH, CR, false, PK>;
    static SmemLimit shared;
    const cudaError_t e = shared.raise((const void*)k, W * per_warp);
    if (e != cudaSuccess) return (int)e;
    return launch_chained(k, dim3((p.Tq + PK * W - 1) / (PK * W), p.B * p.Hkv), dim3(W * 32), W * per_warp, st, p);
}

template <typename T, int D, bool X3, int NH, int CR>
static int launch_acc_cr(const AttnParams& p, cudaStream_t st) {
    // Few groups: one block of 8 warps per group.  Below two groups per SM the chip has room for all their warps at once, and
    // a single warp's walk over its chunks (about 1 us each) would be the whole time of the call.  Calls whose state the
    // backward reads (they keep their selections) always take one warp per group: a query's result then does not depend on
    // how many queries share the call.
    const int64_t groups = (int64_t)p.Tq * p.B * p.Hkv;
    const size_t split_smem = kAccSplitWarps * (AccRings<D, X3, NH, CR, 1, true>::kBytes + 48 * sizeof(float)) + 64 + walk_lists_bytes(walk_layout(p, CR));
    if ((p.flags & kFlagSplitOk) && groups <= 2 * 148 && split_smem <= 227 * 1024) {
        auto* k = acc_mma_kernel<T, D, X3, NH, CR, true, 1>;
        static SmemLimit shared;
        const cudaError_t e = shared.raise((const void*)k, split_smem);
        if (e != cudaSuccess) return (int)e;
        // Blocks per group: while each has an SM, and as a level has chunks for their warps.  A round of chunks ends in a barrier of the
        // cluster, and a walk over 128 chunks was 16 rounds of one block: 4 x 1 queries against 16384 positions, 16 heads of 128, 8 blocks
        // each: 29 -> 20 us; 5 queries of one head against 512 leaf parents: the call 118 -> 71 us.
        // (Chunks of 4 KB pass so fast that a cluster's barriers have to be shared by four rounds.)
        constexpr int rounds = TForm<D, X3, CR>::VSLOT >= 4096 ? 1 : 4;
        const int leaf = (p.ln[0] + CR - 1) / CR, chunks = ((p.TK < leaf ? p.TK : leaf) * CR + 15) / 16;
        int CL = 1;
        while (CL < 8 && 2 * CL * groups <= 148 && 2 * CL * kAccSplitWarps * rounds <= chunks) CL *= 2;
        return launch_clusters(k, CL, dim3(p.Tq, p.B * p.Hkv), dim3(kAccSplitWarps * 32), split_smem, st, p);
    }
    if constexpr (NH == 1 && CR == 16) {
        const int PK = queries_per_warp(CR, p.G, p.TK, (p.ln[0] + CR - 1) / CR, groups);
        int rc = HTREE_E_UNSUPPORTED;
        if (PK == 2) rc = launch_acc_warps<T, D, X3, NH, CR, 2>(p, st);
        if (PK == 4) rc = launch_acc_warps<T, D, X3, NH, CR, 4>(p, st);
        if (rc != HTREE_E_UNSUPPORTED) return rc;
    }
    return launch_acc_warps<T, D, X3, NH, CR, 1>(p, st);
}

template <typename T, int D, bool X3>
static int launch_acc_t(const AttnParams& p, cudaStream_t st) {
    if (p.CR == 16) return p.G <= 8 ? launch_acc_cr<T, D, X3, 1, 16>(p, st) : launch_acc_cr<T, D, X3, 2, 16>(p, st);
    return p.G <= 8 ? launch_acc_cr<T, D, X3, 1, 8>(p, st) : launch_acc_cr<T, D, X3, 2, 8>(p, st);
}
template <typename T>
static int launch_acc_d(const AttnParams& p, cudaStream_t st) {
    constexpr bool F32 = std::is_same<T, float>::value;
    return p.K == 128 ? launch_acc_t<T, 128, F32>(p, st) : p.K == 64 ? launch_acc_t<T, 64, F32>(p, st) : launch_acc_t<T, 32, true>(p, st);
}

// The per-warp parent list, kept bits and ring must fit one warp into an SM's shared memory.
bool acc_mma_supported(const AttnParams& p, int dtype) {
    if (!pack_supported(dtype, p.K, p.V, p.CR) || p.G > 16 || !p.tab) return false;
    for (int l = 0; l < p.L; ++l) if (!p.blk[l]) return false;
    const size_t slot = (pack_split(dtype, p.K) ? 2 : 1) * (size_t)p.K * 64 + 4 * p.K;
    return 3 * slot + 512 + walk_layout(p, p.CR).list + walk_layout(p, p.CR).bits <= 227 * 1024;
}

int launch_acc_mma(const AttnParams& p, int dtype, cudaStream_t st) {
    switch (dtype) {
        case HTREE_F32: return launch_acc_d<float>(p, st);
        case HTREE_BF16: return launch_acc_d<__nv_bfloat16>(p, st);
        default: return launch_acc_d<__half>(p, st);
    }
}

}  // namespace htree
