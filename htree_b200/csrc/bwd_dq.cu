// Query-stationary pass of the backward: dq, and P and dS of every visit for the parent-stationary pass (bwd_tform.cuh).
// One warp per (batch, query position, KV head) group, all levels in one launch.  Replaces
// htree_bwd_preprocess_delta_kernel, htree_bwd_build_parent_mask_kernel and htree_bwd_dq_bottom/upper_kernel
// (src/backward.py:45-436); arithmetic of src/naive.py:333-384 with the forward's scores, bit for bit.  Per chunk:
//   dP^T = V dO^T,  S^T = K' q^,  P = exp(S - gmax) / gsum,  dS = P (dP - D),  dq^T += K~^T dS^T
// with K~ = scale R(-distance) K', its fragments transposed by the load: rotated back into the query's frame in registers, or, split-half,
// dq^T += R(-distance) (K'^T dS^T), which leaves the keys' planes as they are.
//
// Bound by shared-memory reads (69% of the pipe with 16 heads of 128 a group, 83% with 8): values and keys once each, the keys once more
// transposed, table rows.  4 x 65536 positions, 64 heads of 128: this pass 129 ms and the parent-stationary one 86 ms, where the single
// kernel with reductions took 360 ms.
#include "bwd_tform.cuh"

namespace htree {

template <int D, bool X3, int PK>
constexpr int dq_stages() { return D * (X3 ? 2 : 1) >= 128 ? 2 : PK > 1 ? 2 : 3; }     // slots of 8 KB: warps matter more than depth
// A slot: the keys with their table rows, 16-bit: those rows in lane order too (bwd_tform.cuh), the values.
template <int D, bool X3, int CR, int PK>
constexpr int dq_values() { using C = TForm<D, X3, CR, PK>; return C::KSLOT + (X3 ? 0 : C::NTAB * C::TAB); }
// Warps per block and blocks per SM: registers first.  The ring takes nearly all of the SM's L1, so anything that spills is
// re-read from L2 in every chunk: with 180 bytes of spills, groups of 16 heads of 128 spent 4.6 of 9.4 cycles per instruction
// waiting for it.  Those run as blocks of one warp (at most 20 bytes of spills at 12 warps per SM; the compiler keeps 150 in larger
// blocks): 64K positions, 4 KV heads 53 -> 31.6 ms, against 33.3 ms for 8 warps per SM with nothing spilled.  32-wide heads fit
// 16 warps (10.2 -> 9.9 ms at 12000 positions, 512 nodes per layer).
template <int D, bool X3, int NH>
constexpr int dq_warps() { return D == 128 && !X3 && NH == 2 ? 1 : 4; }
template <int D, bool X3, int NH>
constexpr int dq_min_blocks() { return D == 32 && NH == 1 ? 4 : (D == 128 && (X3 || NH == 2)) ? (X3 ? 2 : 12) : (X3 && NH == 2) ? 2 : 3; }

// SUMS: 16-bit dq takes R(-distance) (K'^T dS^T) too, whose distance may differ by query.  Calls whose queries could share a warp
// take it however many there are, so that dq does not depend on that; elsewhere rotating the keys is 4% faster.
template <typename T, int D, bool X3, int NH, int CR, int PK, bool SUMS>
__global__ void __launch_bounds__(dq_warps<D, X3, NH>() * 32, dq_min_blocks<D, X3, NH>()) bwd_dq_kernel(const __grid_constant__ BwdParams bp) {
    chain_enter();
    static_assert(PK == 1 || (NH == 1 && CR == 16 && (X3 || SUMS)), "several queries share a warp's 8 columns");
    using C = TForm<D, X3, CR, PK>;
    using QC = Cols<PK>;
    using BF = BForm<D, X3, NH, CR>;
    using F = Frag<typename std::conditional<X3, __half, T>::type>;
    using FT = typename std::conditional<X3, __half, T>::type;
    using FS = Frag<__half>;
    constexpr int KS = C::KS, PPT = C::PPT, PPC = C::PPC, HALF = C::HALF, GP = QC::GP;
    constexpr int NSTG = dq_stages<D, X3, PK>();
    using Ring = WarpRing<NSTG, dq_values<D, X3, CR, PK>() + C::VSLOT>;
    constexpr int VOFF = dq_values<D, X3, CR, PK>();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const AttnParams& p = bp.a;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, r = lane & 3;
    const int W = blockDim.x >> 5;
    const int gi = (int)(gridDim.x - 1 - blockIdx.x) * W + warp;      // the longest walks first: they would be the tail of the launch
    const int qi = gi * PK;
    const int sub = bp.sub0 + blockIdx.y, unit = sub / bp.nw;
    const int tl = (sub % bp.nw) * bp.subq + qi;
    if (qi >= bp.subq || tl >= p.Tq) return;
    const int b = unit / p.Hkv, hk = unit % p.Hkv;
    const int G = p.G, TK = p.TK, L = p.L;
    const int grp = blockIdx.y * bp.ng + gi;

    const WalkLayout lay = walk_layout(p, CR);
    const size_t per_warp = walk_warp_bytes<Ring, PK>(lay);
    unsigned char* wbase = smem_raw + warp * per_warp;
    Ring ring;
    ring.init(wbase);
    auto list_of = [&](int j) { return ParentList{wbase + Ring::kBytes + j * lay.list, lay.narrow}; };        // query tl + j
    auto bits_of = [&](int j) { return reinterpret_cast<uint32_t*>(wbase + Ring::kBytes + PK * lay.list + j * lay.bits); };
    const ParentList par = list_of(0);
    uint32_t* selw = bits_of(0);
    const int64_t hbase = ((int64_t)b * p.Tq + tl) * p.H + (int64_t)hk * G;
    const int64_t qidx = ((int64_t)b * p.Tq + tl) * p.Hkv + hk;

    QueryRegs<T, D, X3, NH> q;
    // the rows of column 8h + g (operands) and of columns 8h + 2r, + 1 (results), or -1
    auto row_of_lane = [&](int h) -> int64_t {
        const int j = QC::of_lane(g), head = PK == 1 ? 8 * h + g : g % GP;
        return head < G && (PK == 1 || tl + j < p.Tq) ? hbase + (int64_t)j * p.H + head : -1;
    };
    auto row_of_pair = [&](int h, int e) -> int64_t {
        const int j = QC::of_pair(r), head = PK == 1 ? 8 * h + 2 * r + e : (2 * r + e) % GP;
        return head < G && (PK == 1 || tl + j < p.Tq) ? hbase + (int64_t)j * p.H + head : -1;
    };
    const uint32_t tab_of_lane = PK == 1 ? 0 : QC::of_lane(g) * C::TAB, tab_of_pair = PK == 1 ? 0 : QC::of_pair(r) * C::TAB;
    load_query<T, D, X3, NH, PK>([&](int h) -> const T* { const int64_t at = row_of_lane(h); return at < 0 ? nullptr : reinterpret_cast<const T*>(p.q) + at * D; },
                                 r, p.scale, q);
    uint32_t dO[NH][2][KS], dOl[X3 ? NH : 1][2][X3 ? KS : 1];
    float Drow[NH][2], lse[NH][2], ginv[NH][2];
    bool zero = true;                                   // is this lane's dO all zero?
    bool finite = true;                                 // are its dO, dO . out and q finite?
    constexpr float kPScale = 16384.f;                  // split-half: P is carried times 2^14
    float dscale = 1.f, dinv = 1.f;                     // split-half: dO times dscale; dinv = 1 / (dscale kPScale), for P dO and for dS
    float bound_v = 0.f, bound_d = 0.f;                 // |P (dP - D)| as carried <= bound_v * the value block's factor + bound_d
    float vtop = 0.f, sscale = 1.f;                     // the largest such factor so far; the scale of dS
    if constexpr (X3) {
        float most = 0.f;
#pragma unroll
        for (int h = 0; h < NH; ++h)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                float x[D / 8];
                load_row_piece_f32<T, D>(reinterpret_cast<const T*>(p.dO) + row_of_lane(h) * D + hf * HALF + PPT * r, row_of_lane(h) >= 0, x);
#pragma unroll
                for (int i = 0; i < D / 8; ++i) most = fmaxf(most, fabsf(x[i]));
            }
        dscale = range_scale_coarse(QC::max_of(most));
        dinv = QC::for_pair(pow2_inverse(dscale), r) * (1.f / kPScale);
    }
#pragma unroll
    for (int h = 0; h < NH; ++h) {
        const int64_t row = row_of_lane(h);
        const bool on = row >= 0;
        float sum = 0.f, l1 = 0.f;                      // dO . out and |dO|_1 of this lane's head
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int64_t off = row * D + hf * HALF + PPT * r;
            if constexpr (X3) {
                float x[D / 8], o[D / 8];
                load_row_piece_f32<T, D>(reinterpret_cast<const T*>(p.dO) + off, on, x);
                load_row_piece_f32<T, D>(reinterpret_cast<const T*>(p.out) + off, on, o);
#pragma unroll
                for (int i = 0; i < D / 16; ++i) {
                    x[2 * i] *= dscale; x[2 * i + 1] *= dscale;
                    l1 += fabsf(x[2 * i]) + fabsf(x[2 * i + 1]);
                    sum += x[2 * i] * o[2 * i] + x[2 * i + 1] * o[2 * i + 1];
                    split_half2(x[2 * i], x[2 * i + 1], dO[h][hf][i], dOl[X3 ? h : 0][hf][X3 ? i : 0]);
                }
            } else {
                uint32_t o[KS];
                ldg_vec<PPT / 8>(reinterpret_cast<const T*>(p.dO) + off, on, dO[h][hf]);
                ldg_vec<PPT / 8>(reinterpret_cast<const T*>(p.out) + off, on, o);
#pragma unroll
                for (int i = 0; i < KS; ++i) {
                    const float2 x = F::unpack(dO[h][hf][i]), y = F::unpack(o[i]);
                    sum += x.x * y.x + x.y * y.y;
                    l1 += fabsf(x.x) + fabsf(x.y);
                }
            }
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
        l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
        zero = zero && l1 == 0.f;
        finite = finite && l1 < INFINITY && fabsf(sum) < INFINITY;      // (a sum that overflows counts as one that is not)
        if constexpr (!X3) {
            bound_v = fmaxf(bound_v, QC::max_of(l1));
        } else {
            bound_v = fmaxf(bound_v, kPScale * 16384.f * QC::max_of(l1));      // values are carried below 2^14
            bound_d = fmaxf(bound_d, kPScale * QC::max_of(fabsf(sum)));
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int64_t at = row_of_pair(h, e);
            Drow[h][e] = __shfl_sync(0xffffffffu, sum, 4 * (2 * r + e));
            const float gm = at >= 0 ? p.gmax[at] : 0.f, gs = at >= 0 ? p.gsum[at] : 1.f;
            // 16-bit: P = 2^(S log2 e - lse); split-half: exp(S - gmax) * ginv (an exponent re-based by log2 e rounds at 1e-6)
            lse[h][e] = X3 ? gm : (at >= 0 ? gm * kLog2e + __log2f(gs) : INFINITY);
            ginv[h][e] = at >= 0 ? kPScale / gs : 0.f;
        }
    }

    bound_v = QC::for_pair(bound_v, r); bound_d = QC::for_pair(bound_d, r);
    if constexpr (X3) {                                 // a query without a gradient: factors of zero, which no product has to be made for
        // (and a dS of zeros that is not scaled: the largest scale times a value factor would be infinite)
        if (QC::all_of(zero, r)) { dinv = 0.f; bound_d = 8192.f; }
    }
    // Several queries: those with a dO or q that is not finite.  Their columns of the blocked operands must not meet the records of parents
    // that only a neighbour visited: 0 times infinity is NaN.
    uint32_t spoilt = 0u;
    if constexpr (PK > 1) {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf)
#pragma unroll
            for (int i = 0; i < QueryRegs<T, D, X3, NH>::N; ++i) {
                const uint32_t x = q.v[0][hf][i];
                finite = finite && (X3 ? fabsf(__uint_as_float(x)) < INFINITY : (x & 0x7c00u) != 0x7c00u && (x & 0x7c000000u) != 0x7c000000u);
            }
        const uint32_t off = __ballot_sync(0xffffffffu, !finite);
#pragma unroll
        for (int j = 0; j < PK; ++j) spoilt |= (off >> (4 * GP * j) & ((1u << (4 * GP)) - 1u)) != 0u ? 1u << j : 0u;
    }
    float rescale = 1.f;                                // 16-bit: from dS as carried for dq to dS as carried in the records
    if constexpr (!X3) {
        const uint32_t v = __ldg(bp.range + 1 + unit);
        const float call = ds_scale(__ldg(bp.range), v);
        sscale = fmaxf(ds_scale(__float_as_uint(bound_v), v), call);      // (not smaller: sums of the same row may round differently)
        rescale = call * pow2_inverse(sscale);
#pragma unroll
        for (int h = 0; h < NH; ++h) { Drow[h][0] *= sscale; Drow[h][1] *= sscale; }
    }

    // ---- blocked copies of q and dO for the parent-stationary pass: pairs of heads per word, [half][i][lane]{lo, hi} with
    //      dims x(i, g) = PPT*(g/2) + 2i + (g & 1) (and + D/2) and heads 2r, 2r + 1 ----
#pragma unroll
    for (int h = 0; h < NH; ++h) {
        unsigned char* dst = bp.dob + ((int64_t)grp * NH + h) * BF::QB;
#pragma unroll
        for (int i = 0; i < KS; ++i) {
            *reinterpret_cast<uint2*>(dst + i * 256 + lane * 8) = make_uint2(movm(dO[h][0][i]), movm(dO[h][1][i]));
            if constexpr (X3)
                *reinterpret_cast<uint2*>(dst + D * 16 + i * 256 + lane * 8) =
                    make_uint2(movm(dOl[X3 ? h : 0][0][X3 ? i : 0]), movm(dOl[X3 ? h : 0][1][X3 ? i : 0]));
        }
        unsigned char* qd = bp.qb + ((int64_t)grp * NH + h) * BF::QB;
        if constexpr (X3) {
            // fp32: 16 bytes per lane and tile {lo(2r), lo(2r+1), hi(2r), hi(2r+1)}; this lane has head g, dims PPT*r + j
#pragma unroll
            for (int hf = 0; hf < 2; ++hf)
#pragma unroll
                for (int j = 0; j < PPT; ++j)
                    reinterpret_cast<uint32_t*>(qd)[((j >> 1) * 32 + 4 * (2 * r + (j & 1)) + (g >> 1)) * 4 + 2 * hf + (g & 1)] = q.v[h][hf][j];
        } else {
#pragma unroll
            for (int i = 0; i < KS; ++i)
                *reinterpret_cast<uint2*>(qd + i * 256 + lane * 8) = make_uint2(movm(q.v[h][0][i]), movm(q.v[h][1][i]));
        }
    }

    float dq[NH][KS][4];      // dq^T: dims x(ks, g) (elements 0, 1) and + D/2 (2, 3), heads 2r, 2r + 1
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
        for (int i = 0; i < KS; ++i) dq[h][i][0] = dq[h][i][1] = dq[h][i][2] = dq[h][i][3] = 0.f;

    float back = dinv;                                                // split-half: times dS as carried = dS
    bool select_dS = !X3;                                             // several queries: may dP be infinite where a query has no part in a block?
    bool over = false;                                                // several queries, split-half: does the factor of this one's dK overflow?
    for (int l = L - 1; l >= 0; --l) {
        if (bp.voff[l] < 0) continue;
        const int Nl = p.ln[l];
        const int nblk = (Nl + CR - 1) / CR;
        __syncwarp();
        int np, rp, nchunk = 0;
        UnionWalk<PK> walk;
        if constexpr (PK == 1) {
            np = par.load(p, l, qidx * TK, nblk, 8, lane);
            rp = (np - 1) * CR + (int)(((int64_t)(p.t0 + tl) / p.lpow[l]) % CR);
            if (np <= 0 || (l > 0 && rp + 1 <= TK)) continue;
            nchunk = (np + PPC - 1) / PPC;
            __syncwarp();
        } else {
            np = rp = 0;                                              // of query lane mod PK
            for (int j = 0; j < PK; ++j) {
                if (tl + j >= p.Tq) break;
                int n = list_of(j).load(p, l, (qidx + (int64_t)j * p.Hkv) * TK, nblk, 8, lane);
                n = list_of(j).ascending(p, n, 8, lane);
                const int right = (n - 1) * CR + (int)(((int64_t)(p.t0 + tl + j) / p.lpow[l]) % CR);
                if (l > 0 && right < TK) n = 0;
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
        const int64_t blk0 = (int64_t)b * nblk * p.Hkv + hk;
        const unsigned char* kblk = reinterpret_cast<const unsigned char*>(p.blk[l]) + blk0 * C::BLOCK;
        const unsigned char* vblk = reinterpret_cast<const unsigned char*>(p.vkblk[l]) + blk0 * (C::PL * C::PART);
        const uint32_t kstride = (uint32_t)p.Hkv * C::BLOCK;
        auto fill = [&](int c, int p0) {                              // chunk c; several queries: of parent p0, c being this lane's row
            constexpr int PB = C::PB;
            const uint32_t vstride = (uint32_t)p.Hkv * PB;
            if constexpr (PK == 1) p0 = par[c * PPC];
            ring.template copy<PB>(0, kblk + (uint64_t)(uint32_t)p0 * kstride, lane);
            ring.template copy<PB>(VOFF, vblk + (uint64_t)(uint32_t)p0 * vstride, lane);
            if constexpr (CR == 8) {
                const int p1 = c * PPC + 1 < np ? par[c * PPC + 1] : p0;
                ring.template copy<PB>(C::PB, kblk + (uint64_t)(uint32_t)p1 * kstride + 2 * C::ODD, lane);
                ring.template copy<PB>(VOFF + C::PB, vblk + (uint64_t)(uint32_t)p1 * vstride, lane);
                if constexpr (X3) ring.template copy<16>(C::DATA + 16, kblk + (uint64_t)(uint32_t)p1 * kstride + C::FACS_OFF, lane);
            }
            if constexpr (X3) ring.template copy<16>(C::DATA, kblk + (uint64_t)(uint32_t)p0 * kstride + C::FACS_OFF, lane);
            if constexpr (X3) {
                if constexpr (PK > 1) copy_tab_rows<PK, C::TAB>(ring, C::TAB_OFF, p.tab, c, lane);
                else ring.template copy<C::TAB>(C::TAB_OFF, reinterpret_cast<const unsigned char*>(p.tab) + (uint32_t)(rp - 16 * c) * C::TAB, lane);
            } else {
                // the rows for the scores, then those in lane order for dq, in as few instructions as they fit
                constexpr int PER = C::TAB / 16;
                const int d0 = PK > 1 ? c : rp - 16 * c, d1 = C::DUAL && d0 >= 8 ? d0 - 8 : d0;
#pragma unroll
                for (int i = 0; i < 2 * C::NTAB * PER; i += 32) {
                    const int piece = i + lane, k = piece / PER, j = k % C::NTAB;
                    const int row = PK > 1 ? __shfl_sync(0xffffffffu, d0, j) : j ? d1 : d0;
                    const unsigned char* from = k < C::NTAB ? reinterpret_cast<const unsigned char*>(p.tab) : bp.xtab;
                    if (2 * C::NTAB * PER % 32 == 0 || piece < 2 * C::NTAB * PER)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(ring.fill + C::TAB_OFF + 16 * piece),
                                     "l"(from + (uint32_t)row * C::TAB + 16 * (piece % PER)) : "memory");
                }
            }
        };
        ring.start();
        // this visit's place in its parent's list
        int32_t* cnt = bp.cnt + (int64_t)blockIdx.y * bp.NK + bp.koff[l];
        const int visit0 = grp * bp.MV + bp.voff[l];
        constexpr int AHEAD = NSTG - 1;
        uint32_t masks[AHEAD];                                        // several queries: of the chunks on their way, for this lane's
        uint4 placed = make_uint4(0u, 0u, 0u, 0u);                    // the visit fetched last (its rank arrives during a chunk)
        int next = 0, pending = 0;
        bool more = true;
        auto fetch = [&](int slot) {
            if constexpr (PK == 1) {
                if (next < nchunk) fill(next, 0);
                ++next;
            } else {
                const int parent = more ? walk.step() : -1;
                more = parent >= 0;
                masks[slot] = more ? walk.mask() : 0u;
                if (more) {
                    const int row = walk.row();
                    fill(row, parent);
                    uint32_t rows[2] = {0u, 0u};
#pragma unroll
                    for (int j = 0; j < PK; ++j) rows[j >> 1] |= (uint32_t)__shfl_sync(0xffffffffu, row, j) << (16 * (j & 1));
                    const uint32_t skip = spoilt ? spoilt & ~__ballot_sync(0xffffffffu, walk.rank >= 0) : 0u;
                    if (lane == 0) {
                        if (next) bp.vis[visit0 + next - 1] = placed;
                        placed = make_uint4((uint32_t)parent | skip << 16, (uint32_t)atomicAdd(cnt + parent, 1), rows[0], rows[1]);
                    }
                    ++next; ++pending;
                }
            }
            ring.commit();
        };
#pragma unroll
        for (int s = 0; s < AHEAD; ++s) fetch(s);
        float v = 0.f;                                                // split-half: the largest factor of the values that will be met
        if constexpr (PK == 1) {
            for (int i = lane; i < np; i += 32) {
                bp.rank[visit0 + i] = atomicAdd(cnt + par[i], 1);
                if constexpr (X3) v = fmaxf(v, __ldg(reinterpret_cast<const float*>(kblk + (uint64_t)(uint32_t)par[i] * kstride + C::FACS_OFF) + 1));
            }
            if constexpr (X3) v = redux_max_f32(v, 0xffffffffu);
        } else if constexpr (X3) {
#pragma unroll
            for (int j = 0; j < PK; ++j) {
                const int n = __shfl_sync(0xffffffffu, np, j);
                float x = 0.f;
                for (int i = lane; i < n; i += 32) x = fmaxf(x, __ldg(reinterpret_cast<const float*>(kblk + (uint64_t)(uint32_t)list_of(j)[i] * kstride + C::FACS_OFF) + 1));
                x = redux_max_f32(x, 0xffffffffu);
                if (QC::of_pair(r) == j) v = x;
            }
        }
        if constexpr (X3) {
            // dS's scale follows from a bound, 2^4 to 2^8 above what ordinary data reach at P = 1.  Found per level: per chunk, from the
            // largest |dS| or from the chunk's own factor, cost the pass 5 to 7% (32-wide heads)
            if (v > vtop) {
                const float s = range_scale_coarse(fmaf(bound_v, v, bound_d)), f = s * pow2_inverse(sscale);
                vtop = v; sscale = s; back = dinv * pow2_inverse(s);
#pragma unroll
                for (int h = 0; h < NH; ++h) { Drow[h][0] *= f; Drow[h][1] *= f; }
            }
            float fk = back * q.inv;
            if constexpr (PK > 1) {
                // a block that only a neighbour visits may have values beyond this query's bound: an infinite dP
                select_dS = spoilt != 0u || __any_sync(0xffffffffu, !(bound_v * sscale * redux_max_f32(v, 0xffffffffu) < INFINITY));
                over = fk == INFINITY;                                // (0 of a query that has no part in a visit times it is NaN)
                if (over) fk = 0x1p127f;
            }
            if (g == 0 && r * PK % 4 == 0) bp.fac[((int64_t)grp * L + l) * PK + QC::of_pair(r)] = make_float2(fk, dinv);
        }
        if (PK == 1 && l > 0) {
            for (int i = lane; i < (rp + 32) / 32; i += 32) selw[i] = 0u;
            __syncwarp();
            mark_kept<32>(p, l, qidx * TK, par, np, CR, selw, lane);
        }
#pragma unroll 1
        for (int c = 0; PK > 1 ? pending > 0 : c < nchunk; ++c) {
            uint32_t mask = 0xffffu;
            bool any;
            if constexpr (PK > 1) {
                any = __any_sync(0xffffffffu, masks[0] != 0u);
                mask = __shfl_sync(0xffffffffu, masks[0], QC::of_pair(r));        // of the lane's columns
                --pending;
#pragma unroll
                for (int s = 0; s + 1 < AHEAD; ++s) masks[s] = masks[s + 1];
            }
            __syncwarp();
            fetch(AHEAD - 1);
            if constexpr (PK == 1) {
                if (l > 0) mask &= ~(selw[c >> 1] >> ((16 * c) & 31));
                if (16 * c + 15 > rp) mask &= (2u << (rp - 16 * c)) - 1u;
                any = mask != 0u;
            }
            const uint32_t slot = ring.wait();
            const LaneBase<D, X3, CR> lb(slot, slot + VOFF, lane);
            const uint32_t tabs = slot + C::TAB_OFF;

            uint32_t pw[NH][2], sw[NH][2], pwl[X3 ? NH : 1][2], swl[X3 ? NH : 1][2];   // P^T, dS^T: word w = child g + 8w, heads 2r, 2r+1
            if (!any) {
#pragma unroll
                for (int h = 0; h < NH; ++h)
#pragma unroll
                    for (int w = 0; w < 2; ++w) {
                        pw[h][w] = sw[h][w] = 0u;
                        if constexpr (X3) pwl[X3 ? h : 0][w] = swl[X3 ? h : 0][w] = 0u;
                    }
            } else {
                float dP[NH][4];
#pragma unroll
                for (int ks = 0; ks < KS; ++ks) {
                    uint32_t a[4], al[4];
                    vk_frag<D, X3, CR>(lb, 0, ks, a);
                    if constexpr (X3) vk_frag<D, X3, CR>(lb, 1, ks, al);
#pragma unroll
                    for (int h = 0; h < NH; ++h) {
                        if (ks == 0) mma_zero<FT>(dP[h], a, dO[h][0][0], dO[h][1][0]);
                        else mma_acc<FT>(dP[h], a, dO[h][0][ks], dO[h][1][ks]);
                        if constexpr (X3) {
                            mma_acc<FT>(dP[h], al, dO[h][0][ks], dO[h][1][ks]);
                            mma_acc<FT>(dP[h], a, dOl[X3 ? h : 0][0][X3 ? ks : 0], dOl[X3 ? h : 0][1][X3 ? ks : 0]);
                        }
                    }
                }
                float S[NH][4];
                float2 fac[2];
                chunk_factors<D, X3, CR>(slot, fac);
                score_t<T, D, X3, NH, CR>(lb, slot, r, q, S, tab_of_lane);
                const float sfac[2] = {fac[0].x * q.inv, fac[1].x * q.inv};
                const bool c0 = (mask >> g) & 1, c1 = (mask >> (g + 8)) & 1;
                uint32_t db[NH][2], dbl[X3 ? NH : 1][2];       // dS^T as B fragments (children x heads)
                if constexpr (X3) { fac[0].y *= sscale; fac[1].y *= sscale; }
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    float P[4], dS[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        P[i] = X3 ? __expf(fmaf(S[h][i], sfac[i >> 1], -lse[h][i & 1])) * ginv[h][i & 1] : ex2_approx(fmaf(S[h][i], kLog2e, -lse[h][i & 1]));
                        P[i] = (i < 2 ? c0 : c1) ? P[i] : 0.f;
                        dS[i] = P[i] * fmaf(dP[h][i], X3 ? fac[i >> 1].y : sscale, -Drow[h][i & 1]);
                    }
                    if (PK > 1 && select_dS) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) dS[i] = mask ? dS[i] : 0.f;
                    }
                    if constexpr (X3) {
                        split_half2(P[0], P[1], pw[h][0], pwl[X3 ? h : 0][0]); split_half2(P[2], P[3], pw[h][1], pwl[X3 ? h : 0][1]);
                        split_half2(dS[0], dS[1], sw[h][0], swl[X3 ? h : 0][0]); split_half2(dS[2], dS[3], sw[h][1], swl[X3 ? h : 0][1]);
                        dbl[X3 ? h : 0][0] = movm(swl[X3 ? h : 0][0]); dbl[X3 ? h : 0][1] = movm(swl[X3 ? h : 0][1]);
                    } else {
                        pw[h][0] = F::pack(P[0], P[1]); pw[h][1] = F::pack(P[2], P[3]);
                        sw[h][0] = FS::pack(dS[0], dS[1]); sw[h][1] = FS::pack(dS[2], dS[3]);
                    }
                    db[h][0] = movm(sw[h][0]); db[h][1] = movm(sw[h][1]);
                    if (PK > 1 && X3 && over) {                // what the factor no longer says is in the record
#pragma unroll
                        for (int i = 0; i < 4; ++i) dS[i] = dS[i] == 0.f ? 0.f : dS[i] * INFINITY;
                        sw[h][0] = FS::pack(dS[0], dS[1]); sw[h][1] = FS::pack(dS[2], dS[3]);
                        swl[X3 ? h : 0][0] = swl[X3 ? h : 0][1] = 0u;
                    }
                    if (!X3 && rescale != 1.f) {
                        sw[h][0] = FS::pack(dS[0] * rescale, dS[1] * rescale); sw[h][1] = FS::pack(dS[2] * rescale, dS[3] * rescale);
                    }
                }
                // dq^T += K~^T dS^T: transposed key fragments (rows x(ks, g)), rotated back by the chunk's distance
                if constexpr (!X3) {
                    const uint32_t tx = tabs + (C::NTAB * C::TAB + 2 * KS * (4 * (g & 1) + (g >> 1))) + tab_of_pair;
                    uint32_t cw[KS / 2], sn[KS / 2], cv[C::DUAL ? KS / 2 : 1], sv[C::DUAL ? KS / 2 : 1];      // (cv, sv: the odd parent's distance)
                    lds_x<D>(tx, cw, sn);
                    if constexpr (C::DUAL) lds_x<D>(tx + C::TAB, cv, sv);
#pragma unroll
                    for (int ks = 0; ks < KS; ++ks) {
                        uint32_t m[4], a[4];
                        key_frag_trans<D, X3, CR>(lb, 0, ks, m);
                        const __half2 c2 = half_of(cw[ks / 2], ks & 1), s2 = half_of(sn[ks / 2], ks & 1);
                        if constexpr (SUMS) {            // the chunk's sums are rotated, in fp32
                            const uint32_t am[4] = {m[0], m[2], m[1], m[3]};
                            const float cf = __low2float(c2), sf = __low2float(s2);
                            float acc[4];
                            mma_zero<__half>(acc, am, db[0][0], db[0][1]);
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                dq[0][ks][e] = fmaf(acc[2 + e], sf, fmaf(acc[e], cf, dq[0][ks][e]));
                                dq[0][ks][2 + e] = fmaf(acc[e], -sf, fmaf(acc[2 + e], cf, dq[0][ks][2 + e]));
                            }
                        } else {
                            rotate_x<true>(m[0], m[2], c2, s2, a[0], a[1]);
                            if constexpr (C::DUAL) rotate_x<true>(m[1], m[3], half_of(cv[ks / 2], ks & 1), half_of(sv[ks / 2], ks & 1), a[2], a[3]);
                            else rotate_x<true>(m[1], m[3], c2, s2, a[2], a[3]);
#pragma unroll
                            for (int h = 0; h < NH; ++h) mma_acc<__half>(dq[h][ks], a, db[h][0], db[h][1]);
                        }
                    }
                } else {
                    // Split-half: the keys' planes go into the product as they are, and the chunk's sums are rotated back in fp32 as they
                    // join dq: 8 multiply-adds a tile and half, where rotating the keys put both planes together and split them again.
                    // 2 x 16384 positions, 8 heads of 64: 4.55 -> 3.84 ms; 4096 positions, 8 heads of 128: 652 -> 575 us; 32-wide heads
                    // 1080 -> 914 us; groups of 16 heads within 2% either way.  The same distance from an fp32 evaluation as before.
                    float ratio[2] = {1.f, 1.f}, kfac = fac[0].x;
                    if constexpr (CR == 8 && C::KSCALED) {
                        kfac = common_factor(fac[0].x, fac[1].x, ratio);
                        if (ratio[0] != ratio[1]) {
#pragma unroll
                            for (int h = 0; h < NH; ++h)
#pragma unroll
                                for (int w = 0; w < 2; ++w) {
                                    const __half2 f = __float2half2_rn(ratio[w]);       // (a power of two, at most 1)
                                    db[h][w] = as_u32(__hmul2(as_h2(db[h][w]), f));
                                    dbl[X3 ? h : 0][w] = as_u32(__hmul2(as_h2(dbl[X3 ? h : 0][w]), f));
                                }
                        }
                    }
                    kfac *= back;
                    if (PK > 1 && !mask) kfac = 0.f;           // (the product of another query's range may be infinite, and the sums are zero)
#pragma unroll
                    for (int ks = 0; ks < KS; ++ks) {
                        uint32_t mh[4], ml[4];
                        key_frag_trans<D, X3, CR>(lb, 0, ks, mh);
                        key_frag_trans<D, X3, CR>(lb, 1, ks, ml);
                        float cs, sn;
                        const uint32_t tb = tabs + 4 * (PPT * (g >> 1) + 2 * ks + (g & 1)) + tab_of_pair;
                        asm("ld.shared.f32 %0, [%1];" : "=f"(cs) : "r"(tb));
                        asm("ld.shared.f32 %0, [%1];" : "=f"(sn) : "r"(tb + 4 * HALF));
                        cs *= kfac; sn *= kfac;
                        const uint32_t ah[4] = {mh[0], mh[2], mh[1], mh[3]}, al[4] = {ml[0], ml[2], ml[1], ml[3]};
#pragma unroll
                        for (int h = 0; h < NH; ++h) {
                            // from zero, then round-to-nearest fp32 multiply-adds (the tensor core's accumulation truncates)
                            float acc[4];
                            mma_zero<__half>(acc, ah, dbl[X3 ? h : 0][0], dbl[X3 ? h : 0][1]);
                            mma_acc<__half>(acc, al, db[h][0], db[h][1]);
                            mma_acc<__half>(acc, ah, db[h][0], db[h][1]);
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                dq[h][ks][e] = fmaf(acc[2 + e], sn, fmaf(acc[e], cs, dq[h][ks][e]));
                                dq[h][ks][2 + e] = fmaf(acc[e], -sn, fmaf(acc[2 + e], cs, dq[h][ks][2 + e]));
                            }
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < NH; ++h)
#pragma unroll
                    for (int ks = 0; ks < KS; ++ks) consumed(dq[h][ks]);       // (dP and the scores end in the records)
            }
            // ---- leave P and dS behind, one record per visit ----
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                if constexpr (CR == 16) {
                    const int64_t o = ((int64_t)(visit0 + c) * NH + h) * BF::SB + lane * 8;
                    *reinterpret_cast<uint2*>(bp.stp + o) = make_uint2(pw[h][0], pw[h][1]);
                    *reinterpret_cast<uint2*>(bp.sts + o) = make_uint2(sw[h][0], sw[h][1]);
                    if constexpr (X3) {
                        *reinterpret_cast<uint2*>(bp.stp + o + 256) = make_uint2(pwl[X3 ? h : 0][0], pwl[X3 ? h : 0][1]);
                        *reinterpret_cast<uint2*>(bp.sts + o + 256) = make_uint2(swl[X3 ? h : 0][0], swl[X3 ? h : 0][1]);
                    }
                } else {
#pragma unroll
                    for (int w = 0; w < 2; ++w) {
                        if (2 * c + w < np) {      // (PK == 1)
                            const int64_t o = ((int64_t)(visit0 + 2 * c + w) * NH + h) * BF::SB + lane * 4;
                            *reinterpret_cast<uint32_t*>(bp.stp + o) = pw[h][w];
                            *reinterpret_cast<uint32_t*>(bp.sts + o) = sw[h][w];
                            if constexpr (X3) {
                                *reinterpret_cast<uint32_t*>(bp.stp + o + 128) = pwl[X3 ? h : 0][w];
                                *reinterpret_cast<uint32_t*>(bp.sts + o + 128) = swl[X3 ? h : 0][w];
                            }
                        }
                    }
                }
            }
        }
        if constexpr (PK > 1) {
            if (lane == 0) {
                if (next) bp.vis[visit0 + next - 1] = placed;
                bp.nvis[(int64_t)grp * L + l] = next;
            }
        }
    }

    ring.idle();
    // ---- dq through shared memory (the ring is idle), rows written whole: fp32, or rounded once to the storage type ----
    __syncwarp();
    float* sm = reinterpret_cast<float*>(wbase);
    // 128 dims of 16-bit storage: rows and every 16 floats of a row are 4 floats further apart (unpadded, 8 lanes of a store met in
    // one bank).  With 32 and 64 dims 2 and 4 lanes meet and the padded addresses cost more than they give.
    constexpr bool PADDED = D == 128 && !X3;
    constexpr int ROW = D + (PADDED ? D / 4 + 4 : 0);
    static_assert(8 * NH * ROW * sizeof(float) <= Ring::kBytes, "the rows fit the ring");
    const float post = X3 ? p.scale : pow2_inverse(sscale);           // 16-bit: the softmax scale is in the tables
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if constexpr (PADDED) sm[(8 * h + 2 * r + (i & 1)) * ROW + ((i >> 1) * HALF + PPT * (g >> 1)) / 16 * 20 + 2 * ks + (g & 1)] = dq[h][ks][i] * post;
                else sm[(8 * h + 2 * r + (i & 1)) * D + (i >> 1) * HALF + PPT * (g >> 1) + 2 * ks + (g & 1)] = dq[h][ks][i] * post;
            }
    __syncwarp();
    for (int j = 0; j < PK; ++j) {                                    // query by query: its G rows are in one piece
        if (PK > 1 && tl + j >= p.Tq) break;
        const int64_t first = (hbase + (int64_t)j * p.H) * D;
        for (int i0 = lane; i0 < G * D / 4; i0 += 32) {
            const int i = i0 + j * GP * (D / 4);
            const float4 x = reinterpret_cast<const float4*>(sm)[PADDED ? i / (D / 4) * (ROW / 4) + i % (D / 4) / 4 * 5 + i % 4 : i];
            if (p.dq_typed == nullptr) {
                reinterpret_cast<float4*>(p.dq + first)[i0] = x;
            } else if constexpr (sizeof(T) == 4) {
                reinterpret_cast<float4*>(reinterpret_cast<float*>(p.dq_typed) + first)[i0] = x;
            } else {
                using FP = Frag<typename std::conditional<sizeof(T) == 4, __half, T>::type>;
                reinterpret_cast<uint2*>(reinterpret_cast<T*>(p.dq_typed) + first)[i0] = make_uint2(FP::pack(x.x, x.y), FP::pack(x.z, x.w));
            }
        }
    }
}

template <typename T, int D, bool X3, int NH, int CR, int PK, bool SUMS>
static int launch_dq_warps(const BwdParams& bp, cudaStream_t st) {
    using C = TForm<D, X3, CR, PK>;
    using Ring = WarpRing<dq_stages<D, X3, PK>(), dq_values<D, X3, CR, PK>() + C::VSLOT>;
    const size_t per_warp = walk_warp_bytes<Ring, PK>(walk_layout(bp.a, CR));
    constexpr int max_w = dq_warps<D, X3, NH>(), max_warps = max_w * dq_min_blocks<D, X3, NH>();
    int W = 1, best = 0;
    for (int w = max_w; w >= 1; w >>= 1) {
        int blocks = (int)(228 * 1024 / (w * per_warp + 1024));
        if (blocks * w > max_warps) blocks = max_warps / w;
        if (blocks > 0 && blocks * w > best) { best = blocks * w; W = w; }
    }
    if (best == 0 || W * per_warp > 227 * 1024) return HTREE_E_UNSUPPORTED;
    auto* k = bwd_dq_kernel<T, D, X3, NH, CR, PK, SUMS>;
    static SmemLimit shared;
    const cudaError_t e = shared.raise((const void*)k, W * per_warp);
    if (e != cudaSuccess) return (int)e;
    return launch_chained(k, dim3((bp.ng + W - 1) / W, bp.nsub), dim3(W * 32), W * per_warp, st, bp);
}
template <typename T, int D, bool X3, int NH, int CR>
static int launch_dq_cr(const BwdParams& bp, cudaStream_t st) {
    if constexpr (NH == 1 && CR == 16) {
        if (bp.PK == 2) return launch_dq_warps<T, D, X3, NH, CR, 2, !X3>(bp, st);
        if (bp.PK == 4) return launch_dq_warps<T, D, X3, NH, CR, 4, !X3>(bp, st);
        if (!X3 && sharing_queries(CR, bp.a.G, bp.a.TK, (bp.a.ln[0] + CR - 1) / CR) > 1) return launch_dq_warps<T, D, X3, NH, CR, 1, !X3>(bp, st);
    }
    return launch_dq_warps<T, D, X3, NH, CR, 1, false>(bp, st);
}

template <typename T, int D, bool X3>
static int launch_dq_t(const BwdParams& bp, cudaStream_t st) {
    if (bp.a.CR == 16) return bp.a.G <= 8 ? launch_dq_cr<T, D, X3, 1, 16>(bp, st) : launch_dq_cr<T, D, X3, 2, 16>(bp, st);
    return bp.a.G <= 8 ? launch_dq_cr<T, D, X3, 1, 8>(bp, st) : launch_dq_cr<T, D, X3, 2, 8>(bp, st);
}
template <typename T>
static int launch_dq_d(const BwdParams& bp, cudaStream_t st) {
    constexpr bool F32 = std::is_same<T, float>::value;
    return bp.a.K == 128 ? launch_dq_t<T, 128, F32>(bp, st) : bp.a.K == 64 ? launch_dq_t<T, 64, F32>(bp, st) : launch_dq_t<T, 32, true>(bp, st);
}
int launch_bwd_dq(const BwdParams& bp, int dtype, cudaStream_t st) {
    switch (dtype) {
        case HTREE_F32: return launch_dq_d<float>(bp, st);
        case HTREE_BF16: return launch_dq_d<__nv_bfloat16>(bp, st);
        default: return launch_dq_d<__half>(bp, st);
    }
}

}  // namespace htree
