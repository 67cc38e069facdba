// Selection: shared-importance Top-K of every pooled level, in one launch.  Replaces htree_recompute_selection_kernel and the
// selecting half of htree_select_accumulate_gqa_kernel (src/parallel.py:537-867, 1167-1399).  Products, chunks and operand blocks
// of tform.cuh; writes the parent list that each level consumes.
//
// One warp per (batch, query position, KV head) group; with SPLIT the 8 warps of a block, or of up to 8 blocks, share a group's chunks.
// A candidate's importance does not depend on which: every chunk is evaluated alike (the query rotated in fp32 and rounded once to half per
// parent, two accumulation chains, the chunk's own maximum as reference, heads summed in one fixed tree) and the search is exact.
//
// Bound by the shared-memory read pipe (61% busy at 8 heads of 128, 76% before the third part of the table rows was left out) and latency
// at 12 to 16 warps per SM; of its time the copies are a third, the Top-K search and the rotation a tenth each.  Measured against the
// kernel that gathers rows: 4 x 65536 positions, 64 heads of 128: 49 -> 42 ms.
#include "tform.cuh"

namespace htree {

template <int D, bool X3, int CR>
struct SelForm {
    using C = TForm<D, X3, CR>;
    static constexpr int PPC = C::PPC, KPART = C::PL * C::PART;     // keys of one parent (the version without the odd slot's rotation)
    static constexpr int DATA = PPC * KPART, TAB_ROW = D * 6, TAB = D * 4, SLOT = DATA + PPC * TAB;
    // a table row is [cos | sin | -sin] in fp32, each part ordered [k-step pair][r][4]: the four lanes of a quad read 64 consecutive
    // bytes (rows in natural order cost 8 wavefronts a load, a third of the kernel's shared-memory traffic).  A 16-byte load takes 4
    // wavefronts however many lanes share its words, so the third part, which the C interface's tables have, is not fetched but formed,
    // one packed multiply for two values: 16 of 88 wavefronts a chunk and an eighth of the bytes.  8 heads of 128, 65536 positions:
    // 8.08 -> 7.08 ms (6.84 with the shorter Top-K loops below); 16 heads 1.43 -> 1.38.
    static constexpr int NSTG = SLOT > 4096 ? 2 : 3;
};
// Queries up to here take the longest walks first, so that these are not the tail of the call; in longer ones nearly all walks
// have full length and the forward order was 2% faster (16384 to 65536 positions).
constexpr int kSelReverse = 8192;
// Above this many candidates a group gets a whole block: their importances (16 KB for 4096) leave room for few warps per SM where
// each has its own, below it the block-wide Top-K costs more in barriers than it gives.  128-wide heads, one warp against eight:
// 2500 candidates 2.20 / 2.91 ms (40000 positions, 16 heads), 5000 candidates 11.3 / 9.3 ms (80000 positions).
constexpr int kSelLong = 4096;
constexpr int kSelSplitWarps = 8, kSelSplitKeys = 32 * 32 * kSelSplitWarps;      // SPLIT keeps 32 keys per thread

// The most candidates a group has on any level that selects: the children of TK parents, or of all there are.
static int sel_max_candidates(const AttnParams& p) {
    int most = p.CR;
    for (int l = 1; l < p.L; ++l) {
        const int parents = (p.ln[l] + p.CR - 1) / p.CR;
        const int n = (parents < p.TK ? parents : p.TK) * p.CR;
        if (n > most) most = n;
    }
    return most;
}
// shared memory besides the rings: importances, chunk maxima, two parent lists, counters
__host__ __device__ inline size_t sel_scratch_bytes(int maxc, int TK, int CR) {
    return ((size_t)maxc * 4 + (size_t)(maxc / CR) * 4 + 8 * (size_t)TK + 16 + 64 + 127) & ~size_t(127);
}

template <int D, bool X3, int NH>
constexpr int sel_min_blocks() { return NH == 2 && (X3 || D == 128) ? 3 : 4; }

// Scores of a chunk: S[h] as in score_t, multiplied by the softmax scale.  qf: fp32 query values of this lane.
template <int D, bool X3, int NH, int CR>
__device__ __forceinline__ void select_scores(uint32_t slot, int lane, const float (&qf)[NH][2][D / 8], float scale, float (&S)[NH][4]) {
    using SF = SelForm<D, X3, CR>;
    using C = TForm<D, X3, CR>;
    using FS = Frag<__half>;
    constexpr int KS = D / 16, HALF = D / 2, PPC = SF::PPC;
    const int r = lane & 3;
    // ldmatrix rows: 16 children in one part, or lo / hi matrices of two parents
    const uint32_t kb = CR == 16 ? slot + 16 * lane : slot + ((lane >> 3) & 1) * SF::KPART + (lane >> 4) * 128 + (lane & 7) * 16;
    const uint32_t tab = slot + SF::DATA + 16 * r;
    float U[PPC][NH][4], V[PPC][NH][4], B[PPC][NH][4];     // 16-bit: chains of even and odd k-steps (U, V); split-half: hi*hi (U), hi*lo (V), lo*hi (B)
#pragma unroll
    for (int kp = 0; kp < KS / 2; ++kp) {
        float cs[PPC][4], sn[PPC][4];
#pragma unroll
        for (int w = 0; w < PPC; ++w) {
            const uint4 c4 = lds_u4(tab + w * SF::TAB + 64 * kp), s4 = lds_u4(tab + w * SF::TAB + 4 * HALF + 64 * kp);
            const float tsc = X3 ? scale : 1.f;            // split-half: the scale goes into the table values
            cs[w][0] = __uint_as_float(c4.x) * tsc; cs[w][1] = __uint_as_float(c4.y) * tsc; cs[w][2] = __uint_as_float(c4.z) * tsc; cs[w][3] = __uint_as_float(c4.w) * tsc;
            sn[w][0] = __uint_as_float(s4.x) * tsc; sn[w][1] = __uint_as_float(s4.y) * tsc; sn[w][2] = __uint_as_float(s4.z) * tsc; sn[w][3] = __uint_as_float(s4.w) * tsc;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int ks = 2 * kp + u;
            uint32_t a[4], al[4];
            ldmatrix_frag(kb + ks * (CR * 32), a);
            if constexpr (X3) ldmatrix_frag(kb + C::PART + ks * (CR * 32), al);
#pragma unroll
            for (int w = 0; w < PPC; ++w) {
                const float2 c2 = make_float2(cs[w][2 * u], cs[w][2 * u + 1]), s2 = make_float2(sn[w][2 * u], sn[w][2 * u + 1]);
                const float2 n2 = fmul2(s2, make_float2(-1.f, -1.f));
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    float2 x, y;
                    rotate_pairs_f32(make_float2(qf[h][0][2 * ks], qf[h][0][2 * ks + 1]), make_float2(qf[h][1][2 * ks], qf[h][1][2 * ks + 1]), c2, s2, n2, x, y);
                    if constexpr (X3) {
                        uint32_t b0h, b0l, b1h, b1l;
                        split_half2(x.x, x.y, b0h, b0l);
                        split_half2(y.x, y.y, b1h, b1l);
                        float t[4];
                        mma_zero<__half>(t, a, b0h, b1h);
                        if (ks == 0) {
                            mma_zero<__half>(V[w][h], al, b0h, b1h);
                            mma_zero<__half>(B[w][h], a, b0l, b1l);
#pragma unroll
                            for (int i = 0; i < 4; ++i) U[w][h][i] = t[i];
                        } else {
                            mma_acc<__half>(V[w][h], al, b0h, b1h);
                            mma_acc<__half>(B[w][h], a, b0l, b1l);
#pragma unroll
                            for (int i = 0; i < 4; ++i) U[w][h][i] += t[i];
                        }
                    } else {
                        const uint32_t b0 = FS::pack(x.x, x.y), b1 = FS::pack(y.x, y.y);
                        float (&acc)[4] = u ? V[w][h] : U[w][h];
                        if (kp == 0) mma_zero<__half>(acc, a, b0, b1);
                        else mma_acc<__half>(acc, a, b0, b1);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int w = PPC == 2 ? i >> 1 : 0;           // rows 8..15 are the second parent's children
            if constexpr (X3) S[h][i] = U[w][h][i] + (V[w][h][i] + B[w][h][i]);
            else S[h][i] = (U[w][h][i] + V[w][h][i]) * scale;
        }
}

template <typename T, int D, bool X3, int NH, int CR, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? kSelSplitWarps * 32 : 128, SPLIT ? 2 : sel_min_blocks<D, X3, NH>())
select_mma_kernel(const __grid_constant__ AttnParams p) {
    chain_enter();
    using SF = SelForm<D, X3, CR>;
    using C = TForm<D, X3, CR>;
    constexpr int PPC = SF::PPC, NSTG = SF::NSTG, HALF = D / 2, PPT = HALF / 4;
    using Ring = WarpRing<NSTG, SF::SLOT>;
    extern __shared__ __align__(128) unsigned char smem_raw[];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, r = lane & 3;
    const int W = blockDim.x >> 5;
    // SPLIT: the blocks of a cluster score a group's chunks; the first of them finds the Top-K and hands the list to the others
    const int CL = SPLIT ? (int)cluster_blocks() : 1, rank = SPLIT ? (int)cluster_rank() : 0;
    const int at = SPLIT ? (int)blockIdx.x / CL : (int)(blockIdx.x * W + warp);
    if (!SPLIT && at >= p.Tq) return;
    const int tl = p.Tq <= kSelReverse ? p.Tq - 1 - at : at;
    const int t = p.t0 + tl;
    const int b = blockIdx.y / p.Hkv, hk = blockIdx.y % p.Hkv;
    const int G = p.G, TK = p.TK, L = p.L, maxc = p.sel_maxc;
    const int first = SPLIT ? rank * W + warp : 0, step = SPLIT ? CL * W : 1;
    const int tid = SPLIT ? (int)threadIdx.x : lane, nthr = SPLIT ? kSelSplitWarps * 32 : 32;   // the threads that share a group
    auto sync = [&]() { if constexpr (SPLIT) __syncthreads(); else __syncwarp(); };

    const size_t scratch = sel_scratch_bytes(maxc, TK, CR);
    unsigned char* wbase = smem_raw + (SPLIT ? warp * Ring::kBytes : warp * (Ring::kBytes + scratch));
    unsigned char* sbase = SPLIT ? smem_raw + W * Ring::kBytes : wbase + Ring::kBytes;
    Ring ring;
    ring.init(wbase);
    float* imp = reinterpret_cast<float*>(sbase);
    float* cmax = imp + maxc;
    int32_t* par = reinterpret_cast<int32_t*>(cmax + maxc / CR);
    int32_t* nxt = par + TK;
    int* cnt = reinterpret_cast<int*>(nxt + TK);       // SPLIT: three rotating counters
    int* wtot = cnt + 4;                               // SPLIT: one per warp
    if (SPLIT && threadIdx.x < 4) cnt[threadIdx.x] = 0;
    if (CL > 1) cluster_sync();                        // every block has started: its shared memory may be written

    const int64_t hbase = ((int64_t)b * p.Tq + tl) * p.H + (int64_t)hk * G;
    const int64_t qidx = ((int64_t)b * p.Tq + tl) * p.Hkv + hk;
    float qf[NH][2][D / 8];
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            load_row_piece_f32<T, D>(reinterpret_cast<const T*>(p.q) + (hbase + 8 * h + g) * D + hf * HALF + PPT * r, 8 * h + g < G, qf[h][hf]);
            if constexpr (!X3) {       // the 16-bit kernels take the query as IEEE half
#pragma unroll
                for (int i = 0; i < D / 8; ++i) qf[h][hf][i] = __half2float(__float2half_rn(fminf(fmaxf(qf[h][hf][i], -65504.f), 65504.f)));
            }
        }

    {   // virtual parents of the top level (src/parallel.py:1026-1038)
        int np0 = (int)(((int64_t)t / p.lpow[L - 1]) / CR) + 1;
        if (np0 > TK) np0 = TK;
        for (int i = tid; i < TK; i += nthr) par[i] = i < np0 ? i : -1;
    }
    int np = (int)(((int64_t)t / p.lpow[L - 1]) / CR) + 1;
    if (np > TK) np = TK;
    sync();

    for (int l = L - 1; l >= 0; --l) {
        if (rank == 0) for (int i = tid; i < TK; i += nthr) store_parent(p, l, qidx * TK + i, par[i]);
        if (l == 0) break;
        const int Nl = p.ln[l];
        const int rc = (int)(((int64_t)t / p.lpow[l]) % CR);
        const int nc = (np - 1) * CR + rc + 1, rp = nc - 1;
        if (nc <= TK) {       // every candidate is kept
            sync();
            for (int j = tid; j < TK; j += nthr) nxt[j] = j < nc ? par[j / CR] * CR + j % CR : -1;
            np = nc;
        } else {
            const int nchunk = (np + PPC - 1) / PPC;
            const int nblk = (Nl + CR - 1) / CR;
            const uint32_t bstride = (uint32_t)p.Hkv * C::BLOCK;
            const unsigned char* blk = reinterpret_cast<const unsigned char*>(p.blk[l]) + ((int64_t)b * nblk * p.Hkv + hk) * C::BLOCK;
            // Every parent here is below nblk and needs no check (one in this loop cost 2 to 9%): lists ascend and none of them passes
            // the query's own ancestor, position t / lpow[l + 1] of the level above; only a list that ends there has it as its last
            // parent, and then the candidates stop at t / lpow[l], which is a node of this level for every t < T.
            auto fill = [&](int c) {
#pragma unroll
                for (int w = 0; w < PPC; ++w) {
                    const int a = PPC == 1 ? c : min(c * PPC + w, np - 1);     // past the end of the list: masked, any finite block
                    ring.template copy<SF::KPART>(w * SF::KPART, blk + (uint64_t)(uint32_t)par[a] * bstride, lane);
                    ring.template copy<SF::TAB>(SF::DATA + w * SF::TAB, reinterpret_cast<const unsigned char*>(p.tab32) + (uint32_t)(rp - CR * a) * SF::TAB_ROW, lane);
                }
            };
            ring.start();
            int next = first;
#pragma unroll 1
            for (int s = 0; s < NSTG - 1; ++s, next += step) {
                if (next < nchunk) fill(next);
                ring.commit();
            }
#pragma unroll 1
            for (int c = first; c < nchunk; c += step) {
                __syncwarp();                                 // everybody is done with the slot that is refilled now
                if (next < nchunk) fill(next);
                ring.commit();
                next += step;
                const uint32_t slot = ring.wait();
                float S[NH][4];
                select_scores<D, X3, NH, CR>(slot, lane, qf, p.scale, S);
                if (G < 8 * NH || 16 * c + 16 > nc) {          // heads or candidates that do not exist
                    const bool v0 = 16 * c + g < nc, v1 = 16 * c + 8 + g < nc;
#pragma unroll
                    for (int h = 0; h < NH; ++h)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const bool on = 8 * h + 2 * r + e < G;
                            S[h][e] = on && v0 ? S[h][e] : -INFINITY; S[h][2 + e] = on && v1 ? S[h][2 + e] : -INFINITY;
                        }
                }
                float m0 = fmaxf(S[0][0], S[0][1]), m1 = fmaxf(S[0][2], S[0][3]);
                if constexpr (NH == 2) {
                    m0 = fmaxf(m0, fmaxf(S[NH - 1][0], S[NH - 1][1])); m1 = fmaxf(m1, fmaxf(S[NH - 1][2], S[NH - 1][3]));
                }
                if constexpr (CR == 16) m0 = m1 = redux_max_f32(fmaxf(m0, m1), 0xffffffffu);
                else { m0 = redux_max_f32(m0, 0xffffffffu); m1 = redux_max_f32(m1, 0xffffffffu); }
                const float n0 = m0 * kLog2e, n1 = m1 * kLog2e;
                auto ex = [&](float s, float m, float n) { return X3 ? __expf(s - m) : ex2_approx(fmaf(s, kLog2e, -n)); };
                // heads summed as ((h0 + h8) + (h1 + h9)) + ... over the group
                float e0, e1;
                if constexpr (NH == 2) {
                    e0 = (ex(S[0][0], m0, n0) + ex(S[NH - 1][0], m0, n0)) + (ex(S[0][1], m0, n0) + ex(S[NH - 1][1], m0, n0));
                    e1 = (ex(S[0][2], m1, n1) + ex(S[NH - 1][2], m1, n1)) + (ex(S[0][3], m1, n1) + ex(S[NH - 1][3], m1, n1));
                } else {
                    e0 = ex(S[0][0], m0, n0) + ex(S[0][1], m0, n0);
                    e1 = ex(S[0][2], m1, n1) + ex(S[0][3], m1, n1);
                }
                e0 += __shfl_xor_sync(0xffffffffu, e0, 1); e1 += __shfl_xor_sync(0xffffffffu, e1, 1);
                e0 += __shfl_xor_sync(0xffffffffu, e0, 2); e1 += __shfl_xor_sync(0xffffffffu, e1, 2);
                // (all of the chunk's loads end in these stores, ahead of the copies that refill the slot)
                if (rank == 0) {
                    if (r < 2 && 16 * c + 8 * r + g < maxc) imp[16 * c + 8 * r + g] = r ? e1 : e0;
                    if (lane < PPC && c * PPC + lane < np) cmax[c * PPC + lane] = lane ? m1 : m0;
                } else {
                    if (r < 2 && 16 * c + 8 * r + g < maxc) st_cluster(cluster_addr(imp + 16 * c + 8 * r + g, 0), __float_as_uint(r ? e1 : e0));
                    if (lane < PPC && c * PPC + lane < np) st_cluster(cluster_addr(cmax + c * PPC + lane, 0), __float_as_uint(lane ? m1 : m0));
                }
            }
            if (CL > 1) cluster_sync(); else sync();
            if (rank == 0) {
            // common reference maximum (src/naive.py:204-205), right-most candidate forced (src/naive.py:93)
            float M = -INFINITY;
            for (int a = lane; a < np; a += 32) M = fmaxf(M, cmax[a]);
            M = warp_max(M);
            if constexpr (SPLIT) __syncthreads();           // every warp has read the maxima before they become factors
            uint32_t* key = reinterpret_cast<uint32_t*>(imp);
            __syncwarp();
            for (int a = SPLIT ? (int)threadIdx.x : lane; a < np; a += nthr) cmax[a] = __expf(cmax[a] - M);
            sync();
            auto value = [&](int j) {
                const float v = imp[j] * cmax[j / CR];
                return __float_as_uint(j == rp ? kForcedImportance : v);
            };
            const bool in_regs = SPLIT || maxc <= 1024;
            uint32_t kreg[32];
            // over the thread's keys, whole eights of them that hold none left out: levels of few candidates spent more on the search
            // among 1024 than on their scores (fp16, 7777 positions, top_k 32: 567 -> 517 us)
            auto each = [&](auto f) {
#pragma unroll
                for (int i0 = 0; i0 < 32; i0 += 8) {
                    if (nthr * i0 < nc) {
#pragma unroll
                        for (int i = i0; i < i0 + 8; ++i) f(i);
                    }
                }
            };
            if (in_regs) {
                each([&](int i) {
                    const int j = tid + nthr * i;
                    kreg[i] = j < nc ? value(j) : 0u;          // padding is below every probe
                });
            } else {
                for (int j = tid; j < nc; j += nthr) key[j] = value(j);
                sync();
            }
            int rot = 0;
            auto count = [&](uint32_t x) {
                int c = 0;
                if (in_regs) {
                    each([&](int i) { c += kreg[i] >= x; });
                } else {
                    for (int j = tid; j < nc; j += nthr) c += key[j] >= x;
                }
                c = __reduce_add_sync(0xffffffffu, c);
                if constexpr (SPLIT) {                         // sum over the warps of the group
                    if (lane == 0 && c) atomicAdd(&cnt[rot], c);
                    __syncthreads();
                    c = cnt[rot];
                    if (threadIdx.x == 0) cnt[rot == 0 ? 2 : rot - 1] = 0;      // used two calls ago
                    rot = rot == 2 ? 0 : rot + 1;
                }
                return c;
            };
            // the smallest and the largest key (the forced candidate, the largest by far, is left out)
            uint32_t lo = 0xffffffffu, hi = 0u;
            if (in_regs) {
                each([&](int i) {
                    const int j = tid + nthr * i;
                    if (j < nc && j != rp) { lo = min(lo, kreg[i]); hi = max(hi, kreg[i]); }
                });
            } else {
                for (int j = tid; j < nc; j += nthr) if (j != rp) { lo = min(lo, key[j]); hi = max(hi, key[j]); }
            }
            lo = __reduce_min_sync(0xffffffffu, lo); hi = __reduce_max_sync(0xffffffffu, hi);
            if constexpr (SPLIT) {
                if (lane == 0) { wtot[2 * warp] = (int)lo; wtot[2 * warp + 1] = (int)hi; }
                __syncthreads();
#pragma unroll
                for (int w = 0; w < kSelSplitWarps; ++w) { lo = min(lo, (uint32_t)wtot[2 * w]); hi = max(hi, (uint32_t)wtot[2 * w + 1]); }
                __syncthreads();       // the placement below writes wtot, and where all importances are equal no count comes between
            }
            const TopKBound bound = topk_search(count, lo, hi + 1u, nc, TK);
            const uint32_t tau = bound.tau;
            const int need = bound.need;
            const bool exact = bound.exact;
            int base_eq = 0, base_out = 0;
            auto place = [&](int j, uint32_t kx) {
                const bool gt = j < nc && kx > tau, eq = !exact && j < nc && kx == tau;
                int tot_eq = 0, tot_k, pos;
                bool keep = gt;
                if constexpr (SPLIT) {
                    if (!exact) {
                        const int rank = base_eq + block_scan_flag<kSelSplitWarps * 32>(eq, wtot, &tot_eq);
                        keep = gt || (eq && rank < need);
                    }
                    pos = base_out + block_scan_flag<kSelSplitWarps * 32>(keep, wtot, &tot_k);
                } else {
                    const uint32_t below = (1u << lane) - 1u;
                    if (!exact) {
                        const uint32_t meq = __ballot_sync(0xffffffffu, eq);
                        keep = gt || (eq && base_eq + __popc(meq & below) < need);
                        tot_eq = __popc(meq);
                    }
                    const uint32_t mk = __ballot_sync(0xffffffffu, keep);
                    pos = base_out + __popc(mk & below);
                    tot_k = __popc(mk);
                }
                if (keep) nxt[pos] = par[j / CR] * CR + j % CR;
                base_eq += tot_eq; base_out += tot_k;
            };
            if (in_regs) {
                each([&](int i) { if (nthr * i < nc) place(tid + nthr * i, kreg[i]); });
            } else {
                for (int j0 = 0; j0 < nc; j0 += nthr) { const int j = j0 + tid; place(j, j < nc ? key[j] : 0u); }
            }
            for (int i = base_out + tid; i < TK; i += nthr) nxt[i] = -1;
            if (SPLIT && threadIdx.x < 3) cnt[threadIdx.x] = 0;
            np = base_out;
            if (CL > 1) {                                       // the kept list and its length to the other blocks
                __syncthreads();
                for (int i = threadIdx.x; i < TK * (CL - 1); i += nthr) st_cluster(cluster_addr(nxt + i % TK, 1 + i / TK), (uint32_t)nxt[i % TK]);
                if ((int)threadIdx.x < CL - 1) st_cluster(cluster_addr(cnt + 3, 1 + threadIdx.x), (uint32_t)np);
            }
            }
            if (CL > 1) {
                cluster_sync();
                if (rank) np = cnt[3];
            }
        }
        sync();
        int32_t* tmp = par; par = nxt; nxt = tmp;
    }
}

template <typename T, int D, bool X3, int NH, int CR>
static int launch_select_cr(const AttnParams& in, cudaStream_t st) {
    AttnParams p = in;
    using SF = SelForm<D, X3, CR>;
    using Ring = WarpRing<SF::NSTG, SF::SLOT>;
    const int maxc = p.sel_maxc = sel_max_candidates(p);
    const size_t scratch = sel_scratch_bytes(maxc, p.TK, CR), limit = 227 * 1024;
    const int64_t groups = (int64_t)p.Tq * p.B * p.Hkv;
    // A block of 8 warps per group where there are few groups (below two per SM a single warp's walk over its chunks is the whole
    // time of the call), and for lists above kSelLong.
    const size_t split_smem = kSelSplitWarps * Ring::kBytes + scratch;
    if ((groups <= 2 * 148 || maxc > kSelLong) && maxc <= kSelSplitKeys && split_smem <= limit) {
        auto* k = select_mma_kernel<T, D, X3, NH, CR, true>;
        static SmemLimit shared;
        const cudaError_t e = shared.raise((const void*)k, split_smem);
        if (e != cudaSuccess) return (int)e;
        // Blocks per group, while each has an SM and as a level has chunks for their warps (long lists of many groups: one).  With the
        // accumulation alone on clusters a decode call took 63.5 us, with both 60.9.
        int CL = 1;
        while (CL < 8 && 2 * CL * groups <= 148 && 2 * CL * kSelSplitWarps <= maxc / 16) CL *= 2;
        return launch_clusters(k, CL, dim3(p.Tq, p.B * p.Hkv), dim3(kSelSplitWarps * 32), split_smem, st, p);
    }
    const size_t per_warp = Ring::kBytes + scratch;
    constexpr int max_warps = 4 * sel_min_blocks<D, X3, NH>();
    int W = 1, best = 0;
    for (int w = 4; w >= 1; w >>= 1) {
        int blocks = (int)(228 * 1024 / (w * per_warp + 1024));
        if (blocks * w > max_warps) blocks = max_warps / w;
        if (blocks > 0 && blocks * w > best) { best = blocks * w; W = w; }
    }
    if (best == 0 || W * per_warp > limit) return HTREE_E_UNSUPPORTED;
    auto* k = select_mma_kernel<T, D, X3, NH, CR, false>;
    static SmemLimit shared;
    const cudaError_t e = shared.raise((const void*)k, W * per_warp);
    if (e != cudaSuccess) return (int)e;
    return launch_chained(k, dim3((p.Tq + W - 1) / W, p.B * p.Hkv), dim3(W * 32), W * per_warp, st, p);
}

template <typename T, int D, bool X3>
static int launch_select_t(const AttnParams& p, cudaStream_t st) {
    if (p.CR == 16) return p.G <= 8 ? launch_select_cr<T, D, X3, 1, 16>(p, st) : launch_select_cr<T, D, X3, 2, 16>(p, st);
    return p.G <= 8 ? launch_select_cr<T, D, X3, 1, 8>(p, st) : launch_select_cr<T, D, X3, 2, 8>(p, st);
}

// Storage types and head sizes whose selections this kernel makes (the others keep the fp32-arithmetic kernel's).
bool select_blk_supported(const AttnParams& p, int dtype) {
    if (p.K != p.V || (p.K != 64 && (p.K != 128 || dtype == HTREE_F32)) || p.G > 16 || (p.CR != 8 && p.CR != 16) || !p.tab32) return false;
    for (int l = 1; l < p.L; ++l) if (!p.blk[l]) return false;
    const bool x3 = dtype == HTREE_F32;
    const size_t ring = 3 * ((x3 ? 2 : 1) * (size_t)p.K * 32 + 8 * p.K) + 128;
    return ring + sel_scratch_bytes(sel_max_candidates(p), p.TK, p.CR) <= 227 * 1024;
}

int launch_select_blk(const AttnParams& p, int dtype, cudaStream_t st) {
    if (dtype == HTREE_F32) return launch_select_t<float, 64, true>(p, st);
    if (dtype == HTREE_BF16) return p.K == 128 ? launch_select_t<__nv_bfloat16, 128, false>(p, st) : launch_select_t<__nv_bfloat16, 64, false>(p, st);
    return p.K == 128 ? launch_select_t<__half, 128, false>(p, st) : launch_select_t<__half, 64, false>(p, st);
}

}  // namespace htree
