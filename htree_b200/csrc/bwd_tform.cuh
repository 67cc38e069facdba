// Parameters and layouts shared by the kernels of the two-pass backward (bwd_dq.cu, bwd_dkv.cu).
//
// The query-stationary pass (bwd_dq.cu) forms S, P, dP, dS of every accumulated chunk and sums dq in registers.  Pushing dK
// and dV from there costs one fp32 reduction of CR rows per visit (a query's visit to a parent), 16 KB each at 128-wide heads,
// and runs at the L2's reduction rate whatever the arithmetic does.  So it only leaves P and dS behind, in the storage
// precision of the products that consume them (1 KB a visit for 16 heads), and the parent-stationary pass (bwd_dkv.cu) walks the
// visits of one parent with dK, dV in registers: it fetches the queries (4 KB) and that kilobyte, and reduces once per 64 or so
// visits.  The order of a parent's visits comes from a counting sort (ranks taken by the first pass, one scan, one fill).
//
// Split-half operands are brought to the top of half's range by powers of two (range_scale): the heads and the output gradients of a
// group by one each, P (at most 1) by 2^14, dS by one per group and level, from a bound on it.  What undoes them is one factor for dK and
// one for dV, which travel in a visit's entry and are applied where its product joins the fp32 sum: gradients of a mean-reduced loss
// keep their digits, and a visit does not depend on other groups.
//
// 16-bit operands go as they are, but dS is formed here and is a half, carried times a power of two from what bounds it: the largest
// |dO|_1 of a row and the largest value of the (batch, KV head) unit (bwd_range_kernel).  For dq the row is one of the group, so that
// a query's dq does not depend on the others; in a record for dK it is one of the whole call, since the sums over visits run inside
// the products.  The two are the same wherever the magnitudes of dO differ by less than 2^4.
//
// Where several queries share a warp (PK > 1, tform.cuh) they are one group here: eight columns of blocked heads, one record for all who
// visit a parent, a table row per query.  12000 positions, 16 heads of 32, top_k 512: dq 8.1 -> 6.8 ms, dK and dV 4.4 -> 2.6 ms, half the
// records.  A query's scales are its own, in a record too, and the sums over visits undo each query's by itself (dkv_item).
//
// Work is cut into windows of `subq` queries of one (batch, KV head) unit, small enough for a window's blocked queries to stay
// in L2 while its parents gather from them, and into launches of `nsub` windows, whose P and dS fit the caller's buffer.
#pragma once
#include "tform.cuh"

namespace htree {

// A visit in its parent's list: visit slot, group | table row << 15, and, split-half, the factors {dK, dV}.  Where PK queries share a warp a
// group is all of them and a visit one of any of them: group | queries << 16 whose columns are left out, a table row per query in 16 bits
// each, and factors per query.
template <bool X3, int PK> struct __align__(16) BwdEntry { uint32_t visit, where, rows[2]; };
template <int PK> struct __align__(16) BwdEntry<true, PK> { uint32_t visit, where, rows[2]; float2 f[PK]; };
template <> struct __align__(8) BwdEntry<false, 1> { uint32_t visit, where; };
template <> struct __align__(16) BwdEntry<true, 1> { uint32_t visit, where; float2 f[1]; };
constexpr int64_t entry_bytes(bool x3, int PK) { return (PK > 1 ? 16 : 8) + (x3 ? 8 * PK : 0); }
static_assert(sizeof(BwdEntry<true, 4>) == entry_bytes(true, 4) && sizeof(BwdEntry<true, 2>) == entry_bytes(true, 2) && sizeof(BwdEntry<true, 1>) == entry_bytes(true, 1) &&
              sizeof(BwdEntry<false, 2>) == entry_bytes(false, 2) && sizeof(BwdEntry<false, 1>) == entry_bytes(false, 1), "");

struct BwdItem { int32_t key, start, len, pad; };     // a piece of one parent's visit list

struct BwdParams {
    AttnParams a;
    int32_t sub0, nsub, subq, nw;            // windows of this launch: [sub0, sub0 + nsub) of units * nw
    int32_t MV, NK, seg, cap;                // visit slots per group, parents per unit over all levels, longest item, items per window
    int32_t PK, ng;                          // queries per group, groups per window (subq / PK)
    int32_t voff[HTREE_MAX_LEVELS];          // first visit slot of a level, -1: the level accumulates nothing
    int32_t koff[HTREE_MAX_LEVELS];          // first parent of a level among the NK
    unsigned char* qb;                       // blocked queries [group][half]
    unsigned char* dob;                      // blocked output gradients [group][half]
    unsigned char* stp;                      // P  [group * MV + visit][half]
    unsigned char* sts;                      // dS
    const unsigned char* xtab;               // 16-bit: the rotary table by dimensions of a lane (x_index), [distance][cos | sin], behind the accumulators
    uint32_t* range;                         // 16-bit: bits of the largest |dO|_1 of a row, and of every unit's largest |v|; else unused
    float2* fac;                             // split-half: {dK, dV} factors of a query's visits on a level, [(group * L + level) * PK + query]; else NULL
    int32_t* rank;                           // [group * MV + visit], or
    uint4* vis;                              // PK > 1: {parent | queries << 16 to leave out, rank, rows} [group * MV + visit]
    int32_t* nvis;                           // PK > 1: visits [group * L + level]
    int32_t* cnt;                            // [nsub][NK]
    int2* base;                              // [nsub][NK]: first entry, first item
    void* entries;                           // [nsub][ng * MV] BwdEntry
    BwdItem* items;                          // [nsub][cap]
    int32_t* nitems;                         // [nsub]
    float* acck[HTREE_MAX_LEVELS];           // dK', dV of every level in accumulator order, [block][i][child tile][lane][4]
    float* accv[HTREE_MAX_LEVELS];
};

// Products over heads or children put dims x = PPT (g / 2) + 2 ks + (g & 1) on the rows of lane (g, *): a lane needs KS cosines and sines
// that the table has in twice as many words, interleaved with its neighbour's.  Rows in lane order (written once per backward, a row per
// distance) are half the shared-memory reads, and which half of a word is used is known to the compiler, whose packed multiply-adds
// broadcast it: no permutes.
template <int D>
__host__ __device__ constexpr int x_index(int i) {                  // the dimension at place i of a row's cosines (or sines)
    constexpr int KS = D / 16, PPT = D / 8;
    return PPT * ((i / KS) & 3) + 2 * (i % KS) + i / (4 * KS);
}
// this lane's words: KS halves of cosines at `at`, of sines D bytes behind
template <int D>
__device__ __forceinline__ void lds_x(uint32_t at, uint32_t (&c)[D / 32], uint32_t (&s)[D / 32]) {
    if constexpr (D == 128) {
        const uint4 a = lds_u4(at), b = lds_u4(at + D);
        c[0] = a.x; c[1] = a.y; c[2] = a.z; c[3] = a.w;
        s[0] = b.x; s[1] = b.y; s[2] = b.z; s[3] = b.w;
    } else {
        static_assert(D == 64, "16-bit operands of 64 or 128 dims");
        asm("ld.shared.v2.b32 {%0,%1}, [%2];\n" : "=r"(c[0]), "=r"(c[1]) : "r"(at));
        asm("ld.shared.v2.b32 {%0,%1}, [%2];\n" : "=r"(s[0]), "=r"(s[1]) : "r"(at + D));
    }
}
__device__ __forceinline__ __half2 half_of(uint32_t w, int odd) { return odd ? __high2half2(as_h2(w)) : __low2half2(as_h2(w)); }
// (lo, hi) rotated by the angle (c, s) or, BACK, by its opposite; the roundings of rotate_h2
template <bool BACK>
__device__ __forceinline__ void rotate_x(uint32_t lo, uint32_t hi, __half2 c, __half2 s, uint32_t& x, uint32_t& y) {
    x = as_u32(__hfma2(as_h2(lo), c, __hmul2(as_h2(hi), BACK ? s : __hneg2(s))));
    y = as_u32(__hfma2(as_h2(hi), c, __hmul2(as_h2(lo), BACK ? __hneg2(s) : s)));
}

// The power of two that 16-bit dS is carried with, in steps of 2^4: brings |P (dP - D)| <= 2 max|dO|_1 max|v| below 2^15.
__device__ __forceinline__ float ds_scale(uint32_t dO_l1, uint32_t v) {
    const int e = 393 - (int)(dO_l1 >> 23) - (int)(v >> 23);
    return __int_as_float((((min(max(e, 27), 227) + 1) & ~3) - 1) << 23);
}

int launch_bwd_begin(const BwdParams& bp, int dtype, void* zero, int64_t zero_bytes, cudaStream_t st);
int launch_bwd_dq(const BwdParams& bp, int dtype, cudaStream_t st);
int launch_bwd_dkv(const BwdParams& bp, int dtype, cudaStream_t st);
int launch_bwd_fold(const BwdParams& bp, int dtype, void* dk, void* dv, bool typed, cudaStream_t st);
int launch_bwd_clear(void* p, int64_t bytes, const void* tab, void* xtab, int rows, int D, cudaStream_t st);

template <int D, bool X3, int NH, int CR>
struct BForm {
    static constexpr int KS = D / 16, NT = CR / 8;
    static constexpr int QB = D * 16 * (X3 ? 2 : 1);        // bytes of 8 heads of blocked queries (split-half: fp32) or gradients
    static constexpr int SB = NT * 128 * (X3 ? 2 : 1);      // bytes of P or dS of 8 heads of one visit
    static constexpr int ACC = D * CR;                      // floats of one parent's accumulator
};

}  // namespace htree
