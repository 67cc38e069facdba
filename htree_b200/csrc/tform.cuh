// Shared pieces of the transposed tensor-core kernels (forward accumulation, backward): one warp owns one (batch, query
// position, KV head) group and walks its candidates in chunks of 16 positions (the children of one parent with 16 children
// per parent, of two consecutive parents with 8).
//
// Every product puts the candidates (or the head dimension) on the M = 16 side of mma.sync.m16n8k16 and the query HEADS on
// the N = 8 side: S^T = K' q^, O^T += V^T P^T.  A group of at most 8 heads then needs half the instructions of the
// heads-on-M form, whose other 8 rows would be padding; 9..16 heads are two halves (NH = 2) that share every A fragment, at
// the instruction count of the heads-on-M form.
//
// Operand blocks (written by pack_blocks_kernel, read here as whole blocks by asynchronous copies): per parent and KV
// head the children's pre-rotated keys K' and values in the order in which the lanes consume them as A fragments, so that a
// fragment is one conflict-free 16-byte shared load.  With lane = 4g + r, KS = D/16, PPT = D/8, VB = D/8:
//   K    8x8 matrices [ks][m][lane] of 4-byte words, m = lo / hi dims (8 children), or children 0-7 lo, 8-15 lo, 0-7 hi, 8-15 hi
//        (16 children); word of lane (g, r) = K'[child g][lo], lo = dims PPT*r + 2ks + {0,1}, hi = lo + D/2.  ldmatrix gives the
//        A fragments of S^T = K' q^, ldmatrix.trans those of dq^T = K~^T dS^T
//   V    16 children: [i][lane] = { b0(2i), b0(2i+1), b1(2i), b1(2i+1) },  8 children: [w][lane] = b0(w),
//        bj(w) = { V[8j+2r][VB*g+w], V[8j+2r+1][VB*g+w] }
//        A fragments land in four consecutive registers in their order: a 16-byte load whose registers had to be swapped cost
//        4 moves per fragment, a quarter of the loop's instructions.
//   16 children   block = [K | V]
//    8 children   block = [K | V]; a chunk's two parents have distances 8 apart and the query is rotated for each.
//    8 children, split-half   block = [K even | V | K odd]: keys also stored rotated by 8 more positions, for parents in odd slots
//                 of the query's list, which hold positions 8..15 of their chunk: one query rotation per chunk.  (16-bit storage
//                 does not: a score's rounding is the rounding of these half-precision operands, 2^-11 |q||k|, and with scores of
//                 70 another choice of operands moves probabilities by a percent.)
//   split-half (fp32 storage, and every storage type with 32-wide heads): each part is a hi plane followed by a lo plane.  The keys
//                 and the values of a block are multiplied by powers of two that bring their largest magnitudes to the top of half's range
//                 (range_scale; not the keys of 64-wide heads, whose selection works on the plain ones), and the block ends in a line
//                 with the inverse factors {keys, values}.  They belong to the block, so that no row depends on other blocks.
#pragma once
#include "mma_common.cuh"

namespace htree {

// Several queries in one warp (PK > 1; groups of at most 4 heads, 16 children): consecutive positions share the 8 columns, GP = 8 / PK
// of them each.  The warp walks the union of their parent lists; a block that several of them selected is fetched, read and multiplied
// once, each column rotated by its own query's distance (PK table rows a chunk).  A query that did not select it has P = 0 there,
// which changes nothing while the block's values are finite (16-bit values that are not: acc_mma.cu walks again; the backward leaves out what
// does not belong, bwd_dq.cu): rows are those of a walk alone, bit for bit.
template <int D, bool X3, int CR, int PK = 1>
struct TForm {
    static constexpr int KS = D / 16, HALF = D / 2, PPT = HALF / 4, VB = D / 8, MT = D / 16;
    static constexpr int PL = X3 ? 2 : 1;                                  // planes
    static constexpr int PART = D * 2 * CR;                                // bytes of one plane of one part of a block
    static constexpr bool DUAL = CR == 8 && !X3;                           // two query rotations per chunk
    static constexpr int FACS = X3 ? 128 : 0;                              // the line of factors (a whole one: blocks stay aligned to lines)
    static constexpr int BLOCK = PL * PART * (CR == 16 || DUAL ? 2 : 3) + FACS;   // bytes of a block in global memory
    static constexpr int FACS_OFF = BLOCK - FACS;
    static constexpr bool KSCALED = X3 && D != 64;                         // are a block's keys multiplied by their factor?
    static constexpr int ODD = DUAL ? 0 : PL * PART;                       // where an odd parent's copy starts in its block
    static constexpr int NTAB = DUAL ? 2 : PK;
    static constexpr int PPC = 16 / CR;                                    // parents per chunk
    static constexpr int PB = PL * PART;                                   // bytes of one part of a block
    static constexpr int DATA = PB * PPC;                                  // bytes of the keys, or of the values, of a chunk in shared memory
    static constexpr int TAB = X3 ? D * 4 : D * 2;                         // one row of the rotary table: [cos | sin]
    // a slot of keys: the parents' keys, {key factor, value factor, -, -} per parent, table rows, all at whole lines like their
    // sources; a slot of values: the parents' values
    static constexpr int TAB_OFF = DATA + (X3 ? 128 : 0);
    static constexpr int KSLOT = TAB_OFF + NTAB * TAB, VSLOT = DATA;
};

// Shared-memory addresses of a chunk slot that differ by lane, as 32-bit shared addresses.
template <int D, bool X3, int CR>
struct LaneBase {
    uint32_t k, v, vk;   // ldmatrix rows of the key part; value part (16 children: 16-byte pieces, 8: ldmatrix rows); values in key order
    __device__ __forceinline__ LaneBase(uint32_t keys, uint32_t values, int lane) {
        using C = TForm<D, X3, CR>;
        if constexpr (CR == 16) {
            k = keys + 16 * lane; v = vk = values + 16 * lane;
        } else {
            const int j = lane >> 3, row = lane & 7;
            k = keys + ((j & 1) ? C::PB : 0) + (j >> 1) * 128 + row * 16;
            v = values + ((j >> 1) ? C::PB : 0) + (j & 1) * 128 + row * 16;
            vk = values + ((j & 1) ? C::PB : 0) + (j >> 1) * 128 + row * 16;
        }
    }
};
__device__ __forceinline__ void lds_frag(uint32_t addr, uint32_t (&a)[4]) {
    asm("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];\n" : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_frag(uint32_t addr, uint32_t (&a)[4]) {
    asm("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_trans_frag(uint32_t addr, uint32_t (&a)[4]) {
    asm("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(addr));
}
__device__ __forceinline__ float2 lds_f2(uint32_t addr) {
    float2 x;
    asm("ld.shared.v2.f32 {%0,%1}, [%2];\n" : "=f"(x.x), "=f"(x.y) : "r"(addr));
    return x;
}
__device__ __forceinline__ uint4 lds_u4(uint32_t addr) {
    uint4 x;
    asm("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];\n" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(addr));
    return x;
}
// A fragments of k-step ks of the key part (plane pl)
template <int D, bool X3, int CR>
__device__ __forceinline__ void key_frag(const LaneBase<D, X3, CR>& s, int pl, int ks, uint32_t (&a)[4]) {
    using C = TForm<D, X3, CR>;
    ldmatrix_frag(s.k + pl * C::PART + ks * (CR * 32), a);
}
// the same matrices transposed: { children 0-7 lo, 8-15 lo, 0-7 hi, 8-15 hi }, lane (g, r) = { K'[2r][x], K'[2r+1][x] } (+ 8 children),
// x = lo or hi dim PPT*(g/2) + 2ks + (g & 1)
template <int D, bool X3, int CR>
__device__ __forceinline__ void key_frag_trans(const LaneBase<D, X3, CR>& s, int pl, int ks, uint32_t (&a)[4]) {
    ldmatrix_trans_frag(s.k + pl * TForm<D, X3, CR>::PART + ks * (CR * 32), a);
}
// A fragments of k-step ks of the values in key order (backward slots)
template <int D, bool X3, int CR>
__device__ __forceinline__ void vk_frag(const LaneBase<D, X3, CR>& s, int pl, int ks, uint32_t (&a)[4]) {
    ldmatrix_frag(s.vk + pl * TForm<D, X3, CR>::PART + ks * (CR * 32), a);
}
// A fragments of output tile i of the value part: dims VB*g + 2i (row g) and VB*g + 2i + 1 (row g + 8)
template <int D, bool X3, int CR>
__device__ __forceinline__ void value_frag(const LaneBase<D, X3, CR>& s, int pl, int i, uint32_t (&a)[4]) {
    using C = TForm<D, X3, CR>;
    if constexpr (CR == 16) lds_frag(s.v + pl * C::PART + i * 512, a);
    else ldmatrix_frag(s.v + pl * C::PART + i * 256, a);
}
// The loads from a slot and the products below are not volatile, so that the compiler may overlap one step's loads and
// rotations with another's products.  What orders the loads after the slot's wait is the slot address, which comes out of it; what
// orders them before the copies that refill the slot is that everything they went into exists by then: stored to memory, or passed
// to consumed() at the end of the chunk.  (consumed() is no instruction, and the registers it names are carried to the next chunk.)
__device__ __forceinline__ void consumed(const float (&x)[4]) {
    asm volatile("" ::"f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]) : "memory");
}
template <typename T> __device__ __forceinline__ void mma_acc(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma_acc<__half>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <> __device__ __forceinline__ void mma_acc<__nv_bfloat16>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t movm(uint32_t a) {
    uint32_t d;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(d) : "r"(a));
    return d;
}
// d = A B with a zero accumulator (no registers to clear)
template <typename T> __device__ __forceinline__ void mma_zero(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma_zero<__half>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
template <> __device__ __forceinline__ void mma_zero<__nv_bfloat16>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// The query heads of a group as B fragments of the score product: lane (g, r) holds dims PPT*r + [0, PPT) of both halves of
// head 8h + g.  16-bit path: IEEE half pairs; split-half path: fp32 values, already multiplied by the softmax scale and by the power
// of two that brings the query's largest one to the top of half's range; `inv` is its inverse (for the columns 2r, 2r + 1).
template <typename T, int D, bool X3, int NH>
struct QueryRegs {
    static constexpr int N = X3 ? D / 8 : D / 16;
    uint32_t v[NH][2][N];
    float inv;
};

template <typename T, int D>
__device__ __forceinline__ void load_row_piece_f32(const T* p, bool on, float (&o)[D / 8]) {
#pragma unroll
    for (int i = 0; i < D / 8; i += 4) {
        float x[4] = {0.f, 0.f, 0.f, 0.f};
        if (on) load4<T>(p + i, x);
#pragma unroll
        for (int u = 0; u < 4; ++u) o[i + u] = x[u];
    }
}

// Columns of a warp and the queries they belong to.
template <int PK>
struct Cols {
    static constexpr int GP = 8 / PK;                                                       // columns of a query
    static __device__ __forceinline__ int of_lane(int g) { return PK == 1 ? 0 : g / GP; }       // query of column g (B fragments)
    static __device__ __forceinline__ int of_pair(int r) { return PK == 1 ? 0 : 2 * r / GP; }   // query of columns 2r, 2r + 1 (C fragments)
    // over the lanes (g, *) of a query's columns
    static __device__ __forceinline__ float max_of(float x) {
        if constexpr (PK == 1) return redux_max_f32(x, 0xffffffffu);
#pragma unroll
        for (int o = 1; o < 4 * GP; o <<= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
        return x;
    }
    // a value per query held by the lanes (g, *) of its columns, for the lanes (*, r)
    static __device__ __forceinline__ float for_pair(float x, int r) { return PK == 1 ? x : __shfl_sync(0xffffffffu, x, 4 * GP * of_pair(r)); }
    // for the lanes (*, r): is `x` true for every lane (g, *) of the columns of their query?
    static __device__ __forceinline__ bool all_of(bool x, int r) {
        const uint32_t off = __ballot_sync(0xffffffffu, !x);
        return PK == 1 ? off == 0u : (off >> (4 * GP * of_pair(r)) & ((uint32_t)((uint64_t(1) << (4 * GP)) - 1u))) == 0u;
    }
    // the lanes (*, r) of the query of columns 2r, 2r + 1
    static __device__ __forceinline__ uint32_t lanes_of_pair(int r) {
        return PK == 1 ? 0xffffffffu : PK == 2 ? 0x33333333u << (r & 2) : 0x11111111u << r;
    }
};

// row(h): the row of column 8h + g, or NULL.
template <typename T, int D, bool X3, int NH, int PK = 1, typename Row>
__device__ __forceinline__ void load_query(Row row, int r, float scale, QueryRegs<T, D, X3, NH>& q) {
    constexpr int HALF = D / 2, PPT = HALF / 4;
    float most = 0.f;
#pragma unroll
    for (int h = 0; h < NH; ++h) {
        const T* base = row(h);
        const bool on = base != nullptr;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const T* p = base + hf * HALF + PPT * r;
            if constexpr (X3) {
                float x[D / 8];
                load_row_piece_f32<T, D>(p, on, x);
#pragma unroll
                for (int i = 0; i < D / 8; ++i) { q.v[h][hf][i] = __float_as_uint(x[i] * scale); most = fmaxf(most, fabsf(x[i] * scale)); }
            } else {
                ldg_vec<PPT / 8>(p, on, q.v[h][hf]);
                if (!std::is_same<T, __half>::value) {
#pragma unroll
                    for (int i = 0; i < D / 16; ++i) {
                        const float2 f = Frag<__nv_bfloat16>::unpack(q.v[h][hf][i]);
                        q.v[h][hf][i] = Frag<__half>::pack(fminf(fmaxf(f.x, -65504.f), 65504.f), fminf(fmaxf(f.y, -65504.f), 65504.f));
                    }
                }
            }
        }
    }
    if constexpr (X3) {
        const float s = range_scale_coarse(Cols<PK>::max_of(most));
        q.inv = Cols<PK>::for_pair(pow2_inverse(s), r);
#pragma unroll
        for (int h = 0; h < NH; ++h)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf)
#pragma unroll
                for (int i = 0; i < D / 8; ++i) q.v[h][hf][i] = __float_as_uint(__uint_as_float(q.v[h][hf][i]) * s);
    }
}

// B fragments of k-step ks: the query rotated by the chunk's distance.  `tab` is the chunk's table row in shared memory.
__device__ __forceinline__ __half2 as_h2(uint32_t x) { return *reinterpret_cast<const __half2*>(&x); }
__device__ __forceinline__ uint32_t as_u32(__half2 x) { return *reinterpret_cast<const uint32_t*>(&x); }
// (lo, hi) rotated by (c, s): lo*c - hi*s, lo*s + hi*c, four packed instructions (which negate an operand for nothing)
__device__ __forceinline__ void rotate_h2(uint32_t lo, uint32_t hi, uint32_t c, uint32_t s, uint32_t& x, uint32_t& y) {
    x = as_u32(__hfma2(as_h2(lo), as_h2(c), __hmul2(as_h2(hi), __hneg2(as_h2(s)))));
    y = as_u32(__hfma2(as_h2(hi), as_h2(c), __hmul2(as_h2(lo), as_h2(s))));
}

// S^T of one chunk: S[h] = C fragment, rows = children g and g + 8, columns = heads 8h + 2r, 8h + 2r + 1.
template <typename T, int D, int NH, int CR>
__device__ __forceinline__ void score16(const LaneBase<D, false, CR>& s, uint32_t tab, int r, const QueryRegs<T, D, false, NH>& q, float (&S)[NH][4]) {
    using FS = Frag<__half>;
    constexpr int KS = D / 16;
    constexpr int HALF = D / 2, PPT = HALF / 4;
    constexpr bool DUAL = TForm<D, false, CR>::DUAL;
    constexpr bool TWO = NH == 1 && !DUAL;     // two accumulation chains per half; two halves or two parents are two chains anyway
    tab += 2 * (PPT * r);
    float U[TWO || DUAL ? NH : 1][4];          // second chain, or the odd parent's scores
#pragma unroll
    for (int k4 = 0; k4 < KS; k4 += 4) {
        const uint4 c4 = lds_u4(tab + 4 * k4), s4 = lds_u4(tab + 2 * HALF + 4 * k4);
        const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
        uint32_t c2[4], sn2[4];
        if constexpr (DUAL) {
            const uint4 d4 = lds_u4(tab + 2 * D + 4 * k4), t4 = lds_u4(tab + 2 * D + 2 * HALF + 4 * k4);
            c2[0] = d4.x; c2[1] = d4.y; c2[2] = d4.z; c2[3] = d4.w;
            sn2[0] = t4.x; sn2[1] = t4.y; sn2[2] = t4.z; sn2[3] = t4.w;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int ks = k4 + u;
            uint32_t a[4];
            key_frag<D, false, CR>(s, 0, ks, a);
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                uint32_t b0, b1;
                rotate_h2(q.v[h][0][ks], q.v[h][1][ks], c[u], sn[u], b0, b1);
                float (&acc)[4] = TWO && (ks & 1) ? U[TWO ? h : 0] : S[h];
                if (ks < (TWO ? 2 : 1)) mma_zero<__half>(acc, a, b0, b1);
                else mma_acc<__half>(acc, a, b0, b1);
                if constexpr (DUAL) {
                    rotate_h2(q.v[h][0][ks], q.v[h][1][ks], c2[u], sn2[u], b0, b1);
                    if (ks == 0) mma_zero<__half>(U[DUAL ? h : 0], a, b0, b1);
                    else mma_acc<__half>(U[DUAL ? h : 0], a, b0, b1);
                }
            }
        }
    }
#pragma unroll
    for (int h = 0; h < NH; ++h) {
        if constexpr (DUAL) { S[h][2] = U[DUAL ? h : 0][2]; S[h][3] = U[DUAL ? h : 0][3]; }     // rows 8..15 are the odd parent's children
        else if constexpr (TWO) {
#pragma unroll
            for (int i = 0; i < 4; ++i) S[h][i] += U[TWO ? h : 0][i];
        }
    }
}

// Split-half form (see mma_common.cuh for why the leading product of every k-step is summed with ordinary fp32 adds).
template <typename T, int D, int NH, int CR>
__device__ __forceinline__ void score_x3(const LaneBase<D, true, CR>& s, uint32_t tab, int r, const QueryRegs<T, D, true, NH>& q, float (&S)[NH][4]) {
    using FS = Frag<__half>;
    constexpr int KS = D / 16, HALF = D / 2, PPT = HALF / 4;
    tab += 4 * PPT * r;
    float B[NH][4], C[NH][4];
#pragma unroll
    for (int kp = 0; kp < KS / 2; ++kp) {
        const uint4 c4 = lds_u4(tab + 16 * kp), s4 = lds_u4(tab + 4 * HALF + 16 * kp);
        const float cs[4] = {__uint_as_float(c4.x), __uint_as_float(c4.y), __uint_as_float(c4.z), __uint_as_float(c4.w)};
        const float sn[4] = {__uint_as_float(s4.x), __uint_as_float(s4.y), __uint_as_float(s4.z), __uint_as_float(s4.w)};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int ks = 2 * kp + u;
            uint32_t ah[4], al[4];
            key_frag<D, true, CR>(s, 0, ks, ah);
            key_frag<D, true, CR>(s, 1, ks, al);
            const float2 c2 = make_float2(cs[2 * u], cs[2 * u + 1]), s2 = make_float2(sn[2 * u], sn[2 * u + 1]);
            const float2 n2 = make_float2(-s2.x, -s2.y);
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                const float2 lo = make_float2(__uint_as_float(q.v[h][0][2 * ks]), __uint_as_float(q.v[h][0][2 * ks + 1]));
                const float2 hi = make_float2(__uint_as_float(q.v[h][1][2 * ks]), __uint_as_float(q.v[h][1][2 * ks + 1]));
                float2 x, y;
                rotate_pairs_f32(lo, hi, c2, s2, n2, x, y);
                uint32_t b0h, b0l, b1h, b1l;
                split_half2(x.x, x.y, b0h, b0l);
                split_half2(y.x, y.y, b1h, b1l);
                if (ks == 0) {
                    mma_zero<__half>(S[h], ah, b0h, b1h);
                    mma_zero<__half>(B[h], al, b0h, b1h);
                    mma_zero<__half>(C[h], ah, b0l, b1l);
                } else {
                    float t[4];
                    mma_zero<__half>(t, ah, b0h, b1h);
                    mma_acc<__half>(B[h], al, b0h, b1h);
                    mma_acc<__half>(C[h], ah, b0l, b1l);
#pragma unroll
                    for (int i = 0; i < 4; ++i) S[h][i] += t[i];
                }
            }
        }
    }
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) S[h][i] += B[h][i] + C[h][i];
}

// The factors of a chunk's parents, .x of the keys and .y of the values: f[0] of rows 0..7, f[1] of rows 8..15 (one parent: the same).
template <int D, bool X3, int CR>
__device__ __forceinline__ void chunk_factors(uint32_t slot, float2 (&f)[2]) {
    using C = TForm<D, X3, CR>;
    f[0] = f[1] = make_float2(1.f, 1.f);
    if constexpr (X3) {
        f[0] = f[1] = lds_f2(slot + C::DATA);
        if constexpr (CR == 8) f[1] = lds_f2(slot + C::DATA + 16);
    }
}
// Two parents in one product over children: their common factor (the larger one) and what each parent's rows are multiplied by.
__device__ __forceinline__ float common_factor(float a, float b, float (&ratio)[2]) {
    const float f = fmaxf(a, b), inv = pow2_inverse(f);
    ratio[0] = a * inv; ratio[1] = b * inv;
    return f;
}
// Scores; split-half ones still have to be multiplied by f[row / 8].x * q.inv, a power of two.
template <typename T, int D, bool X3, int NH, int CR>
__device__ __forceinline__ void score_t(const LaneBase<D, X3, CR>& s, uint32_t slot, int r, const QueryRegs<T, D, X3, NH>& q, float (&S)[NH][4],
                                        uint32_t tab_of_lane = 0) {
    const uint32_t tab = slot + TForm<D, X3, CR>::TAB_OFF + tab_of_lane;
    if constexpr (X3) score_x3<T, D, NH, CR>(s, tab, r, q, S);
    else score16<T, D, NH, CR>(s, tab, r, q, S);
}

// One warp's ring of chunk slots in shared memory, filled NSTG - 1 chunks ahead by 16-byte asynchronous copies of all lanes
// (cp.async): one instruction per 512 bytes, no barrier object and no single-lane section.  With one bulk copy per operand,
// issued by one lane and completing on an mbarrier, the single-lane section (addresses into uniform registers, barrier
// arithmetic) cost 14 % of the selection kernel.
template <int NSTG, int SLOT>
struct WarpRing {
    uint32_t base;                 // 32-bit shared address of NSTG * SLOT bytes
    uint32_t fill, use;            // addresses of the stages that the next fill / the next use takes
    static constexpr size_t kBytes = ((size_t)NSTG * SLOT + 127) & ~size_t(127);

    __device__ __forceinline__ void init(unsigned char* b) { base = smem_u32(b); start(); }
    __device__ __forceinline__ void start() { fill = use = base; }       // before the first fill of a walk; nothing is in flight
    __device__ __forceinline__ uint32_t after(uint32_t a) const {
        return NSTG == 1 ? a : NSTG == 2 ? 2 * base + SLOT - a : a == base + (NSTG - 1) * SLOT ? base : a + SLOT;
    }
    // BYTES (a multiple of 16) from `src` to offset OFF of the stage being filled
    template <int BYTES>
    __device__ __forceinline__ void copy(uint32_t off, const void* src, int lane) const { copy_to<BYTES>(fill + off, src, lane); }
    template <int BYTES>
    static __device__ __forceinline__ void copy_to(uint32_t at, const void* src, int lane) {
        const uint32_t dst = at + 16 * lane;
        const unsigned char* s = static_cast<const unsigned char*>(src) + 16 * lane;
#pragma unroll
        for (int i = 0; i < BYTES / 512; ++i)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + 512 * i), "l"(s + 512 * i) : "memory");
        if constexpr (BYTES % 512 != 0) {
            if (lane < (BYTES % 512) / 16)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + BYTES / 512 * 512), "l"(s + BYTES / 512 * 512) : "memory");
        }
    }
    // closes one fill (an empty one where nothing is left to fetch: fills and uses are counted alike)
    __device__ __forceinline__ void commit() {
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        fill = after(fill);
    }
    // the oldest fill, complete and visible to every lane: YOUNGER fills (of any ring of the warp) were closed after it
    template <int YOUNGER = NSTG - 1>
    __device__ __forceinline__ uint32_t wait() {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(YOUNGER) : "memory");
        __syncwarp();
        uint32_t slot = use;
        asm volatile("" : "+r"(slot)::"memory");
        use = after(use);
        return slot;
    }
    __device__ __forceinline__ void idle() const { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
};

// A query's parent list of one level in shared memory, 16 bits an entry where every level's parents can be numbered with them
// (with 512 nodes per layer 1 KB instead of 2 beside 17 KB of ring: lists and bits decide whether 11 or 12 warps share an SM).
struct ParentList {
    unsigned char* at;
    bool narrow;
    __device__ __forceinline__ int operator[](int i) const {
        return narrow ? (int)reinterpret_cast<const uint16_t*>(at)[i] : reinterpret_cast<const int32_t*>(at)[i];
    }
    // A query's list of one level: returns the number of its parents, looking at no more entries than the level has parents.  Entries
    // that are no parent of the level become 0 and set `bit`, and so do holes before the last parent: a backward's lists come from
    // its caller, and a slot left as it was would index blocks and counters with what the shared memory held before.
    __device__ __forceinline__ int load(const AttnParams& p, int l, int64_t list, int nblk, int bit, int lane) const {
        int np = 0, end = 0;
        for (int i = lane; i < min(p.TK, nblk); i += 32) {
            int x = load_parent(p, l, list + i);
            if (x >= 0) { ++np; end = i + 1; }
            if (x >= nblk) { if (p.status) atomicOr(p.status, bit); x = 0; }
            x = max(x, 0);
            if (narrow) reinterpret_cast<uint16_t*>(at)[i] = (uint16_t)x; else reinterpret_cast<int32_t*>(at)[i] = x;
        }
        np = __reduce_add_sync(0xffffffffu, np);
        if (end > np && p.status) atomicOr(p.status, bit);
        return np;
    }
    // For a list (of 16-bit entries) that goes into a union of several: strictly ascending from here on, entries that are not above the
    // one before dropped and reported; returns how many are left.  A union of such lists has no more steps than the level has parents,
    // which is what its visits' slots are sized for.  Checked once per list: passing over such entries in UnionWalk::step cost the backward 3%.
    __device__ __forceinline__ int ascending(const AttnParams& p, int np, int bit, int lane) const {
        uint16_t* x = reinterpret_cast<uint16_t*>(at);
        __syncwarp();
        bool bad = false;
        for (int i = lane + 1; i < np; i += 32) bad |= x[i] <= x[i - 1];
        if (!__any_sync(0xffffffffu, bad)) return np;
        int left = 0;
        if (lane == 0) {
            for (int i = 0, last = -1; i < np; ++i)
                if ((int)x[i] > last) { last = x[i]; x[left++] = (uint16_t)last; }
            if (p.status) atomicOr(p.status, bit);
        }
        __syncwarp();
        return __shfl_sync(0xffffffffu, left, 0);
    }
};
// The union of PK queries' ascending lists (of 16-bit entries), walked in that order.  Lane j (mod PK) holds query j's list and place in it.
template <int PK>
struct UnionWalk {
    const uint16_t* list;         // of this lane's query
    const uint32_t* selw;         // its kept-candidate bits (levels that select), or NULL
    int np, rp, at;               // its parents, its right-most position, the next entry
    uint32_t head;                // that entry's parent: read a step ahead
    int rank;                     // of the step taken last: its rank in this lane's list, or -1
    __device__ __forceinline__ void start(const ParentList& par, const uint32_t* bits, int n, int right) {
        list = reinterpret_cast<const uint16_t*>(par.at); selw = bits; np = n; rp = right; at = 0;
        head = n > 0 ? list[0] : 0xffffffffu;
    }
    // the next parent of any list, or -1
    __device__ __forceinline__ int step() {
        const uint32_t least = __reduce_min_sync(0xffffffffu, head);
        const bool mine = head == least && least != 0xffffffffu;
        rank = mine ? at : -1;
        if (mine) { ++at; head = at < np ? list[at] : 0xffffffffu; }
        return (int)least;
    }
    __device__ __forceinline__ uint32_t mask() const {               // the step's candidates that accumulate for this lane's query
        if (rank < 0) return 0u;
        uint32_t m = 0xffffu;
        if (selw) m &= ~(selw[rank >> 1] >> ((16 * rank) & 31));
        if (16 * rank + 15 > rp) m &= (2u << (rp - 16 * rank)) - 1u;
        return m;
    }
    __device__ __forceinline__ int row() const { return rank < 0 ? 0 : rp - 16 * rank; }       // its distance (any row where it has no part)
};
// the step's table rows, one after the other
template <int PK, int TAB, typename Ring>
__device__ __forceinline__ void copy_tab_rows(const Ring& ring, uint32_t off, const void* tab, int row, int lane) {
    constexpr int PER = TAB / 16;
#pragma unroll
    for (int i = 0; i < PK * PER; i += 32) {
        const int piece = i + lane;
        const int of = __shfl_sync(0xffffffffu, row, piece / PER);
        if (PK * PER >= 32 || piece < PK * PER)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(ring.fill + off + 16 * piece),
                         "l"(static_cast<const unsigned char*>(tab) + (int64_t)of * TAB + 16 * (piece % PER)) : "memory");
    }
}

// What the walk over a level's candidates keeps per warp beside the ring: the parent list and one bit per candidate of a level
// that selects.  Both are bounded by the parents that the levels have.
struct WalkLayout { int list, bits; bool narrow; };      // bytes
__host__ __device__ __forceinline__ WalkLayout walk_layout(const AttnParams& p, int CR) {
    const int leaf = (p.ln[0] + CR - 1) / CR, up = p.L > 1 ? (p.ln[1] + CR - 1) / CR : 1;
    WalkLayout w;
    w.narrow = leaf <= 65536;
    w.list = ((leaf < p.TK ? leaf : p.TK) * (w.narrow ? 2 : 4) + 3) & ~3;
    w.bits = ((up < p.TK ? up : p.TK) * CR + 31) / 32 * 4;
    return w;
}
template <typename Ring, int PK = 1>
__host__ __device__ __forceinline__ size_t walk_warp_bytes(const WalkLayout& w) { return (Ring::kBytes + PK * (w.list + w.bits) + 127) & ~size_t(127); }
__host__ __device__ __forceinline__ size_t walk_lists_bytes(const WalkLayout& w) { return ((size_t)w.list + w.bits + 127) & ~size_t(127); }
// one bit per candidate of a level that the next level kept, from its list (both lists ascending); the bits are clear and the list there
template <int NT>
__device__ __forceinline__ void mark_kept(const AttnParams& p, int l, int64_t list, const ParentList& par, int np, int CR, uint32_t* selw, int thread) {
    for (int i = thread; i < p.TK; i += NT) {
        const int node = load_parent(p, l - 1, list + i);
        if (node < 0) continue;
        const int parent = node / CR;
        int lo = 0, hi = np;
        while (lo < hi) { const int mid = (lo + hi) >> 1; if (par[mid] < parent) lo = mid + 1; else hi = mid; }
        if (lo < np && par[lo] == parent) {
            const int j = lo * CR + node % CR;
            atomicOr(&selw[j >> 5], 1u << (j & 31));
        }
    }
}
// How many queries may share a warp (see the head of this file).  It pays where they select many of the same parents: with TK of n leaf
// parents selected, PK queries meet n (1 - (1 - TK/n)^PK) of them, or all the same ones while there are no more than TK.  At TK = n/4
// two queries still meet 12% fewer blocks than one by one; further down a step's extra work (5 to 10%) eats what is saved.
inline int sharing_queries(int CR, int G, int TK, int leaf_parents) {
    return CR != 16 || G > 4 || TK * 16 > 65536 || 4 * (int64_t)TK < leaf_parents ? 1 : G > 2 ? 2 : 4;
}
// ... and how many do: as long as their warps fill half of the chip's places, since each walks up to PK times as far.  (fp32, 2048 positions
// of 2 x 4 heads of 64, 2048 warps instead of 4096: 84.7 -> 77.8 us.)
inline int queries_per_warp(int CR, int G, int TK, int leaf_parents, int64_t groups) {
    const int PK = sharing_queries(CR, G, TK, leaf_parents);
    return groups >= (int64_t)PK * 148 * 8 ? PK : 1;
}

}  // namespace htree
