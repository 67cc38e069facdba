// Operand preparation of the transposed tensor-core kernels: one warp per (batch, parent, KV head) reads the parent's
// children once and writes everything that is derived from them: the parent's own pooled row (the next level), the operand
// blocks of the forward and of the backward (layouts in tform.cuh).  One launch per level.
// HBM / L2 streaming: per 16-bit block of 16 children and 128-wide heads it
// reads 8 KB and writes 8.5 KB (12.5 KB with the backward's part); the launches it replaces (pooling, rotation, two blockings
// per level) read the same rows four times and cost a launch each, which is what short sequences spent their time on.
#include "tform.cuh"

namespace htree {

struct PackArgs {
    const void* k;
    const void* v;
    void* blk;          // forward blocks
    void* vkblk;        // backward: values as A fragments of dP^T, or NULL
    void* pk;           // pooled rows of the next level, or NULL
    void* pv;
    const float* cosc;
    const float* sinc;
    const void* list;       // NULL, or parents [B, Tq, Hkv, TK] (uint16 with `narrow`): only the blocks they name are packed
    int64_t total;      // B * NBLK * Hkv blocks, or list entries
    int32_t Tq, TK;
    int32_t N, NBLK, Hkv, narrow;
};

template <typename T> struct V16;
template <> struct V16<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void unpack(const uint4& r, float* o) {
        o[0] = __uint_as_float(r.x); o[1] = __uint_as_float(r.y); o[2] = __uint_as_float(r.z); o[3] = __uint_as_float(r.w);
    }
    static __device__ __forceinline__ uint4 pack(const float* o) {
        return make_uint4(__float_as_uint(o[0]), __float_as_uint(o[1]), __float_as_uint(o[2]), __float_as_uint(o[3]));
    }
};
template <typename T> struct V16h {
    static constexpr int N = 8;
    static __device__ __forceinline__ void unpack(const uint4& r, float* o) {
        const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { const float2 f = Frag<T>::unpack(w[i]); o[2 * i] = f.x; o[2 * i + 1] = f.y; }
    }
    static __device__ __forceinline__ uint4 pack(const float* o) {
        return make_uint4(Frag<T>::pack(o[0], o[1]), Frag<T>::pack(o[2], o[3]), Frag<T>::pack(o[4], o[5]), Frag<T>::pack(o[6], o[7]));
    }
};
template <> struct V16<__nv_bfloat16> : V16h<__nv_bfloat16> {};
template <> struct V16<__half> : V16h<__half> {};

__device__ __forceinline__ float clamp_half(float x) { return fminf(fmaxf(x, -65504.f), 65504.f); }

// N elements as floats (16-byte loads)
template <typename T, int N>
__device__ __forceinline__ void load_piece(const T* p, bool on, float (&o)[N]) {
    constexpr int VN = V16<T>::N < N ? V16<T>::N : N;
#pragma unroll
    for (int i = 0; i < N; i += VN) {
        if constexpr (VN == V16<T>::N) {
            uint4 x = make_uint4(0u, 0u, 0u, 0u);
            if (on) x = __ldg(reinterpret_cast<const uint4*>(p + i));
            V16<T>::unpack(x, o + i);
        } else {
            float t[4] = {0.f, 0.f, 0.f, 0.f};
            if (on) load4<T>(p + i, t);
#pragma unroll
            for (int u = 0; u < 4; ++u) o[i + u] = t[u];
        }
    }
}

// x[0..N) -> half pairs: hi = half(x) and, split-half, lo = half(x - hi)
template <bool X3, int N>
__device__ __forceinline__ void to_half_words(const float (&x)[N], uint32_t (&hi)[N / 2], uint32_t (&lo)[X3 ? N / 2 : 1]) {
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        if constexpr (X3) split_half2(x[2 * i], x[2 * i + 1], hi[i], lo[i]);
        else hi[i] = Frag<__half>::pack(x[2 * i], x[2 * i + 1]);
    }
}

template <typename T, int D, bool X3, int CR>
__global__ void __launch_bounds__(128) pack_blocks_kernel(const __grid_constant__ PackArgs a) {
    chain_enter();
    using C = TForm<D, X3, CR>;
    constexpr int HALF = C::HALF, PPT = C::PPT, KS = C::KS, VB = C::VB;
    int64_t blk = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (blk >= a.total) return;
    const int lane = threadIdx.x & 31, g = lane >> 2, r = lane & 3;
    if (a.list) {
        // (HTREE_PARENTS_U16: no level has 65536 parents, and "none" is past their end like -1)
        const uint32_t node = a.narrow ? static_cast<const uint16_t*>(a.list)[blk] : static_cast<const uint32_t*>(a.list)[blk];
        if (node >= (uint32_t)a.NBLK) return;
        const int64_t grp = blk / a.TK;
        blk = ((grp / ((int64_t)a.Hkv * a.Tq)) * a.NBLK + node) * a.Hkv + grp % a.Hkv;
    }
    const int h = (int)(blk % a.Hkv);
    const int p = (int)((blk / a.Hkv) % a.NBLK);
    const int64_t b = blk / ((int64_t)a.Hkv * a.NBLK);
    const int row0 = p * CR, cnt = min(CR, a.N - row0);
    const int64_t rs = (int64_t)a.Hkv * D;                               // elements between consecutive nodes
    const int64_t base = ((b * a.N + row0) * a.Hkv + h) * (int64_t)D;    // first child's row
    const T* ks_ = reinterpret_cast<const T*>(a.k) + base;
    const T* vs_ = reinterpret_cast<const T*>(a.v) + base;
    unsigned char* dst = reinterpret_cast<unsigned char*>(a.blk) + blk * C::BLOCK;

    // ---- split-half: the block's factors, from the largest magnitudes of its rows (read here and, from L1, again below) ----
    constexpr int NB = CR / 8;
    float kscale = 1.f, vscale = 1.f;
    if constexpr (X3) {
        float km = 0.f, vm = 0.f;
#pragma unroll
        for (int tl = 0; tl < NB; ++tl) {
            const int child = 8 * tl + g;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                float x[PPT];
                if constexpr (C::KSCALED) {
                    load_piece<T, PPT>(ks_ + child * rs + hf * HALF + PPT * r, child < cnt, x);
#pragma unroll
                    for (int i = 0; i < PPT; ++i) km = fmaxf(km, fabsf(x[i]));
                }
                load_piece<T, PPT>(vs_ + child * rs + hf * HALF + PPT * r, child < cnt, x);
#pragma unroll
                for (int i = 0; i < PPT; ++i) vm = fmaxf(vm, fabsf(x[i]));
            }
        }
        if constexpr (C::KSCALED) kscale = range_scale(redux_max_f32(km, 0xffffffffu));
        vscale = range_scale(redux_max_f32(vm, 0xffffffffu));
        if (lane == 0) *reinterpret_cast<float2*>(dst + C::FACS_OFF) = make_float2(pow2_inverse(kscale), pow2_inverse(vscale));
    }

    // ---- keys: rotate by the position inside the chunk ----
    uint32_t kw[2][2][PPT / 2], kl[2][2][X3 ? PPT / 2 : 1];   // [tile or version][half][pair of pairs]
#pragma unroll
    for (int tl = 0; tl < (C::DUAL ? 1 : 2); ++tl) {
        const int child = CR == 16 ? 8 * tl + g : g;          // 8 children, split-half: tl = 1 is the version for odd slots
        const bool on = child < cnt;
        float lo[PPT], hi[PPT], x[PPT], y[PPT];
        load_piece<T, PPT>(ks_ + child * rs + PPT * r, on, lo);
        load_piece<T, PPT>(ks_ + child * rs + HALF + PPT * r, on, hi);
        if constexpr (C::KSCALED) {
#pragma unroll
            for (int i = 0; i < PPT; ++i) { lo[i] *= kscale; hi[i] *= kscale; }
        }
        const float4* cp = reinterpret_cast<const float4*>(a.cosc + (8 * tl + g) * HALF + PPT * r);
        const float4* sp = reinterpret_cast<const float4*>(a.sinc + (8 * tl + g) * HALF + PPT * r);
#pragma unroll
        for (int i = 0; i < PPT / 4; ++i) {
            const float4 c4 = __ldg(cp + i), s4 = __ldg(sp + i);
            const float cs[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = 4 * i + u;
                x[j] = clamp_half(lo[j] * cs[u] - hi[j] * sn[u]);
                y[j] = clamp_half(lo[j] * sn[u] + hi[j] * cs[u]);
            }
        }
        to_half_words<X3, PPT>(x, kw[tl][0], kl[tl][0]);
        to_half_words<X3, PPT>(y, kw[tl][1], kl[tl][1]);
    }
#pragma unroll
    for (int pl = 0; pl < C::PL; ++pl) {
        auto K = [&](int tl, int hf, int i) { return (X3 && pl) ? kl[tl][hf][X3 ? i : 0] : kw[tl][hf][i]; };
        if constexpr (CR == 16) {
            uint32_t* d = reinterpret_cast<uint32_t*>(dst + pl * C::PART);
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                for (int m = 0; m < 4; ++m) d[(4 * ks + m) * 32 + lane] = K(m & 1, m >> 1, ks);
        } else {
#pragma unroll
            for (int vv = 0; vv < (C::DUAL ? 1 : 2); ++vv) {      // even-slot version first, odd-slot version after the values
                uint32_t* d = reinterpret_cast<uint32_t*>(dst + (vv ? 2 * C::PL * C::PART : 0) + pl * C::PART);
#pragma unroll
                for (int ks = 0; ks < KS; ++ks) { d[(2 * ks) * 32 + lane] = K(vv, 0, ks); d[(2 * ks + 1) * 32 + lane] = K(vv, 1, ks); }
            }
        }
    }

    // ---- values: pairs of children per word ----
    uint32_t vw[NB][VB], vl[X3 ? NB : 1][X3 ? VB : 1];
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        const int c0 = 8 * j + 2 * r;
        float x0[VB], x1[VB];
        load_piece<T, VB>(vs_ + c0 * rs + VB * g, c0 < cnt, x0);
        load_piece<T, VB>(vs_ + (c0 + 1) * rs + VB * g, c0 + 1 < cnt, x1);
#pragma unroll
        for (int w = 0; w < VB; ++w) {
            if constexpr (X3) split_half2(clamp_half(x0[w] * vscale), clamp_half(x1[w] * vscale), vw[j][w], vl[X3 ? j : 0][X3 ? w : 0]);
            else vw[j][w] = Frag<T>::pack(x0[w], x1[w]);      // exact: the values are of this type
        }
    }
#pragma unroll
    for (int pl = 0; pl < C::PL; ++pl) {
        auto W = [&](int j, int w) { return (X3 && pl) ? vl[X3 ? j : 0][X3 ? w : 0] : vw[j][w]; };
        unsigned char* vd = dst + C::PL * C::PART + pl * C::PART;
        if constexpr (CR == 16) {
#pragma unroll
            for (int i = 0; i < VB / 2; ++i)
                reinterpret_cast<uint4*>(vd)[i * 32 + lane] = make_uint4(W(0, 2 * i), W(0, 2 * i + 1), W(NB - 1, 2 * i), W(NB - 1, 2 * i + 1));
        } else {
#pragma unroll
            for (int w = 0; w < VB; ++w) reinterpret_cast<uint32_t*>(vd)[w * 32 + lane] = W(0, w);
        }
    }

    // ---- the pooled row: fp32 sum in child order, one division, one rounding (src/naive.py:53-57) ----
    if (a.pk) {
        constexpr int VN = V16<T>::N, NV = D / VN;
#pragma unroll
        for (int i0 = 0; i0 < 2 * NV; i0 += 32) {
            const int i = i0 + lane;
            if (2 * NV < 32 && i >= 2 * NV) break;
            const bool isv = i >= NV;
            const int col = isv ? i - NV : i;
            const uint4* s = reinterpret_cast<const uint4*>(isv ? vs_ : ks_) + col;
            float acc[VN];
#pragma unroll
            for (int u = 0; u < VN; ++u) acc[u] = 0.f;
#pragma unroll
            for (int c0 = 0; c0 < CR; c0 += 8) {
                uint4 x[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) x[c] = c0 + c < cnt ? __ldg(s + (int64_t)(c0 + c) * (rs / VN)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    if (c0 + c < cnt) {
                        float f[VN];
                        V16<T>::unpack(x[c], f);
#pragma unroll
                        for (int u = 0; u < VN; ++u) acc[u] += f[u];
                    }
                }
            }
            const float n = (float)cnt;
#pragma unroll
            for (int u = 0; u < VN; ++u) acc[u] = acc[u] / n;
            reinterpret_cast<uint4*>(isv ? a.pv : a.pk)[blk * NV + col] = V16<T>::pack(acc);     // row (b, p, h) of the next level
        }
    }

    // ---- backward: value rows in the key-part order (A fragments of dP^T = V dO^T; contraction over the head dimension) ----
    if (a.vkblk) {
        unsigned char* vd = reinterpret_cast<unsigned char*>(a.vkblk) + blk * (C::PL * C::PART);
        uint32_t rw[NB][2][PPT / 2], rl[X3 ? NB : 1][2][X3 ? PPT / 2 : 1];
#pragma unroll
        for (int tl = 0; tl < NB; ++tl) {
            const int child = 8 * tl + g;
            const bool on = child < cnt;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                float x[PPT];
                load_piece<T, PPT>(vs_ + child * rs + hf * HALF + PPT * r, on, x);
#pragma unroll
                for (int i = 0; i < PPT / 2; ++i) {
                    if constexpr (X3) split_half2(clamp_half(x[2 * i] * vscale), clamp_half(x[2 * i + 1] * vscale), rw[tl][hf][i], rl[X3 ? tl : 0][hf][X3 ? i : 0]);
                    else rw[tl][hf][i] = Frag<T>::pack(x[2 * i], x[2 * i + 1]);
                }
            }
        }
#pragma unroll
        for (int pl = 0; pl < C::PL; ++pl) {
            auto R = [&](int tl, int hf, int i) { return (X3 && pl) ? rl[X3 ? tl : 0][hf][X3 ? i : 0] : rw[tl][hf][i]; };
            if constexpr (CR == 16) {
                uint32_t* d = reinterpret_cast<uint32_t*>(vd + pl * C::PART);
#pragma unroll
                for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                    for (int m = 0; m < 4; ++m) d[(4 * ks + m) * 32 + lane] = R((NB - 1) * (m & 1), m >> 1, ks);
            } else {
                uint32_t* d = reinterpret_cast<uint32_t*>(vd + pl * C::PART);
#pragma unroll
                for (int ks = 0; ks < KS; ++ks) { d[(2 * ks) * 32 + lane] = R(0, 0, ks); d[(2 * ks + 1) * 32 + lane] = R(0, 1, ks); }
            }
        }
    }
}

size_t pack_block_bytes(int D, bool x3, int CR) { return (size_t)(x3 ? 2 : 1) * D * 2 * CR * (CR == 16 || !x3 ? 2 : 3) + (x3 ? 128 : 0); }

bool pack_supported(int dtype, int K, int V, int CR) {
    (void)dtype;
    return K == V && (K == 32 || K == 64 || K == 128) && (CR == 8 || CR == 16);
}
bool pack_split(int dtype, int D) { return dtype == HTREE_F32 || D == 32; }

template <typename T, int D, bool X3>
static int launch_pack_t(const PackArgs& a, int CR, cudaStream_t st) {
    return launch_chained(CR == 16 ? pack_blocks_kernel<T, D, X3, 16> : pack_blocks_kernel<T, D, X3, 8>, dim3((unsigned)((a.total + 3) / 4)), dim3(128), 0, st, a);
}
template <typename T>
static int launch_pack_d(const PackArgs& a, int D, int CR, cudaStream_t st) {
    constexpr bool F32 = std::is_same<T, float>::value;
    return D == 128 ? launch_pack_t<T, 128, F32>(a, CR, st) : D == 64 ? launch_pack_t<T, 64, F32>(a, CR, st) : launch_pack_t<T, 32, true>(a, CR, st);
}

static int launch_pack(const PackArgs& a, const HtreeShape& s, cudaStream_t st) {
    switch (s.dtype) {
        case HTREE_F32: return launch_pack_d<float>(a, s.K, s.compression_rate, st);
        case HTREE_BF16: return launch_pack_d<__nv_bfloat16>(a, s.K, s.compression_rate, st);
        default: return launch_pack_d<__half>(a, s.K, s.compression_rate, st);
    }
}

static PackArgs pack_args(const HtreeShape& s, int N, const void* k, const void* v, void* blk, const float* cosc, const float* sinc) {
    PackArgs a{};
    a.k = k; a.v = v; a.blk = blk; a.cosc = cosc; a.sinc = sinc;
    a.N = N; a.Hkv = s.H_kv; a.NBLK = (N + s.compression_rate - 1) / s.compression_rate;
    a.total = (int64_t)s.B * a.NBLK * s.H_kv;
    return a;
}

// blk[l] of the levels from `first` up, and, where asked for, the pooled levels lk[l + 1] / lv[l + 1] and vkblk[l].
int launch_pack_blocks(const HtreeShape& s, int first, int L, const int32_t* ln, void* const* lk, void* const* lv, void* const* blk,
                       void* const* vkblk, bool pool, const float* cosc, const float* sinc, cudaStream_t st) {
    for (int l = first; l < L; ++l) {
        PackArgs a = pack_args(s, ln[l], lk[l], lv[l], blk[l], cosc, sinc);
        a.vkblk = vkblk ? vkblk[l] : nullptr;
        a.pk = pool && l + 1 < L ? lk[l + 1] : nullptr; a.pv = pool && l + 1 < L ? lv[l + 1] : nullptr;
        const int rc = launch_pack(a, s, st);
        if (rc) return rc;
    }
    return 0;
}

// The leaf blocks that the parent lists of level 0 name, [B, Tq, H_kv, top_k] (a block named twice is written twice, alike).
int launch_pack_listed(const HtreeShape& s, int Tq, const void* k, const void* v, void* blk, const void* parents, bool narrow,
                       const float* cosc, const float* sinc, cudaStream_t st) {
    PackArgs a = pack_args(s, s.T, k, v, blk, cosc, sinc);
    a.list = parents; a.narrow = narrow; a.Tq = Tq; a.TK = s.top_k;
    a.total = (int64_t)s.B * Tq * s.H_kv * s.top_k;
    return launch_pack(a, s, st);
}

}  // namespace htree
