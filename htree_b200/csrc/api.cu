// extern "C" boundary of libhtree_b200: argument validation, parameter blocks, kernel dispatch.
#include <atomic>
#include <cstring>

#include "bwd_tform.cuh"

namespace htree {

static std::atomic<unsigned long long> g_launches{0};
void note_launch(int n) { g_launches.fetch_add((unsigned long long)n, std::memory_order_relaxed); }

static int esize(int dtype) { return dtype == HTREE_F32 ? 4 : 2; }
static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
// the tensor-core kernels move 32-byte pieces with 256-bit loads
static bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }

static int level_sizes(int T, int CR, int MTN, int32_t* ln) {
    if (T <= 0 || CR < 2 || MTN < 1) return HTREE_E_SHAPE;
    int L = 1, n = T;
    ln[0] = T;
    while (n > MTN) {
        n = (n + CR - 1) / CR;
        if (L >= HTREE_MAX_LEVELS) return HTREE_E_LEVELS;
        ln[L++] = n;
    }
    return L;
}

static int check_shape(const HtreeShape* s, int32_t* ln, bool check_top = true) {
    if (!s) return HTREE_E_NULL;
    if (s->B <= 0 || s->T <= 0 || s->H <= 0 || s->H_kv <= 0 || s->K <= 0 || s->V <= 0 || s->top_k <= 0) return HTREE_E_SHAPE;
    if (s->H % s->H_kv != 0 || (s->K & 1)) return HTREE_E_SHAPE;
    if (s->dtype != HTREE_F32 && s->dtype != HTREE_BF16 && s->dtype != HTREE_F16) return HTREE_E_DTYPE;
    if ((int64_t)s->B * s->H_kv > 65535) return HTREE_E_UNSUPPORTED;
    const int L = level_sizes(s->T, s->compression_rate, s->max_top_nodes, ln);
    if (L < 0) return L;
    if (check_top && (int64_t)ln[L - 1] > (int64_t)s->top_k * s->compression_rate) return HTREE_E_TOPLEVEL;
    // 16-byte rows: K, V multiples of 8 keep every vector load of every kernel aligned for all storage types
    if (s->K % 8 != 0 || s->V % 8 != 0) return HTREE_E_ALIGN;
    if (s->T_q < 0 || s->t_offset < 0 || (s->T_q == 0 && s->t_offset != 0) ||
        (int64_t)s->t_offset + s->T_q > s->T) return HTREE_E_WINDOW;
    return L;
}

static int fill_params(AttnParams& p, const HtreeShape* s, int L, const int32_t* ln, const void* q, void* const* lk,
                       void* const* lv, const float* cosc, const float* sinc, int32_t n_pos, float scale,
                       int32_t* const* parents, int32_t* status, uint32_t flags) {
    std::memset(&p, 0, sizeof(p));
    if (!q || !lk || !lv || !cosc || !sinc) return HTREE_E_NULL;
    if ((int64_t)n_pos < (int64_t)s->top_k * s->compression_rate) return HTREE_E_ROPE;
    if (!aligned16(q) || !aligned16(cosc) || !aligned16(sinc)) return HTREE_E_ALIGN;
    if ((flags & HTREE_PARENTS_U16) && parents) {   // ids of level l+1 (or of the virtual parents) must fit, 0xFFFF = none
        if (s->top_k > 65535) return HTREE_E_UNSUPPORTED;
        for (int l = 1; l < L; ++l) if (ln[l] > 65535) return HTREE_E_UNSUPPORTED;
    }
    p.q = q;
    int64_t pw = 1;
    for (int l = 0; l < L; ++l) {
        if (!lk[l] || !lv[l]) return HTREE_E_NULL;
        if (!aligned16(lk[l]) || !aligned16(lv[l])) return HTREE_E_ALIGN;
        p.lk[l] = lk[l]; p.lv[l] = lv[l]; p.ln[l] = ln[l]; p.lpow[l] = pw;
        p.parents[l] = parents ? parents[l] : nullptr;
        pw *= s->compression_rate;
    }
    p.cosc = cosc; p.sinc = sinc; p.status = status;
    p.B = s->B; p.T = s->T; p.H = s->H; p.Hkv = s->H_kv; p.K = s->K; p.V = s->V;
    p.CR = s->compression_rate; p.TK = s->top_k; p.L = L; p.G = s->H / s->H_kv; p.n_pos = n_pos;
    p.Tq = s->T_q > 0 ? s->T_q : s->T; p.t0 = s->t_offset;
    p.scale = scale; p.flags = flags;
    return 0;
}

// Windows, launches and buffers of the two-pass backward for a shape and a scratch size.
struct BwdLayout {
    BwdParams bp;
    int64_t acc_bytes, scratch_bytes, zero_bytes;
    int64_t acck[HTREE_MAX_LEVELS], accv[HTREE_MAX_LEVELS], xtab;      // in the accumulators' buffer; xtab < 0: none
    int64_t o_qb, o_dob, o_stp, o_sts, o_fac, o_rank, o_nvis, o_cnt, o_base, o_entries, o_items, o_nitems;
    int total, per_launch;
};

// the counters of `windows` windows, in whole 16-byte pieces; the words of the range stand behind those of a whole launch
static int64_t cnt_words(int64_t windows, int64_t NK) { return (windows * NK + 3) & ~int64_t(3); }

static int bwd_layout(const HtreeShape* s, int L, const int32_t* ln, int64_t budget, BwdLayout& y) {
    std::memset(&y, 0, sizeof(y));
    const int CR = s->compression_rate, TK = s->top_k, D = s->K, G = s->H / s->H_kv;
    if (!pack_supported(s->dtype, s->K, s->V, CR) || G > 16 || (int64_t)TK * CR > 131072) return HTREE_E_UNSUPPORTED;
    const bool x3 = pack_split(s->dtype, D);
    const int NH = G > 8 ? 2 : 1, Tq = s->T_q > 0 ? s->T_q : s->T;
    BwdParams& bp = y.bp;
    auto up = [](int64_t x) { return (x + 255) & ~int64_t(255); };
    const int64_t units = (int64_t)s->B * s->H_kv;
    const int PK = bp.PK = queries_per_warp(CR, G, TK, (ln[0] + CR - 1) / CR, units * Tq);
    const bool many = PK > 1;
    int64_t at = 0, MV = 0, NK = 0;
    for (int l = L - 1; l >= 0; --l) {
        const int64_t nblk = (ln[l] + CR - 1) / CR, one = nblk < TK ? nblk : TK, np = nblk < (int64_t)PK * TK ? nblk : (int64_t)PK * TK;
        const bool used = l == 0 || one * CR > TK;     // does any query accumulate here?
        bp.voff[l] = used ? (int32_t)MV : -1;
        bp.koff[l] = (int32_t)NK;
        if (used) { MV += np; NK += nblk; }
        const int64_t blocks = (int64_t)s->B * nblk * s->H_kv;
        y.acck[l] = at; at += up(blocks * D * CR * 4);
        y.accv[l] = at; at += up(blocks * D * CR * 4);
    }
    y.zero_bytes = at;
    // The rotary rows stand behind the accumulators, whose size is no part of the budget: windows of any size of one backward find them
    // at the same place, and a budget for little more than a window is not taken up by 2 MB of table.
    y.xtab = x3 ? -1 : at;
    y.acc_bytes = x3 ? at : at + up((int64_t)TK * CR * D * 2);
    const int64_t qb = (int64_t)NH * D * 16 * (x3 ? 2 : 1), sb = (int64_t)NH * (CR / 8) * 128 * (x3 ? 2 : 1);
    const int64_t entry = entry_bytes(x3, PK);
    // A window's blocked queries (4 KB each at 16 heads of 128) should stay in the L2 while its parents gather them: 8192 queries
    // are 33 MB; longer windows mean longer visit lists and fewer reductions.
    int64_t subq = 0, ng = 0, bytes = 0;
    const int64_t fixed = up(4 + units * 4);                    // besides the windows: the words of the range
    for (int64_t most = 8192; most >= 8; most >>= 1) {
        const int64_t nw = (Tq + most - 1) / most;
        subq = ((Tq + nw - 1) / nw + PK - 1) / PK * PK;
        ng = subq / PK;
        const int64_t visits = ng * MV;
        // of a window; the buffers below hold no more than `per` times that and the words
        bytes = up(ng * qb) * 2 + up(visits * sb) * 2 + up(visits * (many ? 16 : 4)) + up(visits * entry) + (x3 ? up(ng * PK * L * 8) : 0) + (many ? up(ng * L * 4) : 0) +
                up(NK * 4) + up(NK * 8) + up((visits / 8 + NK) * (int64_t)sizeof(BwdItem)) + up(4);
        if (fixed + bytes <= budget && visits < (int64_t(1) << 31)) { bp.nw = (int32_t)nw; break; }
    }
    if (bp.nw == 0) return HTREE_E_SCRATCH;
    bp.subq = (int32_t)subq; bp.ng = (int32_t)ng; bp.MV = (int32_t)MV; bp.NK = (int32_t)NK;
    y.total = (int)(units * bp.nw);
    int64_t per = (budget - fixed) / bytes;
    if (per > 32767 / ng) per = 32767 / ng;
    if (per * ng * MV >= (int64_t(1) << 31)) per = ((int64_t(1) << 31) - 1) / (ng * MV);
    if (per > y.total) per = y.total;
    if (per < 1) per = 1;
    const int64_t launches = (y.total + per - 1) / per;
    per = (y.total + launches - 1) / launches;
    y.per_launch = (int)per;
    // items long enough to pay for their reduction (64 visits: 128 bytes of it a visit), short enough to fill the chip
    int64_t seg = per * ng * MV / (148 * 16 * 3);
    bp.seg = (int32_t)(seg < 8 ? 8 : seg > 64 ? 64 : seg);
    bp.cap = (int32_t)(ng * MV / bp.seg + NK);
    at = 0;
    auto take = [&](int64_t n) { const int64_t o = at; at += up(n); return o; };
    y.o_qb = take(per * ng * qb); y.o_dob = take(per * ng * qb);
    y.o_stp = take(per * ng * MV * sb); y.o_sts = take(per * ng * MV * sb);
    y.o_fac = x3 ? take(per * ng * PK * L * 8) : -1;
    y.o_nvis = many ? take(per * ng * L * 4) : -1;
    y.o_rank = take(per * ng * MV * (many ? 16 : 4)); y.o_entries = take(per * ng * MV * entry);
    y.o_cnt = take(cnt_words(per, NK) * 4 + 4 + units * 4); y.o_base = take(per * NK * 8);
    y.o_items = take(per * bp.cap * (int64_t)sizeof(BwdItem)); y.o_nitems = take(per * 4);
    y.scratch_bytes = at;
    return 0;
}

}  // namespace htree

using namespace htree;

extern "C" {

int htree_b200_version(void) { return HTREE_B200_VERSION; }

uint64_t htree_b200_launch_count(void) { return (uint64_t)htree::g_launches.load(std::memory_order_relaxed); }

const char* htree_b200_error_string(int code) {
    switch (code) {
        case 0: return "success";
        case HTREE_E_NULL: return "a required pointer is NULL";
        case HTREE_E_SHAPE: return "invalid shape: sizes must be positive, H divisible by H_kv, K even";
        case HTREE_E_DTYPE: return "unknown storage type";
        case HTREE_E_LEVELS: return "too many tree levels";
        case HTREE_E_TOPLEVEL: return "top tree level is longer than top_k*compression_rate";
        case HTREE_E_ROPE: return "cos/sin tables have fewer than top_k*compression_rate rows";
        case HTREE_E_ALIGN: return "pointers must be 16-byte aligned and K, V multiples of 8";
        case HTREE_E_UNSUPPORTED: return "shape not supported by the compiled kernels";
        case HTREE_E_NODEVICE: return "no usable CUDA device";
        case HTREE_E_WINDOW: return "query window outside the sequence, or a backward window without HTREE_BWD_KEEP_ACCUM / HTREE_BWD_NO_FOLD";
        case HTREE_E_SCRATCH: return "pooled tree levels do not fit the built-in scratch array (see htree_b200_static_scratch_bytes)";
        default: return code > 0 ? cudaGetErrorString((cudaError_t)code) : "unknown htree_b200 error";
    }
}

int htree_b200_num_levels(int32_t T, int32_t CR, int32_t MTN) {
    int32_t ln[HTREE_MAX_LEVELS];
    return level_sizes(T, CR, MTN, ln);
}

int htree_b200_level_sizes(int32_t T, int32_t CR, int32_t MTN, int32_t* sizes, int32_t cap) {
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = level_sizes(T, CR, MTN, ln);
    if (L < 0) return L;
    if (!sizes) return HTREE_E_NULL;
    for (int l = 0; l < L && l < cap; ++l) sizes[l] = ln[l];
    return L;
}

int htree_b200_build_tree(const HtreeShape* shape, void* const* layers_k, void* const* layers_v,
                          void* const* layers_k_rot, void* const* layers_k_blk, void* const* layers_v_blk,
                          const float* cos_cache, const float* sin_cache, void* stream) {
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln, false);   // top_k plays no role in the tree
    if (L < 0) return L;
    if (!layers_k || !layers_v) return HTREE_E_NULL;
    for (int l = 0; l < L; ++l) {
        if (!layers_k[l] || !layers_v[l]) return HTREE_E_NULL;
        if (!aligned16(layers_k[l]) || !aligned16(layers_v[l])) return HTREE_E_ALIGN;
    }
    const int es = esize(shape->dtype);
    if ((shape->H_kv * shape->K * es) % 16 || (shape->H_kv * shape->V * es) % 16) return HTREE_E_ALIGN;
    if (layers_k_rot) {
        if (!cos_cache || !sin_cache) return HTREE_E_NULL;
        if (!aligned16(cos_cache) || !aligned16(sin_cache)) return HTREE_E_ALIGN;
        for (int l = 0; l < L; ++l) {
            if (!layers_k_rot[l]) return HTREE_E_NULL;
            if (!aligned16(layers_k_rot[l])) return HTREE_E_ALIGN;
        }
    }
    if (layers_v_blk) {
        if ((shape->V != 64 && shape->V != 128) || (shape->compression_rate != 8 && shape->compression_rate != 16) ||
            (shape->dtype == HTREE_F32 && shape->V != 64))
            return HTREE_E_UNSUPPORTED;
        for (int l = 0; l < L; ++l) {
            if (!layers_v_blk[l]) return HTREE_E_NULL;
            if (!aligned32(layers_v_blk[l])) return HTREE_E_ALIGN;
        }
    }
    if (layers_k_blk) {
        if (!layers_k_rot) return HTREE_E_NULL;       // the blocked keys are built from the rotated keys
        if (shape->dtype == HTREE_F32 || shape->K != 128 || shape->compression_rate != 16) return HTREE_E_UNSUPPORTED;
        for (int l = 0; l < L; ++l) {
            if (!layers_k_blk[l]) return HTREE_E_NULL;
            if (!aligned32(layers_k_blk[l])) return HTREE_E_ALIGN;
        }
    }
    int rc = launch_tree_build(*shape, L, ln, layers_k, layers_v, (cudaStream_t)stream);
    if (rc == 0 && layers_k_rot)
        rc = launch_rotate_keys(*shape, L, ln, layers_k, layers_k_rot, cos_cache, sin_cache, (cudaStream_t)stream);
    if (rc == 0 && layers_k_blk)
        rc = launch_block_keys(*shape, L, ln, layers_k_rot, layers_k_blk, (cudaStream_t)stream);
    if (rc == 0 && layers_v_blk)
        rc = launch_block_values(*shape, L, ln, layers_v, layers_v_blk, (cudaStream_t)stream);
    return rc;
}

int64_t htree_b200_operand_block_bytes(const HtreeShape* shape, int32_t level, int32_t backward) {
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln, false);
    if (L < 0) return L;
    if (level < 0 || level >= L) return HTREE_E_LEVELS;
    if (!pack_supported(shape->dtype, shape->K, shape->V, shape->compression_rate)) return HTREE_E_UNSUPPORTED;
    const int CR = shape->compression_rate;
    const bool x3 = pack_split(shape->dtype, shape->K);
    const int64_t blocks = (int64_t)shape->B * ((ln[level] + CR - 1) / CR) * shape->H_kv;
    return blocks * (backward ? (int64_t)(x3 ? 2 : 1) * shape->K * 2 * CR : (int64_t)pack_block_bytes(shape->K, x3, CR));
}

int htree_b200_prepare(const HtreeShape* shape, void* const* layers_k, void* const* layers_v, void* const* blocks,
                       void* const* blocks_bwd, int32_t pool, const float* cos_cache, const float* sin_cache, void* stream) {
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln, false);
    if (L < 0) return L;
    if (!layers_k || !layers_v || !blocks || !cos_cache || !sin_cache) return HTREE_E_NULL;
    if (!pack_supported(shape->dtype, shape->K, shape->V, shape->compression_rate)) return HTREE_E_UNSUPPORTED;
    if (!aligned16(cos_cache) || !aligned16(sin_cache)) return HTREE_E_ALIGN;
    for (int l = 0; l < L; ++l) {
        if (!layers_k[l] || !layers_v[l] || !blocks[l] || (blocks_bwd && !blocks_bwd[l])) return HTREE_E_NULL;
        if (!aligned16(layers_k[l]) || !aligned16(layers_v[l]) || !aligned16(blocks[l]) || (blocks_bwd && !aligned16(blocks_bwd[l])))
            return HTREE_E_ALIGN;
    }
    return launch_pack_blocks(*shape, 0, L, ln, layers_k, layers_v, blocks, blocks_bwd, pool != 0, cos_cache, sin_cache,
                              (cudaStream_t)stream);
}

// `pack_leaves`: the leaf blocks are still to be packed, those that the selections name
static int attend(const HtreeShape* shape, const void* q, void* const* layers_k, void* const* layers_v, void* const* blocks,
                  const float* cos_cache, const float* sin_cache, const void* table, const void* table_f32, int32_t n_pos, float scale,
                  void* out, float* gmax, float* gsum, int32_t* const* parents, int32_t* status, uint32_t flags, bool pack_leaves,
                  float* top_keys, void* stream) {
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln);
    if (L < 0) return L;
    AttnParams p;
    int rc = fill_params(p, shape, L, ln, q, layers_k, layers_v, cos_cache, sin_cache, n_pos, scale, parents, status, flags);
    if (rc) return rc;
    const bool select_only = (flags & HTREE_FWD_SELECT_ONLY) != 0;
    if (!blocks || !table || !table_f32 || !parents || (!select_only && (!out || !gmax || !gsum))) return HTREE_E_NULL;
    if (!aligned16(out) || !aligned16(table) || !aligned16(table_f32) || !aligned32(q)) return HTREE_E_ALIGN;
    p.out = out; p.gmax = gmax; p.gsum = gsum; p.tab = table; p.tab32 = table_f32;
    for (int l = 0; l < L; ++l) {
        if (!parents[l] || !blocks[l]) return HTREE_E_NULL;
        if (!aligned16(blocks[l])) return HTREE_E_ALIGN;
        p.blk[l] = blocks[l];
    }
    if (!acc_mma_supported(p, shape->dtype)) return HTREE_E_UNSUPPORTED;
    p.flags = flags | HTREE_FWD_SELECT_ONLY;
    if (select_blk_supported(p, shape->dtype)) {
        rc = launch_select_blk(p, shape->dtype, (cudaStream_t)stream);
    } else {
        p.ktop = top_keys;
        rc = launch_select_top(p, shape->dtype, !fwd_generic_tiled(p), (cudaStream_t)stream);
        if (rc == 0) p.first_level = L - 2;       // (0: two levels, nothing below selects)
        if (rc == HTREE_E_UNSUPPORTED || (rc == 0 && L > 2)) rc = launch_fwd_generic(p, shape->dtype, (cudaStream_t)stream);
        p.first_level = 0;
    }
    if (rc || select_only) return rc;
    if (pack_leaves) {
        rc = launch_pack_listed(*shape, p.Tq, layers_k[0], layers_v[0], blocks[0], parents[0], (flags & HTREE_PARENTS_U16) != 0, cos_cache, sin_cache,
                                (cudaStream_t)stream);
        if (rc) return rc;
    }
    p.flags = flags | ((flags & HTREE_FWD_INFERENCE) ? kFlagSplitOk : 0u);
    return launch_acc_mma(p, shape->dtype, (cudaStream_t)stream);
}

int htree_b200_attend(const HtreeShape* shape, const void* q, void* const* layers_k, void* const* layers_v, void* const* blocks,
                      const float* cos_cache, const float* sin_cache, const void* table, const void* table_f32, int32_t n_pos, float scale,
                      void* out, float* gmax, float* gsum, int32_t* const* parents, int32_t* status, uint32_t flags, void* stream) {
    return attend(shape, q, layers_k, layers_v, blocks, cos_cache, sin_cache, table, table_f32, n_pos, scale, out, gmax, gsum, parents,
                  status, flags, false, nullptr, stream);
}

int htree_b200_plan(const HtreeShape* shape, uint32_t flags, HtreePlan* plan) {
    if (!plan) return HTREE_E_NULL;
    std::memset(plan, 0, sizeof(*plan));
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln);
    if (L < 0) return L;
    if (!pack_supported(shape->dtype, shape->K, shape->V, shape->compression_rate) || shape->H / shape->H_kv > 16) return HTREE_E_UNSUPPORTED;
    const int es = esize(shape->dtype), CR = shape->compression_rate;
    const bool x3 = pack_split(shape->dtype, shape->K);
    const int64_t Tq = shape->T_q > 0 ? shape->T_q : shape->T;
    int64_t at = 0;
    auto take = [&](int64_t bytes) { const int64_t o = at; at += (bytes + 255) & ~int64_t(255); return o; };
    plan->levels = L;
    for (int l = 0; l < L; ++l) {
        const int64_t rows = (int64_t)shape->B * ln[l] * shape->H_kv, blocks = (int64_t)shape->B * ((ln[l] + CR - 1) / CR) * shape->H_kv;
        plan->nodes[l] = ln[l];
        plan->layers_k[l] = l ? take(rows * shape->K * es) : -1;
        plan->layers_v[l] = l ? take(rows * shape->V * es) : -1;
        plan->blocks[l] = take(blocks * (int64_t)pack_block_bytes(shape->K, x3, CR));
        plan->blocks_bwd[l] = flags & HTREE_PLAN_BACKWARD ? take(blocks * (x3 ? 2 : 1) * shape->K * 2 * CR) : -1;
        plan->parents[l] = flags & HTREE_PLAN_PARENTS ? take((int64_t)shape->B * Tq * shape->H_kv * shape->top_k * 4) : -1;
    }
    take(top_keys_bytes(*shape, L, ln));       // at the workspace's end
    plan->bytes = at;
    return 0;
}

int htree_b200_run_forward(const HtreeShape* shape, const HtreePlan* plan, const void* q, const void* k, const void* v,
                           const float* cos_cache, const float* sin_cache, const void* table, const void* table_f32, int32_t n_pos,
                           float scale, void* workspace, void* out, float* gmax, float* gsum, int32_t* const* parents, int32_t* status,
                           uint32_t flags, void* stream) {
    if (!shape || !plan || !k || !v || !workspace) return HTREE_E_NULL;
    if (plan->levels <= 0 || plan->levels > HTREE_MAX_LEVELS) return HTREE_E_LEVELS;
    void *lk[HTREE_MAX_LEVELS], *lv[HTREE_MAX_LEVELS], *bl[HTREE_MAX_LEVELS], *bb[HTREE_MAX_LEVELS];
    int32_t* par[HTREE_MAX_LEVELS];
    unsigned char* w = static_cast<unsigned char*>(workspace);
    auto at = [&](int64_t o) { return o < 0 ? nullptr : w + o; };
    for (int l = 0; l < plan->levels; ++l) {
        lk[l] = l ? (void*)at(plan->layers_k[l]) : const_cast<void*>(k);
        lv[l] = l ? (void*)at(plan->layers_v[l]) : const_cast<void*>(v);
        bl[l] = at(plan->blocks[l]); bb[l] = at(plan->blocks_bwd[l]);
        par[l] = parents ? parents[l] : reinterpret_cast<int32_t*>(at(plan->parents[l]));
    }
    // A window of few queries against a long sequence reads a small part of the leaves' blocks: when the selections can name at most
    // half of them, the leaves are only pooled (read once, a sixteenth or an eighth written) and the named blocks packed afterwards.
    // The blocks of all leaves are twice the bytes to move and were a third of a call with one new query against 16K positions.
    const int32_t Tq = shape->T_q > 0 ? shape->T_q : shape->T;
    const int64_t nblk = (shape->T + shape->compression_rate - 1) / shape->compression_rate;
    int rc;
    const bool few = (flags & HTREE_FWD_INFERENCE) && plan->levels > 1 && 2 * (int64_t)Tq * shape->top_k <= nblk;
    if (few) {
        int32_t ln[HTREE_MAX_LEVELS];
        const int L = check_shape(shape, ln);
        if (L < 0) return L;
        if (L != plan->levels || !cos_cache || !sin_cache) return HTREE_E_NULL;
        if (!aligned16(k) || !aligned16(v) || !aligned16(workspace) || !aligned16(cos_cache) || !aligned16(sin_cache)) return HTREE_E_ALIGN;
        rc = launch_tree_build(*shape, 2, ln, lk, lv, (cudaStream_t)stream);
        if (rc == 0) rc = launch_pack_blocks(*shape, 1, L, ln, lk, lv, bl, nullptr, true, cos_cache, sin_cache, (cudaStream_t)stream);
    } else {
        rc = htree_b200_prepare(shape, lk, lv, bl, plan->blocks_bwd[0] >= 0 ? bb : nullptr, 1, cos_cache, sin_cache, stream);
    }
    if (rc) return rc;
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln);
    const int64_t top = L < 0 ? 0 : (top_keys_bytes(*shape, L, ln) + 255) & ~int64_t(255);
    return attend(shape, q, lk, lv, bl, cos_cache, sin_cache, table, table_f32, n_pos, scale, out, gmax, gsum, par, status, flags, few,
                  top ? reinterpret_cast<float*>(w + plan->bytes - top) : nullptr, stream);
}

int htree_b200_block_keys(const HtreeShape* shape, void* const* layers_k_rot, void* const* layers_k_blk, void* stream) {
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln, false);
    if (L < 0) return L;
    if (!layers_k_rot || !layers_k_blk) return HTREE_E_NULL;
    if (shape->dtype == HTREE_F32 || shape->K != 128 || shape->compression_rate != 16) return HTREE_E_UNSUPPORTED;
    for (int l = 0; l < L; ++l) {
        if (!layers_k_rot[l] || !layers_k_blk[l]) return HTREE_E_NULL;
        if (!aligned16(layers_k_rot[l]) || !aligned32(layers_k_blk[l])) return HTREE_E_ALIGN;
    }
    return launch_block_keys(*shape, L, ln, layers_k_rot, layers_k_blk, (cudaStream_t)stream);
}

int htree_b200_block_values(const HtreeShape* shape, void* const* layers_v, void* const* layers_v_blk, void* stream) {
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln, false);
    if (L < 0) return L;
    if (!layers_v || !layers_v_blk) return HTREE_E_NULL;
    if ((shape->V != 64 && shape->V != 128) || (shape->compression_rate != 8 && shape->compression_rate != 16) ||
        (shape->dtype == HTREE_F32 && shape->V != 64))
        return HTREE_E_UNSUPPORTED;
    for (int l = 0; l < L; ++l) {
        if (!layers_v[l] || !layers_v_blk[l]) return HTREE_E_NULL;
        if (!aligned16(layers_v[l]) || !aligned32(layers_v_blk[l])) return HTREE_E_ALIGN;
    }
    return launch_block_values(*shape, L, ln, layers_v, layers_v_blk, (cudaStream_t)stream);
}

int htree_b200_rotate_keys(const HtreeShape* shape, void* const* layers_k, void* const* layers_k_rot,
                           const float* cos_cache, const float* sin_cache, void* stream) {
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln, false);
    if (L < 0) return L;
    if (!layers_k || !layers_k_rot || !cos_cache || !sin_cache) return HTREE_E_NULL;
    if (!aligned16(cos_cache) || !aligned16(sin_cache)) return HTREE_E_ALIGN;
    for (int l = 0; l < L; ++l) {
        if (!layers_k[l] || !layers_k_rot[l]) return HTREE_E_NULL;
        if (!aligned16(layers_k[l]) || !aligned16(layers_k_rot[l])) return HTREE_E_ALIGN;
    }
    return launch_rotate_keys(*shape, L, ln, layers_k, layers_k_rot, cos_cache, sin_cache, (cudaStream_t)stream);
}

int htree_b200_forward(const HtreeShape* shape, const void* q, void* const* layers_k, void* const* layers_v,
                       void* const* layers_k_rot, void* const* layers_k_blk, void* const* layers_v_blk, const float* cos_cache,
                       const float* sin_cache, const void* cos_half,
                       const void* sin_half, int32_t n_pos, float scale, void* out,
                       float* gmax, float* gsum, int32_t* const* parents, const HtreeTrace* trace, int32_t* status,
                       uint32_t flags, void* stream) {
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln);
    if (L < 0) return L;
    AttnParams p;
    int rc = fill_params(p, shape, L, ln, q, layers_k, layers_v, cos_cache, sin_cache, n_pos, scale, parents, status, flags);
    if (rc) return rc;
    const bool select_only = (flags & HTREE_FWD_SELECT_ONLY) != 0;
    if (select_only) {
        if (!parents) return HTREE_E_NULL;
    } else {
        if (!out || !gmax || !gsum) return HTREE_E_NULL;
        if (!aligned16(out)) return HTREE_E_ALIGN;
    }
    p.out = out; p.gmax = gmax; p.gsum = gsum;
    if (cos_half && sin_half && aligned32(cos_half) && aligned32(sin_half)) {
        p.cosh = static_cast<const __half*>(cos_half); p.sinh = static_cast<const __half*>(sin_half);
    }
    if (trace) { p.tr_max = trace->layer_max; p.tr_sum = trace->layer_sum; p.tr_out = trace->layer_out; }
    if (layers_k_rot && !trace && !(flags & HTREE_FWD_GENERIC)) {
        bool all = true;
        for (int l = 0; l < L; ++l) {
            if ((l > 0 || !select_only) && (!layers_k_rot[l] || !aligned32(layers_k_rot[l]))) all = false;   // the leaves select nothing
            p.lkr[l] = layers_k_rot[l];
            if (!select_only) {   // the accumulating passes read the blocked values
                if (!layers_v_blk || !layers_v_blk[l] || !aligned32(layers_v_blk[l])) all = false;
                else p.lvb[l] = layers_v_blk[l];
            }
            // optional: with the blocked keys of every level the pipelined kernels run (bulk copies need 16-byte alignment)
            if (layers_k_blk && layers_k_blk[l] && aligned32(layers_k_blk[l])) p.lkb[l] = layers_k_blk[l];
        }
        all = all && aligned32(q) && aligned32(cos_cache) && aligned32(sin_cache);
        if (all && (select_only ? select_mma_supported(p, shape->dtype) : fwd_mma_supported(p, shape->dtype))) return launch_fwd_mma(p, shape->dtype, (cudaStream_t)stream);
    }
    return launch_fwd_generic(p, shape->dtype, (cudaStream_t)stream);
}

int htree_b200_level_forward(const HtreeShape* s, int32_t level, int32_t n_level, const void* q, const void* layer_k,
                             const void* layer_v, const int32_t* prev_parents, const float* cos_cache,
                             const float* sin_cache, int32_t n_pos, float scale, float* layer_max, float* layer_sum,
                             float* layer_out, int32_t* next_parents, int32_t* status, void* stream) {
    if (!s || !q || !layer_k || !layer_v || !prev_parents || !cos_cache || !sin_cache || !layer_max || !layer_sum || !layer_out)
        return HTREE_E_NULL;
    if (s->B <= 0 || s->T <= 0 || s->H <= 0 || s->H_kv <= 0 || s->K <= 0 || s->V <= 0 || s->top_k <= 0 || n_level <= 0 ||
        s->compression_rate < 2 || s->H % s->H_kv != 0 || (s->K & 1))
        return HTREE_E_SHAPE;
    if (level < 0 || level >= HTREE_MAX_LEVELS) return HTREE_E_LEVELS;
    if (level > 0 && !next_parents) return HTREE_E_NULL;
    if (s->dtype != HTREE_F32 && s->dtype != HTREE_BF16 && s->dtype != HTREE_F16) return HTREE_E_DTYPE;
    if (s->K % 8 != 0 || s->V % 8 != 0 || !aligned16(q) || !aligned16(layer_k) || !aligned16(layer_v) || !aligned16(cos_cache) ||
        !aligned16(sin_cache))
        return HTREE_E_ALIGN;
    if ((int64_t)n_pos < (int64_t)s->top_k * s->compression_rate) return HTREE_E_ROPE;
    if ((int64_t)s->B * s->H_kv > 65535) return HTREE_E_UNSUPPORTED;
    AttnParams p;
    std::memset(&p, 0, sizeof(p));
    p.q = q; p.lk[level] = layer_k; p.lv[level] = layer_v; p.ln[level] = n_level;
    int64_t pw = 1;
    for (int l = 0; l < level; ++l) pw *= s->compression_rate;
    p.lpow[level] = pw;
    p.cosc = cos_cache; p.sinc = sin_cache; p.status = status;
    p.B = s->B; p.T = s->T; p.H = s->H; p.Hkv = s->H_kv; p.K = s->K; p.V = s->V;
    p.CR = s->compression_rate; p.TK = s->top_k; p.L = level + 1; p.G = s->H / s->H_kv; p.n_pos = n_pos;
    p.Tq = s->T; p.t0 = 0; p.scale = scale; p.flags = 0;
    p.level_mode = 1; p.level_index = level; p.parents_in = prev_parents; p.next_out = next_parents;
    p.tr_max = layer_max; p.tr_sum = layer_sum; p.tr_out = layer_out;
    return launch_fwd_generic(p, s->dtype, (cudaStream_t)stream);
}

int htree_b200_merge_to_global(const float* layer_max, const float* layer_sum, const float* layer_out, float* global_max,
                               float* global_sum, float* global_out, int64_t rows, int32_t V, void* stream) {
    if (!layer_max || !layer_sum || !layer_out || !global_max || !global_sum || !global_out) return HTREE_E_NULL;
    if (rows <= 0 || V <= 0) return HTREE_E_SHAPE;
    return launch_merge_to_global(layer_max, layer_sum, layer_out, global_max, global_sum, global_out, rows, V, (cudaStream_t)stream);
}

int htree_b200_final_normalize(const float* global_out, const float* global_sum, void* out, int32_t dtype, int64_t rows,
                               int32_t V, void* stream) {
    if (!global_out || !global_sum || !out) return HTREE_E_NULL;
    if (rows <= 0 || V <= 0) return HTREE_E_SHAPE;
    if (dtype != HTREE_F32 && dtype != HTREE_BF16 && dtype != HTREE_F16) return HTREE_E_DTYPE;
    return launch_final_normalize(global_out, global_sum, out, dtype, rows, V, (cudaStream_t)stream);
}

int htree_b200_copy_rows(void* dst, int64_t dpitch, const void* src, int64_t spitch, int64_t width, int64_t height,
                         void* stream) {
    if (!dst || !src) return HTREE_E_NULL;
    if (width <= 0 || height <= 0 || dpitch < width || spitch < width) return HTREE_E_SHAPE;
    return (int)cudaMemcpy2DAsync(dst, (size_t)dpitch, src, (size_t)spitch, (size_t)width, (size_t)height, cudaMemcpyDefault,
                                  (cudaStream_t)stream);
}

int htree_b200_backward_plan(const HtreeShape* shape, int64_t budget, int64_t* acc_bytes, int64_t* scratch_bytes) {
    if (!acc_bytes || !scratch_bytes) return HTREE_E_NULL;
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln);
    if (L < 0) return L;
    BwdLayout y;
    const int rc = bwd_layout(shape, L, ln, budget, y);
    if (rc) return rc;
    *acc_bytes = y.acc_bytes; *scratch_bytes = y.scratch_bytes;
    return 0;
}

int htree_b200_run_backward(const HtreeShape* shape, const void* q, void* const* blocks, void* const* blocks_bwd,
                            const float* cos_cache, const float* sin_cache, const void* table, int32_t n_pos, float scale,
                            const void* out, const void* dO, const float* gmax, const float* gsum, int32_t* const* parents,
                            void* acc, void* scratch, int64_t budget, void* dq, void* dk, void* dv, int32_t typed, int32_t* status,
                            uint32_t flags, void* stream) {
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln);
    if (L < 0) return L;
    if (!q || !blocks || !blocks_bwd || !cos_cache || !sin_cache || !table || !out || !dO || !gmax || !gsum || !parents || !acc || !scratch || !dq)
        return HTREE_E_NULL;
    if (!(flags & HTREE_BWD_NO_FOLD) && (!dk || !dv)) return HTREE_E_NULL;
    const bool windowed = shape->T_q != 0 && (shape->T_q != shape->T || shape->t_offset != 0);
    if (windowed && !(flags & (HTREE_BWD_KEEP_ACCUM | HTREE_BWD_NO_FOLD))) return HTREE_E_WINDOW;
    if ((int64_t)n_pos < (int64_t)shape->top_k * shape->compression_rate) return HTREE_E_ROPE;
    if (!aligned32(q) || !aligned32(out) || !aligned32(dO) || !aligned16(table) || !aligned16(acc) || !aligned16(scratch) || !aligned16(dq) ||
        !aligned16(dk) || !aligned16(dv) || !aligned16(cos_cache) || !aligned16(sin_cache))
        return HTREE_E_ALIGN;
    BwdLayout y;
    int rc = bwd_layout(shape, L, ln, budget, y);
    if (rc) return rc;
    BwdParams& bp = y.bp;
    // the levels themselves are not read: the block pointers stand in for them in the common checks
    rc = fill_params(bp.a, shape, L, ln, q, blocks, blocks, cos_cache, sin_cache, n_pos, scale, parents, status, flags);
    if (rc) return rc;
    AttnParams& p = bp.a;
    unsigned char *ab = static_cast<unsigned char*>(acc), *sb = static_cast<unsigned char*>(scratch);
    for (int l = 0; l < L; ++l) {
        if (!parents[l] || !blocks_bwd[l]) return HTREE_E_NULL;
        if (!aligned16(blocks_bwd[l])) return HTREE_E_ALIGN;
        p.blk[l] = blocks[l]; p.vkblk[l] = blocks_bwd[l];
        bp.acck[l] = reinterpret_cast<float*>(ab + y.acck[l]); bp.accv[l] = reinterpret_cast<float*>(ab + y.accv[l]);
    }
    p.tab = table; p.out = const_cast<void*>(out); p.dO = dO; p.gmax = const_cast<float*>(gmax); p.gsum = const_cast<float*>(gsum);
    p.dq = typed ? nullptr : static_cast<float*>(dq); p.dq_typed = typed ? dq : nullptr;
    bp.qb = sb + y.o_qb; bp.dob = sb + y.o_dob; bp.stp = sb + y.o_stp; bp.sts = sb + y.o_sts;
    bp.fac = y.o_fac < 0 ? nullptr : reinterpret_cast<float2*>(sb + y.o_fac);
    bp.rank = reinterpret_cast<int32_t*>(sb + y.o_rank); bp.vis = reinterpret_cast<uint4*>(sb + y.o_rank);
    bp.xtab = y.xtab < 0 ? nullptr : ab + y.xtab;
    bp.nvis = y.o_nvis < 0 ? nullptr : reinterpret_cast<int32_t*>(sb + y.o_nvis); bp.entries = sb + y.o_entries;
    bp.cnt = reinterpret_cast<int32_t*>(sb + y.o_cnt); bp.range = reinterpret_cast<uint32_t*>(bp.cnt + cnt_words(y.per_launch, bp.NK)); bp.base = reinterpret_cast<int2*>(sb + y.o_base);
    bp.items = reinterpret_cast<BwdItem*>(sb + y.o_items); bp.nitems = reinterpret_cast<int32_t*>(sb + y.o_nitems);
    cudaStream_t st = (cudaStream_t)stream;
    for (int s0 = 0; s0 < y.total; s0 += y.per_launch) {
        bp.sub0 = s0; bp.nsub = y.total - s0 < y.per_launch ? y.total - s0 : y.per_launch;
        // the counters, and ahead of the first launch (which has the most windows) the words of the range behind them
        rc = launch_bwd_clear(bp.cnt, cnt_words(bp.nsub, bp.NK) * 4 + (s0 == 0 ? (1 + (int64_t)shape->B * shape->H_kv) * 4 : 0), table,
                              s0 == 0 ? const_cast<unsigned char*>(bp.xtab) : nullptr, shape->top_k * shape->compression_rate, shape->K, st);
        if (rc == 0 && s0 == 0) rc = launch_bwd_begin(bp, shape->dtype, acc, flags & HTREE_BWD_KEEP_ACCUM ? 0 : y.zero_bytes, st);
        if (rc == 0) rc = launch_bwd_dq(bp, shape->dtype, st);
        if (rc == 0) rc = launch_bwd_dkv(bp, shape->dtype, st);
        if (rc) return rc;
    }
    if (flags & HTREE_BWD_NO_FOLD) return 0;
    return launch_bwd_fold(bp, shape->dtype, dk, dv, typed != 0, st);
}

int htree_b200_backward(const HtreeShape* shape, const void* q, void* const* layers_k, void* const* layers_v,
                        void* const* layers_k_rot, const float* cos_cache, const float* sin_cache, const void* cos_half,
                        const void* sin_half, int32_t n_pos, float scale, const void* out,
                        const void* dO, const float* gmax, const float* gsum, int32_t* const* parents, float* dq,
                        float* const* dk_levels, float* const* dv_levels, const HtreeTypedGrads* typed, int32_t* status,
                        uint32_t flags, void* stream) {
    int32_t ln[HTREE_MAX_LEVELS];
    const int L = check_shape(shape, ln);
    if (L < 0) return L;
    if (!out || !dO || !gmax || !gsum || !parents || !dk_levels || !dv_levels) return HTREE_E_NULL;
    if (typed) {
        if (!typed->dq || !typed->dk || !typed->dv) return HTREE_E_NULL;
        if (!aligned16(typed->dq) || !aligned16(typed->dk) || !aligned16(typed->dv)) return HTREE_E_ALIGN;
    } else if (!dq) {
        return HTREE_E_NULL;
    }
    // a query window is one part of a backward that the caller runs window by window over the same accumulators: only
    // meaningful with the flags that say which part it is
    const bool windowed = shape->T_q != 0 && (shape->T_q != shape->T || shape->t_offset != 0);
    if (windowed && !(flags & (HTREE_BWD_KEEP_ACCUM | HTREE_BWD_NO_FOLD))) return HTREE_E_WINDOW;
    AttnParams p;
    int rc = fill_params(p, shape, L, ln, q, layers_k, layers_v, cos_cache, sin_cache, n_pos, scale, parents, status, flags);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    for (int l = 0; l < L; ++l) {
        if (!parents[l] || !dk_levels[l] || !dv_levels[l]) return HTREE_E_NULL;
        if (!aligned16(dk_levels[l]) || !aligned16(dv_levels[l])) return HTREE_E_ALIGN;
        p.dk[l] = dk_levels[l]; p.dv[l] = dv_levels[l];
    }
    p.out = const_cast<void*>(out); p.dO = dO; p.gmax = const_cast<float*>(gmax); p.gsum = const_cast<float*>(gsum);
    p.dq = typed ? nullptr : dq;
    p.dq_typed = typed ? typed->dq : nullptr;
    if (cos_half && sin_half && aligned32(cos_half) && aligned32(sin_half)) {
        p.cosh = static_cast<const __half*>(cos_half); p.sinh = static_cast<const __half*>(sin_half);
    }
    // choose the kernel before anything is queued: a shape that neither kernel takes is refused with nothing launched
    bool fast = layers_k_rot != nullptr && !(flags & HTREE_FWD_GENERIC);
    if (fast) {
        for (int l = 0; l < L; ++l) {
            if (!layers_k_rot[l] || !aligned32(layers_k_rot[l]) || !aligned32(layers_v[l])) fast = false;
            p.lkr[l] = layers_k_rot[l];
        }
        fast = fast && aligned32(q) && aligned32(dO) && aligned32(out) && aligned16(typed ? typed->dq : (void*)dq) &&
               aligned32(cos_cache) && aligned32(sin_cache) && bwd_mma_supported(p, shape->dtype);
    }
    if (!fast && !bwd_generic_supported(p, shape->dtype)) return HTREE_E_UNSUPPORTED;
    for (int l = 0; l < L && !(flags & HTREE_BWD_KEEP_ACCUM); ++l) {   // gradient accumulators start at zero (src/backward.py:979-981)
        const size_t rows = (size_t)shape->B * ln[l] * shape->H_kv;
        cudaError_t e = cudaMemsetAsync(dk_levels[l], 0, rows * shape->K * sizeof(float), st);
        if (e == cudaSuccess) e = cudaMemsetAsync(dv_levels[l], 0, rows * shape->V * sizeof(float), st);
        if (e != cudaSuccess) return (int)e;
    }
    rc = fast ? launch_bwd_mma(p, shape->dtype, st) : launch_bwd_generic(p, shape->dtype, st);
    if (rc || (flags & HTREE_BWD_NO_FOLD)) return rc;
    return launch_tree_backward(*shape, L, ln, dk_levels, dv_levels, st, typed ? typed->dk : nullptr, typed ? typed->dv : nullptr);
}

}  // extern "C"
