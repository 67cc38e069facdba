// The calls a training or inference program makes once per layer, over the C ABI, without the interpreter in between: allocation,
// argument blocks, the stream, and an autograd node whose backward runs on the engine's thread without taking the GIL.  Python
// (ops.py) validates, keeps the rotary tables and falls back to its own path for whatever this file declines (returns None).
// For a training step of a thousand positions the interpreter's share, 200 us a step, was twice the kernels' time.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "../../include/htree_b200.h"

namespace {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

bool aligned(const at::Tensor& t, uintptr_t n) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & (n - 1)) == 0; }

int dtype_code(at::ScalarType t) { return t == at::kFloat ? HTREE_F32 : t == at::kBFloat16 ? HTREE_BF16 : t == at::kHalf ? HTREE_F16 : -1; }

void check(int rc, const char* what) {
    TORCH_CHECK(rc == 0, "htree_b200 ", what, " failed with code ", rc, ": ", htree_b200_error_string(rc));
}

HtreeShape make_shape(const at::Tensor& q, const at::Tensor& k, int64_t cr, int64_t mtn, int64_t tk, int64_t offset) {
    HtreeShape s{};
    s.B = (int32_t)q.size(0); s.T = (int32_t)k.size(1); s.H = (int32_t)q.size(2); s.H_kv = (int32_t)k.size(2);
    s.K = s.V = (int32_t)q.size(3);
    s.compression_rate = (int32_t)cr; s.top_k = (int32_t)tk; s.max_top_nodes = (int32_t)mtn; s.dtype = dtype_code(q.scalar_type());
    if (offset >= 0) { s.T_q = (int32_t)q.size(1); s.t_offset = (int32_t)offset; }
    return s;
}

// One workspace: the plan's, the softmax statistics and the parent lists behind it (an allocation and a saved tensor each cost a
// microsecond or two of a step).
struct Forward {
    at::Tensor out, ws;
    HtreePlan plan;
    int64_t stats, parents;       // where they start
};
int64_t up256(int64_t x) { return (x + 255) & ~int64_t(255); }
void place(Forward& f, const HtreeShape& s, int64_t Tq) {
    f.stats = up256(f.plan.bytes);
    f.parents = f.stats + up256(2 * (int64_t)s.B * Tq * s.H * 4);
}
int64_t lists(const HtreeShape& s, int64_t Tq) { return (int64_t)s.B * Tq * s.H_kv * s.top_k; }       // entries of a level

// tables: cos, sin, rows of the transposed kernels, rows of the selection kernel, status word
bool run_forward(const HtreeShape& s, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const std::vector<at::Tensor>& tables,
                 double scale, bool save, int64_t budget, Forward& f) {
    if (htree_b200_plan(&s, save ? HTREE_PLAN_BACKWARD : 0u, &f.plan) != 0) return false;
    const int64_t B = s.B, Tq = q.size(1), H = s.H, L = f.plan.levels;
    if (!save && L * B * Tq * s.H_kv * s.top_k * 4 > budget) return false;
    const auto bytes = at::TensorOptions().device(q.device()).dtype(at::kByte);
    f.out = at::empty(q.sizes(), q.options());
    place(f, s, Tq);
    f.ws = at::empty({f.parents + L * lists(s, Tq) * 4}, bytes);
    unsigned char* w = static_cast<unsigned char*>(f.ws.data_ptr());
    int32_t* par[HTREE_MAX_LEVELS];
    for (int64_t l = 0; l < L; ++l) par[l] = reinterpret_cast<int32_t*>(w + f.parents) + l * lists(s, Tq);
    float* gmax = reinterpret_cast<float*>(w + f.stats);
    check(htree_b200_run_forward(&s, &f.plan, q.data_ptr(), k.data_ptr(), v.data_ptr(), tables[0].data_ptr<float>(), tables[1].data_ptr<float>(),
                                 tables[2].data_ptr(), tables[3].data_ptr(), (int32_t)tables[0].size(0), (float)scale, f.ws.data_ptr(),
                                 f.out.data_ptr(), gmax, gmax + B * Tq * H, par, tables[4].data_ptr<int32_t>(), save ? 0u : HTREE_FWD_INFERENCE,
                                 at::cuda::getCurrentCUDAStream().stream()),
          "forward");
    return true;
}

struct HTreeNode : public torch::autograd::Function<HTreeNode> {
    static at::Tensor forward(AutogradContext* ctx, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                              const std::vector<at::Tensor>& tables, int64_t cr, int64_t mtn, int64_t tk, double scale, int64_t budget) {
        c10::cuda::CUDAGuard guard(q.device());
        const HtreeShape s = make_shape(q, k, cr, mtn, tk, -1);
        Forward f;
        TORCH_CHECK(run_forward(s, q, k, v, tables, scale, true, 0, f), "htree_b200: unsupported shape");
        ctx->save_for_backward({q, k, v, f.out, f.ws, tables[0], tables[1], tables[2], tables[4]});
        ctx->saved_data["cr"] = cr; ctx->saved_data["mtn"] = mtn; ctx->saved_data["tk"] = tk;
        ctx->saved_data["scale"] = scale; ctx->saved_data["budget"] = budget;
        return f.out;
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto sv = ctx->get_saved_variables();
        const at::Tensor &q = sv[0], &k = sv[1], &out = sv[3], &ws = sv[4];
        c10::cuda::CUDAGuard guard(q.device());
        at::Tensor dO = grads[0].to(q.scalar_type()).contiguous();
        if (!aligned(dO, 32)) dO = dO.clone();
        const double scale = ctx->saved_data["scale"].toDouble();
        const int64_t budget = ctx->saved_data["budget"].toInt();
        const HtreeShape s = make_shape(q, k, ctx->saved_data["cr"].toInt(), ctx->saved_data["mtn"].toInt(), ctx->saved_data["tk"].toInt(), -1);
        Forward f;
        HtreePlan& plan = f.plan;
        int64_t acc_bytes = 0, scratch_bytes = 0;
        check(htree_b200_plan(&s, HTREE_PLAN_BACKWARD, &plan), "plan");
        check(htree_b200_backward_plan(&s, budget, &acc_bytes, &scratch_bytes), "backward plan");
        acc_bytes = (acc_bytes + 255) / 256 * 256;
        const at::Tensor scratch = at::empty({acc_bytes + scratch_bytes}, ws.options());
        at::Tensor dq = at::empty(q.sizes(), q.options()), dk = at::empty(k.sizes(), k.options()), dv = at::empty(k.sizes(), k.options());
        void *blk[HTREE_MAX_LEVELS], *bwd[HTREE_MAX_LEVELS];
        int32_t* par[HTREE_MAX_LEVELS];
        unsigned char *w = static_cast<unsigned char*>(ws.data_ptr()), *a = static_cast<unsigned char*>(scratch.data_ptr());
        place(f, s, q.size(1));
        for (int l = 0; l < plan.levels; ++l) {
            blk[l] = w + plan.blocks[l]; bwd[l] = w + plan.blocks_bwd[l];
            par[l] = reinterpret_cast<int32_t*>(w + f.parents) + l * lists(s, q.size(1));
        }
        const float* gmax = reinterpret_cast<const float*>(w + f.stats);
        check(htree_b200_run_backward(&s, q.data_ptr(), blk, bwd, sv[5].data_ptr<float>(), sv[6].data_ptr<float>(), sv[7].data_ptr(),
                                      (int32_t)sv[5].size(0), (float)scale, out.data_ptr(), dO.data_ptr(), gmax, gmax + (int64_t)s.B * q.size(1) * s.H, par, a,
                                      a + acc_bytes, budget, dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), 1, sv[8].data_ptr<int32_t>(), 0u,
                                      at::cuda::getCurrentCUDAStream().stream()),
              "backward");
        variable_list r(13);        // q, k, v, then tables and options, which have no gradient
        r[0] = dq; r[1] = dk; r[2] = dv;
        return r;
    }
};

bool takes(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v) {
    return q.is_contiguous() && k.is_contiguous() && v.is_contiguous() && aligned(q, 32) && aligned(k, 16) && aligned(v, 16);
}

// The differentiable forward; None where the Python path has to take the call.
c10::optional<at::Tensor> autograd_forward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const std::vector<at::Tensor>& tables,
                                           int64_t cr, int64_t mtn, int64_t tk, double scale, int64_t budget) {
    if (!takes(q, k, v)) return c10::nullopt;
    const HtreeShape s = make_shape(q, k, cr, mtn, tk, -1);
    HtreePlan plan;
    int64_t a = 0, b = 0;
    if (htree_b200_plan(&s, HTREE_PLAN_BACKWARD, &plan) != 0 || htree_b200_backward_plan(&s, budget, &a, &b) != 0) return c10::nullopt;
    return HTreeNode::apply(q, k, v, tables, cr, mtn, tk, scale, budget);
}

// The forward alone (no selections kept); offset >= 0: q is a window of query positions.
c10::optional<at::Tensor> plain_forward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const std::vector<at::Tensor>& tables,
                                        int64_t cr, int64_t mtn, int64_t tk, double scale, int64_t offset, int64_t budget) {
    if (!takes(q, k, v)) return c10::nullopt;
    c10::cuda::CUDAGuard guard(q.device());
    Forward f;
    if (!run_forward(make_shape(q, k, cr, mtn, tk, offset), q, k, v, tables, scale, false, budget, f)) return c10::nullopt;
    return f.out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("autograd_forward", &autograd_forward, py::call_guard<py::gil_scoped_release>());
    m.def("plain_forward", &plain_forward, py::call_guard<py::gil_scoped_release>());
}
