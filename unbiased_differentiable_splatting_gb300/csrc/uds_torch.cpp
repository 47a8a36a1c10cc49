// The CUDA kernels of torch.ops.uds and their autograd formulas in native
// code.  library.py defines every op (schema, fake implementation, the
// implementation for every device and the autograd formula in Python); this
// library registers the same for CUDA tensors only, so an eager call on the
// GPU runs no Python below the op: on a Grace host a forward + backward of
// the renderer at 128 x 128 spent 2.1 ms in Python for 0.4 ms of kernels.
// CPU, meta and fake tensors keep the Python definitions, and so do traces
// (the autograd formulas here call the ops, which a tracer sees).
//
// Inputs are checked as the Python wrappers check them, with the same
// exception types.  Scratch memory comes from torch's caching allocator per
// call, so it follows the current stream.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/autograd_not_implemented_fallback.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include "../../include/uds.h"

namespace {

using at::Tensor;
using c10::SymInt;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// ------------------------------------------------------------------ checks
const Tensor& need(const Tensor& t, const char* name, const Tensor* like = nullptr, at::ScalarType type = at::kFloat) {
    TORCH_CHECK_VALUE(t.is_cuda(), name, " must be a CUDA tensor");
    if (like)
        TORCH_CHECK_VALUE(t.device() == like->device(), name, " is on ", t.device(), ", expected ", like->device());
    TORCH_CHECK_TYPE(t.scalar_type() == type, name, " must be ", type == at::kInt ? "torch.int32" : "torch.float32",
                     ", got ", t.scalar_type());
    TORCH_CHECK_VALUE(t.is_contiguous(), name, " must be contiguous");
    return t;
}

// The kernels index an array by the sizes of the others.
void need_numel(const Tensor& t, int64_t count, const char* name) {
    TORCH_CHECK_VALUE(t.numel() == count, name, " must have ", count, " elements, got shape ", t.sizes());
}

// The UdsError of _lib.py, raised for a failing status of the C ABI.
void check(int status, const char* what) {
    if (status == UDS_OK) return;
    std::string msg = std::string(what) + ": " + uds_status_string(status);
    if (status == UDS_ERR_CUDA || status == UDS_ERR_LAUNCH) msg += std::string(" (") + uds_last_error() + ")";
    PyGILState_STATE gil = PyGILState_Ensure();
    PyObject* mod = PyImport_ImportModule("unbiased_differentiable_splatting_gb300._lib");
    PyObject* type = mod ? PyObject_GetAttrString(mod, "UdsError") : nullptr;
    if (type) PyErr_SetString(type, msg.c_str());
    Py_XDECREF(type);
    Py_XDECREF(mod);
    python_error err;
    err.persist();
    PyGILState_Release(gil);
    throw err;
}

int i32(int64_t x) { return static_cast<int>(x); }
const float* f(const Tensor& t) { return t.const_data_ptr<float>(); }
float* fm(const Tensor& t) { return t.mutable_data_ptr<float>(); }
const float* fo(const OptTensor& t) { return t.has_value() && t->defined() ? t->const_data_ptr<float>() : nullptr; }
const int* idx(const Tensor& t) { return t.const_data_ptr<int>(); }

// Current stream on the tensor's device, which becomes the current device.
struct On {
    explicit On(const Tensor& t) : guard(t.device()) {}
    void* stream() const { return c10::cuda::getCurrentCUDAStream(guard.current_device().index()).stream(); }
    c10::cuda::CUDAGuard guard;
};
Tensor scratch(size_t bytes, const Tensor& like) {
    return at::empty({static_cast<int64_t>(bytes > 256 ? bytes : 256)}, like.options().dtype(at::kByte));
}

template <class Sig>
auto op(const char* name) {
    return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Sig>();
}
bool any_grad(std::initializer_list<const Tensor*> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : ts)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}

// --------------------------------------------------------------- transform
template <bool AFFINE>
struct Transform {
    static constexpr const char* fwd = AFFINE ? "uds::affine_forward" : "uds::linear_forward";
    static constexpr const char* bwd = AFFINE ? "uds::affine_backward" : "uds::linear_backward";
    using Fwd = Tensor(const Tensor&, const Tensor&);
    using Bwd = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&);

    static Tensor forward_cuda(const Tensor& M, const Tensor& v) {
        need(M, "transformation");
        need(v, "vector", &M);
        TORCH_CHECK_VALUE(M.dim() == 3 && M.size(1) == 4 && M.size(2) == 4 && v.dim() == 3 && v.size(2) == 3,
                          "expected transformation (B,4,4) and vector (1|B,N,3)");
        On on(v);
        Tensor out = at::empty({M.size(0), v.size(1), 3}, v.options());
        check(uds_transform_forward(AFFINE, i32(M.size(0)), f(M), i32(v.size(0)), i32(v.size(1)), f(v), fm(out),
                                    on.stream()),
              "transform forward");
        return out;
    }
    static std::tuple<Tensor, Tensor> backward_cuda(const Tensor& g, const Tensor& M, const Tensor& v) {
        need(g, "gradIn");
        need(M, "transformation", &g);
        need(v, "vector", &g);
        TORCH_CHECK_VALUE(M.dim() == 3 && M.size(1) == 4 && M.size(2) == 4 && v.dim() == 3 && v.size(2) == 3,
                          "expected transformation (B,4,4) and vector (1|B,N,3)");
        TORCH_CHECK_VALUE(g.dim() == 3 && g.size(0) == M.size(0) && g.size(1) == v.size(1) && g.size(2) == 3,
                          "gradIn must have shape (B,N,3)");
        On on(v);
        Tensor gM = at::empty_like(M), gv = at::empty_like(v);
        check(uds_transform_backward(AFFINE, i32(M.size(0)), f(g), f(M), i32(v.size(0)), i32(v.size(1)), f(v), fm(gM),
                                     fm(gv), on.stream()),
              "transform backward");
        return {gM, gv};
    }
    struct Fn : Function<Fn> {
        static Tensor forward(AutogradContext* ctx, const Tensor& M, const Tensor& v) {
            at::AutoDispatchBelowADInplaceOrView below;
            ctx->save_for_backward({M, v});
            static auto call = op<Fwd>(fwd);
            return call.call(M, v);
        }
        static variable_list backward(AutogradContext* ctx, variable_list g) {
            auto s = ctx->get_saved_variables();
            static auto call = op<Bwd>(bwd);
            auto [gM, gv] = call.call(g[0].contiguous(), s[0], s[1]);
            return {gM, gv};
        }
    };
    static Tensor autograd(const Tensor& M, const Tensor& v) {
        if (any_grad({&M, &v})) return Fn::apply(M, v);
        at::AutoDispatchBelowADInplaceOrView below;
        static auto call = op<Fwd>(fwd);
        return call.call(M, v);
    }
};

// ------------------------------------------------------------- view matrix
using ViewFwd = Tensor(const Tensor&, const Tensor&);
using ViewBwd = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&);
Tensor view_forward_cuda(const Tensor& pos, const Tensor& quat) {
    need(pos, "positions");
    need(quat, "quaternions", &pos);
    need_numel(pos, 3 * quat.size(0), "positions");
    need_numel(quat, 4 * quat.size(0), "quaternions");
    On on(pos);
    Tensor out = at::empty({quat.size(0), 1, 4, 4}, pos.options());
    check(uds_view_matrix_forward(i32(quat.size(0)), f(pos), f(quat), fm(out), on.stream()), "view matrix forward");
    return out;
}
std::tuple<Tensor, Tensor> view_backward_cuda(const Tensor& g, const Tensor& quat) {
    need(g, "gradIn");
    need(quat, "quaternions", &g);
    need_numel(g, 16 * quat.size(0), "gradIn");
    need_numel(quat, 4 * quat.size(0), "quaternions");
    On on(g);
    Tensor gp = at::empty({quat.size(0), 3}, g.options()), gq = at::empty_like(quat);
    check(uds_view_matrix_backward(i32(quat.size(0)), f(g), f(quat), fm(gp), fm(gq), on.stream()),
          "view matrix backward");
    return {gp, gq};
}
struct ViewFn : Function<ViewFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& pos, const Tensor& quat) {
        at::AutoDispatchBelowADInplaceOrView below;
        ctx->save_for_backward({quat});
        static auto call = op<ViewFwd>("uds::view_matrix_forward");
        return call.call(pos, quat);
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        static auto call = op<ViewBwd>("uds::view_matrix_backward");
        auto [gp, gq] = call.call(g[0].contiguous(), ctx->get_saved_variables()[0]);
        return {gp, gq};
    }
};
Tensor view_autograd(const Tensor& pos, const Tensor& quat) {
    if (any_grad({&pos, &quat})) return ViewFn::apply(pos, quat);
    at::AutoDispatchBelowADInplaceOrView below;
    static auto call = op<ViewFwd>("uds::view_matrix_forward");
    return call.call(pos, quat);
}

// ---------------------------------------------------------------- backface
using FaceFwd = std::vector<Tensor>(const Tensor&, const OptTensor&);
using FaceBwd = std::vector<Tensor>(const Tensor&, const Tensor&, const OptTensor&, SymInt);
std::vector<Tensor> backface_cuda(const Tensor& cam, const OptTensor& nrm) {
    need(cam, "camNormals");
    TORCH_CHECK_VALUE(cam.dim() == 3 && cam.size(2) == 3, "camNormals must be (B,N,3)");
    const bool world = nrm.has_value() && nrm->defined();
    On on(cam);
    std::vector<Tensor> out{at::empty_like(cam)};
    if (world) {
        need(*nrm, "normals", &cam);
        TORCH_CHECK_VALUE(nrm->dim() == 3 && nrm->size(1) == cam.size(1) && nrm->size(2) == 3 &&
                              (nrm->size(0) == 1 || nrm->size(0) == cam.size(0)),
                          "normals must be (1|B,N,3)");
        out.push_back(at::empty_like(cam));
    }
    check(uds_backface_forward(i32(cam.size(0)), i32(cam.size(1)), f(cam), world ? i32(nrm->size(0)) : 1, fo(nrm),
                               fm(out[0]), world ? fm(out[1]) : nullptr, on.stream()),
          "backface forward");
    return out;
}
std::vector<Tensor> backface_backward_cuda(const Tensor& cam, const Tensor& gcam, const OptTensor& gnrm,
                                           int64_t batch) {
    need(cam, "camNormals");
    TORCH_CHECK_VALUE(cam.dim() == 3 && cam.size(2) == 3, "camNormals must be (B,N,3)");
    need(gcam, "gradCam", &cam);
    need_numel(gcam, cam.numel(), "gradCam");
    On on(cam);
    std::vector<Tensor> out{at::empty_like(cam)};
    const bool world = gnrm.has_value() && gnrm->defined();
    if (world) {
        need(*gnrm, "gradNormals", &cam);
        need_numel(*gnrm, cam.numel(), "gradNormals");
        out.push_back(at::empty({batch, cam.size(1), 3}, cam.options()));
    }
    check(uds_backface_backward(i32(cam.size(0)), i32(cam.size(1)), f(cam), f(gcam), i32(batch), fo(gnrm), fm(out[0]),
                                world ? fm(out[1]) : nullptr, on.stream()),
          "backface backward");
    return out;
}
struct FaceFn : Function<FaceFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& cam, const OptTensor& nrm) {
        at::AutoDispatchBelowADInplaceOrView below;
        ctx->set_materialize_grads(false);
        ctx->save_for_backward({cam});
        const bool world = nrm.has_value() && nrm->defined();
        ctx->saved_data["world"] = world;
        ctx->saved_data["batch"] = world ? nrm->sym_size(0) : SymInt(1);
        static auto call = op<FaceFwd>("uds::backface");
        return call.call(cam, nrm);
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        Tensor cam = ctx->get_saved_variables()[0];
        const bool world = ctx->saved_data["world"].toBool();
        Tensor gcam = g[0].defined() ? g[0].contiguous() : at::zeros_like(cam);
        OptTensor gnrm;
        if (world && g.size() > 1 && g[1].defined()) gnrm = g[1].contiguous();
        static auto call = op<FaceBwd>("uds::backface_backward");
        auto out = call.call(cam, gcam, gnrm, ctx->saved_data["batch"].toSymInt());
        return {out[0], gnrm.has_value() ? out[1] : Tensor()};
    }
};
std::vector<Tensor> backface_autograd(const Tensor& cam, const OptTensor& nrm) {
    if (any_grad({&cam}) || (nrm.has_value() && any_grad({&*nrm}))) return FaceFn::apply(cam, nrm);
    at::AutoDispatchBelowADInplaceOrView below;
    static auto call = op<FaceFwd>("uds::backface");
    return call.call(cam, nrm);
}

// ------------------------------------------------------- EWA, fused render
using SplatFwd = Tensor(SymInt, SymInt, double, const Tensor&, const Tensor&, const Tensor&, const Tensor&, double);
using SplatBwd = std::tuple<Tensor, Tensor, Tensor>(SymInt, SymInt, double, const Tensor&, const Tensor&, const Tensor&,
                                                    const Tensor&, const Tensor&, double);
using RenderFwd = std::tuple<Tensor, Tensor, Tensor>(SymInt, SymInt, double, const Tensor&, const Tensor&,
                                                     const Tensor&, const Tensor&, double, const Tensor&);
using RenderBwd = std::vector<Tensor>(SymInt, SymInt, double, const Tensor&, const OptTensor&, const OptTensor&,
                                      const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, double,
                                      const Tensor&);
using SplatGrads = std::tuple<Tensor, Tensor>(SymInt, SymInt, double, const Tensor&, const Tensor&, const Tensor&,
                                              const Tensor&, const Tensor&, double);
using RenderGrads = std::tuple<Tensor, Tensor, Tensor>(SymInt, SymInt, double, const Tensor&, const OptTensor&,
                                                       const OptTensor&, const Tensor&, const Tensor&, const Tensor&,
                                                       const Tensor&, const Tensor&, double, const Tensor&);

void check_splats(const Tensor& ids, const Tensor& pts, const Tensor& nrm, const Tensor& sd) {
    need(ids, "indices", nullptr, at::kInt);
    need(pts, "points", &ids);
    need(nrm, "normals", &ids);
    need(sd, "stdDevs", &ids);
    TORCH_CHECK_VALUE(ids.dim() == 4 && pts.dim() == 3 && pts.sizes() == nrm.sizes() && sd.dim() == 3,
                      "expected indices (B,W,H,K), points/normals (B,N,3), stdDevs (1|B,N,2)");
    TORCH_CHECK_VALUE(ids.size(0) == pts.size(0) && sd.size(1) == pts.size(1) &&
                          (sd.size(0) == 1 || sd.size(0) == pts.size(0)),
                      "batch / splat counts of indices, points and stdDevs disagree");
    TORCH_CHECK_VALUE(pts.size(2) == 3 && sd.size(2) == 2, "expected points/normals (B,N,3) and stdDevs (1|B,N,2)");
}
Tensor splat_forward_cuda(int64_t width, int64_t height, double focal, const Tensor& ids, const Tensor& pts,
                          const Tensor& nrm, const Tensor& sd, double smoothing) {
    check_splats(ids, pts, nrm, sd);
    TORCH_CHECK_VALUE(ids.size(1) == width && ids.size(2) == height, "indices shape does not match width/height");
    const int B = i32(ids.size(0)), N = i32(pts.size(1));
    On on(pts);
    Tensor ws = scratch(uds_splat_workspace_size(B, N), pts);
    Tensor w = at::empty(ids.sizes(), pts.options());
    check(uds_splat_forward(B, i32(width), i32(height), i32(ids.size(3)), (float)focal, idx(ids), f(pts), f(nrm),
                            i32(sd.size(0)), N, f(sd), (float)smoothing, fm(w), ws.mutable_data_ptr(),
                            (size_t)ws.numel(), on.stream()),
          "splatting forward");
    return w;
}
std::tuple<Tensor, Tensor, Tensor> splat_backward_cuda(int64_t, int64_t, double focal, const Tensor& g,
                                                       const Tensor& ids, const Tensor& pts, const Tensor& nrm,
                                                       const Tensor& sd, double smoothing) {
    check_splats(ids, pts, nrm, sd);
    need(g, "gradIn", &pts);
    TORCH_CHECK_VALUE(g.sizes() == ids.sizes(), "gradIn must match indices");
    const int B = i32(ids.size(0)), N = i32(pts.size(1));
    On on(pts);
    Tensor ws = scratch(uds_splat_workspace_size(B, N), pts);
    Tensor gp = at::empty_like(pts), gn = at::empty_like(nrm), gs = at::empty_like(sd);
    check(uds_splat_backward(B, i32(ids.size(1)), i32(ids.size(2)), i32(ids.size(3)), (float)focal, f(g), idx(ids),
                             f(pts), f(nrm), i32(sd.size(0)), N, f(sd), (float)smoothing, fm(gp), fm(gn), fm(gs),
                             ws.mutable_data_ptr(), (size_t)ws.numel(), on.stream()),
          "splatting backward");
    return {gp, gn, gs};
}
std::tuple<Tensor, Tensor> splat_gradients_cuda(int64_t, int64_t, double focal, const Tensor& g, const Tensor& ids,
                                                const Tensor& pts, const Tensor& nrm, const Tensor& sd,
                                                double smoothing) {
    check_splats(ids, pts, nrm, sd);
    need(g, "gradIn", &pts);
    TORCH_CHECK_VALUE(g.sizes() == ids.sizes(), "gradIn must match indices");
    const int B = i32(ids.size(0)), N = i32(pts.size(1));
    On on(pts);
    Tensor ws = scratch(uds_splat_workspace_size(B, N), pts);
    Tensor gp = at::empty_like(pts), gs = at::empty_like(sd);
    check(uds_splat_gradients(B, i32(ids.size(1)), i32(ids.size(2)), i32(ids.size(3)), (float)focal, f(g), idx(ids),
                              f(pts), f(nrm), i32(sd.size(0)), N, f(sd), (float)smoothing, fm(gp), fm(gs),
                              ws.mutable_data_ptr(), (size_t)ws.numel(), on.stream()),
          "splatting backward");
    return {gp, gs};
}
std::tuple<Tensor, Tensor, Tensor> render_forward_cuda(int64_t width, int64_t height, double focal, const Tensor& ids,
                                                       const Tensor& pts, const Tensor& nrm, const Tensor& sd,
                                                       double smoothing, const Tensor& attr) {
    check_splats(ids, pts, nrm, sd);
    need(attr, "attribute", &pts);
    TORCH_CHECK_VALUE(ids.size(1) == width && ids.size(2) == height, "indices shape does not match width/height");
    const int B = i32(ids.size(0)), N = i32(pts.size(1));
    TORCH_CHECK_VALUE(attr.dim() == 3 && attr.size(1) == N && (attr.size(0) == 1 || attr.size(0) == B),
                      "attribute must be (1|B,N,C)");
    On on(pts);
    Tensor ws = scratch(uds_splat_workspace_size(B, N), pts);
    Tensor w = at::empty(ids.sizes(), pts.options()), depth = at::empty(ids.sizes(), pts.options());
    Tensor img = at::empty({B, width, height, attr.size(2)}, pts.options());
    check(uds_render_fused_forward(B, i32(width), i32(height), i32(ids.size(3)), (float)focal, idx(ids), f(pts), f(nrm),
                                   i32(sd.size(0)), N, f(sd), (float)smoothing, i32(attr.size(0)), i32(attr.size(2)),
                                   f(attr), fm(w), fm(depth), fm(img), ws.mutable_data_ptr(), (size_t)ws.numel(),
                                   on.stream()),
          "render forward");
    return {img, depth, w};
}
// CLAMP: render_splats_gradients ({points, std-devs, attribute} with the
// reference's post-processing), else the raw gradients.
template <bool CLAMP>
std::vector<Tensor> render_gradients(double focal, const Tensor& gimg, const OptTensor& gdepth, const OptTensor& gw,
                                     const Tensor& ids, const Tensor& w, const Tensor& pts, const Tensor& nrm,
                                     const Tensor& sd, double smoothing, const Tensor& attr) {
    check_splats(ids, pts, nrm, sd);
    need(gimg, "gradImage", &pts);
    need(w, "weights", &pts);
    need(attr, "attribute", &pts);
    const std::pair<const char*, const OptTensor*> more[] = {{"gradDepthWeights", &gdepth}, {"gradWeights", &gw}};
    for (auto& [name, g] : more)
        if (g->has_value() && (*g)->defined()) {
            need(**g, name, &pts);
            TORCH_CHECK_VALUE((*g)->sizes() == ids.sizes(), name, " must match indices");
        }
    const int B = i32(ids.size(0)), N = i32(pts.size(1));
    TORCH_CHECK_VALUE(attr.dim() == 3 && attr.size(1) == N && (attr.size(0) == 1 || attr.size(0) == B),
                      "attribute must be (1|B,N,C)");
    const int C = i32(attr.size(2));
    TORCH_CHECK_VALUE(gimg.dim() == 4 && gimg.size(0) == B && gimg.size(1) == ids.size(1) &&
                          gimg.size(2) == ids.size(2) && gimg.size(3) == C && w.sizes() == ids.sizes(),
                      "gradImage must be (B,W,H,C) and weights (B,W,H,K)");
    On on(pts);
    Tensor ws = scratch(uds_splat_workspace_size(B, N), pts);
    Tensor gp = at::empty_like(pts), gs = at::empty_like(sd), ga = at::empty_like(attr);
    if constexpr (CLAMP) {
        check(uds_render_fused_gradients(B, i32(ids.size(1)), i32(ids.size(2)), i32(ids.size(3)), (float)focal, f(gimg),
                                         fo(gdepth), fo(gw), idx(ids), f(w), f(pts), f(nrm), i32(sd.size(0)), N, f(sd),
                                         (float)smoothing, i32(attr.size(0)), C, f(attr), fm(gp), fm(gs), fm(ga),
                                         ws.mutable_data_ptr(), (size_t)ws.numel(), on.stream()),
              "render backward");
        return {gp, gs, ga};
    } else {
        Tensor gn = at::empty_like(nrm);
        check(uds_render_fused_backward(B, i32(ids.size(1)), i32(ids.size(2)), i32(ids.size(3)), (float)focal, f(gimg),
                                        fo(gdepth), fo(gw), idx(ids), f(w), f(pts), f(nrm), i32(sd.size(0)), N, f(sd),
                                        (float)smoothing, i32(attr.size(0)), C, f(attr), fm(gp), fm(gn), fm(gs), fm(ga),
                                        ws.mutable_data_ptr(), (size_t)ws.numel(), on.stream()),
              "render backward");
        return {gp, gn, gs, ga};
    }
}
std::vector<Tensor> render_backward_cuda(int64_t, int64_t, double focal, const Tensor& gimg, const OptTensor& gdepth,
                                         const OptTensor& gw, const Tensor& ids, const Tensor& w, const Tensor& pts,
                                         const Tensor& nrm, const Tensor& sd, double smoothing, const Tensor& attr) {
    return render_gradients<false>(focal, gimg, gdepth, gw, ids, w, pts, nrm, sd, smoothing, attr);
}
std::tuple<Tensor, Tensor, Tensor> render_gradients_cuda(int64_t, int64_t, double focal, const Tensor& gimg,
                                                         const OptTensor& gdepth, const OptTensor& gw,
                                                         const Tensor& ids, const Tensor& w, const Tensor& pts,
                                                         const Tensor& nrm, const Tensor& sd, double smoothing,
                                                         const Tensor& attr) {
    auto r = render_gradients<true>(focal, gimg, gdepth, gw, ids, w, pts, nrm, sd, smoothing, attr);
    return {r[0], r[1], r[2]};
}

void save_view(AutogradContext* ctx, const SymInt& width, const SymInt& height, double focal, double smoothing) {
    ctx->saved_data["width"] = width;
    ctx->saved_data["height"] = height;
    ctx->saved_data["focal"] = focal;
    ctx->saved_data["smoothing"] = smoothing;
}

// RAW: splat_forward (the kernels' raw gradients); else ewa_weights
template <bool RAW>
struct SplatFn : Function<SplatFn<RAW>> {
    static constexpr const char* name = RAW ? "uds::splat_forward" : "uds::ewa_weights";
    static Tensor forward(AutogradContext* ctx, SymInt width, SymInt height, double focal, const Tensor& ids,
                          const Tensor& pts, const Tensor& nrm, const Tensor& sd, double smoothing) {
        at::AutoDispatchBelowADInplaceOrView below;
        ctx->save_for_backward({ids, pts, nrm, sd});
        save_view(ctx, width, height, focal, smoothing);
        static auto call = op<SplatFwd>(name);
        return call.call(width, height, focal, ids, pts, nrm, sd, smoothing);
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        auto s = ctx->get_saved_variables();
        auto& d = ctx->saved_data;
        if constexpr (RAW) {
            static auto call = op<SplatBwd>("uds::splat_backward");
            auto [gp, gn, gs] = call.call(d["width"].toSymInt(), d["height"].toSymInt(), d["focal"].toDouble(),
                                          g[0].contiguous(), s[0], s[1], s[2], s[3], d["smoothing"].toDouble());
            return {Tensor(), Tensor(), Tensor(), Tensor(), gp, gn, gs, Tensor()};
        } else {
            static auto call = op<SplatGrads>("uds::splat_gradients");
            auto [gp, gs] = call.call(d["width"].toSymInt(), d["height"].toSymInt(), d["focal"].toDouble(),
                                      g[0].contiguous(), s[0], s[1], s[2], s[3], d["smoothing"].toDouble());
            return {Tensor(), Tensor(), Tensor(), Tensor(), gp, Tensor(), gs, Tensor()};
        }
    }
    static Tensor autograd(SymInt width, SymInt height, double focal, const Tensor& ids, const Tensor& pts,
                           const Tensor& nrm, const Tensor& sd, double smoothing) {
        if (any_grad({&pts, &nrm, &sd}))
            return SplatFn::apply(width, height, focal, ids, pts, nrm, sd, smoothing);
        at::AutoDispatchBelowADInplaceOrView below;
        static auto call = op<SplatFwd>(name);
        return call.call(width, height, focal, ids, pts, nrm, sd, smoothing);
    }
};

struct RenderFn : Function<RenderFn> {
    static variable_list forward(AutogradContext* ctx, SymInt width, SymInt height, double focal, const Tensor& ids,
                                 const Tensor& pts, const Tensor& nrm, const Tensor& sd, double smoothing,
                                 const Tensor& attr) {
        at::AutoDispatchBelowADInplaceOrView below;
        static auto call = op<RenderFwd>("uds::render_splats");
        auto [img, depth, w] = call.call(width, height, focal, ids, pts, nrm, sd, smoothing, attr);
        ctx->set_materialize_grads(false);
        ctx->save_for_backward({ids, pts, nrm, sd, attr, w});
        save_view(ctx, width, height, focal, smoothing);
        return {img, depth, w};
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        auto s = ctx->get_saved_variables();
        auto& d = ctx->saved_data;
        auto opt = [](const Tensor& t) { return t.defined() ? OptTensor(t.contiguous()) : OptTensor(); };
        Tensor gimg = g[0].defined() ? g[0].contiguous()
                                     : at::zeros_symint({s[0].sym_size(0), s[0].sym_size(1), s[0].sym_size(2),
                                                         s[4].sym_size(2)}, s[5].options());
        static auto call = op<RenderGrads>("uds::render_splats_gradients");
        auto [gp, gs, ga] = call.call(d["width"].toSymInt(), d["height"].toSymInt(), d["focal"].toDouble(), gimg,
                                      opt(g[1]), opt(g[2]), s[0], s[5], s[1], s[2], s[3], d["smoothing"].toDouble(),
                                      s[4]);
        return {Tensor(), Tensor(), Tensor(), Tensor(), gp, Tensor(), gs, Tensor(), ga};
    }
};
std::tuple<Tensor, Tensor, Tensor> render_autograd(SymInt width, SymInt height, double focal, const Tensor& ids,
                                                   const Tensor& pts, const Tensor& nrm, const Tensor& sd,
                                                   double smoothing, const Tensor& attr) {
    if (any_grad({&pts, &nrm, &sd, &attr})) {
        auto r = RenderFn::apply(width, height, focal, ids, pts, nrm, sd, smoothing, attr);
        return {r[0], r[1], r[2]};
    }
    at::AutoDispatchBelowADInplaceOrView below;
    static auto call = op<RenderFwd>("uds::render_splats");
    return call.call(width, height, focal, ids, pts, nrm, sd, smoothing, attr);
}

// ------------------------------------------------------------- compositing
using FilterFwd = Tensor(const Tensor&, const Tensor&, SymInt, SymInt, double, const Tensor&, const Tensor&);
using FilterBwd = Tensor(const Tensor&, const Tensor&, const Tensor&, SymInt, SymInt, double, const Tensor&,
                         const Tensor&);
void check_filter(const Tensor& ids, const Tensor& w, const Tensor& pts, const Tensor& nrm) {
    need(ids, "indices", nullptr, at::kInt);
    need(w, "weights", &ids);
    need(pts, "points", &ids);
    need(nrm, "normals", &ids);
    TORCH_CHECK_VALUE(ids.sizes() == w.sizes() && ids.dim() == 4, "indices and weights must both be (B,W,H,K)");
    TORCH_CHECK_VALUE(pts.sizes() == nrm.sizes() && (pts.size(0) == 1 || pts.size(0) == ids.size(0)),
                      "points/normals must be (1|B,N,3)");
    need_numel(pts, 3 * pts.size(0) * pts.size(1), "points");
}
Tensor filter_forward_cuda(const Tensor& ids, const Tensor& w, int64_t, int64_t, double focal, const Tensor& pts,
                           const Tensor& nrm) {
    check_filter(ids, w, pts, nrm);
    On on(pts);
    Tensor out = at::empty_like(w);
    check(uds_filter_forward(i32(ids.size(0)), i32(ids.size(1)), i32(ids.size(2)), i32(ids.size(3)), idx(ids), f(w),
                             (float)focal, i32(pts.size(0)), i32(pts.size(1)), f(pts), f(nrm), fm(out), on.stream()),
          "filtering forward");
    return out;
}
Tensor filter_backward_cuda(const Tensor& ids, const Tensor& w, const Tensor& g, int64_t, int64_t, double focal,
                            const Tensor& pts, const Tensor& nrm) {
    check_filter(ids, w, pts, nrm);
    need(g, "gradIn", &ids);
    need_numel(g, ids.numel(), "gradIn");
    On on(pts);
    Tensor out = at::empty_like(w);
    check(uds_filter_backward(i32(ids.size(0)), i32(ids.size(1)), i32(ids.size(2)), i32(ids.size(3)), idx(ids), f(w),
                              f(g), (float)focal, i32(pts.size(0)), i32(pts.size(1)), f(pts), f(nrm), fm(out),
                              on.stream()),
          "filtering backward");
    return out;
}
struct FilterFn : Function<FilterFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& ids, const Tensor& w, SymInt width, SymInt height,
                          double focal, const Tensor& pts, const Tensor& nrm) {
        at::AutoDispatchBelowADInplaceOrView below;
        ctx->save_for_backward({ids, w, pts, nrm});
        save_view(ctx, width, height, focal, 0.0);
        static auto call = op<FilterFwd>("uds::filter_forward");
        return call.call(ids, w, width, height, focal, pts, nrm);
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        auto s = ctx->get_saved_variables();
        auto& d = ctx->saved_data;
        static auto call = op<FilterBwd>("uds::filter_backward");
        Tensor gw = call.call(s[0], s[1], g[0].contiguous(), d["width"].toSymInt(), d["height"].toSymInt(),
                              d["focal"].toDouble(), s[2], s[3]);
        return {Tensor(), gw, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};
Tensor filter_autograd(const Tensor& ids, const Tensor& w, SymInt width, SymInt height, double focal, const Tensor& pts,
                       const Tensor& nrm) {
    if (any_grad({&w, &pts, &nrm})) return FilterFn::apply(ids, w, width, height, focal, pts, nrm);
    at::AutoDispatchBelowADInplaceOrView below;
    static auto call = op<FilterFwd>("uds::filter_forward");
    return call.call(ids, w, width, height, focal, pts, nrm);
}

// ----------------------------------------------------------- interpolation
using InterpFwd = Tensor(const Tensor&, const Tensor&, const Tensor&);
using InterpBwd = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&);
void check_interp(const Tensor& ids, const Tensor& w, const Tensor& attr) {
    need(ids, "indices", nullptr, at::kInt);
    need(w, "weights", &ids);
    need(attr, "attribute", &ids);
    TORCH_CHECK_VALUE(ids.sizes() == w.sizes() && ids.dim() == 4 && attr.dim() == 3,
                      "expected indices/weights (B,W,H,K) and attribute (1|B,N,C)");
    TORCH_CHECK_VALUE(attr.size(0) == 1 || attr.size(0) == ids.size(0), "attribute batch must be 1 or B");
}
Tensor interp_forward_cuda(const Tensor& ids, const Tensor& w, const Tensor& attr) {
    check_interp(ids, w, attr);
    On on(ids);
    Tensor out = at::empty({ids.size(0), ids.size(1), ids.size(2), attr.size(2)}, w.options());
    check(uds_interp_forward(i32(ids.size(0)), i32(ids.size(1)), i32(ids.size(2)), i32(ids.size(3)), idx(ids), f(w),
                             i32(attr.size(0)), i32(attr.size(1)), i32(attr.size(2)), f(attr), fm(out), on.stream()),
          "interpolation forward");
    return out;
}
std::tuple<Tensor, Tensor> interp_backward_cuda(const Tensor& g, const Tensor& ids, const Tensor& w,
                                                const Tensor& attr) {
    check_interp(ids, w, attr);
    need(g, "gradIn", &ids);
    need_numel(g, ids.size(0) * ids.size(1) * ids.size(2) * attr.size(2), "gradIn");
    On on(ids);
    Tensor gw = at::empty_like(w), ga = at::empty_like(attr);
    check(uds_interp_backward(i32(ids.size(0)), i32(ids.size(1)), i32(ids.size(2)), i32(ids.size(3)), f(g), idx(ids),
                              f(w), i32(attr.size(0)), i32(attr.size(1)), i32(attr.size(2)), f(attr), fm(gw), fm(ga),
                              on.stream()),
          "interpolation backward");
    return {gw, ga};
}
struct InterpFn : Function<InterpFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& ids, const Tensor& w, const Tensor& attr) {
        at::AutoDispatchBelowADInplaceOrView below;
        ctx->save_for_backward({ids, w, attr});
        static auto call = op<InterpFwd>("uds::interp_forward");
        return call.call(ids, w, attr);
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        auto s = ctx->get_saved_variables();
        static auto call = op<InterpBwd>("uds::interp_backward");
        auto [gw, ga] = call.call(g[0].contiguous(), s[0], s[1], s[2]);
        return {Tensor(), gw, ga};
    }
};
Tensor interp_autograd(const Tensor& ids, const Tensor& w, const Tensor& attr) {
    if (any_grad({&w, &attr})) return InterpFn::apply(ids, w, attr);
    at::AutoDispatchBelowADInplaceOrView below;
    static auto call = op<InterpFwd>("uds::interp_forward");
    return call.call(ids, w, attr);
}

// ----------------------------------------------------------------- shading
using Shade4 = Tensor(const Tensor&, const Tensor&, const Tensor&, const Tensor&);
using Shade3 = Tensor(const Tensor&, const Tensor&, const Tensor&);
using Shade5 = Tensor(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&);
using ShadeBwd = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&);
using ShBwd = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&);
using LambertBwd = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                       const Tensor&);
std::pair<int, int> pixels(const Tensor& nrm, const Tensor& dif) {
    need(nrm, "normals");
    need(dif, "diffuse", &nrm);
    TORCH_CHECK_VALUE(nrm.sizes() == dif.sizes() && nrm.dim() > 0 && nrm.size(-1) == 3,
                      "normals and diffuse must both be (B,W,H,3)");
    const int64_t B = nrm.size(0);
    return {i32(B), B > 0 ? i32(nrm.numel() / (3 * B)) : 0};
}
void check_lamps(const Tensor& dirs, const Tensor& power, const Tensor& nrm) {
    need(dirs, "directions", &nrm);
    need(power, "intensities", &nrm);
    need_numel(dirs, 3 * power.size(1) * nrm.size(0), "directions");
    need_numel(power, 3 * power.size(1) * power.size(0), "intensities");
}
void check_sh(const Tensor& coef, const Tensor& nrm) {
    need(coef, "coefficients", &nrm);
    need_numel(coef, 27 * coef.size(0), "coefficients");
}
void check_grad(const Tensor& g, const Tensor& nrm) {
    need(g, "gradIn", &nrm);
    need_numel(g, nrm.numel(), "gradIn");
}
Tensor shade_forward_cuda(const Tensor& dirs, const Tensor& power, const Tensor& nrm, const Tensor& dif) {
    auto [B, P] = pixels(nrm, dif);
    check_lamps(dirs, power, nrm);
    On on(nrm);
    Tensor out = at::empty_like(nrm);
    check(uds_shade_forward(B, P, i32(power.size(1)), f(dirs), f(power), i32(power.size(0)), f(nrm), f(dif), fm(out),
                            on.stream()),
          "shading forward");
    return out;
}
std::vector<Tensor> shade_backward_cuda(const Tensor& g, const Tensor& dirs, const Tensor& power, const Tensor& nrm,
                                        const Tensor& dif) {
    auto [B, P] = pixels(nrm, dif);
    check_grad(g, nrm);
    check_lamps(dirs, power, nrm);
    On on(nrm);
    Tensor gd = at::empty_like(dirs), gI = at::empty_like(power), gn = at::empty_like(nrm), gf = at::empty_like(dif);
    check(uds_shade_backward(B, P, i32(power.size(1)), f(g), f(dirs), f(power), i32(power.size(0)), f(nrm), f(dif),
                             fm(gd), fm(gI), fm(gn), fm(gf), on.stream()),
          "shading backward");
    return {gd, gI, gn, gf};
}
Tensor sh_forward_cuda(const Tensor& coef, const Tensor& nrm, const Tensor& dif) {
    auto [B, P] = pixels(nrm, dif);
    check_sh(coef, nrm);
    On on(nrm);
    Tensor out = at::empty_like(nrm);
    check(uds_shade_sh_forward(B, P, f(coef), i32(coef.size(0)), f(nrm), f(dif), fm(out), on.stream()),
          "shading forwardSh");
    return out;
}
std::vector<Tensor> sh_backward_cuda(const Tensor& g, const Tensor& coef, const Tensor& nrm, const Tensor& dif) {
    auto [B, P] = pixels(nrm, dif);
    check_grad(g, nrm);
    check_sh(coef, nrm);
    On on(nrm);
    Tensor gc = at::empty_like(coef), gn = at::empty_like(nrm), gd = at::empty_like(dif);
    check(uds_shade_sh_backward(B, P, f(g), f(coef), i32(coef.size(0)), f(nrm), f(dif), fm(gc), fm(gn), fm(gd),
                                on.stream()),
          "shading backwardSh");
    return {gc, gn, gd};
}
// (B, N, L, ambient, intensity and diffuse batches): shading.lambert_shapes
struct LambertShape {
    int B, N, L, aB, IB, dB;
};
LambertShape lambert_shape(const Tensor& amb, const Tensor& dirs, const Tensor& power, const Tensor& nrm,
                           const Tensor& dif) {
    const Tensor* ts[] = {&amb, &dirs, &power, &nrm, &dif};
    bool ok = nrm.dim() == 3 && nrm.size(2) == 3;
    for (auto* t : ts) ok = ok && t->is_cuda() && t->scalar_type() == at::kFloat && t->device() == nrm.device();
    LambertShape s{};
    if (ok) {
        s.B = i32(nrm.size(0));
        s.N = i32(nrm.size(1));
        ok = dirs.dim() == 3 && dirs.size(0) == s.B && dirs.size(2) == 3 && power.dim() == 3 &&
             power.size(1) == dirs.size(1) && power.size(2) == 3 && dirs.size(1) <= 4 && dif.dim() == 3 &&
             dif.size(1) == s.N && dif.size(2) == 3 && amb.dim() >= 1 && amb.dim() <= 3 && amb.size(-1) == 3;
    }
    if (ok) {
        s.L = i32(dirs.size(1));
        s.IB = i32(power.size(0));
        s.dB = i32(dif.size(0));
        s.aB = amb.dim() == 3 ? i32(amb.size(0)) : 1;
        ok = !(amb.dim() == 3 && amb.size(1) != 1) && !(amb.dim() == 2 && amb.size(0) != 1);
        for (int x : {s.IB, s.dB, s.aB}) ok = ok && (x == 1 || x == s.B);
    }
    // the Python wrapper fails to unpack lambert_shapes' None
    TORCH_CHECK_TYPE(ok, "lambert: operands of shapes or types the kernel does not take");
    return s;
}
Tensor lambert_forward_cuda(const Tensor& amb, const Tensor& dirs, const Tensor& power, const Tensor& nrm,
                            const Tensor& dif) {
    LambertShape s = lambert_shape(amb, dirs, power, nrm, dif);
    On on(nrm);
    Tensor out = at::empty_like(nrm);
    check(uds_lambert_forward(s.B, s.N, s.L, f(amb), s.aB, f(dirs), f(power), s.IB, f(nrm), f(dif), s.dB, fm(out),
                              on.stream()),
          "lambert forward");
    return out;
}
std::vector<Tensor> lambert_backward_cuda(const Tensor& g, const Tensor& amb, const Tensor& dirs, const Tensor& power,
                                          const Tensor& nrm, const Tensor& dif) {
    LambertShape s = lambert_shape(amb, dirs, power, nrm, dif);
    check_grad(g, nrm);
    On on(nrm);
    Tensor ga = at::empty_like(amb), gd = at::empty_like(dirs), gI = at::empty_like(power);
    Tensor gn = at::empty_like(nrm), gf = at::empty_like(dif);
    check(uds_lambert_backward(s.B, s.N, s.L, f(g), f(amb), s.aB, f(dirs), f(power), s.IB, f(nrm), f(dif), s.dB, fm(ga),
                               fm(gd), fm(gI), fm(gn), fm(gf), on.stream()),
          "lambert backward");
    return {ga, gd, gI, gn, gf};
}

// Ops whose backward takes the gradient and every input.
struct ShadeOps {
    static constexpr const char *fwd = "uds::shade_forward", *bwd = "uds::shade_backward";
    using Fwd = Shade4;
    using Bwd = ShadeBwd;
};
struct ShOps {
    static constexpr const char *fwd = "uds::shade_sh_forward", *bwd = "uds::shade_sh_backward";
    using Fwd = Shade3;
    using Bwd = ShBwd;
};
struct LambertOps {
    static constexpr const char *fwd = "uds::lambert_forward", *bwd = "uds::lambert_backward";
    using Fwd = Shade5;
    using Bwd = LambertBwd;
};
template <class Ops, class... T>
struct AllFn : Function<AllFn<Ops, T...>> {
    static Tensor forward(AutogradContext* ctx, const T&... in) {
        at::AutoDispatchBelowADInplaceOrView below;
        ctx->save_for_backward({in...});
        static auto call = op<typename Ops::Fwd>(Ops::fwd);
        return call.call(in...);
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        auto s = ctx->get_saved_variables();
        static auto call = op<typename Ops::Bwd>(Ops::bwd);
        return invoke(call, g[0].contiguous(), s, std::index_sequence_for<T...>());
    }
    template <class Call, size_t... I>
    static variable_list invoke(const Call& call, const Tensor& g, const variable_list& s, std::index_sequence<I...>) {
        return call.call(g, s[I]...);
    }
    static Tensor autograd(const T&... in) {
        if (any_grad({&in...})) return AllFn::apply(in...);
        at::AutoDispatchBelowADInplaceOrView below;
        static auto call = op<typename Ops::Fwd>(Ops::fwd);
        return call.call(in...);
    }
};
using ShadeFn = AllFn<ShadeOps, Tensor, Tensor, Tensor, Tensor>;
using ShFn = AllFn<ShOps, Tensor, Tensor, Tensor>;
using LambertFn = AllFn<LambertOps, Tensor, Tensor, Tensor, Tensor, Tensor>;

// ----------------------------------------------------- per-splat consumers
Tensor nearest_cuda(const Tensor& ids, const Tensor& w, const Tensor& pts, int64_t M) {
    need(ids, "indices", nullptr, at::kInt);
    need(w, "weights", &ids);
    need(pts, "points", &ids);
    TORCH_CHECK_VALUE(ids.dim() == 4 && w.sizes() == ids.sizes(), "weights must match indices");
    TORCH_CHECK_VALUE(pts.dim() == 3 && pts.size(0) == 1 && pts.size(2) == 3, "points must be (1,N,3)");
    const int B = i32(ids.size(0)), W = i32(ids.size(1)), H = i32(ids.size(2)), K = i32(ids.size(3));
    const int N = i32(pts.size(1));
    On on(ids);
    Tensor out = at::empty({1, N, M}, ids.options());
    Tensor ws = scratch(uds_nearest_workspace_size(B, W, H, K, N), ids);
    check(uds_nearest_samples(B, W, H, K, idx(ids), f(w), N, f(pts), i32(M), out.mutable_data_ptr<int>(),
                              ws.mutable_data_ptr(), (size_t)ws.numel(), on.stream()),
          "nearestsamples nearest");
    return out;
}
std::tuple<Tensor, Tensor, Tensor> regularizer_cuda(const Tensor& nearest, const Tensor& pts, const Tensor& nrm,
                                                    double sigma, bool mean) {
    need(nearest, "nearest", nullptr, at::kInt);
    need(pts, "points", &nearest);
    need(nrm, "normals", &nearest);
    TORCH_CHECK_VALUE(nearest.dim() == 3 && nearest.size(0) == 1 && pts.dim() == 3 && pts.size(0) == 1 &&
                          pts.size(2) == 3 && nrm.sizes() == pts.sizes() && nearest.size(1) == pts.size(1),
                      "nearest must be (1,N,M) and points / normals (1,N,3)");
    const int N = i32(pts.size(1)), M = i32(nearest.size(2));
    On on(pts);
    Tensor losses = at::empty({2}, pts.options());
    Tensor gp = at::empty({1, N, 3}, pts.options()), gn = at::empty({1, N, 3}, pts.options());
    Tensor ws = scratch(uds_nearest_regularizer_workspace_size(N), pts);
    check(uds_nearest_regularizer(N, M, idx(nearest), f(pts), f(nrm), (float)sigma, mean, fm(losses), fm(gp), fm(gn),
                                  ws.mutable_data_ptr(), (size_t)ws.numel(), on.stream()),
          "nearestsamples regularizer");
    return {losses, gp, gn};
}

// Losses that compute their gradients in the forward pass (training.py,
// regularizers.py): the backward scales them by the incoming gradient.
using LossFwd = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, SymInt, double);
std::tuple<Tensor, Tensor> image_loss_cuda(const Tensor& x, const Tensor& y, int64_t kind, double scale) {
    need(x, "image");
    need(y, "target", &x);
    need_numel(y, x.numel(), "target");
    On on(x);
    Tensor loss = at::empty({}, x.options()), grad = at::empty_like(x);
    check(uds_image_loss(i32(kind), (size_t)x.numel(), f(x), f(y), (float)scale, fm(loss), fm(grad), on.stream()),
          "image loss");
    return {loss, grad};
}
struct LossFn : Function<LossFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& y, SymInt kind, double scale) {
        at::AutoDispatchBelowADInplaceOrView below;
        static auto call = op<LossFwd>("uds::image_loss");
        auto [loss, grad] = call.call(x, y, kind, scale);
        ctx->set_materialize_grads(false);
        ctx->mark_non_differentiable({grad});
        ctx->save_for_backward({grad});
        return {loss, grad};
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        return {g[0].defined() ? ctx->get_saved_variables()[0] * g[0] : Tensor(), Tensor(), Tensor(), Tensor()};
    }
};
std::tuple<Tensor, Tensor> image_loss_autograd(const Tensor& x, const Tensor& y, SymInt kind, double scale) {
    if (any_grad({&x, &y})) {
        auto r = LossFn::apply(x, y, kind, scale);
        return {r[0], r[1]};
    }
    at::AutoDispatchBelowADInplaceOrView below;
    static auto call = op<LossFwd>("uds::image_loss");
    return call.call(x, y, kind, scale);
}

using NearFwd = std::tuple<Tensor, Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, double, bool);
std::tuple<Tensor, Tensor, Tensor, Tensor> nearest_losses_cuda(const Tensor& pts, const Tensor& nrm,
                                                               const Tensor& nearest, double sigma, bool mean) {
    auto [losses, gp, gn] = regularizer_cuda(nearest, pts, nrm, sigma, mean);
    return {losses.select(0, 0), losses.select(0, 1).clone(), gp, gn};  // outputs share no storage
}
struct NearFn : Function<NearFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& pts, const Tensor& nrm, const Tensor& nearest,
                                 double sigma, bool mean) {
        at::AutoDispatchBelowADInplaceOrView below;
        static auto call = op<NearFwd>("uds::nearest_losses");
        auto [normal, plane, gp, gn] = call.call(pts, nrm, nearest, sigma, mean);
        ctx->set_materialize_grads(false);
        ctx->mark_non_differentiable({gp, gn});
        ctx->save_for_backward({gp, gn});
        return {normal, plane, gp, gn};
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        auto s = ctx->get_saved_variables();
        return {g[1].defined() ? s[0] * g[1] : at::zeros_like(s[0]),
                g[0].defined() ? s[1] * g[0] : at::zeros_like(s[1]), Tensor(), Tensor(), Tensor()};
    }
};
std::tuple<Tensor, Tensor, Tensor, Tensor> nearest_losses_autograd(const Tensor& pts, const Tensor& nrm,
                                                                   const Tensor& nearest, double sigma, bool mean) {
    if (any_grad({&pts, &nrm})) {
        auto r = NearFn::apply(pts, nrm, nearest, sigma, mean);
        return {r[0], r[1], r[2], r[3]};
    }
    at::AutoDispatchBelowADInplaceOrView below;
    static auto call = op<NearFwd>("uds::nearest_losses");
    return call.call(pts, nrm, nearest, sigma, mean);
}

}  // namespace

TORCH_LIBRARY_IMPL(uds, CUDA, m) {
    m.impl("affine_forward", Transform<true>::forward_cuda);
    m.impl("affine_backward", Transform<true>::backward_cuda);
    m.impl("linear_forward", Transform<false>::forward_cuda);
    m.impl("linear_backward", Transform<false>::backward_cuda);
    m.impl("view_matrix_forward", view_forward_cuda);
    m.impl("view_matrix_backward", view_backward_cuda);
    m.impl("backface", backface_cuda);
    m.impl("backface_backward", backface_backward_cuda);
    m.impl("splat_forward", splat_forward_cuda);
    m.impl("ewa_weights", splat_forward_cuda);
    m.impl("splat_backward", splat_backward_cuda);
    m.impl("splat_gradients", splat_gradients_cuda);
    m.impl("render_splats", render_forward_cuda);
    m.impl("render_splats_gradients", render_gradients_cuda);
    m.impl("render_splats_backward", render_backward_cuda);
    m.impl("filter_forward", filter_forward_cuda);
    m.impl("filter_backward", filter_backward_cuda);
    m.impl("interp_forward", interp_forward_cuda);
    m.impl("interp_backward", interp_backward_cuda);
    m.impl("shade_forward", shade_forward_cuda);
    m.impl("shade_backward", shade_backward_cuda);
    m.impl("shade_sh_forward", sh_forward_cuda);
    m.impl("shade_sh_backward", sh_backward_cuda);
    m.impl("lambert_forward", lambert_forward_cuda);
    m.impl("lambert_backward", lambert_backward_cuda);
    m.impl("nearest", nearest_cuda);
    m.impl("nearest_regularizer", regularizer_cuda);
    m.impl("nearest_losses", nearest_losses_cuda);
    m.impl("image_loss", image_loss_cuda);
}

TORCH_LIBRARY_IMPL(uds, AutogradCUDA, m) {
    m.impl("affine_forward", Transform<true>::autograd);
    m.impl("linear_forward", Transform<false>::autograd);
    m.impl("view_matrix_forward", view_autograd);
    m.impl("backface", backface_autograd);
    m.impl("splat_forward", SplatFn<true>::autograd);
    m.impl("ewa_weights", SplatFn<false>::autograd);
    m.impl("render_splats", render_autograd);
    m.impl("filter_forward", filter_autograd);
    m.impl("interp_forward", interp_autograd);
    m.impl("shade_forward", ShadeFn::autograd);
    m.impl("shade_sh_forward", ShFn::autograd);
    m.impl("lambert_forward", LambertFn::autograd);
    m.impl("nearest_losses", nearest_losses_autograd);
    m.impl("image_loss", image_loss_autograd);
    // no formula: a graph through these fails in its backward pass, as with
    // the Python definitions
    for (const char* name : {"sample", "sample_views", "affine_backward", "linear_backward", "view_matrix_backward",
                             "backface_backward", "splat_backward", "splat_gradients", "render_splats_backward",
                             "render_splats_gradients", "filter_backward",
                             "interp_backward", "shade_backward", "shade_sh_backward", "lambert_backward",
                             "pixel_gather", "nearest", "nearest_regularizer"})
        m.impl(name, torch::autograd::autogradNotImplementedFallback());
}
