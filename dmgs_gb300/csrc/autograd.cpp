// autograd.cpp — the package's autograd functions as native nodes.
//
// Same calls, outputs and gradients as the torch.autograd.Function classes of
// the Python modules, which stay the general form: every entry here takes
// only what needs no conversion (float32 CUDA tensors of one device,
// contiguous, of the expected shapes) and returns None for anything else, so
// that the caller runs the general form with its checks, conversions and
// messages.  What this saves is host time: a forward and backward through the
// Python classes held the interpreter for 0.1-0.3 ms on a Grace core (argument
// marshalling, tensor bookkeeping and the engine thread's wait for the
// interpreter lock), more than most of these kernels run.
#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <c10/cuda/CUDAStream.h>
#include <pybind11/pybind11.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/dmgs.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

namespace {

// Raises dmgs_gb300._lib.DmgsError for a negative code, from any thread.
void check(int code, const char *where) {
  if (code == 0) return;
  const std::string msg = dmgs_last_error() ? dmgs_last_error() : "";
  py::gil_scoped_acquire gil;
  {
    py::object cls = py::module_::import("dmgs_gb300._lib").attr("DmgsError");
    py::object err = cls(code, where, msg);
    PyErr_SetObject(cls.ptr(), err.ptr());
  }
  python_error e;
  e.persist();
  throw e;
}

dmgs_stream_t stream_of(const Tensor &t) {
  return reinterpret_cast<dmgs_stream_t>(c10::cuda::getCurrentCUDAStream(t.get_device()).stream());
}

// Address of a tensor; null when undefined or empty.
template <typename T = float>
T *ptr(const Tensor &t) {
  return t.defined() && t.numel() > 0 ? reinterpret_cast<T *>(t.data_ptr()) : nullptr;
}

// Inputs that may be absent reach a node as optionals: it keeps no edge and no
// metadata for those that are.
using Maybe = std::optional<Tensor>;
Maybe maybe(const Tensor &t) { return t.defined() ? Maybe(t) : Maybe(); }
Tensor of(const Maybe &t) { return t.has_value() ? *t : Tensor(); }

Tensor f32(at::IntArrayRef sizes, const Tensor &like) { return at::empty(sizes, like.options().dtype(at::kFloat)); }
Tensor bytes(size_t n, const Tensor &like) {
  return at::empty({(int64_t)n}, like.options().dtype(at::kByte));
}

// A gradient as the kernels read it: float32, contiguous, zeros if undefined.
Tensor grad_of(const Tensor &g, at::IntArrayRef sizes, const Tensor &like) {
  if (!g.defined()) return at::zeros(sizes, like.options().dtype(at::kFloat));
  return g.to(like.device(), at::kFloat).contiguous();
}

// Under torch.jit.trace the tracer records Python autograd functions, and would
// keep a native node's outputs as constants: such a call takes the general form.
bool traced() { return at::tracer::impl::is_dispatch_enabled(); }

// The tensor of a Python argument: false unless it is None (undefined) or a
// tensor.
bool unpack(py::handle h, Tensor &t) {
  if (h.is_none()) return true;
  if (!THPVariable_Check(h.ptr())) return false;
  t = THPVariable_Unpack(h.ptr());
  return true;
}

bool plain(const Tensor &t, const at::Device &d, at::ScalarType type = at::kFloat) {
  return t.defined() && t.layout() == at::kStrided && t.is_cuda() && t.device() == d && t.scalar_type() == type &&
         t.is_contiguous() && t.numel() > 0;
}
bool plain_or_none(const Tensor &t, const at::Device &d) { return !t.defined() || plain(t, d); }
bool shape(const Tensor &t, at::IntArrayRef s) { return t.sizes() == s; }

py::object wrap(const Tensor &t) { return py::reinterpret_steal<py::object>(THPVariable_Wrap(t)); }

// ---- rasteriser -----------------------------------------------------------------

struct RasterSettings {
  Tensor bg, view, proj, campos;
  int64_t H, W, degree;
  double tanx, tany, modifier;
  bool prefiltered;
};

// The settings' tensors as the kernels read them (cameras often come as
// transposed views or from the host); evaluated again for the backward, as
// the general form does.
void to_device(RasterSettings &s, const Tensor &like) {
  at::NoGradGuard no_grad;
  for (Tensor *t : {&s.bg, &s.view, &s.proj, &s.campos}) *t = t->to(like.device(), at::kFloat).contiguous();
}

DmgsView make_view(const RasterSettings &s) {
  DmgsView v{};
  v.width = (int32_t)s.W; v.height = (int32_t)s.H;
  v.tanfovx = (float)s.tanx; v.tanfovy = (float)s.tany;
  v.scale_modifier = (float)s.modifier; v.sh_degree = (int32_t)s.degree;
  v.prefiltered = s.prefiltered ? 1 : 0; v.debug = 0;
  v.bg = ptr(s.bg); v.viewmatrix = ptr(s.view); v.projmatrix = ptr(s.proj); v.campos = ptr(s.campos);
  return v;
}

DmgsGaussians make_gaussians(const Tensor &means, const Tensor &opac, const Tensor &sh, const Tensor &colors,
                             const Tensor &scales, const Tensor &rots, const Tensor &cov) {
  DmgsGaussians g{};
  g.P = (int32_t)means.size(0);
  g.M = sh.defined() ? (int32_t)sh.size(1) : 0;
  g.means3D = ptr(means); g.opacities = ptr(opac); g.shs = ptr(sh); g.colors_precomp = ptr(colors);
  g.scales = ptr(scales); g.rotations = ptr(rots); g.cov3D_precomp = ptr(cov);
  return g;
}

struct Raster : public Function<Raster> {
  static variable_list forward(AutogradContext *ctx, const Tensor &means, const Maybe &means2D, const Maybe &sh_,
                               const Maybe &colors_, const Tensor &opac, const Maybe &scales_, const Maybe &rots_,
                               const Maybe &cov_, const RasterSettings &given) {
    RasterSettings rs = given;
    to_device(rs, means);
    const Tensor sh = of(sh_), colors = of(colors_), scales = of(scales_), rots = of(rots_), cov = of(cov_);
    const DmgsView view = make_view(rs);
    const DmgsGaussians g = make_gaussians(means, opac, sh, colors, scales, rots, cov);
    const dmgs_stream_t stream = stream_of(means);
    Tensor geom = bytes(dmgs_geom_state_bytes(g.P, view.width, view.height), means);
    Tensor radii = at::empty({g.P}, means.options().dtype(at::kInt));
    int64_t K = 0;
    check(dmgs_raster_fwd_geometry(&view, &g, geom.data_ptr(), geom.numel(), radii.data_ptr<int32_t>(), &K, stream),
          "rasterize_gaussians");
    Tensor bin = bytes(dmgs_binning_state_bytes(K, view.width, view.height), means);
    Tensor img = bytes(dmgs_image_state_bytes(view.width, view.height), means);
    Tensor color = f32({3, rs.H, rs.W}, means);
    check(dmgs_raster_fwd_render(&view, &g, geom.data_ptr(), geom.numel(), bin.data_ptr(), bin.numel(), K,
                                 img.data_ptr(), img.numel(), color.data_ptr<float>(), stream),
          "rasterize_gaussians");
    ctx->save_for_backward({means, sh, colors, opac, scales, rots, cov, geom, bin, img});
    // held as they are, without a version check: the backward reads them again
    ctx->saved_data["camera"] = std::vector<Tensor>{given.bg, given.view, given.proj, given.campos};
    ctx->saved_data["ints"] = std::vector<int64_t>{rs.H, rs.W, rs.degree, rs.prefiltered ? 1 : 0, K};
    ctx->saved_data["floats"] = std::vector<double>{rs.tanx, rs.tany, rs.modifier};
    ctx->mark_non_differentiable({radii});
    ctx->set_materialize_grads(false);
    return {color, radii};
  }

  static variable_list backward(AutogradContext *ctx, variable_list gout) {
    const variable_list sv = ctx->get_saved_variables();
    const Tensor &means = sv[0], &sh = sv[1], &colors = sv[2], &opac = sv[3], &scales = sv[4], &rots = sv[5],
                 &cov = sv[6], &geom = sv[7], &bin = sv[8], &img = sv[9];
    const auto camera = ctx->saved_data["camera"].toTensorVector();
    const auto ints = ctx->saved_data["ints"].toIntVector();
    const auto floats = ctx->saved_data["floats"].toDoubleVector();
    RasterSettings rs;
    rs.bg = camera[0]; rs.view = camera[1]; rs.proj = camera[2]; rs.campos = camera[3];
    rs.H = ints[0]; rs.W = ints[1]; rs.degree = ints[2]; rs.prefiltered = ints[3] != 0;
    rs.tanx = floats[0]; rs.tany = floats[1]; rs.modifier = floats[2];
    to_device(rs, means);
    const DmgsView view = make_view(rs);
    const DmgsGaussians g = make_gaussians(means, opac, sh, colors, scales, rots, cov);
    const int64_t P = g.P;
    const Tensor dout = grad_of(gout[0], {3, rs.H, rs.W}, means);
    Tensor d2 = f32({P, 3}, means), dop = f32(opac.sizes(), means), d3 = f32({P, 3}, means), dcol, dcov, dsh, dsc, drot;
    if (colors.defined()) dcol = f32({P, 3}, means);
    if (cov.defined()) dcov = f32({P, 6}, means);
    if (sh.defined()) dsh = f32({P, g.M, 3}, means);
    if (scales.defined() && !cov.defined()) dsc = f32({P, 3}, means);
    if (rots.defined() && !cov.defined()) drot = f32({P, 4}, means);
    DmgsGrads gr{};
    gr.dL_dmeans2D = ptr(d2); gr.dL_dcolors = ptr(dcol); gr.dL_dopacity = ptr(dop); gr.dL_dmeans3D = ptr(d3);
    gr.dL_dcov3D = ptr(dcov); gr.dL_dsh = ptr(dsh); gr.dL_dscales = ptr(dsc); gr.dL_drotations = ptr(drot);
    Tensor scratch = bytes(dmgs_bwd_scratch_bytes(g.P), means);
    check(dmgs_raster_bwd(&view, &g, dout.data_ptr<float>(), geom.data_ptr(), geom.numel(), bin.data_ptr(), bin.numel(),
                          ints[4], img.data_ptr(), img.numel(), scratch.data_ptr(), scratch.numel(), &gr,
                          stream_of(means)),
          "rasterize_gaussians_backward");
    return {d3, d2, dsh, dcol, dop, dsc, drot, dcov, Tensor()};
  }
};

py::object raster(py::handle means_, py::handle means2D_, py::handle sh_, py::handle colors_, py::handle opac_,
                  py::handle scales_, py::handle rots_, py::handle cov_, py::handle bg_, py::handle view_,
                  py::handle proj_, py::handle campos_, int64_t H, int64_t W, double tanx, double tany,
                  double modifier, int64_t degree, bool prefiltered) {
  if (traced()) return py::none();
  Tensor means, means2D, sh, colors, opac, scales, rots, cov;
  RasterSettings rs;
  if (!unpack(means_, means) || !unpack(means2D_, means2D) || !unpack(sh_, sh) || !unpack(colors_, colors) ||
      !unpack(opac_, opac) || !unpack(scales_, scales) || !unpack(rots_, rots) || !unpack(cov_, cov) ||
      !unpack(bg_, rs.bg) || !unpack(view_, rs.view) || !unpack(proj_, rs.proj) || !unpack(campos_, rs.campos))
    return py::none();
  if (!means.defined()) return py::none();
  const at::Device d = means.device();
  if (!plain(means, d) || means.dim() != 2 || means.size(1) != 3 || !plain(opac, d)) return py::none();
  const int64_t P = means.size(0);
  if (P > INT32_MAX || opac.numel() != P) return py::none();
  for (const Tensor *t : {&sh, &colors, &scales, &rots, &cov})
    if (!plain_or_none(*t, d)) return py::none();
  if (sh.defined() && (sh.dim() != 3 || sh.size(0) != P || sh.size(2) != 3)) return py::none();
  if ((colors.defined() && !shape(colors, {P, 3})) || (scales.defined() && !shape(scales, {P, 3})) ||
      (rots.defined() && !shape(rots, {P, 4})) || (cov.defined() && !shape(cov, {P, 6})))
    return py::none();
  if (rots.defined() && (reinterpret_cast<uintptr_t>(rots.data_ptr()) & 15)) return py::none();
  const std::pair<const Tensor *, int64_t> camera[] = {{&rs.bg, 3}, {&rs.view, 16}, {&rs.proj, 16}, {&rs.campos, 3}};
  for (const auto &[t, n] : camera)
    if (!t->defined() || t->layout() != at::kStrided || !(t->is_cuda() || t->is_cpu()) || t->numel() != n)
      return py::none();
  if (H < INT32_MIN || H > INT32_MAX || W < INT32_MIN || W > INT32_MAX || degree < INT32_MIN || degree > INT32_MAX)
    return py::none();
  rs.H = H; rs.W = W; rs.degree = degree;
  rs.tanx = tanx; rs.tany = tany; rs.modifier = modifier; rs.prefiltered = prefiltered;
  variable_list out;
  {
    py::gil_scoped_release nogil;
    out = Raster::apply(means, maybe(means2D), maybe(sh), maybe(colors), opac, maybe(scales), maybe(rots), maybe(cov), rs);
  }
  return py::make_tuple(wrap(out[0]), wrap(out[1]));
}

// ---- photometric loss -------------------------------------------------------------

struct Loss : public Function<Loss> {
  static Tensor forward(AutogradContext *ctx, const Tensor &x, const Tensor &y, double lambda) {
    const int32_t C = (int32_t)x.size(0), H = (int32_t)x.size(1), W = (int32_t)x.size(2);
    Tensor scratch = bytes(dmgs_l1_ssim_scratch_bytes(C, H, W), x);
    Tensor loss = f32({}, x), grad = at::empty_like(x);
    check(dmgs_l1_ssim(ptr(x), ptr(y), C, H, W, (float)lambda, loss.data_ptr<float>(), grad.data_ptr<float>(),
                       scratch.data_ptr(), scratch.numel(), stream_of(x)),
          "l1_ssim");
    ctx->save_for_backward({grad});
    return loss;
  }
  static variable_list backward(AutogradContext *ctx, variable_list g) {
    return {ctx->get_saved_variables()[0] * g[0], Tensor(), Tensor()};
  }
};

py::object l1_ssim(py::handle x_, py::handle y_, double lambda) {
  if (traced()) return py::none();
  Tensor x, y;
  if (!unpack(x_, x) || !unpack(y_, y) || !x.defined() || !plain(x, x.device()) || !plain(y, x.device()) ||
      x.dim() != 3 || x.sizes() != y.sizes() || x.numel() > INT32_MAX)
    return py::none();
  Tensor out;
  {
    py::gil_scoped_release nogil;
    out = Loss::apply(x, y, lambda);
  }
  return wrap(out);
}

// ---- sigmoid(SH) colours -------------------------------------------------------------

struct ShColors : public Function<ShColors> {
  static Tensor forward(AutogradContext *ctx, const Tensor &sh, const Tensor &xyz, const Tensor &campos, int64_t deg) {
    Tensor out = f32({sh.size(0), 3}, xyz);
    check(dmgs_sh_colors_fwd((int32_t)sh.size(0), (int32_t)deg, (int32_t)sh.size(2), ptr(sh), ptr(xyz), ptr(campos),
                             out.data_ptr<float>(), stream_of(xyz)),
          "sh_colors_fwd");
    ctx->saved_data["deg"] = deg;
    ctx->save_for_backward({sh, xyz, campos});
    return out;
  }
  static variable_list backward(AutogradContext *ctx, variable_list g) {
    const variable_list sv = ctx->get_saved_variables();
    const Tensor &sh = sv[0], &xyz = sv[1], &campos = sv[2];
    const Tensor dcol = grad_of(g[0], {sh.size(0), 3}, xyz);
    Tensor dsh = at::empty_like(sh), dx;
    if (ctx->needs_input_grad(1)) dx = at::empty_like(xyz);
    check(dmgs_sh_colors_bwd((int32_t)sh.size(0), (int32_t)ctx->saved_data["deg"].toInt(), (int32_t)sh.size(2), ptr(sh),
                             ptr(xyz), ptr(campos), dcol.data_ptr<float>(), dsh.data_ptr<float>(), ptr(dx),
                             stream_of(xyz)),
          "sh_colors_bwd");
    return {dsh, dx, Tensor(), Tensor()};
  }
};

py::object sh_colors(py::handle sh_, py::handle xyz_, py::handle campos_, int64_t deg) {
  if (traced()) return py::none();
  Tensor sh, xyz, cam;
  if (!unpack(sh_, sh) || !unpack(xyz_, xyz) || !unpack(campos_, cam) || !xyz.defined()) return py::none();
  const at::Device d = xyz.device();
  if (!plain(sh, d) || !plain(xyz, d) || !plain(cam, d) || sh.dim() != 3 || sh.size(1) != 3 || xyz.dim() != 2 ||
      xyz.size(1) != 3 || sh.size(0) != xyz.size(0) || sh.size(0) > INT32_MAX || cam.numel() != 3)
    return py::none();
  Tensor out;
  {
    py::gil_scoped_release nogil;
    out = ShColors::apply(sh, xyz, cam, deg);
  }
  return wrap(out);
}

// ---- face bindings -------------------------------------------------------------------

struct Bind2Args {
  int64_t G, per_g, adaptive;
  double rad_base, z_scale, max_scale;
};

DmgsFaceBinding bind2_desc(const Tensor &v, const Tensor &sf, const Tensor &f, const Tensor &bc, const Bind2Args &a) {
  DmgsFaceBinding b{};
  b.F = (int32_t)f.size(0); b.V = (int32_t)v.size(0); b.G = (int32_t)a.G;
  b.bc_per_gaussian = (int32_t)a.per_g; b.adaptive_cov = (int32_t)a.adaptive;
  b.rad_base = (float)a.rad_base; b.z_scale = (float)a.z_scale; b.max_scale = (float)a.max_scale;
  b.verts = ptr(v); b.faces = ptr<int64_t>(f); b.bc = ptr(bc); b.scale_factor = ptr(sf);
  return b;
}

struct Bind2 : public Function<Bind2> {
  static variable_list forward(AutogradContext *ctx, const Tensor &v, const Maybe &sf_, const Tensor &f,
                               const Tensor &bc, const Bind2Args &a) {
    const Tensor sf = of(sf_);
    const DmgsFaceBinding b = bind2_desc(v, sf, f, bc, a);
    const int64_t F = b.F, n = F * a.G;
    Tensor xyz = f32({n, 3}, v), cov = f32({n, 6}, v), covL = f32({F, 3, 3}, v);
    check(dmgs_bind_fwd(&b, xyz.data_ptr<float>(), cov.data_ptr<float>(), nullptr, covL.data_ptr<float>(),
                        stream_of(v)),
          "bind_fwd");
    ctx->save_for_backward({v, sf, f, bc});
    ctx->saved_data["ints"] = std::vector<int64_t>{a.G, a.per_g, a.adaptive};
    ctx->saved_data["floats"] = std::vector<double>{a.rad_base, a.z_scale, a.max_scale};
    ctx->mark_non_differentiable({covL});
    ctx->set_materialize_grads(false);
    return {xyz, cov, covL};
  }
  static variable_list backward(AutogradContext *ctx, variable_list g) {
    const variable_list sv = ctx->get_saved_variables();
    const Tensor &v = sv[0], &sf = sv[1], &f = sv[2], &bc = sv[3];
    const auto i = ctx->saved_data["ints"].toIntVector();
    const auto x = ctx->saved_data["floats"].toDoubleVector();
    const DmgsFaceBinding b = bind2_desc(v, sf, f, bc, Bind2Args{i[0], i[1], i[2], x[0], x[1], x[2]});
    const int64_t n = (int64_t)b.F * i[0];
    const Tensor dxyz = grad_of(g[0], {n, 3}, v), dcov = grad_of(g[1], {n, 6}, v);
    Tensor dv = at::empty_like(v), dsf;
    if (sf.defined()) dsf = at::empty_like(sf);
    check(dmgs_bind_bwd(&b, ptr(dxyz), ptr(dcov), dv.data_ptr<float>(), ptr(dsf), stream_of(v)), "bind_bwd");
    return {dv, dsf, Tensor(), Tensor(), Tensor()};
  }
};

py::object bind2(py::handle v_, py::handle sf_, py::handle f_, py::handle bc_, int64_t G, bool per_g, double rad_base,
                 double z_scale, double max_scale, bool adaptive) {
  if (traced()) return py::none();
  Tensor v, sf, f, bc;
  if (!unpack(v_, v) || !unpack(sf_, sf) || !unpack(f_, f) || !unpack(bc_, bc) || !v.defined()) return py::none();
  const at::Device d = v.device();
  if (!plain(v, d) || !plain(f, d, at::kLong) || !plain(bc, d) || !plain_or_none(sf, d) || v.dim() != 2 ||
      v.size(1) != 3 || f.dim() != 2 || f.size(1) != 3 || bc.dim() != 2 || bc.size(1) != 3 || G < 1 ||
      f.size(0) * G > INT32_MAX || v.size(0) > INT32_MAX || bc.size(0) != (per_g ? f.size(0) * G : G) ||
      (sf.defined() && sf.numel() != 1))
    return py::none();
  variable_list out;
  {
    py::gil_scoped_release nogil;
    out = Bind2::apply(v, maybe(sf), f, bc, Bind2Args{G, per_g ? 1 : 0, adaptive ? 1 : 0, rad_base, z_scale, max_scale});
  }
  return py::make_tuple(wrap(out[0]), wrap(out[1]), wrap(out[2]));
}

DmgsFaceBinding3 bind3_desc(const Tensor &v, const Tensor &s2, const Tensor &r2, const Tensor &f, const Tensor &bc,
                            double thin_z) {
  DmgsFaceBinding3 b{};
  b.F = (int32_t)f.size(0); b.V = (int32_t)v.size(0); b.G = (int32_t)bc.size(0); b.thin_z = (float)thin_z;
  b.verts = ptr(v); b.faces = ptr<int64_t>(f); b.bc = ptr(bc); b.scaling2d = ptr(s2); b.rotation2d = ptr(r2);
  return b;
}

struct Bind3 : public Function<Bind3> {
  static variable_list forward(AutogradContext *ctx, const Tensor &v, const Tensor &s2, const Tensor &r2,
                               const Tensor &f, const Tensor &bc, double thin_z) {
    const DmgsFaceBinding3 b = bind3_desc(v, s2, r2, f, bc, thin_z);
    const int64_t n = (int64_t)b.F * b.G;
    Tensor xyz = f32({n, 3}, v), scales = f32({n, 3}, v), rots = f32({n, 4}, v);
    check(dmgs_bind3_fwd(&b, xyz.data_ptr<float>(), scales.data_ptr<float>(), rots.data_ptr<float>(), stream_of(v)),
          "bind3_fwd");
    ctx->save_for_backward({v, s2, r2, f, bc});
    ctx->saved_data["thin_z"] = thin_z;
    return {xyz, scales, rots};
  }
  static variable_list backward(AutogradContext *ctx, variable_list g) {
    const variable_list sv = ctx->get_saved_variables();
    const Tensor &v = sv[0], &s2 = sv[1], &r2 = sv[2], &f = sv[3], &bc = sv[4];
    const DmgsFaceBinding3 b = bind3_desc(v, s2, r2, f, bc, ctx->saved_data["thin_z"].toDouble());
    const int64_t n = (int64_t)b.F * b.G;
    const Tensor dxyz = grad_of(g[0], {n, 3}, v), dsc = grad_of(g[1], {n, 3}, v), drot = grad_of(g[2], {n, 4}, v);
    Tensor dv = at::empty_like(v), ds2 = at::empty_like(s2), dr2 = at::empty_like(r2);
    check(dmgs_bind3_bwd(&b, ptr(dxyz), ptr(dsc), ptr(drot), dv.data_ptr<float>(), ds2.data_ptr<float>(),
                         dr2.data_ptr<float>(), stream_of(v)),
          "bind3_bwd");
    return {dv, ds2, dr2, Tensor(), Tensor(), Tensor()};
  }
};

py::object bind3(py::handle v_, py::handle s2_, py::handle r2_, py::handle f_, py::handle bc_, double thin_z) {
  if (traced()) return py::none();
  Tensor v, s2, r2, f, bc;
  if (!unpack(v_, v) || !unpack(s2_, s2) || !unpack(r2_, r2) || !unpack(f_, f) || !unpack(bc_, bc) || !v.defined())
    return py::none();
  const at::Device d = v.device();
  if (!plain(v, d) || !plain(f, d, at::kLong) || !plain(bc, d) || !plain(s2, d) || !plain(r2, d) || v.dim() != 2 ||
      v.size(1) != 3 || f.dim() != 2 || f.size(1) != 3 || bc.dim() != 2 || bc.size(1) != 3 || v.size(0) > INT32_MAX ||
      f.size(0) * bc.size(0) > INT32_MAX)
    return py::none();
  const int64_t n = f.size(0) * bc.size(0);
  if (s2.numel() != 2 * n || r2.numel() != 2 * n) return py::none();
  variable_list out;
  {
    py::gil_scoped_release nogil;
    out = Bind3::apply(v, s2, r2, f, bc, thin_z);
  }
  return py::make_tuple(wrap(out[0]), wrap(out[1]), wrap(out[2]));
}

// ---- hash-grid texture ---------------------------------------------------------------

struct TexArgs {
  std::vector<double> aabb;
  double per_level_scale;
  bool keep_enc;
};

DmgsTexture tex_desc(const Tensor &t, const Tensor &w1, const Tensor &w2, const Tensor &w3,
                     const std::vector<double> &aabb, double pls) {
  DmgsTexture d{};
  d.table = ptr(t); d.W1 = ptr(w1); d.W2 = ptr(w2); d.W3 = ptr(w3);
  d.channels = (int32_t)w3.size(0);
  for (int k = 0; k < 6; ++k) d.aabb[k] = (float)aabb[k];
  d.per_level_scale = (float)pls;
  return d;
}

struct Texture : public Function<Texture> {
  static Tensor forward(AutogradContext *ctx, const Tensor &x, const Tensor &t, const Tensor &w1, const Tensor &w2,
                        const Tensor &w3, const TexArgs &a) {
    const DmgsTexture d = tex_desc(t, w1, w2, w3, a.aabb, a.per_level_scale);
    const int64_t n = x.size(0);
    Tensor out = f32({n, w3.size(0)}, x), enc;
    if (a.keep_enc) {
      enc = f32({n, 32}, x);
      check(dmgs_tex_fwd_enc(&d, n, ptr(x), out.data_ptr<float>(), enc.data_ptr<float>(), stream_of(x)), "tex_fwd");
    } else {
      check(dmgs_tex_fwd(&d, n, ptr(x), out.data_ptr<float>(), stream_of(x)), "tex_fwd");
    }
    ctx->save_for_backward({x, t, w1, w2, w3, enc});
    std::vector<double> f = a.aabb;
    f.push_back(a.per_level_scale);
    ctx->saved_data["floats"] = f;
    return out;
  }
  static variable_list backward(AutogradContext *ctx, variable_list gout) {
    const variable_list sv = ctx->get_saved_variables();
    const Tensor &x = sv[0], &t = sv[1], &w1 = sv[2], &w2 = sv[3], &w3 = sv[4], &enc = sv[5];
    const std::vector<double> f = ctx->saved_data["floats"].toDoubleVector();
    const DmgsTexture d = tex_desc(t, w1, w2, w3, f, f[6]);
    const int64_t n = x.size(0);
    const Tensor g = grad_of(gout[0], {n, w3.size(0)}, x);
    Tensor dx, dt, dw1 = at::empty_like(w1), dw2 = at::empty_like(w2), dw3 = at::empty_like(w3);
    if (ctx->needs_input_grad(0)) dx = at::empty_like(x);
    if (ctx->needs_input_grad(1)) dt = at::empty_like(t);
    Tensor scratch = bytes(dmgs_tex_bwd_scratch_bytes(n), x);
    if (enc.defined())
      check(dmgs_tex_bwd_enc(&d, n, ptr(x), ptr(enc), ptr(g), ptr(dx), ptr(dt), ptr(dw1), ptr(dw2), ptr(dw3),
                             scratch.data_ptr(), scratch.numel(), stream_of(x)),
            "tex_bwd");
    else
      check(dmgs_tex_bwd(&d, n, ptr(x), ptr(g), ptr(dx), ptr(dt), ptr(dw1), ptr(dw2), ptr(dw3), scratch.data_ptr(),
                         scratch.numel(), stream_of(x)),
            "tex_bwd");
    return {dx, dt, dw1, dw2, dw3, Tensor()};
  }
};

py::object texture(py::handle x_, py::handle t_, py::handle w1_, py::handle w2_, py::handle w3_, py::sequence aabb,
                   double pls, bool keep_enc) {
  if (traced()) return py::none();
  Tensor x, t, w1, w2, w3;
  if (!unpack(x_, x) || !unpack(t_, t) || !unpack(w1_, w1) || !unpack(w2_, w2) || !unpack(w3_, w3) || !x.defined())
    return py::none();
  const at::Device d = x.device();
  if (!plain(x, d) || !plain(t, d) || !plain(w1, d) || !plain(w2, d) || !plain(w3, d) || x.dim() != 2 ||
      x.size(1) != 3 || !shape(w1, {32, 32}) || !shape(w2, {32, 32}) || w3.dim() != 2 || w3.size(1) != 32 ||
      t.numel() != 2 * dmgs_tex_table_entries((float)pls))
    return py::none();
  TexArgs a;
  for (py::handle h : aabb) a.aabb.push_back(h.cast<double>());
  if (a.aabb.size() != 6) return py::none();
  a.per_level_scale = pls;
  a.keep_enc = keep_enc;
  Tensor out;
  {
    py::gil_scoped_release nogil;
    out = Texture::apply(x, t, w1, w2, w3, a);
  }
  return wrap(out);
}

// ---- FlexiCubes ------------------------------------------------------------------------

struct FcArgs {
  int64_t res[3];
  bool training, fused, nocheck;
};

DmgsFcGrid fc_grid(const Tensor &x, const Tensor &s, const Tensor &beta, const Tensor &alpha, const Tensor &gamma,
                   const Tensor &vmask, const FcArgs &a) {
  DmgsFcGrid g{};
  g.vert_mask = ptr<uint8_t>(vmask);
  g.no_ambiguity_check = a.nocheck ? 1 : 0;
  g.x = ptr(x); g.s = ptr(s);
  g.beta = ptr(beta);
  if (a.fused) {  // beta holds all three: columns 0-11, 12-19, 20 of [C, 21]
    g.alpha = g.beta + 12;
    g.gamma = g.beta + 20;
    g.beta_stride = g.alpha_stride = g.gamma_stride = 21;
  } else {
    g.alpha = ptr(alpha);
    g.gamma = ptr(gamma);
  }
  g.rx = (int32_t)a.res[0]; g.ry = (int32_t)a.res[1]; g.rz = (int32_t)a.res[2];
  g.training = a.training ? 1 : 0;
  return g;
}

struct FlexiCubes : public Function<FlexiCubes> {
  static variable_list forward(AutogradContext *ctx, const Tensor &x, const Tensor &s, const Maybe &beta_,
                               const Maybe &alpha_, const Maybe &gamma_, const Maybe &vmask_, const FcArgs &a) {
    const Tensor beta = of(beta_), alpha = of(alpha_), gamma = of(gamma_), vmask = of(vmask_);
    const DmgsFcGrid g = fc_grid(x, s, beta, alpha, gamma, vmask, a);
    const dmgs_stream_t stream = stream_of(x);
    Tensor state = bytes(dmgs_fc_state_bytes(g.rx, g.ry, g.rz), x);
    uint32_t c[8];
    check(dmgs_fc_count(&g, state.data_ptr(), state.numel(), c, stream), "fc_count");
    const int64_t n_surf = c[0], n_vd = c[1], n_ent = c[2], n_edges = c[3], n_quads = c[4];
    Tensor work = bytes(std::max<size_t>(1, dmgs_fc_work_bytes(c)), x);
    const auto longs = x.options().dtype(at::kLong);
    Tensor vertices = f32({n_vd + (a.training ? n_quads : 0), 3}, x);
    Tensor faces = at::empty({(a.training ? 4 : 2) * n_quads, 3}, longs);
    Tensor L = f32({n_ent}, x), edges = at::empty({n_edges, 2}, longs);
    if (n_surf)
      check(dmgs_fc_emit(&g, c, state.data_ptr(), state.numel(), work.data_ptr(), work.numel(),
                         vertices.data_ptr<float>(), ptr<int64_t>(faces), ptr(L), ptr<int64_t>(edges), stream),
            "fc_emit");
    std::vector<int64_t> ints(c, c + 8);
    for (int k = 0; k < 3; ++k) ints.push_back(a.res[k]);
    for (bool b : {a.training, a.fused, a.nocheck}) ints.push_back(b ? 1 : 0);
    ctx->saved_data["ints"] = ints;
    ctx->save_for_backward({x, s, beta, alpha, gamma, vmask, state, work, vertices});
    ctx->mark_non_differentiable({faces, edges});
    ctx->set_materialize_grads(false);
    return {vertices, faces, L, edges};
  }
  static variable_list backward(AutogradContext *ctx, variable_list gout) {
    const variable_list sv = ctx->get_saved_variables();
    const Tensor &x = sv[0], &s = sv[1], &beta = sv[2], &alpha = sv[3], &gamma = sv[4], &vmask = sv[5], &state = sv[6],
                 &work = sv[7], &vertices = sv[8];
    const auto ints = ctx->saved_data["ints"].toIntVector();
    uint32_t c[8];
    for (int k = 0; k < 8; ++k) c[k] = (uint32_t)ints[k];
    const FcArgs a{{ints[8], ints[9], ints[10]}, ints[11] != 0, ints[12] != 0, ints[13] != 0};
    const DmgsFcGrid g = fc_grid(x, s, beta, alpha, gamma, vmask, a);
    // the kernel adds into the vertices' gradient: a copy of its own
    Tensor dv = grad_of(gout[0], vertices.sizes(), x);
    if (gout[0].defined() && dv.is_alias_of(gout[0])) dv = dv.clone();
    const Tensor dL = grad_of(gout[2], {(int64_t)c[2]}, x);
    Tensor dx = at::empty_like(x), ds = at::empty_like(s), db, da, dg;
    size_t edge = 2;  // edges are counted over the inputs that are there
    if (beta.defined() && ctx->needs_input_grad(edge++)) db = at::empty_like(beta);
    if (alpha.defined() && ctx->needs_input_grad(edge++)) da = at::empty_like(alpha);
    if (gamma.defined() && ctx->needs_input_grad(edge++)) dg = at::empty_like(gamma);
    float *pb = ptr(db), *pa = ptr(da), *pg = ptr(dg);
    if (a.fused && pb) {
      pa = pb + 12;
      pg = pb + 20;
    }
    check(dmgs_fc_bwd(&g, c, state.data_ptr(), state.numel(), work.data_ptr(), work.numel(), ptr(vertices), ptr(dv),
                      ptr(dL), dx.data_ptr<float>(), ds.data_ptr<float>(), pb, pa, pg, stream_of(x)),
          "fc_bwd");
    return {dx, ds, db, da, dg, Tensor(), Tensor()};
  }
};

py::object flexicubes(py::handle x_, py::handle s_, py::handle beta_, py::handle alpha_, py::handle gamma_,
                      py::handle vmask_, int64_t rx, int64_t ry, int64_t rz, bool training, bool fused, bool nocheck) {
  if (traced()) return py::none();
  Tensor x, s, beta, alpha, gamma, vmask;
  if (!unpack(x_, x) || !unpack(s_, s) || !unpack(beta_, beta) || !unpack(alpha_, alpha) || !unpack(gamma_, gamma) ||
      !unpack(vmask_, vmask) || !x.defined())
    return py::none();
  const at::Device d = x.device();
  if (!plain(x, d) || !plain(s, d) || !plain_or_none(beta, d) || !plain_or_none(alpha, d) || !plain_or_none(gamma, d) ||
      (vmask.defined() && !plain(vmask, d, at::kByte)) || (fused && (!beta.defined() || alpha.defined() || gamma.defined())))
    return py::none();
  variable_list out;
  {
    py::gil_scoped_release nogil;
    out = FlexiCubes::apply(x, s, maybe(beta), maybe(alpha), maybe(gamma), maybe(vmask), FcArgs{{rx, ry, rz}, training, fused, nocheck});
  }
  return py::make_tuple(wrap(out[0]), wrap(out[1]), wrap(out[2]), wrap(out[3]));
}

}  // namespace

PYBIND11_MODULE(_autograd, m) {
  m.def("raster", &raster);
  m.def("l1_ssim", &l1_ssim);
  m.def("sh_colors", &sh_colors);
  m.def("bind2", &bind2);
  m.def("bind3", &bind3);
  m.def("texture", &texture);
  m.def("flexicubes", &flexicubes);
}
