// The operators of npa_b200 as autograd nodes in C++, over the C ABI of libnpa_b200.so.
//
// What a training step of a small system waits for is the host: with torch.autograd.Function in
// Python and ctypes underneath, one operator costs 30-50 us of argument conversion, checks,
// allocation and node bookkeeping per direction, several times what its kernels take at 4,096
// particles.  Here an operator is one call: checks, output allocation, launch and graph node
// together are a few microseconds, and backward nodes run in the autograd engine without the
// interpreter.  Semantics are those of the reference's Functions (sphops/sph.py:127-464): a
// gradient is produced only for inputs that need it, mass receives one in the reorder only (elsewhere it is an input of
// the node without a gradient, so that outputs require one wherever any input does), and kernels run on the current
// stream of the tensors' device.
#include <torch/extension.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include "../../include/npa_b200.h"

namespace {

namespace py = pybind11;
using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// ---- status codes and argument checks --------------------------------------------------------
void check_status(int rc) {
    if (rc == NPA_OK) return;
    const std::string text = npa_last_error();
    if (rc == NPA_ERR_UNSUPPORTED) throw std::invalid_argument(text);  // ValueError
    throw std::runtime_error(text);
}

std::string shape_text(at::IntArrayRef s) {
    std::string t = "(";
    for (size_t k = 0; k < s.size(); ++k) t += (k ? ", " : "") + std::to_string(s[k]);
    return t + ")";
}

// The checks of the reference's binding: wrong dtype, device or layout is a TypeError (nanobind), a
// wrong shape a RuntimeError with the reference's wording (sphops/utils.cuh:526-567).
void require(const Tensor &t, at::IntArrayRef shape, const char *name, at::ScalarType dtype = at::kFloat) {
    if (!t.is_cuda() || t.scalar_type() != dtype || !t.is_contiguous())
        throw py::type_error(std::string(name) + ": incompatible function arguments; expected a contiguous CUDA tensor of dtype " +
                             (dtype == at::kFloat ? "torch.float32" : "torch.int32") + ", got tensor(dtype=" + toString(t.scalar_type()) +
                             ", device=" + t.device().str() + ", contiguous=" + (t.is_contiguous() ? "True" : "False") + ")");
    if (t.dim() != (int64_t)shape.size())
        throw std::runtime_error(std::string(name) + " must have " + std::to_string(shape.size()) + " dimensions, got " + std::to_string(t.dim()));
    if (t.sizes() != shape)
        throw std::runtime_error(std::string(name) + " must have shape " + shape_text(shape) + ", got " + shape_text(t.sizes()));
}

const float *fptr(const Tensor &t) { return t.defined() ? t.const_data_ptr<float>() : nullptr; }
float *fmut(const Tensor &t) { return t.defined() ? t.mutable_data_ptr<float>() : nullptr; }
const int32_t *iptr(const Tensor &t) { return t.defined() ? t.const_data_ptr<int32_t>() : nullptr; }
int32_t *imut(const Tensor &t) { return t.defined() ? t.mutable_data_ptr<int32_t>() : nullptr; }
Tensor or_none(const OptTensor &t) { return t.has_value() ? *t : Tensor(); }
// An upstream gradient as the kernels read it: contiguous, and at an address that any vector load can use.
Tensor solid(const Tensor &t) {
    if (!t.defined()) return t;
    const Tensor c = t.contiguous();
    return (uintptr_t)c.const_data_ptr() % 16 ? c.clone() : c;
}
void *stream_of(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
// Contiguous memory on the device of another tensor, without the dispatcher: a call here makes 13 to 22 such tensors, and at::empty
// takes 1.6 us for one, twice what the allocator and the tensor object take (host time of a step 159 -> 151 us, of 22 per-operator tensors 237 -> 224).
Tensor fresh(const Tensor &like, at::IntArrayRef shape, at::ScalarType type) {
    return at::detail::empty_cuda(shape, type, like.device(), std::nullopt);
}
Tensor floats(const Tensor &like, at::IntArrayRef shape) { return fresh(like, shape, at::kFloat); }
Tensor ints(const Tensor &like, at::IntArrayRef shape) { return fresh(like, shape, at::kInt); }
Tensor blank(const Tensor &like) { return floats(like, like.sizes()); }
bool wants_grad(const Tensor &t) { return t.defined() && t.requires_grad(); }
// No operator here has a forward-mode derivative: a dual number would lose its tangent without a word.
template <typename... In>
void refuse_tangents(const char *name, const In &...inputs) {
    TORCH_CHECK_NOT_IMPLEMENTED(!((inputs.defined() && inputs._fw_grad(0).defined()) || ...), name, " has no forward-mode derivative");
}

// ---- a grid and the snapshot of one binning pass -------------------------------------------------
struct Grid {
    npa_grid g;
    int64_t cells, max_blocks, scratch_bytes, B, N, P, D;
    Tensor scratch;  // work arrays of the binning, allocated once per device

    explicit Grid(uintptr_t descriptor) : g(*reinterpret_cast<const npa_grid *>(descriptor)) {
        cells = npa_grid_num_cells(&g);
        if (cells < 0) check_status((int)cells);
        max_blocks = npa_grid_max_blocks(&g);
        scratch_bytes = npa_grid_scratch_bytes(&g);
        B = g.batch; N = g.particles; D = g.dim; P = g.dim == 2 ? 2 : 4;
    }
    void positions(const Tensor &x, const char *name) const { require(x, {B, N, P}, name); }
    void rows(const Tensor &t, const char *name) const { require(t, {B, N}, name); }
    void rows(const Tensor &t, const char *name, int64_t c) const { require(t, {B, N, c}, name); }
    void snapshot(const Tensor &offs, const Tensor &info) const {
        require(offs, {B * cells + 1}, "bin_offsets", at::kInt);
        require(info, {max_blocks, 4}, "block_info", at::kInt);
    }
    void bin(const Tensor &x, const Tensor &perm, const Tensor &offs, const Tensor &info, void *st) {
        check_status(npa_grid_build(&g, fptr(x), imut(perm), imut(offs), imut(info), scratch_for(x), scratch_bytes, st));
    }
    void *scratch_for(const Tensor &x) {
        if (!scratch.defined() || scratch.device() != x.device())
            scratch = at::empty({scratch_bytes}, at::TensorOptions().dtype(at::kByte).device(x.device()));
        return scratch.mutable_data_ptr();
    }
    void features(const Tensor &s, const char *name) const { require(s, {B, N, s.dim() == 3 ? s.size(2) : -1}, name); }
};
using GridPtr = std::shared_ptr<Grid>;

py::tuple instantiate(const GridPtr &grid, const Tensor &x) {
    Grid &g = *grid;
    g.positions(x, "positions");
    c10::cuda::CUDAGuard guard(x.device());
    Tensor perm = ints(x, {g.B, g.N}), offs = ints(x, {g.B * g.cells + 1}), info = ints(x, {g.max_blocks, 4});
    g.bin(x, perm, offs, info, stream_of(x));
    return py::make_tuple(offs, perm, info);
}

// ---- node plumbing ------------------------------------------------------------------------------
template <typename T, typename... In>
std::shared_ptr<T> node_for(const In &...inputs) {
    std::shared_ptr<T> n(new T(), torch::autograd::deleteNode);
    n->set_next_edges(torch::autograd::collect_next_edges(inputs...));
    return n;
}
template <typename... In>
bool recording(const In &...inputs) {
    return at::GradMode::is_enabled() && (wants_grad(inputs) || ...);
}

// What a backward reads of the forward is kept as SavedVariable, so that saved-tensor hooks see it: they move it to the
// host, or drop and recompute it (checkpointing), and changes in place are noticed.  Outside are the snapshot's arrays and
// neighbour lists that operators share: whether an operator finds lists may differ between a forward and its recomputation.
SavedVariable saved(const Tensor &t) { return SavedVariable(t, false); }

// What every node of a neighbour sweep keeps: the grid, the snapshot arrays, the neighbour lists.
struct SweepNode : Node {
    GridPtr grid;
    Tensor offs, info, pairs;
    SavedVariable x_, mass_;
    void keep(const GridPtr &g, const Tensor &o, const Tensor &i, const Tensor &p, const Tensor &x, const Tensor &mass) {
        grid = g; offs = o; info = i; pairs = p;
        x_ = saved(x);
        mass_ = saved(mass);
    }
    void release_variables() override {
        x_.reset_data(); mass_.reset_data();
        pairs = Tensor();
    }
    static int list_stride(const Tensor &pairs) { return pairs.defined() ? (int)pairs.size(2) : 0; }
};

struct Snap {  // arguments every sweep shares, checked
    GridPtr grid;
    Tensor offs, info, mass, pairs;
    Snap(const GridPtr &g, const Tensor &o, const Tensor &i, const OptTensor &m, const OptTensor &p)
        : grid(g), offs(o), info(i), mass(or_none(m)), pairs(or_none(p)) {
        grid->snapshot(offs, info);
        if (mass.defined()) grid->rows(mass, "mass");
        if (pairs.defined()) {
            require(pairs, {grid->B, grid->N, pairs.dim() == 3 ? pairs.size(2) : -1}, "pair_cache", at::kInt);
            if (pairs.size(2) < 2 || pairs.size(2) > 513)
                throw std::runtime_error("pair_cache must have between 2 and 513 columns, got " + std::to_string(pairs.size(2)));
            // The lists belong to the snapshot, which drops them with the next binning: an operator on another stream than the
            // one that recorded them may still be reading then (the caller never sees them, and could not do this).
            c10::cuda::CUDACachingAllocator::recordStream(pairs.storage().data_ptr(), c10::cuda::getCurrentCUDAStream(pairs.device().index()));
        }
    }
    int stride() const { return pairs.defined() ? (int)pairs.size(2) : 0; }
};

Tensor new_lists(const Grid &g, const Tensor &like, int64_t columns) {
    return columns ? ints(like, {g.B, g.N, columns}) : Tensor();
}

// The cell-tile engine, when it is switched on for backward sweeps, searches for its pairs itself.
bool by_lists(const Tensor &pairs) { return pairs.defined() && !npa_tile_enabled(1); }

// Work memory of a backward over lists.
Tensor list_scratch(const Grid &g, const Tensor &like, int64_t channels) {
    const int64_t bytes = npa_lists_backward_scratch_bytes(&g.g, (int)channels);
    if (bytes < 0) check_status((int)bytes);
    return floats(like, {bytes / 4});
}

// ---- reorder into cell order (Permute, sph.py:127-184) ---------------------------------------------
struct ReorderNode : Node {
    GridPtr grid;
    Tensor perm;
    std::vector<int64_t> xs, ss, ms;
    at::TensorOptions opt;
    variable_list apply(variable_list &&g) override {
        c10::cuda::CUDAGuard guard(perm.device());
        auto upstream = [&](const Tensor &t, const std::vector<int64_t> &shape, bool need) {
            if (!need) return Tensor();
            return t.defined() ? solid(t) : at::zeros(shape, opt);
        };
        const bool nx = should_compute_output(0), ns = should_compute_output(1), nm = !ms.empty() && should_compute_output(2);
        const Tensor gx = upstream(g[0], xs, nx), gs = upstream(g[1], ss, ns), gm = ms.empty() ? Tensor() : upstream(g[2], ms, nm);
        Tensor ox = nx ? blank(gx) : Tensor(), os = ns ? blank(gs) : Tensor(), om = nm ? blank(gm) : Tensor();
        const int C = (int)ss[2];
        const bool feats = ns && C > 0;
        if (nx || feats || nm)
            check_status(npa_unbin_particles(&grid->g, C, fptr(gx), feats ? fptr(gs) : nullptr, fptr(gm), iptr(perm), fmut(ox),
                                             feats ? fmut(os) : nullptr, fmut(om), stream_of(perm)));
        return {ox, os, om};
    }
};

py::tuple reorder(const GridPtr &grid, const Tensor &perm, const Tensor &x, const Tensor &s, const OptTensor &mass_) {
    refuse_tangents("bin_particles", x, s, or_none(mass_));
    const Tensor mass = or_none(mass_);
    Grid &g = *grid;
    g.positions(x, "input_positions");
    g.features(s, "input_state");
    if (mass.defined()) g.rows(mass, "input_mass");
    require(perm, {g.B, g.N}, "permutation", at::kInt);
    c10::cuda::CUDAGuard guard(x.device());
    const int C = (int)s.size(2);
    Tensor xo = blank(x), so = blank(s), mo = mass.defined() ? blank(mass) : Tensor();
    check_status(npa_bin_particles(&g.g, C, fptr(x), C ? fptr(s) : nullptr, fptr(mass), iptr(perm), fmut(xo), C ? fmut(so) : nullptr, fmut(mo),
                                   stream_of(x)));
    if (recording(x, s, mass)) {
        auto n = node_for<ReorderNode>(x, s, mass);
        n->grid = grid; n->perm = perm; n->opt = x.options().requires_grad(false);
        n->xs = x.sizes().vec(); n->ss = s.sizes().vec();
        if (mass.defined()) n->ms = mass.sizes().vec();
        variable_list outs = {xo, so};
        if (mass.defined()) outs.push_back(mo);
        torch::autograd::set_history(outs, n);
    }
    return mass.defined() ? py::make_tuple(xo, so, mo) : py::make_tuple(xo, so);
}

py::tuple unreorder(const GridPtr &grid, const Tensor &perm, const Tensor &x, const Tensor &s, const OptTensor &mass_) {
    const Tensor mass = or_none(mass_);
    Grid &g = *grid;
    g.positions(x, "grad_output_positions");
    g.features(s, "grad_output_state");
    if (mass.defined()) g.rows(mass, "grad_output_mass");
    require(perm, {g.B, g.N}, "permutation", at::kInt);
    c10::cuda::CUDAGuard guard(x.device());
    const int C = (int)s.size(2);
    Tensor xo = blank(x), so = blank(s), mo = mass.defined() ? blank(mass) : Tensor();
    check_status(npa_unbin_particles(&g.g, C, fptr(x), C ? fptr(s) : nullptr, fptr(mass), iptr(perm), fmut(xo), C ? fmut(so) : nullptr, fmut(mo),
                                     stream_of(x)));
    return mass.defined() ? py::make_tuple(xo, so, mo) : py::make_tuple(xo, so);
}

// ---- neighbour count ------------------------------------------------------------------------------------
// Piecewise constant in the positions: the node is there because a caller may ask the output for its graph, and gives none.
struct CountNode : Node {
    variable_list apply(variable_list &&) override { return {Tensor()}; }
};

Tensor count(const GridPtr &grid, const Tensor &offs, const Tensor &info, const Tensor &x) {
    refuse_tangents("count", x);
    const Grid &g = *grid;
    g.snapshot(offs, info);
    g.positions(x, "binned_positions");
    c10::cuda::CUDAGuard guard(x.device());
    Tensor out = floats(x, {g.B, g.N});
    check_status(npa_count_forward(&g.g, fptr(x), fmut(out), iptr(offs), iptr(info), stream_of(x)));
    if (recording(x)) torch::autograd::set_history(out, node_for<CountNode>(x));
    return out;
}

// ---- density and density gradient -------------------------------------------------------------------
struct DensityNode : SweepNode {
    bool has_rho, has_dg;
    variable_list apply(variable_list &&g) override {
        const Tensor x = x_.unpack(), mass = mass_.unpack();
        const Tensor g_rho = has_rho ? solid(g[0]) : Tensor(), g_dg = has_dg ? solid(g[has_rho ? 1 : 0]) : Tensor();
        if ((!g_rho.defined() && !g_dg.defined()) || !should_compute_output(0)) return {Tensor(), Tensor()};
        c10::cuda::CUDAGuard guard(x.device());
        Tensor gx = blank(x);
        check_status(npa_density_chain_backward(&grid->g, fptr(x), fptr(mass), fptr(g_rho), nullptr, fptr(g_dg), fmut(gx), 0, iptr(offs),
                                                iptr(info), iptr(pairs), list_stride(pairs), stream_of(x)));
        return {gx, Tensor()};
    }
};

// (rho, density gradient); either may be left out.  `pairs` holds lists of these positions to be used by the backward:
// with `write` the forward records them first.
py::tuple density(const GridPtr &grid, const Tensor &offs, const Tensor &info, const Tensor &x, const OptTensor &mass, const OptTensor &pairs,
                  bool want_rho, bool want_dg, bool write) {
    refuse_tangents("density", x, or_none(mass));
    Snap sn(grid, offs, info, mass, pairs);
    Grid &g = *grid;
    g.positions(x, "binned_positions");
    c10::cuda::CUDAGuard guard(x.device());
    Tensor rho = want_rho ? floats(x, {g.B, g.N}) : Tensor(), dg = want_dg ? floats(x, {g.B, g.N, g.D}) : Tensor();
    if (want_rho)
        check_status(npa_perception_forward(&g.g, 0, fptr(x), fptr(sn.mass), nullptr, fmut(rho), nullptr, fmut(dg), nullptr, nullptr, nullptr,
                                            iptr(offs), iptr(info), write ? imut(sn.pairs) : nullptr, write ? sn.stride() : 0, stream_of(x)));
    else if (sn.pairs.defined())
        check_status(npa_density_gradient_forward_lists(&g.g, fptr(x), fptr(sn.mass), fmut(dg), iptr(offs), iptr(sn.pairs), sn.stride(), stream_of(x)));
    else
        check_status(npa_density_gradient_forward(&g.g, fptr(x), fptr(sn.mass), fmut(dg), iptr(offs), iptr(info), stream_of(x)));
    if (recording(x, sn.mass)) {
        auto n = node_for<DensityNode>(x, sn.mass);
        n->keep(grid, offs, info, sn.pairs, x, sn.mass);
        n->has_rho = want_rho; n->has_dg = want_dg;
        if (want_rho) torch::autograd::set_history(rho, n);
        if (want_dg) torch::autograd::set_history(dg, n);
    }
    return py::make_tuple(want_rho ? py::cast(rho) : py::none(), want_dg ? py::cast(dg) : py::none());
}

// ---- blur and feature gradient ----------------------------------------------------------------------
struct FeatureNode : SweepNode {
    SavedVariable s_, rho_;
    bool has_blur, has_grad;
    variable_list apply(variable_list &&g) override {
        const Tensor x = x_.unpack(), s = s_.unpack(), rho = rho_.unpack(), mass = mass_.unpack();
        const bool nx = should_compute_output(0), ns = should_compute_output(1), nr = should_compute_output(2);
        const Tensor gb = has_blur ? solid(g[0]) : Tensor(), gg = has_grad ? solid(g[has_blur ? 1 : 0]) : Tensor();
        if ((!gb.defined() && !gg.defined()) || !(nx || ns || nr)) return variable_list(4);
        c10::cuda::CUDAGuard guard(x.device());
        const int C = (int)s.size(2);
        auto out = [&](const Tensor &t, bool need) { return !need ? Tensor() : C ? blank(t) : at::zeros_like(t); };  // no features: no gradient
        Tensor gx = out(x, nx), gs = out(s, ns), gr = out(rho, nr);
        if (C > 0 && by_lists(pairs)) {
            Tensor work = list_scratch(*grid, s, C);
            check_status(npa_blur_gradient_backward_lists(&grid->g, C, fptr(x), fptr(rho), fptr(mass), fptr(s), fptr(gb), fptr(gg), fmut(gx), fmut(gs),
                                                          fmut(gr), work.mutable_data_ptr(), work.numel() * 4, iptr(offs), iptr(pairs), list_stride(pairs),
                                                          stream_of(x)));
        } else if (C > 0) {
            check_status(npa_blur_gradient_backward(&grid->g, C, fptr(x), fptr(rho), fptr(mass), fptr(s), fptr(gb), fptr(gg), fmut(gx), fmut(gs),
                                                    fmut(gr), iptr(offs), iptr(info), iptr(pairs), list_stride(pairs), stream_of(x)));
        }
        return {gx, gs, gr, Tensor()};
    }
    void release_variables() override {
        SweepNode::release_variables();
        s_.reset_data(); rho_.reset_data();
    }
};

// (blur, gradient, moment matrix) of the requested set; the moment matrix carries no gradient here.  `pairs`: neighbour
// lists, valid when `have_lists`, otherwise recorded by this sweep.
py::tuple blur_gradient(const GridPtr &grid, const Tensor &offs, const Tensor &info, const Tensor &x, const Tensor &rho, const Tensor &s,
                        const OptTensor &mass, const OptTensor &pairs, bool have_lists, bool want_blur, bool want_grad, bool want_moment) {
    refuse_tangents("blur / gradient", x, rho, s, or_none(mass));
    Snap sn(grid, offs, info, mass, pairs);
    Grid &g = *grid;
    g.positions(x, "binned_positions");
    g.rows(rho, "rho");
    g.features(s, "state_in");
    const int64_t C = s.size(2);
    c10::cuda::CUDAGuard guard(x.device());
    Tensor blur = want_blur ? blank(s) : Tensor(), grad = want_grad ? floats(s, {g.B, g.N, C, g.D}) : Tensor();
    Tensor moment = want_moment ? floats(s, {g.B, g.N, g.D, g.D}) : Tensor();
    if (C > 0)
        check_status(npa_blur_gradient_forward(&g.g, (int)C, fptr(x), fptr(rho), fptr(sn.mass), fptr(s), fmut(blur), fmut(grad), fmut(moment),
                                               iptr(offs), iptr(info), imut(sn.pairs), sn.stride(), have_lists ? 1 : 0, stream_of(x)));
    if (recording(x, s, rho, sn.mass)) {
        auto n = node_for<FeatureNode>(x, s, rho, sn.mass);
        n->keep(grid, offs, info, sn.pairs, x, sn.mass);
        n->s_ = saved(s);
        n->rho_ = saved(rho);
        n->has_blur = want_blur; n->has_grad = want_grad;
        if (want_blur) torch::autograd::set_history(blur, n);
        if (want_grad) torch::autograd::set_history(grad, n);
    }
    auto cast = [](const Tensor &t) -> py::object { return t.defined() ? py::cast(t) : py::none(); };
    return py::make_tuple(cast(blur), cast(grad), cast(moment));
}

// gradient_hybrid (sph.py:474-484) over neighbour lists: the value is gradient . inv(moment), the gradient that of the
// raw operator.
Tensor gradient_hybrid(const GridPtr &grid, const Tensor &offs, const Tensor &info, const Tensor &x, const Tensor &rho, const Tensor &s,
                       const OptTensor &mass, const Tensor &pairs, double rtol) {
    refuse_tangents("gradient_hybrid", x, rho, s, or_none(mass));
    Snap sn(grid, offs, info, mass, pairs);
    Grid &g = *grid;
    g.positions(x, "binned_positions");
    g.rows(rho, "rho");
    g.features(s, "state_in");
    const int64_t C = s.size(2);
    c10::cuda::CUDAGuard guard(x.device());
    Tensor out = floats(s, {g.B, g.N, C, g.D});
    if (C > 0)
        check_status(npa_gradient_hybrid_forward_lists(&g.g, (int)C, fptr(x), fptr(rho), fptr(sn.mass), fptr(s), (float)rtol, fmut(out), iptr(offs),
                                                       iptr(sn.pairs), sn.stride(), stream_of(x)));
    if (recording(x, s, rho, sn.mass)) {
        auto n = node_for<FeatureNode>(x, s, rho, sn.mass);
        n->keep(grid, offs, info, sn.pairs, x, sn.mass);
        n->s_ = saved(s);
        n->rho_ = saved(rho);
        n->has_blur = false; n->has_grad = true;
        torch::autograd::set_history(out, n);
    }
    return out;
}

// ---- moment matrix -----------------------------------------------------------------------------------
struct MomentNode : SweepNode {
    SavedVariable rho_;
    variable_list apply(variable_list &&g) override {
        const Tensor x = x_.unpack(), rho = rho_.unpack(), mass = mass_.unpack();
        const bool nx = should_compute_output(0), nr = should_compute_output(1);
        if (!g[0].defined() || !(nx || nr)) return variable_list(3);
        c10::cuda::CUDAGuard guard(x.device());
        Tensor gx = nx ? blank(x) : Tensor(), gr = nr ? blank(rho) : Tensor();
        check_status(npa_moment_matrix_backward(&grid->g, fptr(x), fptr(rho), fptr(mass), fptr(solid(g[0])), fmut(gx), fmut(gr), iptr(offs),
                                                iptr(info), stream_of(x)));
        return {gx, gr, Tensor()};
    }
    void release_variables() override {
        SweepNode::release_variables();
        rho_.reset_data();
    }
};

Tensor moment_matrix(const GridPtr &grid, const Tensor &offs, const Tensor &info, const Tensor &x, const Tensor &rho, const OptTensor &mass) {
    refuse_tangents("moment_matrix", x, rho, or_none(mass));
    Snap sn(grid, offs, info, mass, std::nullopt);
    Grid &g = *grid;
    g.positions(x, "binned_positions");
    g.rows(rho, "rho");
    c10::cuda::CUDAGuard guard(x.device());
    Tensor out = floats(x, {g.B, g.N, g.D, g.D});
    check_status(npa_moment_matrix_forward(&g.g, fptr(x), fptr(rho), fptr(sn.mass), fmut(out), iptr(offs), iptr(info), stream_of(x)));
    if (recording(x, rho, sn.mass)) {
        auto n = node_for<MomentNode>(x, rho, sn.mass);
        n->keep(grid, offs, info, Tensor(), x, sn.mass);
        n->rho_ = saved(rho);
        torch::autograd::set_history(out, n);
    }
    return out;
}

// ---- the same from a gradient and a moment matrix that are there already ------------------------------------
struct StraightThroughNode : Node {
    variable_list apply(variable_list &&g) override { return {g[0]}; }
};

Tensor corrected_gradient(const Tensor &raw, const Tensor &moment, double rtol) {
    refuse_tangents("gradient_hybrid", raw, moment);
    const int64_t B = raw.size(0), N = raw.size(1), C = raw.size(2), D = raw.size(3);
    require(raw, {B, N, C, D}, "gradient");
    require(moment, {B, N, D, D}, "moment_matrix");
    c10::cuda::CUDAGuard guard(raw.device());
    Tensor out = blank(raw);
    if (out.numel() > 0)
        check_status(npa_corrected_gradient((int)D, B * N, (int)C, fptr(raw), fptr(moment), (float)rtol, fmut(out), stream_of(raw)));
    if (recording(raw)) {
        auto n = node_for<StraightThroughNode>(raw);
        torch::autograd::set_history(out, n);
    }
    return out;
}

// ---- the fused perception step -------------------------------------------------------------------------
struct PerceptionNode : SweepNode {
    SavedVariable s_, rho_, packed_, pairs_;  // packed: (x, y, z, m / rho) records of the density sweep
    bool has_dg;
    variable_list apply(variable_list &&g) override {
        const Tensor x = x_.unpack(), s = s_.unpack(), rho = rho_.unpack(shared_from_this()), mass = mass_.unpack(), packed = packed_.unpack(),
                     pairs = pairs_.unpack();
        const bool nx = should_compute_output(0), ns = should_compute_output(1);
        if (!(nx || ns)) return variable_list(3);
        const Tensor g_rho = nx ? solid(g[0]) : Tensor(), gb = solid(g[1]), gg = solid(g[2]), g_dg = nx && has_dg ? solid(g[3]) : Tensor();
        c10::cuda::CUDAGuard guard(x.device());
        Tensor gx = nx ? blank(x) : Tensor(), gs = ns ? blank(s) : Tensor();
        if (by_lists(pairs)) {
            Tensor work = list_scratch(*grid, s, s.size(2));
            check_status(npa_perception_backward_lists(&grid->g, (int)s.size(2), fptr(x), fptr(mass), fptr(s), fptr(rho), fptr(packed), fptr(g_rho),
                                                       fptr(gb), fptr(gg), fptr(g_dg), fmut(gx), fmut(gs), work.mutable_data_ptr(), work.numel() * 4,
                                                       iptr(offs), iptr(pairs), list_stride(pairs), stream_of(x)));
            return {gx, gs, Tensor()};
        }
        Tensor gr = nx ? blank(rho) : Tensor();
        check_status(npa_perception_backward(&grid->g, (int)s.size(2), fptr(x), fptr(mass), fptr(s), fptr(rho), fptr(g_rho), fptr(gb), fptr(gg),
                                             fptr(g_dg), fmut(gx), fmut(gs), fmut(gr), iptr(offs), iptr(info), iptr(pairs), list_stride(pairs), stream_of(x)));
        return {gx, gs, Tensor()};
    }
    void release_variables() override {
        SweepNode::release_variables();
        s_.reset_data(); rho_.reset_data(); packed_.reset_data(); pairs_.reset_data();
    }
};

py::tuple perception(const GridPtr &grid, const Tensor &offs, const Tensor &info, const Tensor &x, const Tensor &s, const OptTensor &mass,
                     bool want_dg, int64_t columns) {
    refuse_tangents("perceive", x, s, or_none(mass));
    Snap sn(grid, offs, info, mass, std::nullopt);
    Grid &g = *grid;
    g.positions(x, "binned_positions");
    g.features(s, "state_in");
    const int64_t C = s.size(2);
    if (C == 0) columns = 0;  // without features the density is all there is
    c10::cuda::CUDAGuard guard(x.device());
    const bool record = recording(x, s, sn.mass);
    Tensor rho = floats(x, {g.B, g.N}), blur = blank(s), grad = floats(s, {g.B, g.N, C, g.D});
    Tensor dg = want_dg ? floats(x, {g.B, g.N, g.D}) : Tensor(), pairs = new_lists(g, x, columns);
    Tensor packed = columns ? floats(x, {g.B, g.N, 4}) : Tensor();
    if (columns)
        check_status(npa_perception_forward_lists(&g.g, (int)C, fptr(x), fptr(sn.mass), fptr(s), fmut(rho), fmut(dg), fmut(blur), fmut(grad),
                                                  fmut(packed), iptr(offs), iptr(info), imut(pairs), (int)columns, stream_of(x)));
    else
        check_status(npa_perception_forward(&g.g, (int)C, fptr(x), fptr(sn.mass), fptr(s), fmut(rho), nullptr, fmut(dg), fmut(blur), fmut(grad),
                                            nullptr, iptr(offs), iptr(info), nullptr, 0, stream_of(x)));
    if (record) {
        auto n = node_for<PerceptionNode>(x, s, sn.mass);
        n->keep(grid, offs, info, Tensor(), x, sn.mass);
        n->pairs_ = saved(pairs);
        n->s_ = saved(s);
        n->has_dg = want_dg;
        n->packed_ = saved(packed);
        torch::autograd::set_history(rho, n);
        torch::autograd::set_history(blur, n);
        torch::autograd::set_history(grad, n);
        if (want_dg) torch::autograd::set_history(dg, n);
        n->rho_ = SavedVariable(rho, true);
    }
    return want_dg ? py::make_tuple(rho, blur, grad, dg) : py::make_tuple(rho, blur, grad);
}

// ---- the packed perception row ---------------------------------------------------------------------------
struct PackedNode : SweepNode {
    SavedVariable s_, rho_, rho_grad_, vgrad_, packed_, pairs_;
    float coef, dg_scale;
    bool ln_grad, ln_dg;
    variable_list apply(variable_list &&g) override {
        const Tensor x = x_.unpack(), s = s_.unpack(), mass = mass_.unpack(), rho = rho_.unpack(), rho_grad = rho_grad_.unpack(), vgrad = vgrad_.unpack(),
                     packed = packed_.unpack(), pairs = pairs_.unpack();
        const bool nx = should_compute_output(0), ns = should_compute_output(1);
        if (!g[0].defined() || !(nx || ns)) return variable_list(3);
        c10::cuda::CUDAGuard guard(x.device());
        const Tensor gz = solid(g[0]);
        if (by_lists(pairs)) {
            Tensor work = list_scratch(*grid, s, s.size(2)), gx = nx ? blank(x) : Tensor(), gs = ns ? blank(s) : Tensor();
            check_status(npa_perceive_features_backward_lists(&grid->g, (int)s.size(2), fptr(x), fptr(mass), fptr(s), fptr(rho), fptr(rho_grad),
                                                              fptr(vgrad), fptr(packed), fptr(gz), coef, dg_scale, ln_grad, ln_dg, nullptr, fmut(gx), fmut(gs),
                                                              work.mutable_data_ptr(), work.numel() * 4, iptr(offs), iptr(pairs), list_stride(pairs),
                                                              stream_of(x)));
            return {gx, gs, Tensor()};
        }
        const int64_t n = s.numel(), D = grid->D, rows = rho.numel();
        // dL/dblur and dL/dgradient of the rows, and with position gradients the two per-particle upstreams, in one buffer
        Tensor work = floats(s, {n * (1 + D) + (nx ? rows * (1 + D) : 0)});
        float *gb = fmut(work), *gg = gb + n, *g_dg = nx ? gg + n * D : nullptr, *gr = nx ? g_dg + rows * D : nullptr;
        Tensor gx = nx ? blank(x) : Tensor(), gs = blank(s);
        check_status(npa_perceive_features_backward(&grid->g, (int)s.size(2), fptr(x), fptr(mass), fptr(s), fptr(rho), fptr(rho_grad), fptr(vgrad),
                                                    fptr(gz), coef, dg_scale, ln_grad, ln_dg, gb, gg, g_dg, gr, fmut(gx), fmut(gs), iptr(offs),
                                                    iptr(info), iptr(pairs), list_stride(pairs), stream_of(x)));
        return {gx, ns ? gs : Tensor(), Tensor()};
    }
    void release_variables() override {
        SweepNode::release_variables();
        s_.reset_data(); rho_.reset_data(); rho_grad_.reset_data(); vgrad_.reset_data(); packed_.reset_data(); pairs_.reset_data();
    }
};

Tensor packed_perception(const GridPtr &grid, const Tensor &offs, const Tensor &info, const Tensor &x, const Tensor &s, const OptTensor &mass,
                         double coef, double dg_scale, double inv_tol, bool ln_grad, bool ln_dg, int64_t columns) {
    refuse_tangents("perceive_features", x, s, or_none(mass));
    Snap sn(grid, offs, info, mass, std::nullopt);
    Grid &g = *grid;
    g.positions(x, "binned_positions");
    g.features(s, "state_in");
    const int64_t C = s.size(2), D = g.D;
    c10::cuda::CUDAGuard guard(x.device());
    const bool record = recording(x, s, sn.mass);
    Tensor rho = floats(x, {g.B, g.N}), rho_grad = floats(x, {g.B, g.N, D}), z = floats(s, {g.B, g.N, 2 * C + C * D + D});
    Tensor vgrad = record ? floats(s, {g.B, g.N, C, D}) : Tensor(), pairs = new_lists(g, x, columns);
    Tensor packed = columns ? floats(x, {g.B, g.N, 4}) : Tensor();
    check_status(npa_perceive_features_forward_lists(&g.g, (int)C, fptr(x), fptr(sn.mass), fptr(s), (float)coef, (float)dg_scale, (float)inv_tol,
                                                     ln_grad, ln_dg, fmut(rho), fmut(rho_grad), fmut(z), fmut(vgrad), fmut(packed), iptr(offs),
                                                     iptr(info), imut(pairs), pairs.defined() ? (int)columns : 0, stream_of(x)));
    if (record) {
        auto n = node_for<PackedNode>(x, s, sn.mass);
        n->keep(grid, offs, info, Tensor(), x, sn.mass);
        n->pairs_ = saved(pairs);
        n->s_ = saved(s);
        n->rho_ = saved(rho); n->rho_grad_ = saved(rho_grad); n->vgrad_ = saved(vgrad); n->packed_ = saved(packed);
        n->coef = (float)coef; n->dg_scale = (float)dg_scale; n->ln_grad = ln_grad; n->ln_dg = ln_dg;
        torch::autograd::set_history(z, n);
    }
    return z;
}

// ---- the Euler update --------------------------------------------------------------------------------------
struct StepNode : Node {
    GridPtr grid;
    SavedVariable y_, mask_;
    int C;
    float alpha, dt, below;  // below >= 0: the mask is uniforms, a particle updates where its value is below it
    variable_list apply(variable_list &&g) override {
        const Tensor y = y_.unpack(), mask = mask_.unpack(), gx = solid(g[0]), gs = solid(g[1]);
        Tensor gy;
        if (should_compute_output(0) && (gx.defined() || gs.defined())) {
            c10::cuda::CUDAGuard guard(y.device());
            gy = blank(y);
            check_status(mask.defined() && below >= 0.f
                             ? npa_step_update_backward_masked(&grid->g, fptr(y), fptr(mask), below, C, alpha, dt, fptr(gx), fptr(gs), fmut(gy), stream_of(y))
                             : npa_step_update_backward(&grid->g, fptr(y), fptr(mask), C, alpha, dt, fptr(gx), fptr(gs), fmut(gy), stream_of(y)));
        }
        return {gy, should_compute_output(1) ? gx : Tensor(), should_compute_output(2) ? gs : Tensor(), Tensor()};
    }
    void release_variables() override {
        y_.reset_data(); mask_.reset_data();
    }
};

py::tuple step_update(const GridPtr &grid, const Tensor &y, const Tensor &x, const Tensor &s, const OptTensor &mask_, double alpha, double dt, bool wrap,
                      double below) {
    refuse_tangents("step_update", y, x, s, or_none(mask_));
    Grid &g = *grid;
    const Tensor mask = or_none(mask_);
    g.positions(x, "binned_positions");
    g.features(s, "state_in");
    g.rows(y, "y", g.D + s.size(2));
    if (mask.defined()) g.rows(mask, "mask");
    c10::cuda::CUDAGuard guard(x.device());
    Tensor xo = blank(x), so = blank(s);
    check_status(mask.defined() && below >= 0.0
                     ? npa_step_update_forward_masked(&g.g, fptr(y), fptr(x), fptr(s), fptr(mask), (float)below, (int)s.size(2), (float)alpha, (float)dt,
                                                      wrap, fmut(xo), fmut(so), stream_of(x))
                     : npa_step_update_forward(&g.g, fptr(y), fptr(x), fptr(s), fptr(mask), (int)s.size(2), (float)alpha, (float)dt, wrap, fmut(xo),
                                               fmut(so), stream_of(x)));
    if (recording(y, x, s, mask)) {
        auto n = node_for<StepNode>(y, x, s, mask);
        n->grid = grid; n->mask_ = saved(mask); n->C = (int)s.size(2); n->alpha = (float)alpha; n->dt = (float)dt; n->below = (float)below;
        n->y_ = saved(y);
        torch::autograd::set_history(xo, n);
        torch::autograd::set_history(so, n);
    }
    return py::make_tuple(xo, so);
}

// ---- the adaptation MLP on the tensor-memory kernels (mlp.py) -------------------------------------------------
constexpr int kHidden = 128;

// Gradients of the MLP's weights and bias from one kernel over the rows.
// (the tensor-memory kernel appends a column of ones to z, 176 columns in all)
int64_t weight_grad_scratch_floats(int64_t m, int64_t k, int64_t o) {
    return k < 176 ? npa_mlp_weight_grad_tcgen05_scratch_floats(m, (int)k, (int)o) : npa_mlp_weight_grad_scratch_floats(m, (int)k, (int)o);
}
void mlp_weight_grads(const float *z, const float *dh, const float *h, const float *dy, int64_t m, const Tensor &w1, const Tensor &w2,
                      float *scratch, Tensor &gw1, Tensor &gb1, Tensor &gw2, void *st, bool partial = false) {
    const int64_t k = w1.size(1), o = w2.size(0);
    gw1 = blank(w1);
    gw2 = blank(w2);
    gb1 = floats(w1, {kHidden});
    if (partial) {  // added up by npa_step_unbin
        check_status(npa_mlp_weight_grad_tcgen05_partial(z, dh, h, dy, m, (int)k, kHidden, (int)o, scratch, weight_grad_scratch_floats(m, k, o), st));
        return;
    }
    check_status((k < 176 ? npa_mlp_weight_grad_tcgen05 : npa_mlp_weight_grad)(z, dh, h, dy, m, (int)k, kHidden, (int)o, scratch,
                                                                               weight_grad_scratch_floats(m, k, o), fmut(gw1), fmut(gw2), fmut(gb1), st));
}

// The arrays that a node keeps to itself, in one allocation: offsets in floats, 256-byte aligned.
struct Slab {
    int64_t floats = 0;
    int64_t add(int64_t count) {
        const int64_t at = floats;
        floats += (count + 63) & ~(int64_t)63;
        return at;
    }
    Tensor make(const Tensor &like) const { return fresh(like, {floats}, at::kFloat); }
};

struct MlpNode : Node {
    SavedVariable z_, w1_, w2_, h_, dz_image_;  // h: hidden layer; dz_image: W1 as the tensor cores read it for dz = dh W1
    std::vector<int64_t> z_shape;
    variable_list apply(variable_list &&g) override {
        const Tensor z = z_.unpack(), w1 = w1_.unpack(), w2 = w2_.unpack(), h = h_.unpack(), dz_image = dz_image_.unpack();
        if (!g[0].defined()) return {Tensor(), Tensor(), Tensor(), Tensor()};
        c10::cuda::CUDAGuard guard(z.device());
        const Tensor dy = solid(g[0]);
        const int64_t k = z.size(-1), m = z.numel() / k, o = w2.size(0);
        void *st = stream_of(z);
        Tensor dh = floats(z, {m, kHidden});
        check_status(npa_mlp_hidden_grad(fptr(dy), fptr(w2), fptr(h), fmut(dh), m, kHidden, (int)o, w2.stride(0), w2.stride(1), st));
        Tensor gz, gw1, gb1, gw2;
        if (should_compute_output(0)) {
            gz = floats(z, z_shape);
            check_status(npa_linear_tcgen05_prepared(fptr(dh), dz_image.const_data_ptr(), dz_image.numel() * 4, fmut(gz), m, kHidden, (int)k, st));
        }
        const bool n1 = should_compute_output(1), nb = should_compute_output(2), n2 = should_compute_output(3);
        if (n1 || nb || n2) {
            Tensor scratch = floats(z, {weight_grad_scratch_floats(m, k, o)});
            mlp_weight_grads(fptr(z), fptr(dh), fptr(h), fptr(dy), m, w1, w2, fmut(scratch), gw1, gb1, gw2, st);
        }
        return {gz, n1 ? gw1 : Tensor(), nb ? gb1 : Tensor(), n2 ? gw2 : Tensor()};
    }
    void release_variables() override {
        z_.reset_data(); w1_.reset_data(); w2_.reset_data(); h_.reset_data(); dz_image_.reset_data();
    }
};

// y = relu(z W1^T + b1) W2^T over the rows of z; the caller has checked the shapes (mlp.supported).
Tensor mlp(const Tensor &z, const Tensor &w1, const Tensor &b1, const Tensor &w2) {
    refuse_tangents("the adaptation MLP", z, w1, b1, w2);
    c10::cuda::CUDAGuard guard(z.device());
    const int64_t k = z.size(-1), m = z.numel() / k, o = w2.size(0);
    std::vector<int64_t> shape = z.sizes().vec();
    shape.back() = o;
    const bool record = recording(z, w1, b1, w2);
    const int64_t bytes = npa_mlp_forward_tcgen05_scratch_bytes((int)k, (int)o);
    const int64_t dz_bytes = record && wants_grad(z) ? npa_linear_tcgen05_scratch_bytes(kHidden, (int)k) : 0;
    // without a backward the hidden layer stays in tensor memory
    Tensor y = floats(z, shape), h = record ? floats(z, {m, kHidden}) : Tensor(), image = floats(z, {bytes / 4});
    Tensor dz_image = dz_bytes ? floats(z, {dz_bytes / 4}) : Tensor();
    check_status(npa_mlp_forward_tcgen05_images(fptr(z), fptr(w1), fptr(b1), fptr(w2), fmut(h), fmut(y), m, (int)k, (int)o, w1.stride(0), w1.stride(1),
                                                w2.stride(0), w2.stride(1), image.mutable_data_ptr(), bytes, fmut(dz_image), dz_bytes,
                                                stream_of(z)));
    if (record) {
        auto n = node_for<MlpNode>(z, w1, b1, w2);
        n->z_ = saved(z); n->w1_ = saved(w1); n->w2_ = saved(w2);
        n->h_ = saved(h); n->dz_image_ = saved(dz_image); n->z_shape = z.sizes().vec();
        torch::autograd::set_history(y, n);
    }
    return y;
}

// ---- a whole Euler step as one node ------------------------------------------------------------------------------
// Binning, reorder, packed perception, MLP and update of stepping.step_euler: the same kernels as the operators above, but
// one crossing from Python and one node.  Four nodes cost ~60 us of host time more per training step (graph bookkeeping,
// the engine's hand-over between nodes, and the addition of the two gradients of the reordered states, which here rides
// the perception's backward).
struct EulerNode : Node {
    GridPtr grid;
    SavedVariable w1_, w2_, slab_, mask_;
    Tensor offs, perm, info;
    int64_t o_x, o_s, o_rho, o_dg, o_v, o_packed, o_z, o_h, o_y, o_dz, o_pairs;  // places in the slab, in floats
    int64_t C, columns, dz_bytes, slab_floats, y_pitch;  // y: rows that begin with the raw displacements
    float coef, dg_scale, alpha, dt, below;
    bool ln_grad, ln_dg, stop_pos, stop_state;
    bool rows;  // the image of W1 is in the order of npa_step_perceive_backward

    variable_list apply(variable_list &&g) override {
        const Tensor w1 = w1_.unpack(), w2 = w2_.unpack(), slab = solid(slab_.unpack()), mask = mask_.unpack();  // raise when the graph was released
        // (a hook may have had it elsewhere: the places below are only good in a block of the same size)
        TORCH_CHECK(slab.numel() == slab_floats && slab.scalar_type() == at::kFloat && slab.device() == w1.device(),
                    "a saved-tensor hook returned another tensor than the step had saved");
        const Tensor gx_new = solid(g[0]), gs_new = solid(g[1]);
        if (!gx_new.defined() && !gs_new.defined()) return variable_list(5);
        const float *kept = fptr(slab), *x_bin = kept + o_x, *s_bin = kept + o_s, *rho = kept + o_rho, *rho_grad = kept + o_dg, *vgrad = kept + o_v,
                    *packed = kept + o_packed, *z = kept + o_z, *h = kept + o_h, *y = kept + o_y, *dz_image = kept + o_dz;
        const int32_t *pairs = reinterpret_cast<const int32_t *>(kept + o_pairs);
        c10::cuda::CUDAGuard guard(slab.device());
        void *st = stream_of(slab);
        Grid &gr = *grid;
        npa_grid *gd = &gr.g;
        const int64_t k = w1.size(1), m = gr.B * gr.N, o = w2.size(0);
        const bool nx = should_compute_output(0), ns = should_compute_output(1);
        const bool n1 = should_compute_output(2), nb = should_compute_output(3), n2 = should_compute_output(4);
        const bool back_x = nx && !stop_pos, back_s = ns && !stop_state, back = back_x || back_s, weights = n1 || nb || n2;
        const int64_t work_bytes = !back ? 0 : rows ? npa_step_perceive_backward_scratch_bytes(gd, (int)C) : npa_lists_backward_scratch_bytes(gd, (int)C);
        if (work_bytes < 0) check_status((int)work_bytes);
        Slab l;
        const int64_t o_gy = l.add(m * o), o_dh = l.add(back || weights ? m * kHidden : 0), o_gz = l.add(back && !rows ? m * k : 0),
                      o_work = l.add(work_bytes / 4), o_gs = l.add(back_s ? m * C : 0),
                      o_scratch = l.add(weights ? weight_grad_scratch_floats(m, k, o) : 0);
        Tensor temporary = l.make(w1);
        float *t = fmut(temporary), *gy = t + o_gy, *dh = t + o_dh, *gz = t + o_gz;
        // update, and the MLP's output layer
        if (back || weights)
            check_status(npa_step_hidden_grad(gd, y, (int)y_pitch, fptr(mask), mask.defined(), below, (int)C, alpha, dt, fptr(gx_new), fptr(gs_new), fptr(w2), h, gy,
                                              dh, kHidden, w2.stride(0), w2.stride(1), st));
        Tensor gw1, gb1, gw2;
        const bool sum_later = weights && k < 176 && (nx || ns);  // the launch of the inverse reorder adds the partial sums up
        if (weights) mlp_weight_grads(z, dh, h, gy, m, w1, w2, t + o_scratch, gw1, gb1, gw2, st, sum_later);
        // perception, with the update's own gradient of the states added
        Tensor gx_bin = gx_new, none;
        const float *gs_bin = fptr(gs_new);
        if (back) {
            if (!rows) check_status(npa_linear_tcgen05_prepared(dh, dz_image, dz_bytes, gz, m, kHidden, (int)k, st));
            Tensor gxp = back_x ? floats(w1, {gr.B, gr.N, gr.P}) : Tensor();
            float *gsp = back_s ? t + o_gs : nullptr;
            if (rows) {  // (the positions want none)
                check_status(npa_step_perceive_backward(gd, (int)C, dh, dz_image, dz_bytes, x_bin, s_bin, rho, vgrad, packed, coef, ln_grad, fptr(gs_new), gsp,
                                                        t + o_work, work_bytes, iptr(offs), pairs, (int)columns, st));
            } else if (npa_tile_enabled(1)) {
                Tensor gsf = floats(w1, {gr.B, gr.N, C}), work = floats(w1, {m * (C + 1) * (1 + gr.D)});
                float *gb = fmut(work), *gg = gb + m * C, *g_dg = gg + m * C * gr.D, *g_rho = g_dg + m * gr.D;
                check_status(npa_perceive_features_backward(gd, (int)C, x_bin, nullptr, s_bin, rho, rho_grad, vgrad, gz, coef, dg_scale, ln_grad, ln_dg,
                                                            gb, gg, back_x ? g_dg : nullptr, back_x ? g_rho : nullptr, fmut(gxp), fmut(gsf), iptr(offs),
                                                            iptr(info), pairs, (int)columns, st));
                if (gs_new.defined()) gsf.add_(gs_new.detach());
                none = gsf;
                gsp = back_s ? fmut(gsf) : nullptr;
            } else {
                check_status(npa_perceive_features_backward_binned(gd, (int)C, x_bin, nullptr, s_bin, rho, rho_grad, vgrad, packed, gz, coef, dg_scale,
                                                                  ln_grad, ln_dg, fptr(gs_new), fmut(gxp), gsp, t + o_work, work_bytes, iptr(offs),
                                                                  pairs, (int)columns, st));
            }
            if (back_s) gs_bin = gsp;
            if (back_x) gx_bin = gx_bin.defined() ? gxp.add_(gx_bin) : gxp;
        }
        // back into the order of the inputs
        Tensor gx, gs;
        if (nx && !gx_bin.defined()) gx_bin = at::zeros({gr.B, gr.N, gr.P}, w1.options().requires_grad(false));
        if (ns && !gs_bin) {
            none = at::zeros({gr.B, gr.N, C}, w1.options().requires_grad(false));
            gs_bin = fptr(none);
        }
        if (nx) gx = floats(w1, {gr.B, gr.N, gr.P});
        if (ns) gs = floats(w1, {gr.B, gr.N, C});
        if (sum_later)
            check_status(npa_step_unbin(gd, (int)C, nx ? fptr(gx_bin) : nullptr, ns ? gs_bin : nullptr, iptr(perm), fmut(gx), fmut(gs), (int)k, (int)o,
                                        t + o_scratch, weight_grad_scratch_floats(m, k, o), fmut(gw1), fmut(gw2), fmut(gb1), st));
        else if (nx || ns)
            check_status(npa_unbin_particles(gd, (int)C, nx ? fptr(gx_bin) : nullptr, ns ? gs_bin : nullptr, nullptr, iptr(perm), fmut(gx), fmut(gs),
                                             nullptr, st));
        return {gx, gs, n1 ? gw1 : Tensor(), nb ? gb1 : Tensor(), n2 ? gw2 : Tensor()};
    }
    void release_variables() override {
        w1_.reset_data(); w2_.reset_data(); slab_.reset_data(); mask_.reset_data();
    }
};

// (x_new, s_new, bin_offsets, permutation, block_info, uniforms or None)
py::tuple euler_step(const GridPtr &grid, const Tensor &x, const Tensor &s, const Tensor &w1, const Tensor &b1, const Tensor &w2, double coef,
                     double dg_scale, double inv_tol, bool ln_grad, bool ln_dg, bool stop_pos, bool stop_state, double alpha, double dt,
                     double update_prob, bool wrap, int64_t columns) {
    refuse_tangents("step_euler", x, s, w1, b1, w2);
    Grid &g = *grid;
    g.positions(x, "positions");
    g.features(s, "input_state");
    c10::cuda::CUDAGuard guard(x.device());
    void *st = stream_of(x);
    const int64_t C = s.size(2), D = g.D, k = 2 * C + C * D + D, o = D + C, m = g.B * g.N;
    const bool record = recording(x, s, w1, b1, w2);
    const bool back = record && ((wants_grad(x) && !stop_pos) || (wants_grad(s) && !stop_state));  // a backward reaches the perception
    Tensor perm = ints(x, {g.B, g.N}), offs = ints(x, {g.B * g.cells + 1}), info = ints(x, {g.max_blocks, 4});
    const int64_t bytes = npa_mlp_forward_tcgen05_scratch_bytes((int)k, (int)o), rows_bytes = back && !npa_tile_enabled(1) && !(wants_grad(x) && !stop_pos) ? npa_step_rows_image_bytes(&g.g, (int)C) : 0;
    const bool rows = rows_bytes > 0;  // the backward takes dL/dz apart as it forms it
    const int64_t dz_bytes = rows ? rows_bytes : back ? npa_linear_tcgen05_scratch_bytes(kHidden, (int)k) : 0;
    const bool in_mlp = C % 4 == 0 && C <= 32;  // the update in the MLP's epilogue, which of y keeps only what the backward reads
    Slab l;
    const int64_t o_x = l.add(m * g.P), o_s = l.add(m * C), o_rho = l.add(m), o_dg = l.add(m * D), o_z = l.add(m * k), o_v = l.add(back ? m * C * D : 0),
                  o_packed = l.add(m * 4), o_y = l.add(!in_mlp ? m * o : record ? m * g.P : 0), o_h = l.add(record ? m * kHidden : 0), o_image = l.add(bytes / 4),
                  o_dz = l.add(dz_bytes / 4), o_pairs = l.add(m * columns);
    Tensor slab = l.make(x);
    float *t = fmut(slab), *x_bin = t + o_x, *s_bin = t + o_s, *rho = t + o_rho, *rho_grad = t + o_dg, *z = t + o_z, *packed = t + o_packed,
          *y = t + o_y, *vgrad = back ? t + o_v : nullptr, *h = record ? t + o_h : nullptr, *dz_image = dz_bytes ? t + o_dz : nullptr;
    int32_t *pairs = reinterpret_cast<int32_t *>(t + o_pairs);
    check_status(npa_step_bin(&g.g, (int)C, fptr(x), fptr(s), imut(perm), imut(offs), imut(info), g.scratch_for(x), g.scratch_bytes, x_bin, s_bin, fptr(w1),
                              fptr(w2), w1.stride(0), w1.stride(1), w2.stride(0), w2.stride(1), t + o_image, bytes, dz_image, dz_bytes, rows, st));
    check_status(npa_perceive_features_forward_lists(&g.g, (int)C, x_bin, nullptr, s_bin, (float)coef, (float)dg_scale, (float)inv_tol, ln_grad, ln_dg,
                                                     rho, rho_grad, z, vgrad, packed, iptr(offs), iptr(info), pairs, (int)columns, st));
    Tensor mask = update_prob < 1.0 ? at::rand({g.B, g.N, 1}, s.options().requires_grad(false)) : Tensor();
    Tensor xo = blank(x), so = blank(s);
    if (in_mlp) {
        check_status(npa_mlp_step_forward(&g.g, z, fptr(b1), h, (int)k, t + o_image, bytes, x_bin, s_bin, fptr(mask), mask.defined(), (float)update_prob,
                                          (int)C, (float)alpha, (float)dt, wrap, record ? y : nullptr, fmut(xo), fmut(so), st));
    } else {
        check_status(npa_mlp_forward_tcgen05_prepared(z, fptr(b1), h, y, m, (int)k, (int)o, t + o_image, bytes, st));
        check_status(mask.defined() ? npa_step_update_forward_masked(&g.g, y, x_bin, s_bin, fptr(mask), (float)update_prob, (int)C, (float)alpha, (float)dt,
                                                                     wrap, fmut(xo), fmut(so), st)
                                    : npa_step_update_forward(&g.g, y, x_bin, s_bin, nullptr, (int)C, (float)alpha, (float)dt, wrap, fmut(xo), fmut(so), st));
    }
    if (record) {
        auto n = node_for<EulerNode>(x, s, w1, b1, w2);
        n->grid = grid; n->offs = offs; n->perm = perm; n->info = info; n->slab_ = saved(slab); n->mask_ = saved(mask);
        n->o_x = o_x; n->o_s = o_s; n->o_rho = o_rho; n->o_dg = o_dg; n->o_v = o_v; n->o_packed = o_packed; n->o_z = o_z; n->o_h = o_h; n->o_y = o_y;
        n->o_dz = o_dz; n->o_pairs = o_pairs; n->slab_floats = l.floats; n->y_pitch = in_mlp ? g.P : o; n->C = C; n->columns = columns; n->dz_bytes = dz_bytes;
        n->w1_ = saved(w1); n->w2_ = saved(w2);
        n->coef = (float)coef; n->dg_scale = (float)dg_scale; n->alpha = (float)alpha; n->dt = (float)dt; n->below = (float)update_prob;
        n->ln_grad = ln_grad; n->ln_dg = ln_dg; n->stop_pos = stop_pos; n->stop_state = stop_state; n->rows = rows;
        torch::autograd::set_history(xo, n);
        torch::autograd::set_history(so, n);
    }
    return py::make_tuple(xo, so, offs, perm, info, mask.defined() ? py::cast(mask) : py::none());
}

// ---- splat renderer ------------------------------------------------------------------------------------------
struct SplatConsts {
    int img, radius, y_up, normalize;
    double sigma, lo, hi, scale;
};

struct SplatNode : Node {
    SavedVariable x_, color_;
    SplatConsts c;
    variable_list apply(variable_list &&g) override {
        const Tensor x = x_.unpack(), color = color_.unpack();
        const bool nx = should_compute_output(0), nc = should_compute_output(1);
        if (!g[0].defined() || !(nx || nc)) return {Tensor(), Tensor()};
        c10::cuda::CUDAGuard guard(x.device());
        const Tensor up = solid(g[0]);
        Tensor gx = nx ? blank(x) : Tensor(), gc = nc ? blank(color) : Tensor();
        check_status(npa_splat_backward(fptr(x), fptr(color), fptr(up), (int)x.size(0), (int)x.size(1), c.img, c.sigma, c.radius, c.lo, c.hi, c.y_up,
                                        c.normalize, c.scale, fmut(gx), fmut(gc), stream_of(x)));
        return {gx, gc};
    }
    void release_variables() override { x_.reset_data(); color_.reset_data(); }
};

Tensor splat(const Tensor &x, const Tensor &color, int img, double sigma, int radius, double lo, double hi, bool y_up, bool normalize, double scale) {
    refuse_tangents("splat_particles", x, color);
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t B = x.size(0), n = x.size(1);
    Tensor out = floats(x, {B, img, img, 4}), scratch = normalize ? floats(x, {B, n}) : Tensor();
    check_status(npa_splat_forward(fptr(x), fptr(color), (int)B, (int)n, img, sigma, radius, lo, hi, y_up, normalize, scale, fmut(scratch), fmut(out),
                                   stream_of(x)));
    if (recording(x, color)) {
        auto node = node_for<SplatNode>(x, color);
        node->x_ = saved(x); node->color_ = saved(color);
        node->c = SplatConsts{img, radius, y_up ? 1 : 0, normalize ? 1 : 0, sigma, lo, hi, scale};
        torch::autograd::set_history(out, node);
    }
    return out;
}

// `fn` as Python calls it.  torch.jit.trace sees no C++ node and would keep the outputs of the traced call as constants: while
// it records, the call is handed to Python, which makes it one node of the trace (npa_b200/_native.py).
template <typename R, typename... A>
auto op(const char *name, R (*fn)(A...)) {
    return [name, fn](A... a) -> py::object {
        if (torch::jit::tracer::isTracing()) return py::module_::import("npa_b200._native").attr("_traced")(name, a...);
        if constexpr (std::is_base_of_v<py::object, R>) return fn(a...);
        else return py::cast(fn(a...));
    };
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.attr("abi_version") = NPA_B200_ABI_VERSION;
    py::class_<Grid, GridPtr>(m, "Grid").def(py::init<uintptr_t>());
    m.def("instantiate", op("instantiate", &instantiate));
    m.def("reorder", op("reorder", &reorder));
    m.def("unreorder", op("unreorder", &unreorder));
    m.def("count", op("count", &count));
    m.def("density", op("density", &density));
    m.def("blur_gradient", op("blur_gradient", &blur_gradient));
    m.def("gradient_hybrid", op("gradient_hybrid", &gradient_hybrid));
    m.def("moment_matrix", op("moment_matrix", &moment_matrix));
    m.def("corrected_gradient", op("corrected_gradient", &corrected_gradient));
    m.def("perception", op("perception", &perception));
    m.def("packed_perception", op("packed_perception", &packed_perception));
    m.def("step_update", op("step_update", &step_update));
    m.def("mlp", op("mlp", &mlp));
    m.def("euler_step", op("euler_step", &euler_step));
    m.def("splat", op("splat", &splat));
}
