// PyTorch side of the encoding: checks, output allocation, launches and the autograd graph in C++.
//
// A README-sized batch runs for a few microseconds on the device, so what a call costs is host work:
// with checks, ctypes marshalling and torch.autograd.Function in Python a forward of 1000 points took
// 14 us and a training step on 4096 points 117 us, most of it in the interpreter.  Nothing here is
// remembered between calls except the scale factors of the encoding on each device.
//
// The two nodes mirror the reference's chained autograd Functions (src/pytorch_modules/funcs.py:8-72).
// Unlike a Python Function, a C++ node can ask the engine which of its inputs the running backward
// needs: autograd.grad(y, positions) does not compute the lattice gradient, and a backward restricted
// to the lattice values does not compute the position gradient.
//
// The C ABI is called through the pointers of the library the Python side has loaded.
#include <torch/extension.h>

#include <ATen/SavedTensorHooks.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <optional>
#include <set>
#include <string>
#include <unordered_map>
#include <vector>

#include "permuto_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct Api {
    decltype(&permuto_last_error) last_error;
    decltype(&permuto_order_pays) order_pays;
    decltype(&permuto_order_bytes) order_bytes;
    decltype(&permuto_order_record_bytes) order_record_bytes;
    decltype(&permuto_order_scratch_bytes) order_scratch_bytes;
    decltype(&permuto_order_records) order_records;
    decltype(&permuto_forward_ordered) forward;
    decltype(&permuto_forward_mlp_ordered) forward_mlp;
    decltype(&permuto_backward_ordered) backward;
    decltype(&permuto_double_backward_ordered) double_backward;
    decltype(&permuto_backward_combined) backward_combined;
    decltype(&permuto_adam_step) adam_step;
} api = {};

template <class F>
void take(F& slot, const std::unordered_map<std::string, uintptr_t>& table, const char* name) {
    const auto it = table.find(name);
    if (it == table.end()) throw std::runtime_error(std::string("missing C ABI symbol ") + name);
    slot = reinterpret_cast<F>(it->second);
}

void bind_api(const std::unordered_map<std::string, uintptr_t>& t) {
    take(api.last_error, t, "permuto_last_error");
    take(api.order_pays, t, "permuto_order_pays");
    take(api.order_bytes, t, "permuto_order_bytes");
    take(api.order_record_bytes, t, "permuto_order_record_bytes");
    take(api.order_scratch_bytes, t, "permuto_order_scratch_bytes");
    take(api.order_records, t, "permuto_order_records");
    take(api.forward, t, "permuto_forward_ordered");
    take(api.forward_mlp, t, "permuto_forward_mlp_ordered");
    take(api.backward, t, "permuto_backward_ordered");
    take(api.double_backward, t, "permuto_double_backward_ordered");
    take(api.backward_combined, t, "permuto_backward_combined");
    take(api.adam_step, t, "permuto_adam_step");
}

void check(int status) {
    if (status != PERMUTO_OK) throw std::runtime_error(api.last_error());
}

std::string sizes_of(const Tensor& t) {
    std::string s = "(";
    for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
    return s + (t.dim() == 1 ? ",)" : ")");
}

[[noreturn]] void fail(const std::string& what) { throw std::runtime_error(what); }

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// fp32, contiguous, on `device`, without a graph
Tensor plain(const Tensor& t, const c10::Device& device) {
    if (t.device() == device && t.scalar_type() == at::kFloat && t.is_contiguous()) return t;
    return t.detach().to(t.options().device(device).dtype(at::kFloat).requires_grad(false)).contiguous();
}

// fp32 (or byte) tensor on the device of `like`, straight from the allocator: the dispatcher is a third of at::empty
Tensor empty(at::IntArrayRef sizes, const Tensor& like, at::ScalarType type = at::kFloat) {
    return Tensor(at::detail::empty_cuda(sizes, type, like.device(), std::nullopt));
}

const void* data(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// Fixed description of an encoding and what it keeps on every device.
struct Lattice : torch::CustomClassHolder {
    permuto_config cfg = {};
    int64_t width = 0;
    bool aggregate = true;
    bool concat_positions_grad = false;
    // data-parallel hooks: callables kept by the Python wrapper, empty objects when not installed
    py::object on_backward, on_double_backward;

    Lattice(int pos_dim, int feat, int levels, int capacity, bool concat, double scaling, int64_t width_, Tensor scale_host)
        : width(width_), scale_host_(std::move(scale_host)) {
        cfg.pos_dim = pos_dim;
        cfg.nr_feat_per_level = feat;
        cfg.nr_levels = levels;
        cfg.capacity = capacity;
        cfg.concat_points = concat ? 1 : 0;
        cfg.points_scaling = (float)scaling;
    }
    ~Lattice() override {
        if ((on_backward || on_double_backward) && Py_IsInitialized()) {
            py::gil_scoped_acquire gil;  // the last owner may be a graph released on the engine's thread
            on_backward = py::object();
            on_double_backward = py::object();
        } else {
            on_backward.release();
            on_double_backward.release();
        }
    }

    Tensor scale_on(const c10::Device& device) {
        std::lock_guard<std::mutex> lock(mutex_);
        Tensor& t = scale_[device.index()];
        if (!t.defined()) t = scale_host_.to(device);
        return t;
    }

  private:
    Tensor scale_host_;
    std::mutex mutex_;
    std::unordered_map<int, Tensor> scale_;
};

// One call's inputs.
struct Inputs {
    c10::intrusive_ptr<Lattice> lattice;
    Tensor values, positions, window, shift, half, order;
    int levels_per_pass = 0;
    bool all_open = false;  // the caller knows the window to be open on every level
};

// What the nodes of one call share.  The tensors of the graph are not here: nodes keep them with
// save_for_backward, so that the engine frees them with the graph and saved-tensor hooks see them.
struct Call : torch::CustomClassHolder {
    c10::intrusive_ptr<Lattice> lattice;
    Tensor shift, half;
    int levels_per_pass = 0;
    bool need_values = false, need_positions = false;
    bool all_open = false;  // as in Inputs
    bool ordered = false;   // the forward ran in spatial order

    // A loss that reaches both the features and the position gradient gives the lattice values two
    // gradients in one backward, from the first-order node and from a second-order one (EncodeBackward).
    // Whichever of the two runs first leaves its part to the other, which adds both to the table in one
    // pass -- instead of two passes, two cleared tables and their sum.  It only does so when the engine
    // is certain to run the other one later in the same backward.
    struct Part {
        Tensor double_positions_grad;  // undefined: the first-order part
        Tensor grad;
    };
    static constexpr int kFirst = 0;  // number of the first-order node; the others are second-order ones

    int reserve_node() {
        std::lock_guard<std::mutex> lock(mutex_);
        nodes_.emplace_back();
        return (int)nodes_.size() - 1;
    }
    void set_node(int number, const std::shared_ptr<torch::autograd::Node>& node) {
        std::lock_guard<std::mutex> lock(mutex_);
        nodes_[number] = node;
    }

    // from the node `number` of the running backward: true when another node has taken over `p`
    bool leave(int number, Part p) {
        const int task = torch::autograd::get_current_graph_task_id();
        const auto* in_graph = torch::autograd::get_current_graph_task_nodes_in_graph();
        if (task < 0 || !in_graph) return false;
        const auto* info = torch::autograd::get_current_graph_task_exec_info();
        std::lock_guard<std::mutex> lock(mutex_);
        const int begin = number == kFirst ? 1 : kFirst, end = number == kFirst ? (int)nodes_.size() : kFirst + 1;
        for (int to = begin; to < end; ++to) {
            const auto node = nodes_[to].lock();
            if (!node || in_graph->count(node.get()) == 0 || ran_.count({task, to}) || parts_.count({task, to})) continue;
            if (info && !info->empty()) {  // a backward restricted to some inputs
                const auto it = info->find(node.get());
                if (it == info->end() || !it->second.should_execute()) continue;
            }
            parts_.emplace(std::make_pair(task, to), std::move(p));
            return true;
        }
        return false;
    }
    // what was left for the node `number` in the running backward; nothing is left for it from here on
    std::optional<Part> collect(int number) {
        const auto key = std::make_pair(torch::autograd::get_current_graph_task_id(), number);
        std::lock_guard<std::mutex> lock(mutex_);
        ran_.insert(key);  // task numbers are never used again
        std::optional<Part> p;
        const auto it = parts_.find(key);
        if (it != parts_.end()) {
            p = std::move(it->second);
            parts_.erase(it);
        }
        return p;
    }

  private:
    std::mutex mutex_;
    std::vector<std::weak_ptr<torch::autograd::Node>> nodes_ = std::vector<std::weak_ptr<torch::autograd::Node>>(1);
    std::map<std::pair<int, int>, Part> parts_;
    std::set<std::pair<int, int>> ran_;
};

// Same checks and messages as the reference (src/Encoding.cu:37-45, :63-66, :119-125).
void check_inputs(const Inputs& c) {
    const permuto_config& cfg = c.lattice->cfg;
    const Tensor& pos = c.positions;
    if (!pos.is_cuda()) fail("positions should be in GPU memory. Please call .cuda() on the tensor");
    if (pos.scalar_type() != at::kFloat) fail("positions should be of type float");
    if (pos.dim() != 2) fail("positions should have dim 2 correspondin to HW. However it has sizes " + sizes_of(pos));
    if (pos.size(0) == 0) fail("Why do we have 0 points");
    if (pos.size(1) != cfg.pos_dim)
        fail("Pos dim for the lattice doesn't correspond with the position of the points. Lattice was initialized with " +
             std::to_string(cfg.pos_dim) + " and points have pos dim " + std::to_string(pos.size(1)));
    const Tensor& lv = c.values;
    if (lv.dim() != 3 || lv.size(0) != cfg.nr_levels || lv.size(1) != cfg.capacity || lv.size(2) != cfg.nr_feat_per_level)
        fail("lattice_values should be nr_levels x capacity x " + std::to_string(cfg.nr_feat_per_level) + ", got " + sizes_of(lv));
    if (!lv.is_contiguous())
        fail("We assume that the lattice_values_monolithic are contiguous because in the cuda code we make a load of 2 float "
             "values at a time");
    if ((lv.scalar_type() != at::kFloat && lv.scalar_type() != at::kHalf) || lv.device() != pos.device())
        fail("lattice_values should be float32 (or float16 storage) on the device of the positions");
    if (c.half.defined() && (c.half.scalar_type() != at::kHalf || c.half.sizes() != lv.sizes() || c.half.device() != lv.device() ||
                             !c.half.is_contiguous()))
        fail("lattice_values_half should be a contiguous float16 tensor of the shape and device of lattice_values");
    if (c.shift.dim() != 2 || c.shift.size(0) != cfg.nr_levels || c.shift.size(1) != cfg.pos_dim)
        fail("Random shift should be nr of resolutions x pos dim");
    if (c.window.dim() != 1 || c.window.size(0) != cfg.nr_levels)
        fail("anneal_window should have the first dimension the same as the nr of resolutions");
    if (c.order.defined()) {
        // one of EncodingWrapper.order, whose size tells pos_dim and the number of points, or a buffer of
        // permuto_order_points
        const Tensor& o = c.order;
        const int64_t n = pos.size(0);
        if (o.device() != pos.device() || o.scalar_type() != at::kByte || o.dim() != 1 || !o.is_contiguous() ||
            (o.numel() != api.order_record_bytes(cfg.pos_dim, n) && o.numel() != api.order_bytes(cfg.pos_dim, n)) ||
            reinterpret_cast<uintptr_t>(o.data_ptr()) % 256 != 0)
            fail("the spatial order does not belong to " + std::to_string(n) + " positions of pos dim " +
                 std::to_string(cfg.pos_dim) + " on their device");
    }
}

// The C ABI's view of a checked call.
struct Bound {
    permuto_config cfg;
    permuto_inputs in;
    c10::cuda::OptionalCUDAGuard guard;
    Tensor scale, shift, window;

    explicit Bound(const Inputs& c) : cfg(c.lattice->cfg) {
        const c10::Device device = c.positions.device();
        if (device.index() != c10::cuda::current_device()) guard.set_device(device);
        scale = c.lattice->scale_on(device);
        shift = plain(c.shift, device);
        window = plain(c.window, device);
        const Tensor& table = c.half.defined() ? c.half : c.values;
        cfg.table_dtype = table.scalar_type() == at::kHalf ? PERMUTO_TABLE_F16 : PERMUTO_TABLE_F32;
        cfg.levels_per_pass = c.levels_per_pass;
        in.nr_positions = c.positions.size(0);
        in.positions = c.positions.data_ptr<float>();
        in.pos_stride_n = c.positions.stride(0);
        in.pos_stride_d = c.positions.stride(1);
        in.lattice_values = table.data_ptr();
        in.scale_factor = scale.data_ptr<float>();
        in.random_shift = shift.data_ptr<float>();
        in.anneal_window = window.data_ptr<float>();
    }
};

// The records alone: the scratch of the sort, a third of it all, goes back to the allocator right away.
Tensor make_order(const Inputs& c, Bound& b) {
    Tensor order = empty({api.order_record_bytes(b.cfg.pos_dim, b.in.nr_positions)}, c.positions, at::kByte);
    const Tensor scratch = empty({api.order_scratch_bytes(b.cfg.pos_dim, b.in.nr_positions)}, c.positions, at::kByte);
    check(api.order_records(&b.cfg, &b.in, order.data_ptr(), scratch.data_ptr(), stream_of(c.positions)));
    return order;
}

// What a call is ordered for: an order is made where order_pays says so.
enum Purpose {
    kAsGiven = -1,
    kInference = PERMUTO_ORDER_FEATURES,
    kTable = PERMUTO_ORDER_TABLE_GRAD,
    kPositions = PERMUTO_ORDER_POS_GRAD
};

// Whether to order a call, as far as the host knows its open levels.  What a closed level takes is far less than
// its share of the order (24 levels with 7 open, 2^20 points: features 74 -> 102 us, both gradients 269 -> 297), so
// a call whose window is on the device, unless it is the module's own, is not ordered.  Letting the sort count
// the open levels there and stand aside was measured too: 10-15 us a call (91 -> 106), and no gain at 0.3.
// Half of the levels have to be open, since rows are read out of order whether their levels are open or not
// (table gradient of 2^21 points, 7 of 24 levels open: 421 -> 477; 14 of 24: 862 -> 649).
bool order_pays(const Inputs& c, const Bound& b, Purpose purpose) {
    permuto_config cfg = b.cfg;
    if (!c.all_open) {
        if (!c.window.is_cpu()) return false;
        const Tensor w = plain(c.window, c.window.device());
        const float* v = w.data_ptr<float>();
        cfg.nr_levels = (int)std::count_if(v, v + w.numel(), [](float x) { return x != 0.f; });
        if (2 * cfg.nr_levels < b.cfg.nr_levels) return false;
    }
    return api.order_pays(&cfg, b.in.nr_positions, purpose) != 0;
}

// An order that a call can do without: where there is no room for its 24 to 44 bytes a point the call runs
// as it would without one (callers allocate their outputs first).
void try_order(Inputs& c, Bound& b, Purpose purpose) {
    if (c.order.defined() || !order_pays(c, b, purpose)) return;
    try {
        c.order = make_order(c, b);
    } catch (const c10::OutOfMemoryError&) {
    }
}

// features [N, W]; where the batch is large enough to be worth it the points are put into spatial order
// first, and the order is left in `c` for the backward passes
Tensor run_forward(Inputs& c, Purpose purpose) {
    check_inputs(c);
    Bound b(c);
    Tensor out = empty({b.in.nr_positions, c.lattice->width}, c.positions);
    if (purpose != kAsGiven) try_order(c, b, purpose);
    check(api.forward(&b.cfg, &b.in, data(c.order), out.data_ptr<float>(), stream_of(c.positions)));
    return out;
}

// Up to this many points the table gradients are summed in spatial order, beyond it in the sequence of the
// batch.  A slot of a coarse level receives up to a million fp32 addends and more, and what their sum rounds
// to follows the sequence and the merging inside the warps.  Two runs of one sequence differ in the 2-norm by
// 2-3e-6 at 2^22 and 2.4-4e-6 at 2^24 points, the two sequences by about 2.5e-9 * sqrt(points): 2-3e-6 at 2^20,
// 3-7e-6 at 2^22, 6.6-11e-6 at 2^24 (pos_dim 2, 3 and 6, 6 to 24 levels).  The line keeps that below 1e-5, on a
// measured size: whether a batch is ordered does not show in its gradient.  Spatial order is closer to a
// float64 sum of the same addends (1.3-3.4e-6 against 2-6.5e-6 at 2^22).
constexpr int64_t kOrderedSums = 1 << 22;
bool ordered_sums(const Inputs& c) { return c.order.defined() && c.positions.size(0) <= kOrderedSums; }

struct Gradients {
    Tensor values, positions;
};

Gradients run_backward(const Inputs& c, const Tensor& grad, bool need_values, bool need_positions, const Tensor& values_out,
                       int level_begin, int level_end, bool zero, const Tensor& positions_out) {
    check_inputs(c);
    const int64_t n = c.positions.size(0);
    if (grad.dim() != 2 || grad.size(0) != n || grad.size(1) != c.lattice->width)
        fail("The nr of positions should match between the input positions and the sliced values: expected (" +
             std::to_string(n) + ", " + std::to_string(c.lattice->width) + "), got " + sizes_of(grad));
    if (!grad.is_contiguous()) fail("Grad sliced values needs to be contiguous. Please call .contiguous() on it");
    Bound b(c);
    uint32_t flags = zero ? PERMUTO_ZERO_OUTPUTS : 0;
    if (!c.lattice->aggregate) flags |= PERMUTO_NO_AGGREGATE;
    if (c.lattice->concat_positions_grad) flags |= PERMUTO_CONCAT_POSITIONS_GRAD;
    Gradients g;
    if (need_values)  // always fp32, whatever the storage type of the values
        g.values = values_out.defined() ? values_out : empty(c.values.sizes(), c.positions);
    if (need_positions) {
        if (positions_out.defined()) {
            g.positions = positions_out;
            flags |= PERMUTO_KEEP_POSITIONS_GRAD;
        } else {  // without ZERO_OUTPUTS nothing clears it natively
            g.positions = zero ? empty({n, b.cfg.pos_dim}, c.positions)
                               : at::zeros({n, b.cfg.pos_dim}, c.positions.options());
        }
    }
    const int end = level_end < 0 ? b.cfg.nr_levels : level_end;
    auto launch = [&](const void* order, const Tensor& values, const Tensor& positions) {
        check(api.backward(&b.cfg, &b.in, order, grad.data_ptr<float>(), values.defined() ? values.data_ptr<float>() : nullptr,
                           positions.defined() ? positions.data_ptr<float>() : nullptr, level_begin, end, flags,
                           stream_of(c.positions)));
    };
    if (c.order.defined() && need_values && !ordered_sums(c)) {
        launch(nullptr, g.values, {});
        if (need_positions) launch(data(c.order), {}, g.positions);
    } else {
        launch(data(c.order), g.values, g.positions);
    }
    return g;
}

struct SecondOrder {
    Tensor values, features;
};

SecondOrder run_double_backward(const Inputs& c, const Tensor& double_positions_grad, const Tensor& grad, bool need_values,
                                bool need_features) {
    check_inputs(c);
    const int64_t n = c.positions.size(0);
    if (double_positions_grad.dim() != 2 || double_positions_grad.size(0) != n ||
        double_positions_grad.size(1) != c.lattice->cfg.pos_dim)
        fail("double_positions_grad should be nr_positions x pos_dim");
    if (grad.dim() != 2 || grad.size(0) != n || grad.size(1) != c.lattice->width)
        fail("The nr of positions should match between the input positions and the sliced values");
    Bound b(c);
    const Tensor dpg = double_positions_grad.contiguous(), gf = grad.contiguous();
    SecondOrder s;
    if (need_values) s.values = empty(c.values.sizes(), c.positions);
    if (need_features) s.features = empty(gf.sizes(), c.positions);
    auto launch = [&](const void* order, const Tensor& values, const Tensor& features) {
        check(api.double_backward(&b.cfg, &b.in, order, dpg.data_ptr<float>(), gf.data_ptr<float>(),
                                  values.defined() ? values.data_ptr<float>() : nullptr,
                                  features.defined() ? features.data_ptr<float>() : nullptr,
                                  PERMUTO_ZERO_OUTPUTS | (c.lattice->aggregate ? 0 : PERMUTO_NO_AGGREGATE),
                                  stream_of(c.positions)));
    };
    if (c.order.defined() && need_values && !ordered_sums(c)) {
        launch(nullptr, s.values, {});
        if (need_features) launch(data(c.order), {}, s.features);
    } else {
        launch(data(c.order), s.values, s.features);
    }
    return s;
}

// table gradient of both orders in one buffer
Tensor run_combined(const Inputs& c, const Tensor& grad, const Call::Part& second) {
    Bound b(c);
    const Tensor dpg = second.double_positions_grad.contiguous();
    Tensor values = empty(c.values.sizes(), c.positions);
    check(api.backward_combined(&b.cfg, &b.in, data(c.order), grad.data_ptr<float>(), dpg.data_ptr<float>(),
                                second.grad.data_ptr<float>(), values.data_ptr<float>(),
                                PERMUTO_ZERO_OUTPUTS | (c.lattice->aggregate ? 0 : PERMUTO_NO_AGGREGATE), stream_of(c.positions)));
    return values;
}

py::object as_python(const Tensor& t) { return t.defined() ? py::cast(t) : py::none(); }
Tensor from_python(const py::handle& h) { return h.is_none() ? Tensor() : py::cast<Tensor>(h); }

Gradients backward_or_hook(const Inputs& c, const Tensor& grad, bool need_values, bool need_positions) {
    if (need_values && c.lattice->on_backward) {
        py::gil_scoped_acquire gil;
        const py::tuple r = c.lattice->on_backward(c.values, c.positions, c.window, as_python(c.half), as_python(c.order), grad,
                                                   need_values, need_positions);
        return {from_python(r[0]), from_python(r[1])};
    }
    return run_backward(c, grad, need_values, need_positions, {}, 0, -1, true, {});
}

// parts of one backward may be merged: no second differentiation, no data-parallel hooks, and not where each
// part is summed in the sequence of the batch (the two sums stay separate there, as without an order)
bool may_merge(const Inputs& c) {
    return !at::GradMode::is_enabled() && !c.lattice->on_backward && !c.lattice->on_double_backward &&
           c.positions.size(0) <= kOrderedSums;
}

// The order goes with the saved tensors, unless hooks look at those: they get what a node without an order
// saves, and the backward makes the order again from the positions that they hand back.
Tensor order_to_save(const Inputs& in) { return at::SavedTensorDefaultHooks::get_tls_state().stack.empty() ? in.order : Tensor(); }

// a node's inputs out of its saved tensors, which start at `first`: values, positions, window, order
Inputs saved_inputs(const Call& call, const variable_list& saved, size_t first) {
    Inputs in{call.lattice, saved[first], saved[first + 1], saved[first + 2], call.shift, call.half, saved[first + 3],
              call.levels_per_pass, call.all_open};
    if (call.ordered && !in.order.defined()) {
        check_inputs(in);
        Bound b(in);
        try_order(in, b, call.need_positions ? kPositions : kTable);
    }
    return in;
}

// The first-order backward as a differentiable function of (upstream gradient, lattice values); its own
// backward is the double backward from the position gradient.
struct EncodeBackward : torch::autograd::Function<EncodeBackward> {
    static variable_list forward(AutogradContext* ctx, const Tensor& grad, const Tensor& values, const Tensor& positions,
                                 const Inputs& in, const c10::intrusive_ptr<Call>& call, bool need_values, bool need_positions,
                                 int64_t number) {
        const Gradients g = backward_or_hook(in, grad, need_values, need_positions);
        ctx->save_for_backward({grad, values, positions, in.window, order_to_save(in)});
        ctx->saved_data["call"] = c10::IValue::make_capsule(call);
        ctx->saved_data["number"] = number;
        ctx->saved_data["position_output"] = need_positions ? (need_values ? 1 : 0) : -1;
        ctx->set_materialize_grads(false);
        variable_list out;
        if (need_values) out.push_back(g.values);
        if (need_positions) out.push_back(g.positions);
        return out;
    }

    static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
        variable_list out(8);
        const variable_list saved = ctx->get_saved_variables();  // checks the version counters
        const auto call = c10::static_intrusive_pointer_cast<Call>(ctx->saved_data["call"].toCapsule());
        const int number = (int)ctx->saved_data["number"].toInt();
        const bool need_features = ctx->needs_input_grad(0), need_values = ctx->needs_input_grad(1);
        const auto first = call->collect(number);
        // As in the reference, only the path through the position gradient is differentiated again; a
        // second-order term through the lattice-value gradient is not propagated.
        const int64_t at = ctx->saved_data["position_output"].toInt();
        const bool second = at >= 0 && grads[at].defined();
        if (!first && !(second && (need_features || need_values))) return out;
        const Inputs in = saved_inputs(*call, saved, 1);
        if (first) {
            out[1] = second ? run_combined(in, first->grad, {grads[at], saved[0]})
                            : run_backward(in, first->grad, true, false, {}, 0, -1, true, {}).values;
        }
        if (!second) return out;
        const bool own_values = need_values && !first && !(may_merge(in) && call->leave(number, {grads[at], saved[0]}));
        if (!need_features && !own_values) return out;
        SecondOrder s = run_double_backward(in, grads[at], saved[0], own_values, need_features);
        // data-parallel use: this second-order lattice gradient is summed over the ranks like the
        // first-order one, otherwise the replicated tables drift apart
        if (s.values.defined() && call->lattice->on_double_backward) {
            py::gil_scoped_acquire gil;
            s.values = from_python(call->lattice->on_double_backward(s.values));
        }
        out[0] = s.features;
        if (own_values) out[1] = s.values;
        return out;
    }
};

struct Encode : torch::autograd::Function<Encode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& values, const Tensor& positions, Inputs& in,
                          const c10::intrusive_ptr<Call>& call) {
        const Tensor out = run_forward(in, call->need_positions ? kPositions : kTable);
        call->ordered = in.order.defined();
        ctx->save_for_backward({values, positions, in.window, order_to_save(in)});
        ctx->saved_data["call"] = c10::IValue::make_capsule(call);
        return out;
    }

    static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
        const variable_list saved = ctx->get_saved_variables();  // checks the version counters
        const auto call = c10::static_intrusive_pointer_cast<Call>(ctx->saved_data["call"].toCapsule());
        const bool need_values = call->need_values && ctx->needs_input_grad(0);
        const bool need_positions = call->need_positions && ctx->needs_input_grad(1);
        variable_list out(4);
        if (!need_values && !need_positions) return out;
        const Tensor grad = grads[0].contiguous();
        const Inputs in = saved_inputs(*call, saved, 0);
        if (at::GradMode::is_enabled()) {
            const int number = call->reserve_node();
            const variable_list g = EncodeBackward::apply(grad, saved[0], saved[1], in, call, need_values, need_positions, number);
            call->set_node(number, g[0].grad_fn());
            if (need_values) out[0] = g[0];
            if (need_positions) out[1] = g[need_values ? 1 : 0];
            return out;
        }
        const auto second = call->collect(Call::kFirst);
        if (second) out[0] = run_combined(in, grad, *second);
        const bool own_values = need_values && !second && !(may_merge(in) && call->leave(Call::kFirst, {{}, grad}));
        if (own_values || need_positions) {
            const Gradients g = backward_or_hook(in, grad, own_values, need_positions);
            if (own_values) out[0] = g.values;
            out[1] = g.positions;
        }
        return out;
    }
};

Inputs make_inputs(const c10::intrusive_ptr<Lattice>& lattice, const Tensor& values, const Tensor& positions, const Tensor& window,
                   const Tensor& shift, const std::optional<Tensor>& half, const std::optional<Tensor>& order,
                   int levels_per_pass, bool all_open) {
    return {lattice, values, positions, window, shift, half ? *half : Tensor(), order ? *order : Tensor(), levels_per_pass,
            all_open};
}

// the module's forward: with a graph where one is wanted
Tensor encode(const c10::intrusive_ptr<Lattice>& lattice, const Tensor& values, const Tensor& positions, const Tensor& window,
              const Tensor& shift, const std::optional<Tensor>& half, int levels_per_pass, bool all_open) {
    Inputs in = make_inputs(lattice, values, positions, window, shift, half, std::nullopt, levels_per_pass, all_open);
    const bool graph = at::GradMode::is_enabled();
    const bool need_values = graph && values.requires_grad(), need_positions = graph && positions.requires_grad();
    if (!need_values && !need_positions) return run_forward(in, kInference);
    auto call = c10::make_intrusive<Call>();
    call->lattice = lattice;
    call->shift = in.shift;
    call->half = in.half;
    call->levels_per_pass = levels_per_pass;
    call->all_open = all_open;
    call->need_values = need_values;
    call->need_positions = need_positions;
    Tensor out = Encode::apply(values, positions, in, call);
    call->set_node(Call::kFirst, out.grad_fn());
    return out;
}

Tensor forward_mlp(const c10::intrusive_ptr<Lattice>& lattice, const Tensor& values, const Tensor& positions,
                   const Tensor& window, const Tensor& shift, const std::optional<Tensor>& half,
                   const std::optional<Tensor>& order, int levels_per_pass, bool all_open, const std::vector<Tensor>& weights,
                   const std::vector<std::optional<Tensor>>& biases, int activation, const std::optional<Tensor>& status) {
    Inputs c = make_inputs(lattice, values, positions, window, shift, half, order, levels_per_pass, all_open);
    check_inputs(c);
    const c10::Device device = positions.device();
    if (weights.empty() || weights.size() > 6)
        fail("the fused network takes 1..6 layers, got " + std::to_string(weights.size()));
    std::vector<permuto_mlp_layer> layers(weights.size());
    std::vector<Tensor> keep;
    int64_t width = lattice->width;
    for (size_t i = 0; i < weights.size(); ++i) {
        const std::string where = weights.size() == 1 ? "" : "layer " + std::to_string(i) + ": ";
        if (weights[i].dim() != 2 || weights[i].size(1) != width)
            fail(where + "weight should be out_features x " + std::to_string(width) + ", got " + sizes_of(weights[i]));
        keep.push_back(plain(weights[i], device));
        layers[i].weight = keep.back().data_ptr<float>();
        layers[i].in_features = (int32_t)width;
        width = weights[i].size(0);
        layers[i].out_features = (int32_t)width;
        layers[i].bias = nullptr;
        if (biases[i]) {
            if (biases[i]->dim() != 1 || biases[i]->size(0) != width)
                fail(where + "bias should have " + std::to_string(width) + " entries");
            keep.push_back(plain(*biases[i], device));
            layers[i].bias = keep.back().data_ptr<float>();
        }
    }
    if (status && (status->scalar_type() != at::kInt || status->device() != device || status->numel() != 1))
        fail("status should be a one-element int32 tensor on the device of the positions");
    Bound b(c);
    // One layer behind the encoding gains 18 % from an order on 2^20 independent points (349 -> 285 us); with
    // a whole network behind it the gathers are less of the time, and the gain (4 %) is what ray samples lose.
    Tensor out = empty({b.in.nr_positions, width}, positions);
    if (layers.size() == 1) try_order(c, b, kInference);
    check(api.forward_mlp(&b.cfg, &b.in, data(c.order), layers.data(), (int32_t)layers.size(), activation,
                          out.data_ptr<float>(), status ? status->data_ptr<int32_t>() : nullptr, stream_of(positions)));
    return out;
}

void adam_step(const Tensor& values, const Tensor& grad, const Tensor& exp_avg, const Tensor& exp_avg_sq, int64_t step, double lr,
               double beta1, double beta2, double eps, double weight_decay, bool skip_untouched, bool zero_grad) {
    const std::pair<const char*, const Tensor*> all[] = {
        {"values", &values}, {"grad", &grad}, {"exp_avg", &exp_avg}, {"exp_avg_sq", &exp_avg_sq}};
    for (const auto& [name, t] : all) {
        if (!t->is_cuda()) fail(std::string(name) + " should be in GPU memory. There is no CPU path");
        if (t->scalar_type() != at::kFloat || !t->is_contiguous() || t->sizes() != values.sizes() || t->device() != values.device())
            fail(std::string(name) + " must be a contiguous float32 tensor of the shape and device of the values");
    }
    c10::cuda::OptionalCUDAGuard guard;
    if (values.device().index() != c10::cuda::current_device()) guard.set_device(values.device());
    check(api.adam_step(values.data_ptr<float>(), grad.data_ptr<float>(), exp_avg.data_ptr<float>(), exp_avg_sq.data_ptr<float>(),
                        values.numel(), lr, beta1, beta2, eps, weight_decay, step,
                        (skip_untouched ? PERMUTO_ADAM_SKIP_UNTOUCHED : 0) | (zero_grad ? PERMUTO_ADAM_ZERO_GRAD : 0),
                        stream_of(values)));
    // the kernel wrote through the raw pointer: tell autograd (and the module's fp16 copy) so
    values.unsafeGetTensorImpl()->bump_version();
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("bind_api", &bind_api);
    py::class_<Lattice, c10::intrusive_ptr<Lattice>>(m, "Lattice")
        .def(py::init<int, int, int, int, bool, double, int64_t, Tensor>())
        .def_readwrite("aggregate", &Lattice::aggregate)
        .def_readwrite("concat_positions_grad", &Lattice::concat_positions_grad)
        .def("scale_on", [](Lattice& l, const c10::Device& d) { return l.scale_on(d); })
        .def("set_hooks", [](Lattice& l, const py::object& backward, const py::object& double_backward) {
            l.on_backward = backward.is_none() ? py::object() : backward;
            l.on_double_backward = double_backward.is_none() ? py::object() : double_backward;
        });
    m.def("encode", &encode);
    m.def("forward", [](const c10::intrusive_ptr<Lattice>& l, const Tensor& v, const Tensor& p, const Tensor& w, const Tensor& s,
                        const std::optional<Tensor>& half, const std::optional<Tensor>& order, int lpp) {
        Inputs c = make_inputs(l, v, p, w, s, half, order, lpp, true);
        return run_forward(c, kAsGiven);
    });
    m.def("check_inputs", [](const c10::intrusive_ptr<Lattice>& l, const Tensor& v, const Tensor& p, const Tensor& w,
                             const Tensor& s, const std::optional<Tensor>& half) {
        check_inputs(make_inputs(l, v, p, w, s, half, std::nullopt, 0, true));
    });
    m.def("order", [](const c10::intrusive_ptr<Lattice>& l, const Tensor& v, const Tensor& p, const Tensor& w, const Tensor& s,
                      const std::optional<Tensor>& half, int lpp, int purpose) -> std::optional<Tensor> {
        Inputs c = make_inputs(l, v, p, w, s, half, std::nullopt, lpp, true);
        check_inputs(c);
        Bound b(c);
        if (purpose >= 0 && !api.order_pays(&b.cfg, b.in.nr_positions, purpose)) return std::nullopt;
        return make_order(c, b);
    });
    m.def("backward", [](const c10::intrusive_ptr<Lattice>& l, const Tensor& v, const Tensor& p, const Tensor& w, const Tensor& s,
                         const std::optional<Tensor>& half, const std::optional<Tensor>& order, int lpp, const Tensor& grad,
                         bool need_values, bool need_positions, const std::optional<Tensor>& values_out, int level_begin,
                         int level_end, bool zero, const std::optional<Tensor>& positions_out) {
        Inputs c = make_inputs(l, v, p, w, s, half, order, lpp, true);
        const Gradients g = run_backward(c, grad, need_values, need_positions, values_out ? *values_out : Tensor(), level_begin,
                                         level_end, zero, positions_out ? *positions_out : Tensor());
        return py::make_tuple(as_python(g.values), as_python(g.positions));
    });
    m.def("double_backward", [](const c10::intrusive_ptr<Lattice>& l, const Tensor& v, const Tensor& p, const Tensor& w,
                                const Tensor& s, const std::optional<Tensor>& half, const std::optional<Tensor>& order, int lpp,
                                const Tensor& dpg, const Tensor& grad, bool need_values, bool need_features) {
        Inputs c = make_inputs(l, v, p, w, s, half, order, lpp, true);
        const SecondOrder r = run_double_backward(c, dpg, grad, need_values, need_features);
        return py::make_tuple(as_python(r.values), as_python(r.features));
    });
    m.def("forward_mlp", &forward_mlp);
    m.def("adam_step", &adam_step);
}
