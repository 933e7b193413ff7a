// Native autograd nodes over the C ABI for the calls whose eager time is host
// time: transform_grid, transform_data and transform_data_mixed.
//
// The Python classes of libcpab_gb300/_autograd.py stay the reference for what
// these calls do (and serve every other call, and these ones under functorch,
// tracing or tensor subclasses).  One image's forward and d(theta) took 280 us
// of Python and ctypes around 75 us of kernels; here it is the dispatch of the
// allocations and launches.  A forward that the C ABI refuses returns None, and
// the Python class then raises with its message.
//
// The solver settings that the Python backward reads from the transformer's
// params when it runs (step count, gradient mode, point gradient, tie counter,
// basis) are read at the same time here, under the GIL, by one call of
// libcpab_gb300._autograd.settings.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/utils/pybind.h>

#include <mutex>
#include <vector>

#include "../../include/cpab_gb300.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

struct Fallback {};   // the Python class takes the call (and reports its error)

void check(int rc) {
    if (rc != CPAB_OK) throw Fallback();
}

struct Cells {
    int ndim = 0;
    int nc[3] = {1, 1, 1};
    int64_t nC = 0;
};

Cells parse_cells(const py::handle &nc) {
    Cells c;
    const auto seq = py::reinterpret_steal<py::object>(PySequence_Fast(nc.ptr(), "nc"));
    if (!seq) throw py::error_already_set();
    c.ndim = (int)PySequence_Fast_GET_SIZE(seq.ptr());
    if (c.ndim < 1 || c.ndim > 3) throw Fallback();
    for (int j = 0; j < c.ndim; ++j) {
        c.nc[j] = (int)PyLong_AsLong(PySequence_Fast_GET_ITEM(seq.ptr(), j));
        if (PyErr_Occurred()) throw py::error_already_set();
    }
    c.nC = cpab_num_cells(c.ndim, c.nc);
    if (c.nC < 0) throw Fallback();
    return c;
}

struct Settings {
    int nsteps = 0, mode = 0;
    bool point_gradient = false;
    Tensor ties, basis;
};

Settings parse_settings(const py::handle &t) {
    Settings s;
    PyObject *p = t.ptr();
    if (!PyTuple_Check(p) || PyTuple_GET_SIZE(p) != 5) throw Fallback();
    s.nsteps = (int)PyLong_AsLong(PyTuple_GET_ITEM(p, 0));
    s.mode = (int)PyLong_AsLong(PyTuple_GET_ITEM(p, 1));
    s.point_gradient = PyTuple_GET_ITEM(p, 2) == Py_True;
    if (PyErr_Occurred()) throw py::error_already_set();
    if (PyTuple_GET_ITEM(p, 3) != Py_None)
        s.ties = py::cast<Tensor>(py::handle(PyTuple_GET_ITEM(p, 3)));
    s.basis = py::cast<Tensor>(py::handle(PyTuple_GET_ITEM(p, 4)));
    return s;
}

// References to params of nodes that went away on a thread without the GIL (the
// autograd engine's): handed to the interpreter as a pending call, so that the
// engine never waits for a busy one (it did, 5 us and more per backward).  Should
// the interpreter's list of those be full, the next native call drops them; every
// node was made by such a call, so no more pile up than there were nodes.  Both
// objects outlive the process's last node.
std::mutex &dropped_mu() {
    static std::mutex *mu = new std::mutex;
    return *mu;
}
std::vector<PyObject *> &dropped() {   // under dropped_mu
    static auto *v = new std::vector<PyObject *>;
    return *v;
}

void drop_params() {   // with the GIL
    std::vector<PyObject *> v;
    {
        std::lock_guard<std::mutex> lock(dropped_mu());
        v.swap(dropped());
    }
    for (PyObject *p : v) Py_DECREF(p);
}

void release_params(PyObject *params) {   // with or without the GIL
    if (!Py_IsInitialized()) return;   // the interpreter and its objects are gone
    if (PyGILState_Check()) {
        Py_DECREF(params);
        return;
    }
    bool first;
    {
        std::lock_guard<std::mutex> lock(dropped_mu());
        first = dropped().empty();
        dropped().push_back(params);
    }
    if (first)
        Py_AddPendingCall(
            [](void *) {
                drop_params();
                return 0;
            },
            nullptr);
}

// What a node keeps beside its saved tensors.
struct Kept : torch::CustomClassHolder {
    PyObject *params = nullptr;
    Cells cells;
    int mode = 0;          // as of the forward
    bool exact = false;    // transform_grid: integration == 'exact'
    int64_t points_dim = 0, theta_dim = 0;
    std::vector<int64_t> outsize;
    // transform_data_mixed
    int64_t C = 0, data_points = 0, total = 0, tiles = 0;
    std::vector<std::vector<int64_t>> shapes, out_shapes;
    std::vector<int64_t> sizes, out_sizes;

    ~Kept() override {
        if (params) release_params(params);
    }
};

[[noreturn]] void raise_native(int rc) {
    const std::string msg =
        "libcpab_gb300 error " + std::to_string(rc) + ": " + cpab_last_error();
    py::gil_scoped_acquire gil;
    const py::object cls = py::module_::import("libcpab_gb300._native").attr("CpabError");
    PyErr_SetString(cls.ptr(), msg.c_str());
    python_error e;
    e.persist();
    throw e;
}

void check_backward(int rc) {
    if (rc != CPAB_OK) raise_native(rc);
}

PyObject *g_settings = nullptr;   // _autograd.settings, held from the module's import on

// The params' settings at the time of a backward.
Settings settings_now(const Kept &k, const at::Device &device) {
    py::gil_scoped_acquire gil;
    try {
        return parse_settings(py::handle(g_settings)(py::handle(k.params), py::cast(device)));
    } catch (py::error_already_set &e) {
        e.restore();
        python_error err;
        err.persist();
        throw err;
    } catch (Fallback &) {
        PyErr_SetString(PyExc_RuntimeError, "libcpab_gb300: malformed solver settings");
        python_error err;
        err.persist();
        throw err;
    }
}

void *stream_of(const Tensor &t) {
    return c10::cuda::getCurrentCUDAStream(t.device().index()).stream();
}

Tensor floats(const Tensor &t) {
    return t.detach().to(at::kFloat).contiguous();
}

float *ptr(const Tensor &t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
unsigned long long *ties_of(const Settings &s) {
    return s.ties.defined() ? static_cast<unsigned long long *>(s.ties.data_ptr()) : nullptr;
}

Tensor make(const Tensor &like, at::IntArrayRef shape) {
    return at::empty(shape, like.options().dtype(at::kFloat).requires_grad(false));
}

Tensor workspace(const Tensor &like, size_t bytes) {
    return at::empty({(int64_t)(bytes > 0 ? bytes : 1)},
                     like.options().dtype(at::kByte).requires_grad(false));
}

// A = B theta and E = expm(dt [A; 0]) - I of every cell (undefined: not wanted).
void tables(const Cells &c, const Settings &s, const Tensor &theta, bool want_A, bool want_E,
            Tensor *A, Tensor *E) {
    if (theta.dim() != 2 || s.basis.dim() != 2 || s.basis.size(1) != theta.size(1) ||
        s.basis.size(0) != c.nC * c.ndim * (c.ndim + 1))
        throw Fallback();
    const int64_t n = theta.size(0);
    if (want_A) *A = make(theta, {n, c.nC, c.ndim, c.ndim + 1});
    if (want_E) *E = make(theta, {n, c.nC, c.ndim, c.ndim + 1});
    check(cpab_cell_tables(c.ndim, c.nc, s.nsteps, ptr(theta), (int)n, (int)theta.size(1),
                           ptr(s.basis), ptr(*A), nullptr, ptr(*E), stream_of(theta)));
}

// Gradients of a node that was differentiated with create_graph: a second
// differentiation raises, as once_differentiable's does.
variable_list once(bool create_graph, const variable_list &grads, variable_list out) {
    if (!create_graph) return out;
    bool any = false;
    for (const Tensor &g : grads) any = any || (g.defined() && g.requires_grad());
    if (!any) return out;
    variable_list in;
    for (Tensor &t : out)
        if (t.defined()) {
            t = t.detach();
            t.set_requires_grad(true);
            in.push_back(t);
        }
    const auto err = std::make_shared<torch::autograd::DelayedError>(
        "trying to differentiate twice a function that was marked with @once_differentiable",
        (int64_t)in.size());
    const variable_list res = err->apply(std::move(in));
    size_t k = 0;
    for (Tensor &t : out)
        if (t.defined()) t = res[k++];
    return out;
}

// f() with the interpreter free for other threads: allocations may synchronise and
// launches wait for room in the queue.  Saved-tensor hooks take the GIL themselves.
template <typename F>
auto without_gil(const F &f) {
    py::gil_scoped_release free;
    return f();
}

bool needs_graph(const Tensor &a, const Tensor &b) {
    return at::GradMode::is_enabled() && (a.requires_grad() || b.requires_grad());
}

using KeptPtr = c10::intrusive_ptr<Kept>;

void keep(AutogradContext *ctx, const KeptPtr &k) {
    ctx->saved_data["kept"] = c10::IValue::make_capsule(k);
}
Kept &kept(AutogradContext *ctx) {
    return static_cast<Kept &>(*ctx->saved_data["kept"].toCapsule());
}

struct Call {
    KeptPtr kept;
    Settings s;
};

// ------------------------------ transform_grid -------------------------------
Tensor grid_forward(const Call &a, const Tensor &points, const Tensor &theta, bool grad, Tensor *A,
                    Tensor *E) {
    const Cells &c = a.kept->cells;
    tables(c, a.s, theta, a.kept->exact || grad, !a.kept->exact, A, E);
    const int64_t n = theta.size(0), nP = points.size(-1);
    const int broadcast = points.dim() == 3 && points.size(0) == n;
    Tensor out = make(points, {n, c.ndim, nP});
    if (a.kept->exact)
        check(cpab_integrate_exact(c.ndim, c.nc, ptr(points), broadcast, nP, ptr(*A), (int)n,
                                   ptr(out), ties_of(a.s), nullptr, stream_of(points)));
    else
        check(cpab_integrate(c.ndim, c.nc, a.s.nsteps, ptr(points), broadcast, nP, ptr(*E), (int)n,
                             ptr(out), ties_of(a.s), stream_of(points)));
    return out;
}

struct TransformGrid : torch::autograd::Function<TransformGrid> {
    static Tensor forward(AutogradContext *ctx, const Tensor &points_in, const Tensor &theta_in,
                          const Call &a) {
        const Tensor points = floats(points_in), theta = floats(theta_in);
        Tensor A, E;
        const Tensor out = grid_forward(a, points, theta, true, &A, &E);
        keep(ctx, a.kept);
        ctx->set_materialize_grads(false);
        if (a.kept->exact) {
            // the exact scheme's backward integrates back from its result
            ctx->save_for_backward({points, A, out});
        } else {
            ctx->save_for_backward({points, A, E});
        }
        return out;
    }

    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const bool create_graph = at::GradMode::is_enabled();
        at::AutoGradMode off(false);
        const auto saved = ctx->get_saved_variables();
        const Tensor &points = saved[0], &A = saved[1], &E = saved[2];
        const Kept &k = kept(ctx);
        const Cells &c = k.cells;
        const bool need_p = ctx->needs_input_grad(0), need_t = ctx->needs_input_grad(1);
        const int64_t n = A.size(0);
        if (!grads[0].defined()) {
            // the reference computes this gradient from a zero cotangent: zeros
            return {Tensor(), need_t ? at::zeros({n, k.theta_dim}, A.options()) : Tensor(), Tensor()};
        }
        const Settings s = settings_now(k, points.device());
        // the reference returns no gradient for the points
        // (libcpab/pytorch/transformer.py:202); params.point_gradient opts in
        const bool want_p = need_p && s.point_gradient;
        if (!want_p && !need_t) return {Tensor(), Tensor(), Tensor()};
        const Tensor g = floats(grads[0]);
        const int64_t nP = points.size(-1);
        Tensor dtheta = make(A, {n, s.basis.size(1)}), dpoints;
        if (want_p) dpoints = make(A, {n, c.ndim, nP});
        void *stream = stream_of(points);
        if (k.exact) {
            const size_t need = cpab_backward_exact_workspace(c.ndim, c.nc, nP, (int)n);
            if (need == 0 && nP > 0 && n > 0) raise_native(3);
            const Tensor ws = workspace(A, need);
            check_backward(cpab_backward_exact(
                c.ndim, c.nc, ptr(E), nP, ptr(A), (int)n, ptr(s.basis), (int)s.basis.size(1),
                ptr(g), ptr(dtheta), ptr(dpoints), ws.data_ptr(), (size_t)ws.numel(), ties_of(s),
                stream));
        } else {
            const size_t need = cpab_backward_workspace(c.ndim, c.nc, s.nsteps, nP, (int)n);
            if (need == 0 && nP > 0 && n > 0) raise_native(3);
            const Tensor ws = workspace(A, need);
            const int broadcast = points.dim() == 3 && points.size(0) == n;
            check_backward(cpab_backward(c.ndim, c.nc, s.nsteps, s.mode, ptr(points), broadcast,
                                         nP, ptr(A), ptr(E), (int)n, ptr(s.basis),
                                         (int)s.basis.size(1), ptr(g), ptr(dtheta), ptr(dpoints),
                                         ws.data_ptr(), (size_t)ws.numel(), ties_of(s), stream));
        }
        if (dpoints.defined() && k.points_dim == 2) dpoints = dpoints.sum(0);
        return once(create_graph, grads, {dpoints, need_t ? dtheta : Tensor(), Tensor()});
    }
};

py::object transform_grid(const Tensor &points, const Tensor &theta, const py::handle &params,
                          const py::handle &nc, const py::handle &settings, bool exact) {
    drop_params();
    try {
        Call a{c10::make_intrusive<Kept>(), parse_settings(settings)};
        a.kept->cells = parse_cells(nc);
        a.kept->exact = exact;
        a.kept->points_dim = points.dim();
        if (theta.dim() != 2 || theta.device() != points.device()) throw Fallback();
        a.kept->theta_dim = theta.size(1);
        const bool graph = needs_graph(points, theta);
        if (graph) a.kept->params = params.inc_ref().ptr();
        return py::cast(without_gil([&] {
            if (graph) return TransformGrid::apply(points, theta, a);
            at::AutoGradMode off(false);
            Tensor A, E;
            return grid_forward(a, floats(points), floats(theta), false, &A, &E);
        }));
    } catch (Fallback &) {
        return py::none();
    }
}

// ------------------------------ transform_data -------------------------------
struct Image {
    Tensor lin;
    std::vector<int64_t> outsize;
};

void to_ints(at::IntArrayRef v, int *out) {
    for (size_t j = 0; j < v.size(); ++j) out[j] = (int)v[j];
}

Tensor image_forward(const Call &a, const Tensor &lin, const Tensor &data, const Tensor &theta,
                     bool grad, Tensor *A, Tensor *E, Tensor *grid) {
    const Cells &c = a.kept->cells;
    tables(c, a.s, theta, grad, true, A, E);
    std::vector<int64_t> shape = {data.size(0), data.size(1)};
    int64_t nP = 1;
    for (int64_t o : a.kept->outsize) {
        shape.push_back(o);
        nP *= o;
    }
    Tensor out = make(data, shape);
    if (grad && a.kept->mode != CPAB_GRAD_EXACT) *grid = make(data, {data.size(0), c.ndim, nP});
    int size[3], outsize[3];
    to_ints(data.sizes().slice(2), size);
    to_ints(a.kept->outsize, outsize);
    check(cpab_transform_data(c.ndim, c.nc, a.s.nsteps, ptr(lin), outsize, ptr(*E),
                              (int)data.size(0), ptr(data), (int)data.size(1), size, ptr(out),
                              ptr(*grid), ties_of(a.s), stream_of(data)));
    return out;
}

struct TransformData : torch::autograd::Function<TransformData> {
    static Tensor forward(AutogradContext *ctx, const Tensor &data_in, const Tensor &theta_in,
                          const Call &a, const Image &im) {
        const Tensor data = floats(data_in), theta = floats(theta_in);
        Tensor A, E, grid;
        const Tensor out = image_forward(a, im.lin, data, theta, true, &A, &E, &grid);
        keep(ctx, a.kept);
        ctx->save_for_backward({data, im.lin, A, E, grid});
        return out;
    }

    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const bool create_graph = at::GradMode::is_enabled();
        at::AutoGradMode off(false);
        const auto saved = ctx->get_saved_variables();
        const Tensor &data = saved[0], &lin = saved[1], &A = saved[2], &E = saved[3],
                     &grid = saved[4];
        const Kept &k = kept(ctx);
        const Cells &c = k.cells;
        const bool want_d = ctx->needs_input_grad(0), want_t = ctx->needs_input_grad(1);
        if (!want_d && !want_t) return {Tensor(), Tensor(), Tensor(), Tensor()};
        const Settings s = settings_now(k, data.device());
        const Tensor g = floats(grads[0]);
        const int nb = (int)data.size(0), C = (int)data.size(1), d = (int)s.basis.size(1);
        int size[3], outsize[3];
        to_ints(data.sizes().slice(2), size);
        to_ints(k.outsize, outsize);
        Tensor dtheta = make(data, {nb, d}), ddata;
        if (want_d) ddata = at::empty_like(data);
        const size_t need =
            cpab_transform_data_backward_workspace(c.ndim, c.nc, s.nsteps, k.mode, outsize, nb);
        if (need == 0 && nb > 0) raise_native(3);
        const Tensor ws = workspace(data, need);
        check_backward(cpab_transform_data_backward(
            c.ndim, c.nc, s.nsteps, k.mode, ptr(lin), outsize, ptr(A), ptr(E), ptr(grid), nb,
            ptr(data), C, size, ptr(s.basis), d, ptr(g), ptr(ddata), ptr(dtheta), ws.data_ptr(),
            (size_t)ws.numel(), ties_of(s), stream_of(data)));
        return once(create_graph, grads, {ddata, want_t ? dtheta : Tensor(), Tensor(), Tensor()});
    }
};

py::object transform_data(const Tensor &data, const Tensor &theta, const py::handle &params,
                          const py::handle &nc, const py::handle &settings, const Tensor &lin,
                          const std::vector<int64_t> &outsize) {
    drop_params();
    try {
        Call a{c10::make_intrusive<Kept>(), parse_settings(settings)};
        a.kept->cells = parse_cells(nc);
        a.kept->mode = a.s.mode;
        a.kept->outsize = outsize;
        if (theta.device() != data.device() || data.dim() != a.kept->cells.ndim + 2 ||
            (int)outsize.size() != a.kept->cells.ndim)
            throw Fallback();
        for (int64_t o : outsize)
            if (o < 1 || o > INT_MAX) throw Fallback();
        for (int64_t o : data.sizes())
            if (o > INT_MAX) throw Fallback();
        const bool graph = needs_graph(data, theta);
        if (graph) a.kept->params = params.inc_ref().ptr();
        return py::cast(without_gil([&] {
            if (graph) return TransformData::apply(data, theta, a, Image{lin, {}});
            at::AutoGradMode off(false);
            Tensor A, E, grid;
            return image_forward(a, lin, floats(data), floats(theta), false, &A, &E, &grid);
        }));
    } catch (Fallback &) {
        return py::none();
    }
}

// --------------------------- transform_data_mixed ----------------------------
struct Layout {
    Tensor plan, offsets, points;
};

Tensor pack(at::TensorList images) {
    std::vector<Tensor> flat;
    flat.reserve(images.size());
    for (const Tensor &t : images) flat.push_back(t.detach().reshape({-1}).to(at::kFloat));
    return at::cat(flat);
}

std::vector<Tensor> unpack(const Tensor &packed, const std::vector<int64_t> &sizes,
                           const std::vector<std::vector<int64_t>> &shapes) {
    std::vector<Tensor> out = packed.split_with_sizes(sizes);
    for (size_t k = 0; k < out.size(); ++k) out[k] = out[k].view(shapes[k]);
    return out;
}

struct TransformMixed : torch::autograd::Function<TransformMixed> {
    static variable_list forward(AutogradContext *ctx, at::TensorList images,
                                 const Tensor &theta_in, const Call &a, const Layout &lay) {
        const Kept &k = *a.kept;
        const Cells &c = k.cells;
        const Tensor theta = floats(theta_in), data = pack(images);
        const int64_t S = theta.size(0);
        if (data.numel() != k.C * k.data_points) throw Fallback();
        Tensor A, E;
        tables(c, a.s, theta, true, true, &A, &E);
        void *stream = stream_of(theta);
        const Tensor grid = make(theta, {c.ndim, k.total});
        const size_t need = cpab_ragged_points_workspace(c.ndim, c.nc, (int)S);
        if (need == 0) throw Fallback();
        const Tensor ws = workspace(theta, need);
        const auto *off = reinterpret_cast<const long long *>(lay.offsets.data_ptr<int64_t>());
        check(cpab_ragged_points_forward(c.ndim, c.nc, a.s.nsteps, ptr(E), (int)S, off, k.total,
                                         ptr(lay.points), ptr(grid), ws.data_ptr(),
                                         (size_t)ws.numel(), ties_of(a.s), stream));
        const Tensor out = make(theta, {k.C * k.total});
        const auto *plan = reinterpret_cast<const long long *>(lay.plan.data_ptr<int64_t>());
        check(cpab_interpolate_ragged(c.ndim, (int)S, (int)k.C, plan, k.data_points, k.total,
                                      k.tiles, ptr(data), ptr(grid), ptr(out), stream));
        keep(ctx, a.kept);
        ctx->save_for_backward({data, grid, lay.plan, lay.offsets, lay.points, A,
                                k.mode == CPAB_GRAD_EXACT ? E : Tensor()});
        return unpack(out, k.out_sizes, k.out_shapes);
    }

    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const bool create_graph = at::GradMode::is_enabled();
        at::AutoGradMode off(false);
        const auto saved = ctx->get_saved_variables();
        const Tensor &data = saved[0], &grid = saved[1], &plan = saved[2], &offsets = saved[3],
                     &points = saved[4], &A = saved[5], &E = saved[6];
        const Kept &k = kept(ctx);
        const Cells &c = k.cells;
        const size_t S = k.sizes.size();
        variable_list res(S + 3);
        bool want_d = false;
        for (size_t i = 0; i < S; ++i) want_d = want_d || ctx->needs_input_grad(i);
        const bool want_t = ctx->needs_input_grad(S);
        if (!want_d && !want_t) return res;
        const Settings s = settings_now(k, data.device());
        std::vector<Tensor> flat;
        flat.reserve(S);
        for (size_t i = 0; i < S; ++i)
            flat.push_back(grads[i].defined()
                               ? grads[i].detach().reshape({-1}).to(at::kFloat)
                               : at::zeros({k.out_sizes[i]}, data.options()));
        const Tensor g = at::cat(flat);
        Tensor ddata, dgrid;
        if (want_d) ddata = at::empty_like(data);
        if (want_t) dgrid = at::empty_like(grid);
        void *stream = stream_of(data);
        check_backward(cpab_interpolate_ragged_backward(
            c.ndim, (int)S, (int)k.C, reinterpret_cast<const long long *>(plan.data_ptr<int64_t>()),
            k.data_points, k.total, k.tiles, ptr(data), ptr(grid), ptr(g), ptr(ddata), ptr(dgrid),
            stream));
        if (want_t) {
            const int d = (int)s.basis.size(1);
            Tensor dtheta = make(data, {(int64_t)S, d});
            const size_t need = cpab_ragged_points_workspace(c.ndim, c.nc, (int)S);
            if (need == 0) raise_native(1);
            const Tensor ws = workspace(data, need);
            check_backward(cpab_ragged_points_backward(
                c.ndim, c.nc, s.nsteps, k.mode, ptr(A), ptr(E), (int)S,
                reinterpret_cast<const long long *>(offsets.data_ptr<int64_t>()), k.total,
                ptr(s.basis), d, ptr(points), ptr(dgrid), ptr(dtheta), nullptr, ws.data_ptr(),
                (size_t)ws.numel(), ties_of(s), stream));
            res[S] = dtheta;
        }
        if (want_d) {
            const std::vector<Tensor> parts = unpack(ddata, k.sizes, k.shapes);
            for (size_t i = 0; i < S; ++i)
                if (ctx->needs_input_grad(i)) res[i] = parts[i];
        }
        return once(create_graph, grads, std::move(res));
    }
};

// layout: functions.ImageLayout; returns the list of outputs, or None.
py::object transform_mixed(const std::vector<Tensor> &images, const Tensor &theta,
                           const py::handle &params, const py::handle &nc,
                           const py::handle &settings, const py::object &layout, int64_t C) {
    drop_params();
    try {
        Call a{c10::make_intrusive<Kept>(), parse_settings(settings)};
        Kept &k = *a.kept;
        k.cells = parse_cells(nc);
        k.mode = a.s.mode;
        k.C = C;
        Layout lay{py::cast<Tensor>(layout.attr("plan")), py::cast<Tensor>(layout.attr("offsets")),
                   py::cast<Tensor>(layout.attr("points"))};
        const auto totals = py::cast<std::vector<int64_t>>(layout.attr("totals"));
        const auto npoints = py::cast<std::vector<int64_t>>(layout.attr("npoints"));
        const auto outsizes =
            py::cast<std::vector<std::vector<int64_t>>>(layout.attr("outsizes"));
        if (totals.size() != 3 || npoints.size() != images.size() ||
            outsizes.size() != images.size() || (size_t)theta.size(0) != images.size() || C < 1)
            throw Fallback();
        k.data_points = totals[0];
        k.total = totals[1];
        k.tiles = totals[2];
        for (size_t i = 0; i < images.size(); ++i) {
            k.shapes.push_back(images[i].sizes().vec());
            k.sizes.push_back(images[i].numel());
            std::vector<int64_t> o = {C};
            o.insert(o.end(), outsizes[i].begin(), outsizes[i].end());
            k.out_shapes.push_back(o);
            k.out_sizes.push_back(C * npoints[i]);
        }
        a.kept->params = params.inc_ref().ptr();
        return py::cast(without_gil(
            [&] { return TransformMixed::apply(at::TensorList(images), theta, a, lay); }));
    } catch (Fallback &) {
        return py::none();
    }
}

}  // namespace

PYBIND11_MODULE(_torch_bind, m) {
    py::object settings = py::module_::import("libcpab_gb300._autograd").attr("settings");
    g_settings = settings.release().ptr();
    m.def("transform_grid", &transform_grid);
    m.def("transform_data", &transform_data);
    m.def("transform_mixed", &transform_mixed);
}
