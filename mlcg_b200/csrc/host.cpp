// The host side of the calls that a small batch waits for: addresses and layouts of lists of tensors, outputs and workspaces, and the
// library calls themselves, without a Python object per argument.  Of the 68 us of host time for an evaluation of 64 x 10 beads 21 went
// around the library call (now 61 us, the kernels take 60), of a step of Langevin dynamics of 54 beads with four priors 228 are 168
// now, of a force-matching step of 12 x 100 beads 590 are 554 (its spread from run to run is as large).  Nothing here computes: the library's entry points come as addresses,
// from the copy that the ctypes binding has loaded.
#include <torch/extension.h>

#include <string>
#include <vector>

#include "../../include/mlcg_b200.h"

namespace py = pybind11;

namespace {

decltype(&mlcgb_schnet_evaluate) g_evaluate = nullptr;
decltype(&mlcgb_schnet_evaluate_workspace_bytes) g_evaluate_bytes = nullptr;
decltype(&mlcgb_prior_eval) g_prior_eval = nullptr;
decltype(&mlcgb_prior_eval_workspace_bytes) g_prior_eval_bytes = nullptr;

void bind(uintptr_t evaluate, uintptr_t evaluate_bytes, uintptr_t prior_eval, uintptr_t prior_eval_bytes) {
    g_evaluate = reinterpret_cast<decltype(g_evaluate)>(evaluate);
    g_evaluate_bytes = reinterpret_cast<decltype(g_evaluate_bytes)>(evaluate_bytes);
    g_prior_eval = reinterpret_cast<decltype(g_prior_eval)>(prior_eval);
    g_prior_eval_bytes = reinterpret_cast<decltype(g_prior_eval_bytes)>(prior_eval_bytes);
}

const at::Tensor &tensor_of(PyObject *o) {
    if (!THPVariable_Check(o)) throw py::type_error("a tensor is wanted");
    return THPVariable_Unpack(o);
}

void *address(const c10::optional<at::Tensor> &t) { return t ? t->data_ptr() : nullptr; }

// every tensor whose address a kernel gets is on the device of the first one
struct SameDevice {
    int device = -1;
    void operator()(const at::Tensor &t) {
        if (!t.is_cuda()) throw std::runtime_error("mlcg_b200 operators run on CUDA tensors only (there is no CPU fallback)");
        if (device < 0) device = t.get_device();
        else if (t.get_device() != device)
            throw std::runtime_error("mlcg_b200: tensors on different devices (cuda:" + std::to_string(device) + " and " + t.device().str() + ")");
    }
    void operator()(const c10::optional<at::Tensor> &t) {
        if (t) (*this)(*t);
    }
};

// addresses of the tensors of a list (None left out) as bytes; None where one of them is not contiguous
py::object pointers(const py::list &list) {
    std::vector<void *> at;
    at.reserve(list.size());
    for (py::handle h : list) {
        if (h.is_none()) continue;
        const at::Tensor &t = tensor_of(h.ptr());
        if (!t.is_contiguous()) return py::none();
        at.push_back(t.data_ptr());
    }
    return py::bytes(reinterpret_cast<const char *>(at.data()), at.size() * sizeof(void *));
}

// address, in-place version, shape and strides of every tensor of a sequence, as bytes; in front of them dtype, device and length of `like`
py::bytes layouts(const py::tuple &list, const c10::optional<at::Tensor> &like) {
    std::vector<int64_t> v;
    v.reserve(8 * list.size() + 4);
    if (like) v = {(int64_t)like->scalar_type(), (int64_t)like->device().type(), (int64_t)like->device().index(), like->size(0)};
    for (py::handle h : list) {
        const at::Tensor &t = tensor_of(h.ptr());
        v.push_back(reinterpret_cast<int64_t>(t.data_ptr()));
        v.push_back(t._version());
        v.push_back(t.dim());
        v.insert(v.end(), t.sizes().begin(), t.sizes().end());
        v.insert(v.end(), t.strides().begin(), t.strides().end());
    }
    return py::bytes(reinterpret_cast<const char *>(v.data()), v.size() * sizeof(int64_t));
}

// one contiguous view of `flat` after the other, shaped like the tensors of `like`
std::vector<at::Tensor> views(const at::Tensor &flat, const py::list &like) {
    std::vector<at::Tensor> out;
    out.reserve(like.size());
    int64_t at = flat.storage_offset();
    std::vector<int64_t> strides;
    for (py::handle h : like) {
        const at::Tensor &t = tensor_of(h.ptr());
        strides.assign(t.dim(), 1);
        for (int64_t d = t.dim() - 2; d >= 0; d--) strides[d] = strides[d + 1] * t.size(d + 1);
        out.push_back(flat.as_strided(t.sizes(), strides, at));
        at += t.numel();
    }
    return out;
}

// mlcgb_schnet_evaluate with its outputs and workspaces: (code, host [5], energy, gradient or forces, workspace, graph workspace)
py::tuple evaluate(const at::Tensor &pos_in, const at::Tensor &types, const c10::optional<at::Tensor> &n_atoms, const c10::optional<at::Tensor> &ptr, double r,
                   int64_t max_nn, uintptr_t spec, int cutoff_kind, double lower, double upper, uintptr_t weights, int precision, bool forces, bool training,
                   int64_t edges, const c10::optional<at::Tensor> &pending, const at::Tensor &status, uintptr_t stream) {
    SameDevice check;
    check(pos_in); check(types); check(n_atoms); check(ptr);
    const at::NoGradGuard guard;
    const at::Tensor pos = pos_in.contiguous();
    const int64_t N = pos.size(0), B = n_atoms ? n_atoms->numel() : ptr->numel() - 1;
    const auto *rbf = reinterpret_cast<const mlcgb_rbf_spec *>(spec);
    const auto *w = reinterpret_cast<const mlcgb_schnet_weights *>(weights);
    const auto floats = pos.options(), bytes = floats.dtype(at::kByte);
    const at::Tensor energy = at::empty({B}, floats), grad = at::empty({N, 3}, floats);
    const int64_t graph_bytes = (int64_t)g_evaluate_bytes(N, B, -1, 0, w, 0);
    int64_t size = (int64_t)g_evaluate_bytes(N, B, edges, rbf->num_rbf, w, training);
    const at::Tensor graph_ws = at::empty({graph_bytes}, bytes);
    at::Tensor ws = at::empty({size}, bytes);
    int64_t host[5] = {0, 0, 0, 0, 0};
    int code;
    while (true) {
        {
            py::gil_scoped_release unlocked;               // (the call waits for the device)
            code = g_evaluate(pos.data_ptr(), types.data_ptr<int64_t>(), (const int64_t *)address(n_atoms), (const int64_t *)address(ptr), N, B, r, max_nn, rbf,
                              cutoff_kind, lower, upper, w, precision, forces, training, graph_ws.data_ptr(), (size_t)graph_bytes, ws.data_ptr(), (size_t)size,
                              energy.data_ptr(), grad.data_ptr(), (const int32_t *)address(pending), (int32_t *)status.data_ptr(), host, (void *)stream);
        }
        if (code || host[4] != MLCGB_EVALUATE_MORE) break;
        ws = at::Tensor();
        size = (int64_t)g_evaluate_bytes(N, B, host[0], rbf->num_rbf, w, training);
        ws = at::empty({size}, bytes);
    }
    return py::make_tuple(code, py::make_tuple(host[0], host[1], host[2], host[3], host[4]), energy, grad, ws, graph_ws);
}

// mlcgb_prior_eval of lists (kind, idx, params, symmetric, sliced): (code, energy [rows, B], gradient [rows, N, 3]), rows = lists and, with
// `totals`, their sums
py::tuple prior_eval(const py::list &lists, const at::Tensor &pos_in, const c10::optional<at::Tensor> &batch_in, int64_t B, bool deterministic, bool forces,
                     bool totals, const at::Tensor &status, uintptr_t stream) {
    SameDevice check;
    check(pos_in); check(batch_in);
    const at::NoGradGuard guard;
    const int n = (int)lists.size();
    const at::Tensor pos = pos_in.contiguous();
    const int64_t N = pos.size(0);
    c10::optional<at::Tensor> batch;
    if (batch_in) {
        batch = batch_in->to(at::kLong).contiguous();
        if (batch->numel() != N) throw py::value_error("batch must have one entry per bead");
    }
    mlcgb_prior_list a[MLCGB_MAX_PRIOR_SEGMENTS] = {};
    std::vector<at::Tensor> keep;
    for (int k = 0; k < n; k++) {
        const py::tuple l = lists[k];
        at::Tensor params;
        if (!l[4].is_none()) {
            const py::tuple s = l[4];
            const at::Tensor &slices = tensor_of(s[0].ptr()), &beads = tensor_of(s[1].ptr()), &offsets = tensor_of(s[2].ptr());
            params = tensor_of(s[3].ptr());
            check(slices); check(beads); check(offsets); check(params);
            a[k].M = offsets.size(0) * 128;
            a[k].n_slices = slices.size(0);
            a[k].steps = offsets.size(0);
            a[k].slices = (const int32_t *)slices.data_ptr();
            a[k].slice_beads = (const int32_t *)beads.data_ptr();
            a[k].offsets = (const uint16_t *)offsets.data_ptr();
            a[k].slice_params = params.data_ptr();
        } else {
            const at::Tensor idx = tensor_of(l[1].ptr()).contiguous();
            params = tensor_of(l[2].ptr()).contiguous();
            check(idx); check(params);
            if (idx.scalar_type() != at::kInt) throw py::type_error("prior lists take int32 indices");
            a[k].M = idx.size(1);
            a[k].idx = (const int32_t *)idx.data_ptr();
            a[k].params = params.data_ptr();
            keep.push_back(idx);
            keep.push_back(params);
        }
        if (params.scalar_type() != pos.scalar_type()) throw py::type_error("prior lists take parameters of the positions' dtype");
        a[k].kind = l[0].cast<int>();
        a[k].n_params = (int)params.size(0);
        a[k].symmetric = l[3].cast<bool>();
    }
    const int64_t rows = totals ? n + 1 : n;
    const int dtype = pos.scalar_type() == at::kFloat ? MLCGB_F32 : MLCGB_F64;
    const at::Tensor buf = at::empty({rows * (3 * N + B)}, pos.options());
    const at::Tensor grad = buf.as_strided({rows, N, 3}, {3 * N, 3, 1}, 0), energy = buf.as_strided({rows, B}, {B, 1}, rows * 3 * N);
    const size_t bytes = g_prior_eval_bytes(n, N, B, dtype), item = (size_t)pos.element_size();
    const at::Tensor ws = at::empty({(int64_t)bytes}, pos.options().dtype(at::kByte));
    char *e = (char *)energy.data_ptr(), *g = (char *)grad.data_ptr();
    int code;
    {
        py::gil_scoped_release unlocked;
        code = g_prior_eval(n, a, pos.data_ptr(), dtype, (const int64_t *)address(batch), N, B, e, g, forces, totals ? e + item * (size_t)(n * B) : nullptr,
                            totals ? g + item * (size_t)(n * 3 * N) : nullptr, deterministic, ws.data_ptr(), bytes, (int32_t *)status.data_ptr(), (void *)stream);
    }
    return py::make_tuple(code, energy, grad);
}

}  // namespace

PYBIND11_MODULE(_native, m) {
    m.def("bind", &bind);
    m.def("pointers", &pointers);
    m.def("layouts", &layouts, py::arg("list"), py::arg("like") = py::none());
    m.def("views", &views);
    m.def("evaluate", &evaluate);
    m.def("prior_eval", &prior_eval);
}
