// The decode loop's calls from Python, without Python in between: the argument
// blocks of include/lily_sampler.h are filled straight from torch tensors, ctypes
// parameter structs and plain lists. A call that this file does not know how to
// read (an argument of another type, a tensor that is not contiguous) returns None,
// and the caller takes its own path, which names what is wrong.
//
// Why: a step over a few rows is some ten microseconds of GPU time; marshalling it
// through ctypes took 9 (an argmax) to 29 us (64 rows) of host time per call.
#include <Python.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <vector>

#include "../../include/lily_sampler.h"

namespace {

PyTypeObject *g_params_type = nullptr;  // SamplingParams, a ctypes structure
PyObject *g_names[32];
enum Name {
    N_UNIFORMS, N_STEPS, N_HISTORY_IDS, N_HISTORY_LEN, N_BIAS_IDS, N_BIAS_VALS, N_BIAS_LEN, N_BAN_IDS, N_BAN_LEN,
    N_FORCED_IDS, N_COUNT_SLOTS, N_OUT_STATUS, N_KEPT_N, N_KEPT_IDS, N_KEPT_PROBS, N_PARAMS_ON_DEVICE, N_MODE, N_Q_DENSE,
    N_Q_IDS, N_Q_PROBS, N_Q_N, N_U_ACCEPT, N_U_RESID, N_STEP0, N_COUNT_SLOT, N_OUT_LSE, N_COUNT
};
const char *const kNames[N_COUNT] = {
    "uniforms", "steps", "history_ids", "history_len", "bias_ids", "bias_vals", "bias_len", "ban_ids", "ban_len",
    "forced_ids", "count_slots", "out_status", "kept_n", "kept_ids", "kept_probs", "params_on_device", "mode", "q_dense",
    "q_ids", "q_probs", "q_n", "u_accept", "u_resid", "step0", "count_slot", "out_lse"};

// A call that has to go the other way.
struct Other {};

const at::Tensor *tensor(PyObject *o) {
    if (o == nullptr || o == Py_None) {
        return nullptr;
    }
    if (!THPVariable_Check(o)) {
        throw Other();
    }
    const at::Tensor &t = THPVariable_Unpack(o);
    if (!t.is_contiguous()) {
        throw Other();
    }
    return &t;
}

template <typename P>
P *address(PyObject *o) {
    const at::Tensor *t = tensor(o);
    return t ? static_cast<P *>(t->data_ptr()) : nullptr;
}

uint64_t pitch(const at::Tensor &t) {
    if (t.dim() == 0) {
        throw Other();
    }
    return (uint64_t)(t.dim() == 2 && t.size(0) > 1 ? t.stride(0) : t.size(-1));
}

uint32_t dtype_code(const at::Tensor &t) {
    if (t.scalar_type() == at::kFloat) {
        return LILY_F32;
    }
    if (t.scalar_type() == at::kBFloat16) {
        return LILY_BF16;
    }
    throw Other();
}

// The call's stream: torch's current one for None, else the object's handle.
void *stream_of(PyObject *o) {
    if (o == Py_None) {
        return c10::cuda::getCurrentCUDAStream().stream();
    }
    PyObject *v = PyObject_GetAttrString(o, "cuda_stream");
    if (v == nullptr) {
        PyErr_Clear();
        throw Other();
    }
    void *p = PyLong_AsVoidPtr(v);
    Py_DECREF(v);
    if (p == nullptr && PyErr_Occurred()) {
        PyErr_Clear();
        throw Other();
    }
    return p;
}

// The items of a list or tuple of exactly n.
PyObject **items(PyObject *o, Py_ssize_t n) {
    if (PyList_CheckExact(o) && PyList_GET_SIZE(o) == n) {
        return reinterpret_cast<PyListObject *>(o)->ob_item;
    }
    if (PyTuple_CheckExact(o) && PyTuple_GET_SIZE(o) == n) {
        return reinterpret_cast<PyTupleObject *>(o)->ob_item;
    }
    throw Other();
}

uint32_t word(PyObject *o) {
    if (!PyLong_CheckExact(o)) {
        throw Other();
    }
    return (uint32_t)PyLong_AsUnsignedLongMask(o);
}

// The bytes of a ctypes structure.
void struct_bytes(PyObject *o, void *to, size_t n) {
    Py_buffer b;
    if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0) {
        PyErr_Clear();
        throw Other();
    }
    const bool fits = b.len == (Py_ssize_t)n;
    if (fits) {
        std::memcpy(to, b.buf, n);
    }
    PyBuffer_Release(&b);
    if (!fits) {
        throw Other();
    }
}

void one_params(PyObject *o, lily_sampling_params_t *to) {
    if (Py_TYPE(o) != g_params_type) {
        throw Other();
    }
    struct_bytes(o, to, sizeof(*to));
}

// Host arrays of a call, kept between calls (one set per thread).
struct Rows {
    std::vector<lily_sampling_params_t> params;
    std::vector<uint32_t> steps, slots;
};
thread_local Rows t_rows;

const lily_sampling_params_t *params_of(PyObject *list, Py_ssize_t rows) {
    PyObject **p = items(list, rows);
    t_rows.params.resize((size_t)rows);
    for (Py_ssize_t r = 0; r < rows; ++r) {
        // (The same request on neighbouring rows is read once.)
        if (r != 0 && p[r] == p[r - 1]) {
            t_rows.params[(size_t)r] = t_rows.params[(size_t)r - 1];
        } else {
            one_params(p[r], &t_rows.params[(size_t)r]);
        }
    }
    return t_rows.params.data();
}

const uint32_t *words_of(PyObject *list, Py_ssize_t rows, std::vector<uint32_t> &to) {
    PyObject **p = items(list, rows);
    to.resize((size_t)rows);
    for (Py_ssize_t r = 0; r < rows; ++r) {
        to[(size_t)r] = word(p[r]);
    }
    return to.data();
}

// Keyword arguments: what is there and not None; `left` counts those not asked for.
struct Keywords {
    PyObject *dict;
    Py_ssize_t left;
    explicit Keywords(PyObject *d) : dict(d), left(PyDict_GET_SIZE(d)) {}
    PyObject *get(Name n) {
        if (left == 0) {
            return nullptr;
        }
        PyObject *v = PyDict_GetItemWithError(dict, g_names[n]);
        if (v == nullptr) {
            if (PyErr_Occurred()) {
                PyErr_Clear();
                throw Other();
            }
            return nullptr;
        }
        --left;
        return v == Py_None ? nullptr : v;
    }
    void done() const {
        if (left != 0) {
            throw Other();  // a name this call does not have
        }
    }
};

lily_sampler_t *handle(PyObject *o) {
    if (!PyLong_Check(o)) {
        throw Other();
    }
    void *p = PyLong_AsVoidPtr(o);
    if (p == nullptr) {
        PyErr_Clear();
        throw Other();
    }
    return static_cast<lily_sampler_t *>(p);
}

template <typename F>
PyObject *guarded(Py_ssize_t n, Py_ssize_t want, F f) {
    try {
        if (n != want) {
            throw Other();
        }
        return PyLong_FromLong(f());
    } catch (const Other &) {
        Py_RETURN_NONE;
    } catch (const std::exception &) {
        Py_RETURN_NONE;
    }
}

template <typename F>
int32_t unlocked(F f) {
    int32_t st;
    Py_BEGIN_ALLOW_THREADS;
    st = f();
    Py_END_ALLOW_THREADS;
    return st;
}

// sample_batch(handle, stream, logits, params, out_ids, keywords)
PyObject *py_sample_batch(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded(n, 6, [&]() -> int32_t {
        const at::Tensor *logits = tensor(v[2]);
        if (logits == nullptr) {
            throw Other();
        }
        Keywords kw(v[5]);
        lily_sample_args_t a;
        std::memset(&a, 0, sizeof a);
        a.struct_size = sizeof a;
        a.rows = (uint32_t)(logits->dim() == 2 ? logits->size(0) : 1);
        a.logits = logits->data_ptr();
        a.logits_dtype = dtype_code(*logits);
        a.logits_ld = pitch(*logits);
        PyObject *on_device = kw.get(N_PARAMS_ON_DEVICE), *steps = kw.get(N_STEPS);
        if (on_device != nullptr && on_device != Py_False && on_device != Py_True) {
            throw Other();
        }
        if (on_device == Py_True) {
            a.params_on_device = 1;
            a.params = address<const lily_sampling_params_t>(v[3]);
            a.steps = address<const uint32_t>(steps);
        } else {
            a.params = params_of(v[3], a.rows);
            if (steps != nullptr) {
                a.steps = words_of(steps, a.rows, t_rows.steps);
            }
        }
        a.uniforms = address<const float>(kw.get(N_UNIFORMS));
        PyObject *hist = kw.get(N_HISTORY_IDS), *hist_len = kw.get(N_HISTORY_LEN);
        if (hist != nullptr) {
            const at::Tensor *t = tensor(hist);
            a.history_ids = static_cast<const uint32_t *>(t->data_ptr());
            a.history_len = address<const uint32_t>(hist_len);
            a.history_ld = pitch(*t);
        }
        PyObject *bias = kw.get(N_BIAS_IDS), *bias_vals = kw.get(N_BIAS_VALS), *bias_len = kw.get(N_BIAS_LEN);
        if (bias != nullptr) {
            const at::Tensor *t = tensor(bias);
            a.bias_ids = static_cast<const uint32_t *>(t->data_ptr());
            a.bias_vals = address<const float>(bias_vals);
            a.bias_len = address<const uint32_t>(bias_len);
            a.bias_ld = pitch(*t);
        }
        PyObject *ban = kw.get(N_BAN_IDS), *ban_len = kw.get(N_BAN_LEN);
        if (ban != nullptr) {
            const at::Tensor *t = tensor(ban);
            a.ban_ids = static_cast<const uint32_t *>(t->data_ptr());
            a.ban_len = address<const uint32_t>(ban_len);
            a.ban_ld = pitch(*t);
        }
        a.forced_ids = address<const int32_t>(kw.get(N_FORCED_IDS));
        if (PyObject *slots = kw.get(N_COUNT_SLOTS)) {
            a.count_slots = words_of(slots, a.rows, t_rows.slots);
        }
        a.out_ids = address<uint32_t>(v[4]);
        a.out_status = address<uint32_t>(kw.get(N_OUT_STATUS));
        PyObject *kept_n = kw.get(N_KEPT_N), *kept_ids = kw.get(N_KEPT_IDS), *kept_probs = kw.get(N_KEPT_PROBS);
        if (kept_n != nullptr) {
            const at::Tensor *t = tensor(kept_ids);
            if (t == nullptr) {
                throw Other();
            }
            a.kept_n = address<uint32_t>(kept_n);
            a.kept_ids = static_cast<uint32_t *>(t->data_ptr());
            a.kept_probs = address<float>(kept_probs);
            a.kept_ld = pitch(*t);
        }
        kw.done();
        lily_sampler_t *h = handle(v[0]);
        void *stream = stream_of(v[1]);
        return unlocked([&] { return lily_sample_batch(h, stream, &a); });
    });
}

// sample_prepared(handle, stream, argument block)
PyObject *py_sample_prepared(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded(n, 3, [&]() -> int32_t {
        lily_sample_args_t a;
        struct_bytes(v[2], &a, sizeof a);
        lily_sampler_t *h = handle(v[0]);
        void *stream = stream_of(v[1]);
        return unlocked([&] { return lily_sample_batch(h, stream, &a); });
    });
}

// sample_one(handle, stream, logits, params, step, out, history or None)
PyObject *py_sample_one(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded(n, 7, [&]() -> int32_t {
        const at::Tensor *logits = tensor(v[2]), *hist = tensor(v[6]);
        if (logits == nullptr) {
            throw Other();
        }
        lily_sampling_params_t p;
        one_params(v[3], &p);
        const uint32_t step = word(v[4]), dtype = dtype_code(*logits);
        uint32_t *out = address<uint32_t>(v[5]);
        lily_sampler_t *h = handle(v[0]);
        void *stream = stream_of(v[1]);
        return unlocked([&] {
            return lily_sample_one(h, stream, logits->data_ptr(), dtype, (uint64_t)logits->numel(), &p, step,
                                   hist ? static_cast<const uint32_t *>(hist->data_ptr()) : nullptr,
                                   hist ? (uint32_t)hist->numel() : 0u, out);
        });
    });
}

// argmax_batch(handle, stream, logits, out_ids)
PyObject *py_argmax_batch(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded(n, 4, [&]() -> int32_t {
        const at::Tensor *logits = tensor(v[2]);
        if (logits == nullptr) {
            throw Other();
        }
        const uint32_t rows = (uint32_t)(logits->dim() == 2 ? logits->size(0) : 1), dtype = dtype_code(*logits);
        const uint64_t ld = pitch(*logits);
        uint32_t *out = address<uint32_t>(v[3]);
        lily_sampler_t *h = handle(v[0]);
        void *stream = stream_of(v[1]);
        return unlocked([&] { return lily_argmax_batch(h, stream, logits->data_ptr(), dtype, ld, rows, out); });
    });
}

// spec_verify(handle, stream, target_logits, params, draft_ids, out_ids, out_accepted, keywords)
PyObject *py_spec_verify(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded(n, 8, [&]() -> int32_t {
        const at::Tensor *target = tensor(v[2]);
        if (target == nullptr || target->dim() == 0) {
            throw Other();
        }
        Keywords kw(v[7]);
        lily_spec_args_t a;
        std::memset(&a, 0, sizeof a);
        a.struct_size = sizeof a;
        a.m = (uint32_t)target->size(0);
        a.target_logits = target->data_ptr();
        a.logits_dtype = dtype_code(*target);
        PyObject *mode = kw.get(N_MODE), *step0 = kw.get(N_STEP0), *slot = kw.get(N_COUNT_SLOT);
        a.mode = mode ? word(mode) : (uint32_t)LILY_SPEC_REJECTION;
        a.logits_ld = pitch(*target);
        lily_sampling_params_t p;
        one_params(v[3], &p);
        a.params = &p;
        a.draft_ids = address<const uint32_t>(v[4]);
        if (PyObject *q = kw.get(N_Q_DENSE)) {
            const at::Tensor *t = tensor(q);
            a.q_dense = static_cast<const float *>(t->data_ptr());
            a.q_ld = pitch(*t);
        }
        a.q_ids = address<const uint32_t>(kw.get(N_Q_IDS));
        a.q_probs = address<const float>(kw.get(N_Q_PROBS));
        a.q_n = address<const uint32_t>(kw.get(N_Q_N));
        a.u_accept = address<const float>(kw.get(N_U_ACCEPT));
        a.u_resid = address<const float>(kw.get(N_U_RESID));
        a.step0 = step0 ? word(step0) : 0u;
        if (PyObject *hist = kw.get(N_HISTORY_IDS)) {
            const at::Tensor *t = tensor(hist);
            a.history_ids = static_cast<const uint32_t *>(t->data_ptr());
            a.history_len = (uint32_t)t->numel();
        }
        uint32_t slot_word = 0;
        if (slot != nullptr) {
            slot_word = word(slot);
            a.count_slot = &slot_word;
        }
        a.out_ids = address<uint32_t>(v[5]);
        a.out_accepted = address<uint32_t>(v[6]);
        a.out_status = address<uint32_t>(kw.get(N_OUT_STATUS));
        kw.done();
        lily_sampler_t *h = handle(v[0]);
        void *stream = stream_of(v[1]);
        return unlocked([&] { return lily_spec_verify(h, stream, &a); });
    });
}

lily_lmhead_t head_of(PyObject *weights, PyObject *scales, PyObject *biases, PyObject *bits) {
    const at::Tensor *w = tensor(weights);
    if (w == nullptr || w->dim() != 2) {
        throw Other();
    }
    lily_lmhead_t hd;
    std::memset(&hd, 0, sizeof hd);
    hd.struct_size = sizeof hd;
    hd.code_bits = word(bits);
    hd.rows = (uint32_t)w->size(0);
    hd.hidden = (uint32_t)w->size(1) * (hd.code_bits == 4u ? 2u : 1u);
    hd.group = 64;
    hd.weights = static_cast<const int8_t *>(w->data_ptr());
    hd.scales_bf16 = address<const void>(scales);
    hd.biases_bf16 = address<const void>(biases);
    return hd;
}

// lmhead_logits(handle, stream, weights, scales, hidden, out_logits, biases, code_bits)
PyObject *py_lmhead_logits(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded(n, 8, [&]() -> int32_t {
        const lily_lmhead_t hd = head_of(v[2], v[3], v[6], v[7]);
        const at::Tensor *hidden = tensor(v[4]), *out = tensor(v[5]);
        if (hidden == nullptr || out == nullptr || hidden->dim() == 0) {
            throw Other();
        }
        const uint64_t hidden_ld = pitch(*hidden), out_ld = pitch(*out);
        lily_sampler_t *h = handle(v[0]);
        void *stream = stream_of(v[1]);
        return unlocked([&] {
            return lily_lmhead_logits(h, stream, &hd, hidden->data_ptr(), hidden_ld, (uint32_t)hidden->size(0),
                                      static_cast<float *>(out->data_ptr()), out_ld);
        });
    });
}

// lmhead_shard_candidates(handle, stream, weights, scales, hidden, params, records, first_id, want_sums, biases, code_bits)
PyObject *py_lmhead_shard_candidates(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded(n, 11, [&]() -> int32_t {
        const lily_lmhead_t hd = head_of(v[2], v[3], v[9], v[10]);
        const at::Tensor *hidden = tensor(v[4]);
        if (hidden == nullptr || hidden->dim() == 0) {
            throw Other();
        }
        lily_sample_args_t a;
        std::memset(&a, 0, sizeof a);
        a.struct_size = sizeof a;
        a.rows = (uint32_t)hidden->size(0);
        a.params = params_of(v[5], a.rows);
        void *records = address<void>(v[6]);
        const uint32_t first_id = word(v[7]);
        const int want_sums = PyObject_IsTrue(v[8]);
        const uint64_t hidden_ld = pitch(*hidden);
        lily_sampler_t *h = handle(v[0]);
        void *stream = stream_of(v[1]);
        return unlocked([&] {
            return lily_lmhead_shard_candidates(h, stream, &hd, hidden->data_ptr(), hidden_ld, &a, first_id,
                                                want_sums > 0 ? 1 : 0, records);
        });
    });
}

// merge_draw(handle, stream, gathered, params, out_ids, keywords)
PyObject *py_merge_draw(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded(n, 6, [&]() -> int32_t {
        const at::Tensor *gathered = tensor(v[2]);
        if (gathered == nullptr || gathered->dim() < 2) {
            throw Other();
        }
        Keywords kw(v[5]);
        lily_sample_args_t a;
        std::memset(&a, 0, sizeof a);
        a.struct_size = sizeof a;
        a.rows = (uint32_t)gathered->size(1);
        a.params = params_of(v[3], a.rows);
        if (PyObject *steps = kw.get(N_STEPS)) {
            a.steps = words_of(steps, a.rows, t_rows.steps);
        }
        a.uniforms = address<const float>(kw.get(N_UNIFORMS));
        a.out_ids = address<uint32_t>(v[4]);
        a.out_status = address<uint32_t>(kw.get(N_OUT_STATUS));
        PyObject *kept_n = kw.get(N_KEPT_N), *kept_ids = kw.get(N_KEPT_IDS), *kept_probs = kw.get(N_KEPT_PROBS);
        if (kept_n != nullptr) {
            const at::Tensor *t = tensor(kept_ids);
            if (t == nullptr) {
                throw Other();
            }
            a.kept_n = address<uint32_t>(kept_n);
            a.kept_ids = static_cast<uint32_t *>(t->data_ptr());
            a.kept_probs = address<float>(kept_probs);
            a.kept_ld = pitch(*t);
        }
        float *lse = address<float>(kw.get(N_OUT_LSE));
        kw.done();
        const uint32_t shards = (uint32_t)gathered->size(0);
        lily_sampler_t *h = handle(v[0]);
        void *stream = stream_of(v[1]);
        return unlocked([&] { return lily_merge_draw(h, stream, gathered->data_ptr(), shards, a.rows, &a, lse); });
    });
}

// bind(SamplingParams)
PyObject *py_bind(PyObject *, PyObject *type) {
    if (!PyType_Check(type)) {
        PyErr_SetString(PyExc_TypeError, "the parameter structure's type");
        return nullptr;
    }
    Py_INCREF(type);
    g_params_type = reinterpret_cast<PyTypeObject *>(type);
    Py_RETURN_NONE;
}

template <PyObject *(*F)(PyObject *, PyObject *const *, Py_ssize_t)>
PyCFunction fast() {
    return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F));
}

PyMethodDef g_methods[] = {{"bind", py_bind, METH_O, nullptr},
                           {"sample_batch", fast<py_sample_batch>(), METH_FASTCALL, nullptr},
                           {"sample_prepared", fast<py_sample_prepared>(), METH_FASTCALL, nullptr},
                           {"sample_one", fast<py_sample_one>(), METH_FASTCALL, nullptr},
                           {"argmax_batch", fast<py_argmax_batch>(), METH_FASTCALL, nullptr},
                           {"spec_verify", fast<py_spec_verify>(), METH_FASTCALL, nullptr},
                           {"lmhead_logits", fast<py_lmhead_logits>(), METH_FASTCALL, nullptr},
                           {"lmhead_shard_candidates", fast<py_lmhead_shard_candidates>(), METH_FASTCALL, nullptr},
                           {"merge_draw", fast<py_merge_draw>(), METH_FASTCALL, nullptr},
                           {nullptr, nullptr, 0, nullptr}};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_lily_calls", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__lily_calls(void) {
    for (int i = 0; i < N_COUNT; ++i) {
        g_names[i] = PyUnicode_InternFromString(kNames[i]);
        if (g_names[i] == nullptr) {
            return nullptr;
        }
    }
    return PyModule_Create(&g_module);
}
