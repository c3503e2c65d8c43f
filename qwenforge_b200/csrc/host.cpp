// The launches of a prompt step's longest stretches, issued from native code: a norm; queries, keys and values, attention and output
// projection; gate, up and down; three recurrent mixers whole. The kernels and the library products are those that the Python entries of
// ops/kernels.py launch one by one, where a layer of few microseconds a kernel waits for its arguments to be made (a launch 4 to 5
// microseconds of host time beside 2 to 3 of the driver's own, a buffer 3 to 5; here 3 and 1).
// Every function looks at its tensors as those entries do and answers None, having done nothing, for what it does not take: the caller then
// goes their way, where the same condition is reported or another kernel chosen. Nothing is kept between calls but the entries' addresses.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

namespace {

typedef cudaStream_t Stream;
struct QkvArgs {   // TcQkvArgs of tc_gemm.cu
    const void* bias;
    const void* angles;
    const int *tok_pos, *tok_seq, *slots;
    void *q_out, *kv_base;
    const int* table;
    long long page_elems;
    int table_stride, n_heads, kv_heads, head_dim, write_cache;
    const float* inv_freq;
};

int (*add_rms_norm)(int, float*, const void*, const void*, void*, int, int, float, int, Stream);
int (*qkv_pairs_pays)(int, int, int, int);
int (*qkv_pairs)(const void*, int, const void*, int, int, int, const QkvArgs*, int*, Stream);
int (*prefill_tc)(const void*, void*, const int*, const int*, const int*, void*, const int*, long long, int, int, int, int, int, int, int, int,
                  float, int, int*, const float*, int, Stream);
int (*tc_is_persistent)(int, int, int);
int (*tc_gemm)(int, const void*, int, const void*, int, void*, int, int, int, int, int*, Stream);
int (*tc_gemm_tail)(const void*, int, const void*, int, void*, int, float*, int, int, int, int, int*, Stream);
int (*stabilized_gates)(const float*, int, const float*, float, const int*, const int*, int, float*, long long, long long, int, float*, float*,
                        float*, Stream);
int (*state_chunks)(const void*, int, const void*, int, const void*, int, const float*, const float*, const float*, const float*, int, const int*,
                    const int*, int, int, float*, long long, long long, long long, int, int, int, int, float, float*, long long, int, float*,
                    float*, Stream);
int (*gated_group_norm)(int, const float*, const void*, int, const void*, float, void*, int, int, int, int, int, int, const float*, const float*,
                        float, const float*, const void*, int, Stream);
int (*rope_cache_write)(int, const void*, const void*, int, const int*, const int*, const int*, const float*, int, int, void*, void*, const int*, long long, int,
                        int, int, int, int, int*, Stream);
int (*swiglu)(int, const void*, void*, int, int, Stream);
int (*causal_conv)(int, const void*, int, const float*, const float*, const int*, const int*, const int*, int, float*, long long, long long, int, int, int,
                   void*, int, int, Stream);
int (*row_chunks)(const void*, int, const void*, int, const void*, int, const float*, const float*, int, float, const float*, const int*, const int*, int, int,
                  float*, long long, long long, int, int, int, float, float*, long long, int, float*, Stream);
PyObject* kernel_error = nullptr;

const struct {
    const char* name;
    void** to;
} entries[] = {{"qf_add_rms_norm", (void**)&add_rms_norm}, {"qf_tc_gemm_qkv_pairs_pays", (void**)&qkv_pairs_pays},
               {"qf_tc_gemm_qkv_pairs", (void**)&qkv_pairs}, {"qf_attention_prefill_tc_ex", (void**)&prefill_tc},
               {"qf_tc_gemm_is_persistent", (void**)&tc_is_persistent}, {"qf_tc_gemm", (void**)&tc_gemm}, {"qf_tc_gemm_tail", (void**)&tc_gemm_tail},
               {"qf_stabilized_gates", (void**)&stabilized_gates}, {"qf_state_chunks", (void**)&state_chunks},
               {"qf_gated_group_norm", (void**)&gated_group_norm}, {"qf_rope_cache_write", (void**)&rope_cache_write}, {"qf_swiglu", (void**)&swiglu},
               {"qf_causal_conv", (void**)&causal_conv}, {"qf_row_chunks", (void**)&row_chunks}};

// setup(KernelError, {name: address}): some of the entries, or more of them later.
PyObject* setup(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 2 || !PyDict_Check(args[1])) return PyErr_Format(PyExc_TypeError, "setup(error, addresses)");
    Py_INCREF(args[0]);
    Py_XDECREF(kernel_error);
    kernel_error = args[0];
    for (const auto& e : entries)
        if (PyObject* at = PyDict_GetItemString(args[1], e.name)) *e.to = PyLong_AsVoidPtr(at);
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
}

// ---- arguments
const at::Tensor* tensor(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }
long long number(PyObject* o) { return PyLong_AsLongLong(o); }

bool whole(const at::Tensor* t, at::ScalarType type) { return t && t->is_cuda() && t->scalar_type() == type && t->is_contiguous(); }
const int* ints(const at::Tensor* t) { return t->const_data_ptr<int>(); }
template <typename T = void> T* at_ptr(const at::Tensor& t) { return static_cast<T*>(t.data_ptr()); }
bool on16(const at::Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }
// What `tc_gemm_takes` asks of a matrix: rows on 16-byte boundaries.
bool rows16(const at::Tensor* t) {
    return t && t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->dim() == 2 && t->stride(1) == 1 && t->size(1) % 8 == 0 && t->stride(0) % 8 == 0 && on16(*t);
}
// Floats of a buffer, up to whole 256 bytes, where small buffers share an allocation. The large ones, rows in float32 and the chunks' records,
// have allocations of their own: a state space of 28 heads, microseconds of a pass, one allocation of parts on 16 bytes / on 256 / apart: 5,003
// tokens 203.5 / 196.8 / 195.5, 2,501 and 2,500 202.4 / 194.7 / 193.6 (a warp's loads meet a fifth line, its stores straddle sectors).
long long whole_lines(long long floats) { return (floats + 63) / 64 * 64; }
Stream stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// What a launch was refused with; said once the interpreter's lock is held again.
struct Refusal {
    int code = 0;
    const char* what = nullptr;
    bool ok(int answer, const char* name) {
        if (answer == 0) return true;
        code = answer, what = name;
        return false;
    }
};
struct Unlocked {   // without the interpreter's lock, however the block is left
    PyThreadState* state = PyEval_SaveThread();
    ~Unlocked() { PyEval_RestoreThread(state); }
};
// What `launch` returns, run without the interpreter's lock, as the calls that it stands for are: a launch into a full queue and an allocation that
// asks the driver may block, and a server's other threads go on meanwhile. (The caller's frame holds the tensors.)
template <typename Launch> PyObject* unlocked(Launch launch) {
    Refusal refused;
    at::Tensor out;
    {
        Unlocked without;
        out = launch(refused);
    }
    if (!refused.what) return THPVariable_Wrap(std::move(out));
    if (refused.code == 801) return PyErr_Format(kernel_error, "%s: the driver offers no tensor-map encoder (cuTensorMapEncodeTiled)", refused.what);
    return PyErr_Format(kernel_error, "%s: CUDA error %d at launch", refused.what, refused.code);
}

// rms_norm(hidden, delta or None, weight, eps) -> out: `add_rms_norm` into a new tensor.
PyObject* rms_norm(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 4) return PyErr_Format(PyExc_TypeError, "rms_norm: 4 arguments");
    const at::Tensor *hidden = tensor(args[0]), *delta = tensor(args[1]), *weight = tensor(args[2]);
    if (!add_rms_norm || !whole(hidden, at::kFloat) || hidden->dim() != 2 || (!delta && args[1] != Py_None) || !weight ||
        (weight->scalar_type() != at::kBFloat16 && weight->scalar_type() != at::kFloat) || !whole(weight, weight->scalar_type()) ||
        weight->dim() != 1 || weight->size(0) != hidden->size(1) || (delta && (!whole(delta, weight->scalar_type()) || delta->sizes() != hidden->sizes())))
        Py_RETURN_NONE;
    const double eps = PyFloat_AsDouble(args[3]);
    if (PyErr_Occurred()) return nullptr;
    return unlocked([&](Refusal& refused) {
        at::Tensor out = at::empty(hidden->sizes(), weight->options());
        if (!refused.ok(add_rms_norm(weight->scalar_type() == at::kBFloat16, at_ptr<float>(*hidden), delta ? delta->data_ptr() : nullptr, weight->data_ptr(),
                             out.data_ptr(), (int)hidden->size(0), (int)hidden->size(1), (float)eps, 0, stream()), "add_rms_norm"))
            return at::Tensor();
        return out;
    });
    END_HANDLE_TH_ERRORS
}

// prompt_attention(x, qkv_weight, bias, inv_freq, o_weight, tok_seq, tok_pos, slots, cu_q, storage, table, err,
//                  n_heads, kv_heads, head_dim, n_seqs, max_q_len, max_kv_len, scale, window, write_cache) -> out
// `qkv_product` where it is the faster way, else the library's product and `rope_cache_write`; `attention_prefill_tc`; the output projection by the library.
PyObject* prompt_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 21) return PyErr_Format(PyExc_TypeError, "prompt_attention: 21 arguments");
    const at::Tensor *x = tensor(args[0]), *w = tensor(args[1]), *bias = tensor(args[2]), *freq = tensor(args[3]), *o = tensor(args[4]);
    const at::Tensor *seq = tensor(args[5]), *pos = tensor(args[6]), *slots = tensor(args[7]), *cu = tensor(args[8]), *storage = tensor(args[9]);
    const at::Tensor *table = tensor(args[10]), *err = tensor(args[11]);
    const long long heads = number(args[12]), kv = number(args[13]), d = number(args[14]), n_seqs = number(args[15]), longest = number(args[16]);
    const long long keys = number(args[17]), window = number(args[19]), write = number(args[20]);
    const double scale = PyFloat_AsDouble(args[18]);
    if (PyErr_Occurred()) return nullptr;
    if (!qkv_pairs_pays || !qkv_pairs || !rope_cache_write || !prefill_tc || !rows16(x) || !rows16(w) || (!bias && args[2] != Py_None) || (!freq && args[3] != Py_None) ||
        !o || !o->is_cuda() || o->scalar_type() != at::kBFloat16 || o->dim() != 2 || o->size(1) != heads * d || !whole(seq, at::kInt) ||
        !whole(pos, at::kInt) || !whole(slots, at::kInt) || !whole(cu, at::kInt) || !whole(storage, at::kBFloat16) || !table || !table->is_cuda() ||
        table->scalar_type() != at::kInt || !whole(err, at::kInt))
        Py_RETURN_NONE;
    const long long m = x->size(0), k = x->size(1), page = storage->stride(0);
    if ((d != 64 && d != 128) || heads <= 0 || kv <= 0 || heads % kv || w->size(0) != (heads + 2 * kv) * d || w->size(1) != k ||
        (bias && (!whole(bias, at::kBFloat16) || bias->numel() != w->size(0) || !on16(*bias))) ||
        (freq && (!whole(freq, at::kFloat) || 2 * freq->numel() > d)) || storage->dim() < 2 || !on16(*storage) || page % 8 ||
        page != 2 * kv * storage->size(-2) * d || seq->numel() != m || pos->numel() != m || slots->numel() < n_seqs || cu->numel() < n_seqs + 1)
        Py_RETURN_NONE;
    return unlocked([&](Refusal& refused) {
        at::Tensor q = at::empty({m, heads * d}, x->options()), attended = at::empty({m, heads * d}, x->options());
        const Stream s = stream();
        const float* angles = freq ? freq->const_data_ptr<float>() : nullptr;
        if ((!freq || 2 * freq->numel() == d) && qkv_pairs_pays((int)m, (int)w->size(0), (int)k, (int)d)) {
            const QkvArgs a = {bias ? bias->data_ptr() : nullptr, nullptr, ints(pos), ints(seq), ints(slots), q.data_ptr(), storage->data_ptr(), ints(table), page,
                               (int)table->stride(0), (int)heads, (int)kv, (int)d, write != 0, angles};
            if (!refused.ok(qkv_pairs(x->data_ptr(), (int)x->stride(0), w->data_ptr(), (int)w->stride(0), (int)m, (int)k, &a, at_ptr<int>(*err), s), "qkv_product")) return at::Tensor();
        } else {
            at::Tensor qkv = at::linear(*x, *w);
            if (!refused.ok(rope_cache_write(1, qkv.data_ptr(), bias ? bias->data_ptr() : nullptr, (int)qkv.stride(0), ints(seq), ints(pos), ints(slots), angles,
                                     freq ? (int)(2 * freq->numel()) : 0, (int)heads, q.data_ptr(), storage->data_ptr(), ints(table), page, (int)table->stride(0),
                                     (int)kv, (int)d, write != 0, (int)m, at_ptr<int>(*err), s), "rope_cache_write"))
                return at::Tensor();
        }
        if (!refused.ok(prefill_tc(q.data_ptr(), attended.data_ptr(), ints(cu), ints(pos), ints(slots), storage->data_ptr(), ints(table), page, (int)table->stride(0),
                           (int)kv, (int)d, (int)heads, (int)n_seqs, (int)m, (int)longest, (int)keys, (float)scale, (int)window, at_ptr<int>(*err), nullptr,
                           0, s), "attention_prefill_tc"))
            return at::Tensor();
        return at::linear(attended, *o);
    });
    END_HANDLE_TH_ERRORS
}

// gated_feed_forward(x, gate_up, down, err) -> out: `tc_gemm` with the gate in its epilogue where it has tiles for every pair of SMs, else the
// library's product and `swiglu`; down by the library.
PyObject* gated_feed_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 4) return PyErr_Format(PyExc_TypeError, "gated_feed_forward: 4 arguments");
    const at::Tensor *x = tensor(args[0]), *gate_up = tensor(args[1]), *down = tensor(args[2]), *err = tensor(args[3]);
    if (!tc_gemm || !tc_is_persistent || !swiglu || !rows16(x) || !rows16(gate_up) || !down || !down->is_cuda() || down->scalar_type() != at::kBFloat16 || down->dim() != 2 ||
        !whole(err, at::kInt))
        Py_RETURN_NONE;
    const long long m = x->size(0), k = x->size(1), inter = gate_up->size(0) / 2;
    if (gate_up->size(0) != 2 * inter || inter % 8 || gate_up->size(1) != k || down->size(1) != inter) Py_RETURN_NONE;
    return unlocked([&](Refusal& refused) {
        at::Tensor act = at::empty({m, inter}, x->options());
        if (tc_is_persistent(1, (int)m, (int)(2 * inter))) {
            if (!refused.ok(tc_gemm(1, x->data_ptr(), (int)x->stride(0), gate_up->data_ptr(), (int)gate_up->stride(0), act.data_ptr(), (int)inter, (int)m, (int)(2 * inter),
                            (int)k, at_ptr<int>(*err), stream()), "tc_gemm"))
                return at::Tensor();
        } else {
            at::Tensor both = at::linear(*x, *gate_up);
            if (!refused.ok(swiglu(1, both.data_ptr(), act.data_ptr(), (int)m, (int)inter, stream()), "swiglu")) return at::Tensor();
        }
        return at::linear(act, *down);
    });
    END_HANDLE_TH_ERRORS
}

// matrix_memory(x, joint, gate_bias, norm, o_weight, state, cu_q, slots, err, heads, dim, vdim, max_q_len, records, each, s_offset, n_offset,
//               m_offset, cap, eps, floor) -> out: `tc_gemm_tail`, `stabilized_gates`, `state_chunks`, `gated_group_norm` and the output
// projection by the library. The caller has found the tail and the chunks to be the ways to go; joint is [q | k | v | gate | i | f].
PyObject* matrix_memory(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 21) return PyErr_Format(PyExc_TypeError, "matrix_memory: 21 arguments");
    const at::Tensor *x = tensor(args[0]), *joint = tensor(args[1]), *gate_bias = tensor(args[2]), *norm = tensor(args[3]), *o = tensor(args[4]);
    const at::Tensor *state = tensor(args[5]), *cu = tensor(args[6]), *slots = tensor(args[7]), *err = tensor(args[8]);
    long long v[9];
    for (int i = 0; i < 9; ++i) v[i] = number(args[9 + i]);
    const long long h = v[0], d = v[1], vd = v[2], longest = v[3], records = v[4], each = v[5], s_at = v[6], n_at = v[7], m_at = v[8];
    const double cap = PyFloat_AsDouble(args[18]), eps = PyFloat_AsDouble(args[19]), floor_add = PyFloat_AsDouble(args[20]);
    if (PyErr_Occurred()) return nullptr;
    if (!tc_gemm_tail || !stabilized_gates || !state_chunks || !gated_group_norm || !rows16(x) || !rows16(joint) || !whole(gate_bias, at::kFloat) ||
        !whole(norm, at::kBFloat16) || !o || !o->is_cuda() || o->scalar_type() != at::kBFloat16 || o->dim() != 2 || !whole(state, at::kFloat) || state->dim() != 2 ||
        !whole(cu, at::kInt) || !whole(slots, at::kInt) || !whole(err, at::kInt))
        Py_RETURN_NONE;
    const long long t = x->size(0), main = 2 * h * (d + vd), inner = h * vd, seqs = cu->numel() - 1, floats = state->size(1);
    if (h <= 0 || (d != 64 && d != 128) || vd <= 0 || vd % 64 || seqs <= 0 || seqs > 65535 || inner / 64 > 65535 || joint->size(0) != main + 2 * h ||
        joint->size(1) != x->size(1) || gate_bias->numel() != 2 * h || norm->numel() != inner || o->size(1) != inner || slots->numel() < seqs ||
        s_at < 0 || s_at + h * d * vd > floats || n_at < 0 || n_at + h * d > floats || m_at < 0 || m_at + h > floats || records <= 0 || each < 0)
        Py_RETURN_NONE;
    return unlocked([&](Refusal& refused) {
        at::Tensor proj = at::empty({t, main}, x->options()), out = at::empty({t, inner}, x->options());
        const long long gates = whole_lines(t * h);
        at::Tensor room = at::empty({6 * gates}, state->options()), made = at::empty({t * inner}, state->options());
        at::Tensor kept = at::empty({records * h * (d * vd + d + 1) + (each ? seqs * h * (d * vd + d) : 0)}, state->options());
        float* decay = at_ptr<float>(room);
        float *take = decay + gates, *floor = take + gates, *nq = floor + gates, *pre = nq + gates, *y = at_ptr<float>(made), *scratch = at_ptr<float>(kept);
        unsigned char* p = at_ptr<unsigned char>(proj);
        const unsigned char *q = p, *k = p + 2 * h * d, *vals = p + 4 * h * d, *gate = vals + 2 * inner;
        const Stream s = stream();
        const long long slot = state->stride(0);
        if (!refused.ok(tc_gemm_tail(x->data_ptr(), (int)x->stride(0), joint->data_ptr(), (int)joint->stride(0), p, (int)main, pre, (int)t, (int)main, (int)(2 * h),
                             (int)x->size(1), at_ptr<int>(*err), s), "tc_gemm_tail") ||
            !refused.ok(stabilized_gates(pre, (int)(2 * h), gate_bias->const_data_ptr<float>(), (float)cap, ints(cu), ints(slots), (int)seqs, at_ptr<float>(*state), slot,
                                 m_at, (int)h, decay, take, floor, s), "stabilized_gates") ||
            !refused.ok(state_chunks(q, (int)main, k, (int)main, vals, (int)main, decay, take, nullptr, nullptr, (int)h, ints(cu), ints(slots), (int)seqs, (int)longest,
                             at_ptr<float>(*state), slot, s_at, n_at, (int)h, (int)h, (int)d, (int)vd, (float)std::pow((double)d, -0.5), scratch, records,
                             (int)each, y, nq, s), "state_chunks") ||
            !refused.ok(gated_group_norm(1, y, gate, (int)main, norm->data_ptr(), (float)eps, out.data_ptr(), (int)t, (int)inner, (int)h, (int)h, 0, 0, nq, floor,
                                 (float)floor_add, nullptr, nullptr, 0, s), "gated_group_norm"))
            return at::Tensor();
        return at::linear(out, *o);
    });
    END_HANDLE_TH_ERRORS
}

// state_space(x, joint, conv_weight, conv_bias, dt_bias, rate_log, skip, norm, o_weight, state, cu_q, tok_seq, slots, err, heads, vdim, state_size,
//             groups, norm_parts, max_q_len, records, each, s_offset, conv_offset, eps) -> out: `tc_gemm_tail`, `causal_conv_silu`,
// `state_chunks` with the gates formed inside, `gated_group_norm` and the output projection by the library; joint is [z | x | B | C | dt].
PyObject* state_space(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 25) return PyErr_Format(PyExc_TypeError, "state_space: 25 arguments");
    const at::Tensor* t[14];
    for (int i = 0; i < 14; ++i) t[i] = tensor(args[i]);
    const at::Tensor *x = t[0], *joint = t[1], *conv_w = t[2], *conv_b = t[3], *dt_bias = t[4], *rate = t[5], *skip = t[6], *norm = t[7], *o = t[8], *state = t[9];
    const at::Tensor *cu = t[10], *seq = t[11], *slots = t[12], *err = t[13];
    long long v[10];
    for (int i = 0; i < 10; ++i) v[i] = number(args[14 + i]);
    const long long h = v[0], vd = v[1], d = v[2], groups = v[3], parts = v[4], longest = v[5], records = v[6], each = v[7], s_at = v[8], conv_at = v[9];
    const double eps = PyFloat_AsDouble(args[24]);
    if (PyErr_Occurred()) return nullptr;
    if (!tc_gemm_tail || !causal_conv || !state_chunks || !gated_group_norm || !rows16(x) || !rows16(joint) || !whole(conv_w, at::kFloat) || conv_w->dim() != 2 ||
        !whole(conv_b, at::kFloat) || !whole(dt_bias, at::kFloat) || !whole(rate, at::kFloat) || !whole(skip, at::kFloat) || !whole(norm, at::kBFloat16) || !o ||
        !o->is_cuda() || o->scalar_type() != at::kBFloat16 || o->dim() != 2 || !whole(state, at::kFloat) || state->dim() != 2 || !whole(cu, at::kInt) ||
        !whole(seq, at::kInt) || !whole(slots, at::kInt) || !whole(err, at::kInt))
        Py_RETURN_NONE;
    const long long m = x->size(0), inner = h * vd, channels = inner + 2 * groups * d, main = inner + channels, seqs = cu->numel() - 1, taps = conv_w->size(1);
    if (h <= 0 || (d != 64 && d != 128) || vd <= 0 || vd % 64 || groups <= 0 || h % groups || parts <= 0 || inner % parts || seqs <= 0 || seqs > 65535 ||
        inner / 64 > 65535 || joint->size(0) != main + h || joint->size(1) != x->size(1) || conv_w->size(0) != channels || taps < 1 || taps > 16 ||
        conv_b->numel() != channels || dt_bias->numel() != h || rate->numel() != h || skip->numel() != h || norm->numel() != inner || o->size(1) != inner ||
        seq->numel() != m || slots->numel() < seqs || s_at < 0 || s_at + h * d * vd > state->size(1) || conv_at < 0 ||
        conv_at + (taps - 1) * channels > state->size(1) || records <= 0 || each < 0)
        Py_RETURN_NONE;
    return unlocked([&](Refusal& refused) {
        at::Tensor made = at::empty({m, main}, x->options()), mixed = at::empty({m, channels}, x->options()), out = at::empty({m, inner}, x->options());
        at::Tensor pre = at::empty({m * h}, state->options()), sums = at::empty({m * inner}, state->options());
        at::Tensor kept = at::empty({records * h * (d * vd + d + 1) + (each ? seqs * h * (d * vd + d) : 0)}, state->options());
        float *dt = at_ptr<float>(pre), *y = at_ptr<float>(sums), *scratch = at_ptr<float>(kept);
        const unsigned char *z = at_ptr<unsigned char>(made), *vals = at_ptr<unsigned char>(mixed), *k = vals + 2 * inner, *q = k + 2 * groups * d;
        const Stream s = stream();
        const long long slot = state->stride(0);
        if (!refused.ok(tc_gemm_tail(x->data_ptr(), (int)x->stride(0), joint->data_ptr(), (int)joint->stride(0), made.data_ptr(), (int)main, dt, (int)m, (int)main, (int)h,
                             (int)x->size(1), at_ptr<int>(*err), s), "tc_gemm_tail") ||
            !refused.ok(causal_conv(1, z + 2 * inner, (int)main, conv_w->const_data_ptr<float>(), conv_b->const_data_ptr<float>(), ints(cu), ints(seq), ints(slots), (int)seqs,
                            at_ptr<float>(*state), slot, conv_at, (int)taps, (int)m, (int)channels, mixed.data_ptr(), 0, 0, s), "causal_conv_silu") ||
            !refused.ok(state_chunks(q, (int)channels, k, (int)channels, vals, (int)channels, dt, nullptr, dt_bias->const_data_ptr<float>(), rate->const_data_ptr<float>(),
                             (int)h, ints(cu), ints(slots), (int)seqs, (int)longest, at_ptr<float>(*state), slot, s_at, -1, (int)h, (int)groups, (int)d, (int)vd, 1.f,
                             scratch, records, (int)each, y, nullptr, s), "state_chunks") ||
            !refused.ok(gated_group_norm(1, y, z, (int)main, norm->data_ptr(), (float)eps, out.data_ptr(), (int)m, (int)inner, (int)parts, (int)h, 1, 1, nullptr, nullptr, 0.f,
                                 skip->const_data_ptr<float>(), vals, (int)channels, s), "gated_group_norm"))
            return at::Tensor();
        return at::linear(out, *o);
    });
    END_HANDLE_TH_ERRORS
}

// gated_linear_attention(x, joint, a2, a2_bias, norm, o_weight, state, cu_q, slots, heads, dim, vdim, max_q_len, records, each, inv_tau, eps) -> out:
// the library's product of [q | k | v | gate | middle] and of the middle in float32, `row_chunks`, `gated_group_norm` and the output projection.
PyObject* gated_linear_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 17) return PyErr_Format(PyExc_TypeError, "gated_linear_attention: 17 arguments");
    const at::Tensor* t[9];
    for (int i = 0; i < 9; ++i) t[i] = tensor(args[i]);
    const at::Tensor *x = t[0], *joint = t[1], *a2 = t[2], *bias = t[3], *norm = t[4], *o = t[5], *state = t[6], *cu = t[7], *slots = t[8];
    long long v[6];
    for (int i = 0; i < 6; ++i) v[i] = number(args[9 + i]);
    const long long h = v[0], d = v[1], vd = v[2], longest = v[3], records = v[4], each = v[5];
    const double inv_tau = PyFloat_AsDouble(args[15]), eps = PyFloat_AsDouble(args[16]);
    if (PyErr_Occurred()) return nullptr;
    if (!row_chunks || !gated_group_norm || !rows16(x) || !rows16(joint) || !rows16(a2) || !whole(bias, at::kFloat) || !whole(norm, at::kBFloat16) || !o ||
        !o->is_cuda() || o->scalar_type() != at::kBFloat16 || o->dim() != 2 || !whole(state, at::kFloat) || state->dim() != 2 || !whole(cu, at::kInt) ||
        !whole(slots, at::kInt))
        Py_RETURN_NONE;
    const long long m = x->size(0), inner = h * vd, main = 2 * h * d + 2 * inner, rank = a2->size(1), seqs = cu->numel() - 1, wide = main + rank;
    if (h <= 0 || d != 64 || vd <= 0 || vd % 64 || vd > 512 || seqs <= 0 || seqs > 65535 || inner / 64 > 65535 || joint->size(0) != wide ||
        joint->size(1) != x->size(1) || a2->size(0) != h * d || bias->numel() != h * d || norm->numel() != inner || o->size(1) != inner ||
        slots->numel() < seqs || h * d * vd > state->size(1) || records <= 0 || each < 0)
        Py_RETURN_NONE;
    return unlocked([&](Refusal& refused) {
        at::Tensor all = at::linear(*x, *joint), pre = at::mm(all.narrow(1, main, rank), a2->t(), at::kFloat), out = at::empty({m, inner}, x->options());
        TORCH_CHECK(on16(all) && on16(pre) && pre.is_contiguous(), "gated_linear_attention: the allocator's rows begin on no 16-byte boundary");
        at::Tensor sums = at::empty({m * inner}, state->options());
        at::Tensor kept = at::empty({records * h * (d * vd + d) + (each ? seqs * h * d * vd : 0) + m * h * d}, state->options());
        float *y = at_ptr<float>(sums), *scratch = at_ptr<float>(kept);
        const unsigned char *q = at_ptr<unsigned char>(all), *k = q + 2 * h * d, *vals = k + 2 * h * d, *gate = vals + 2 * inner;
        const Stream s = stream();
        if (!refused.ok(row_chunks(q, (int)wide, k, (int)wide, vals, (int)wide, pre.const_data_ptr<float>(), bias->const_data_ptr<float>(), 2, (float)inv_tau, nullptr, ints(cu),
                           ints(slots), (int)seqs, (int)longest, at_ptr<float>(*state), state->stride(0), 0, (int)h, (int)d, (int)vd, (float)std::pow((double)d, -0.5),
                           scratch, records, (int)each, y, s), "row_chunks") ||
            !refused.ok(gated_group_norm(1, y, gate, (int)wide, norm->data_ptr(), (float)eps, out.data_ptr(), (int)m, (int)inner, (int)h, (int)h, 1, 0, nullptr, nullptr, 0.f,
                                 nullptr, nullptr, 0, s), "gated_group_norm"))
            return at::Tensor();
        return at::linear(out, *o);
    });
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {{"setup", (PyCFunction)(void (*)())setup, METH_FASTCALL, nullptr},
                         {"rms_norm", (PyCFunction)(void (*)())rms_norm, METH_FASTCALL, nullptr},
                         {"prompt_attention", (PyCFunction)(void (*)())prompt_attention, METH_FASTCALL, nullptr},
                         {"gated_feed_forward", (PyCFunction)(void (*)())gated_feed_forward, METH_FASTCALL, nullptr},
                         {"matrix_memory", (PyCFunction)(void (*)())matrix_memory, METH_FASTCALL, nullptr},
                         {"state_space", (PyCFunction)(void (*)())state_space, METH_FASTCALL, nullptr},
                         {"gated_linear_attention", (PyCFunction)(void (*)())gated_linear_attention, METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "qf_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_qf_host() { return PyModule_Create(&module); }
