// Host path of the Python package in native code: the module polarquant_kv._host, a CPython extension over torch's C++ API
// and the C ABI of libpolarquant_b200.so.
//
// A call of the package used to spend 15 to 40 us in Python and ctypes (argument checks, plan look-up, allocation, the
// conversion of twenty-odd arguments) around kernels of 4 to 15 us.  The functions here do the same for the ordinary
// form of a call (contiguous float16 tensors on the current device, known plan) in 2 to 4 us.  Anything else - other
// types or layouts, an error to report - makes them return None, and the Python function of the same name goes on with
// its complete checks; so every error is raised in one place only.
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include <cmath>
#include <cstring>
#include <deque>
#include <string>

#include "polarquant_b200.h"
#include "polarquant_llama_abi.h"

namespace {

// ------------------------------------------------------------------ what Python registers once
struct Plan {                       // device-side constants of a DevicePlan (kept alive by the Python object)
    int head_dim, device, jl_dim;
    const float* rot;
    const void* rot_split;
    const float* jl;
    const void* jl_split;
};
struct Tables {
    bool set = false;
    float codebook[16], thresholds[16];
};
Tables g_tables[5];                 // by n_bits
PyObject* g_cache_type = nullptr;   // types.CompressedKV
PyObject* g_plan_type = nullptr;    // rotation.DevicePlan
PyObject* g_check = nullptr;        // _ext.check(status, where)
PyObject *s_native, *s_blocks, *s_signs, *s_norms, *s_bits, *s_dim, *s_seq, *s_cap;

constexpr const char* kPlanCapsule = "polarquant_kv.plan";

// New reference, or nullptr with no error set.
PyObject* attr(PyObject* o, PyObject* name) {
    PyObject* v = PyObject_GetAttr(o, name);
    if (!v) PyErr_Clear();
    return v;
}
bool attr_int(PyObject* o, PyObject* name, int64_t* out) {
    PyObject* v = attr(o, name);
    if (!v) return false;
    const bool ok = PyLong_Check(v);
    if (ok) *out = PyLong_AsLongLong(v);
    Py_DECREF(v);
    if (ok && PyErr_Occurred()) { PyErr_Clear(); return false; }
    return ok;
}
const at::Tensor* tensor(PyObject* o) { return o && THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }
bool as_int(PyObject* o, int64_t* v) {
    if (!PyLong_Check(o)) return false;
    *v = PyLong_AsLongLong(o);
    if (PyErr_Occurred()) { PyErr_Clear(); return false; }
    return true;
}

// A copy of a plan object's constants: a launch runs without the GIL, and another thread may change the object meanwhile.
bool plan_of(PyObject* o, Plan* out) {
    if (!g_plan_type || !PyObject_TypeCheck(o, (PyTypeObject*)g_plan_type)) return false;
    PyObject* c = attr(o, s_native);
    if (!c) return false;
    const Plan* p = (const Plan*)PyCapsule_GetPointer(c, kPlanCapsule);
    if (p) *out = *p;
    else PyErr_Clear();
    Py_DECREF(c);
    return p != nullptr;
}

// ------------------------------------------------------------------ plans by the matrices of a call
// A matrix as a call gives it.  On the host (a C-contiguous float array or CPU tensor) it is its type, shape and bytes, all
// of them: an edit in place anywhere is noticed, and an equal matrix in another object is recognised (two of 128 x 128 float64
// take 5 us).  On a device it is the tensor object, its type and layout, and its version counter, which
// every in-place operation of torch moves; reading the contents back would stop the stream.
struct Matrix {
    enum Kind { kNone, kHost, kDevice } kind = kNone;
    int type = 0;                            // format character of an array, or 256 + scalar type of a tensor
    int64_t size[2] = {0, 0}, stride[2] = {0, 0}, version = 0;
    const void* data = nullptr;              // host: valid while the call's view is open
    size_t bytes = 0;                        // host
    PyObject* object = nullptr;              // device
};
constexpr size_t kMatrixLimit = 1 << 20;     // larger ones are left to the caller's digest

class MatrixView {
  public:
    Matrix m;
    bool good;
    explicit MatrixView(PyObject* o) : good(read(o)) {}
    ~MatrixView() { if (open_) PyBuffer_Release(&buf_); }
    MatrixView(const MatrixView&) = delete;
    MatrixView& operator=(const MatrixView&) = delete;

  private:
    Py_buffer buf_;
    bool open_ = false;
    bool read(PyObject* o) {
        if (o == Py_None) return true;
        if (const at::Tensor* t = tensor(o)) {
            if (t->layout() != at::kStrided || t->dim() != 2 || t->is_conj() || t->is_neg()) return false;
            m.type = 256 + (int)t->scalar_type();
            for (int i = 0; i < 2; ++i) { m.size[i] = t->size(i); m.stride[i] = t->stride(i); }
            m.data = t->data_ptr();
            if (t->is_cpu()) {
                m.kind = Matrix::kHost;
                m.bytes = t->nbytes();
                return t->is_contiguous() && m.bytes <= kMatrixLimit;
            }
            if (t->is_inference()) return false;                 // (no version counter)
            m.kind = Matrix::kDevice;
            m.version = t->_version();
            m.object = o;
            return true;
        }
        if (PyObject_GetBuffer(o, &buf_, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT) != 0) {
            PyErr_Clear();
            return false;
        }
        open_ = true;
        const char* f = buf_.format;
        if (buf_.ndim != 2 || !f || f[1] || (*f != 'd' && *f != 'f' && *f != 'e') || (size_t)buf_.len > kMatrixLimit) return false;
        m.kind = Matrix::kHost;
        m.type = *f;
        for (int i = 0; i < 2; ++i) m.size[i] = buf_.shape[i];
        m.data = buf_.buf;
        m.bytes = (size_t)buf_.len;
        return true;
    }
};
// A matrix kept from an earlier call: host bytes copied, a device tensor held (its identity cannot be reused meanwhile).
struct KeptMatrix {
    Matrix m;
    std::string bytes;
    explicit KeptMatrix(const Matrix& v) : m(v) {
        if (m.kind == Matrix::kHost) bytes.assign((const char*)m.data, m.bytes);
        Py_XINCREF(m.object);
    }
    bool operator==(const Matrix& o) const {
        if (m.kind != o.kind || m.type != o.type || m.size[0] != o.size[0] || m.size[1] != o.size[1]) return false;
        if (m.kind == Matrix::kHost) return m.bytes == o.bytes && memcmp(bytes.data(), o.data, m.bytes) == 0;
        return m.object == o.object && m.data == o.data && m.version == o.version && m.stride[0] == o.stride[0] &&
               m.stride[1] == o.stride[1];
    }
};
struct Known {
    KeptMatrix r, p;
    int device;
    PyObject* plan;
};
std::deque<Known> g_known;
constexpr size_t kKnownLimit = 64;

// Borrowed reference or nullptr.
PyObject* known_plan(PyObject* R, PyObject* P, int device) {
    const MatrixView r(R), p(P);
    if (!r.good || !p.good) return nullptr;
    for (auto it = g_known.rbegin(); it != g_known.rend(); ++it)
        if (it->device == device && it->r == r.m && it->p == p.m) return it->plan;
    return nullptr;
}

// plan_get(R, device_index, P) -> DevicePlan or None
PyObject* plan_get(PyObject*, PyObject* const* args, Py_ssize_t n) {
    int64_t dev;
    if (n != 3 || !as_int(args[1], &dev)) Py_RETURN_NONE;
    PyObject* p = known_plan(args[0], args[2], (int)dev);
    if (!p) Py_RETURN_NONE;
    Py_INCREF(p);
    return p;
}
// plan_put(R, device_index, P, plan)
PyObject* plan_put(PyObject*, PyObject* const* args, Py_ssize_t n) {
    int64_t dev;
    if (n != 4 || !as_int(args[1], &dev)) Py_RETURN_NONE;
    const MatrixView r(args[0]), p(args[2]);
    if (!r.good || !p.good || r.m.kind == Matrix::kNone) Py_RETURN_NONE;
    g_known.push_back(Known{KeptMatrix(r.m), KeptMatrix(p.m), (int)dev, args[3]});
    Py_INCREF(args[3]);
    if (g_known.size() > kKnownLimit) {
        const Known old = std::move(g_known.front());
        g_known.pop_front();
        Py_XDECREF(old.r.m.object);
        Py_XDECREF(old.p.m.object);
        Py_DECREF(old.plan);
    }
    Py_RETURN_NONE;
}

// plan_handle(head_dim, device_index, rot, rot_split, jl, jl_split, jl_dim) -> capsule (data pointers as ints)
PyObject* plan_handle(PyObject*, PyObject* const* args, Py_ssize_t n) {
    int64_t v[7];
    if (n != 7) { PyErr_SetString(PyExc_TypeError, "plan_handle takes 7 integers"); return nullptr; }
    for (int i = 0; i < 7; ++i)
        if (!as_int(args[i], &v[i])) { PyErr_SetString(PyExc_TypeError, "plan_handle takes 7 integers"); return nullptr; }
    Plan* p = new Plan{(int)v[0], (int)v[1], (int)v[6], (const float*)v[2], (const void*)v[3], (const float*)v[4], (const void*)v[5]};
    return PyCapsule_New(p, kPlanCapsule, [](PyObject* c) { delete (Plan*)PyCapsule_GetPointer(c, kPlanCapsule); });
}

// set_tables(n_bits, codebook_address, thresholds_address): host float32 arrays
PyObject* set_tables(PyObject*, PyObject* const* args, Py_ssize_t n) {
    int64_t bits, cb, thr;
    if (n != 3 || !as_int(args[0], &bits) || !as_int(args[1], &cb) || !as_int(args[2], &thr) || (bits != 2 && bits != 4)) {
        PyErr_SetString(PyExc_ValueError, "set_tables(n_bits, codebook address, thresholds address)");
        return nullptr;
    }
    Tables& t = g_tables[bits];
    memcpy(t.codebook, (const void*)cb, sizeof(float) << bits);
    memcpy(t.thresholds, (const void*)thr, sizeof(float) * ((1 << bits) - 1));
    t.set = true;
    Py_RETURN_NONE;
}

// register(CompressedKV, DevicePlan, check)
PyObject* register_types(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 3) { PyErr_SetString(PyExc_TypeError, "register(CompressedKV, DevicePlan, check)"); return nullptr; }
    PyObject** slots[3] = {&g_cache_type, &g_plan_type, &g_check};
    for (int i = 0; i < 3; ++i) {
        Py_INCREF(args[i]);
        Py_XSETREF(*slots[i], args[i]);
    }
    Py_RETURN_NONE;
}

// nullptr with the error set, through _ext.check
PyObject* raise_status(int status, const char* where) {
    PyObject* r = PyObject_CallFunction(g_check, "is", status, where);
    if (r) { Py_DECREF(r); PyErr_SetString(PyExc_RuntimeError, where); }
    return nullptr;
}

// A launch waits when the stream's queue is full, so other Python threads go on meanwhile.  What the call uses is held by
// local references or by the caller's arguments.
template <class F>
int launch(F f) {
    struct Released {
        PyThreadState* state = PyEval_SaveThread();
        ~Released() { PyEval_RestoreThread(state); }         // also when an exception passes
    } released;
    return f();
}

void* stream_of(int device) { return (void*)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }

bool half_contiguous(const at::Tensor& t) {
    return t.is_cuda() && t.scalar_type() == at::kHalf && t.is_contiguous() && t.get_device() == c10::cuda::current_device();
}
at::Tensor empty(at::IntArrayRef size, at::ScalarType type, int device) {
    return at::detail::empty_cuda(size, type, c10::Device(c10::kCUDA, (c10::DeviceIndex)device), std::nullopt);
}

// ------------------------------------------------------------------ a CompressedKV, read field by field
struct Cache {
    at::Tensor blocks, signs, norms;          // the last two undefined without a sketch
    int64_t n_bits, dim, seq, cap, rows_b, rows_h;
    bool contiguous, sketch;
};
bool read_cache(PyObject* o, Cache* c) {
    if (!g_cache_type || !PyObject_TypeCheck(o, (PyTypeObject*)g_cache_type)) return false;
    if (!attr_int(o, s_bits, &c->n_bits) || !attr_int(o, s_dim, &c->dim) || !attr_int(o, s_seq, &c->seq)) return false;
    PyObject* b = attr(o, s_blocks);
    const at::Tensor* t = tensor(b);
    const bool ok = t && t->is_cuda() && t->scalar_type() == at::kByte && t->dim() == 5;
    if (ok) c->blocks = *t;
    Py_XDECREF(b);
    if (!ok || (c->n_bits != 2 && c->n_bits != 4) || !g_tables[c->n_bits].set) return false;
    c->rows_b = c->blocks.size(0);
    c->rows_h = c->blocks.size(1);
    // the stated capacity is the tensor's; anything else goes through the Python function's checks
    c->cap = c->blocks.size(2);
    int64_t stated;
    if (!attr_int(o, s_cap, &stated) || stated != c->cap) return false;
    c->contiguous = c->blocks.is_contiguous();
    c->sketch = false;
    PyObject *s = attr(o, s_signs), *m = attr(o, s_norms);
    const at::Tensor *ts = tensor(s), *tm = tensor(m);
    if (ts && tm) {
        c->signs = *ts;
        c->norms = *tm;
        c->sketch = true;
    }
    Py_XDECREF(s);
    Py_XDECREF(m);
    return c->seq >= 0 && c->seq <= c->cap;
}

// A position: an int, or a one-element int64 tensor on `device`.
struct Position {
    int64_t host = 0;
    const int64_t* dev = nullptr;
};
bool read_position(PyObject* o, int device, Position* p) {
    if (const at::Tensor* t = tensor(o)) {
        if (t->scalar_type() != at::kLong || t->numel() != 1 || !t->is_cuda() || t->get_device() != device) return false;
        p->dev = (const int64_t*)t->data_ptr();
        return true;
    }
    return as_int(o, &p->host);
}

int launch_compress(const at::Tensor& x, int64_t rows, int64_t tokens, int64_t cap, const Position& pos, const Plan& plan,
                    int n_bits, const at::Tensor& blocks, const at::Tensor& signs, const at::Tensor& norms, bool sketch) {
    const Tables& t = g_tables[n_bits];
    const void* js = sketch ? plan.jl_split : nullptr;
    const int m = sketch ? plan.jl_dim : 0;
    void *sp = sketch ? signs.data_ptr() : nullptr, *np = sketch ? norms.data_ptr() : nullptr, *st = stream_of(plan.device);
    return launch([&] {
        return pos.dev ? pq_compress_rows_dynamic(x.data_ptr(), rows, tokens, cap, pos.dev, plan.head_dim, n_bits, plan.rot_split,
                                                  t.thresholds, t.codebook, blocks.data_ptr(), js, m, sp, np, st)
                       : pq_compress_rows(x.data_ptr(), rows, tokens, cap, pos.host, plan.head_dim, n_bits, plan.rot_split,
                                          t.thresholds, t.codebook, blocks.data_ptr(), js, m, sp, np, st);
    });
}

bool plan_for(PyObject* R, PyObject* P, int device, Plan* out) {
    if (!plan_of(R, out)) {
        PyObject* known = known_plan(R, P, device);
        if (!known || !plan_of(known, out)) return false;
    }
    return out->device == device;
}

// What an append into `c` needs beyond read_cache: the input's rows and width, room, and the plan's sketch.
bool append_fits(const at::Tensor& x, const Cache& c, const Plan& plan, const Position& pos) {
    if (x.dim() != 4 || x.numel() == 0 || x.size(0) != c.rows_b || x.size(1) != c.rows_h || x.size(3) != c.dim) return false;
    if (plan.head_dim != c.dim || !c.contiguous || c.blocks.get_device() != plan.device) return false;
    if (!pos.dev && (pos.host < 0 || pos.host + x.size(2) > c.cap)) return false;
    if (plan.jl_dim && (!c.sketch || c.signs.size(-1) != plan.jl_dim / 8 || !c.signs.is_contiguous() || !c.norms.is_contiguous()))
        return false;
    return true;
}

bool store_seq(PyObject* o, int64_t seq) {
    PyObject* v = PyLong_FromLongLong(seq);
    const bool ok = v && PyObject_SetAttr(o, s_seq, v) == 0;
    Py_XDECREF(v);
    return ok;
}

// compress(kv, rotation, n_bits, group_size, jl_matrix, out, position) -> CompressedKV or None
PyObject* compress(PyObject*, PyObject* const* args, Py_ssize_t n) {
    int64_t bits, group;
    const at::Tensor* x = n == 7 ? tensor(args[0]) : nullptr;
    if (!x || !as_int(args[2], &bits) || !as_int(args[3], &group) || (bits != 2 && bits != 4) || group != 32 ||
        !g_tables[bits].set || x->dim() != 4 || x->numel() == 0 || !half_contiguous(*x))
        Py_RETURN_NONE;
    const int dev = x->get_device();
    Plan plan;
    if (!plan_for(args[1], args[4], dev, &plan) || plan.head_dim != x->size(3) || (plan.head_dim != 64 && plan.head_dim != 128))
        Py_RETURN_NONE;
    const int64_t B = x->size(0), H = x->size(1), S = x->size(2), D = x->size(3);
    if (args[5] != Py_None) {
        Cache c;
        Position pos;
        if (!read_cache(args[5], &c) || c.n_bits != bits || !read_position(args[6], dev, &pos) ||
            !append_fits(*x, c, plan, pos))
            Py_RETURN_NONE;
        const int st = launch_compress(*x, B * H, S, c.cap, pos, plan, (int)bits, c.blocks, c.signs, c.norms, plan.jl_dim > 0);
        if (st) return raise_status(st, "pq_compress_rows");
        if (!pos.dev && pos.host + S > c.seq && !store_seq(args[5], pos.host + S)) return nullptr;
        Py_INCREF(args[5]);
        return args[5];
    }
    at::Tensor blocks = empty({B, H, S, D / 32, 2 + 4 * bits}, at::kByte, dev), signs, norms;
    if (plan.jl_dim) {
        signs = empty({B, H, S, plan.jl_dim / 8}, at::kByte, dev);
        norms = empty({B, H, S}, at::kHalf, dev);
    }
    const int st = launch_compress(*x, B * H, S, S, Position(), plan, (int)bits, blocks, signs, norms, plan.jl_dim > 0);
    if (st) return raise_status(st, "pq_compress_rows");
    auto wrap = [](const at::Tensor& t) -> PyObject* {
        if (t.defined()) return THPVariable_Wrap(t);
        Py_RETURN_NONE;
    };
    PyObject* a[9] = {nullptr, wrap(blocks), wrap(signs), wrap(norms), args[2], args[3], PyLong_FromLongLong(D),
                      PyLong_FromLongLong(S), PyLong_FromLongLong(S)};
    PyObject* out = nullptr;
    if (a[1] && a[2] && a[3] && a[6] && a[7] && a[8])
        out = PyObject_Vectorcall(g_cache_type, a + 1, 8 | PY_VECTORCALL_ARGUMENTS_OFFSET, nullptr);
    for (int i : {1, 2, 3, 6, 7, 8}) Py_XDECREF(a[i]);
    return out;
}

// append(key, value, key_cache, value_cache, key_plan, value_plan, position) -> True or None: one step of a cache manager
PyObject* append(PyObject*, PyObject* const* args, Py_ssize_t n) {
    const at::Tensor *k = n == 7 ? tensor(args[0]) : nullptr, *v = n == 7 ? tensor(args[1]) : nullptr;
    if (!k || !v || !half_contiguous(*k) || !half_contiguous(*v) || k->get_device() != v->get_device()) Py_RETURN_NONE;
    const int dev = k->get_device();
    Plan pk, pv;
    Cache ck, cv;
    Position pos;
    if (!plan_of(args[4], &pk) || !plan_of(args[5], &pv) || pk.device != dev || pv.device != dev || pv.jl_dim || !read_position(args[6], dev, &pos) ||
        !read_cache(args[2], &ck) || !read_cache(args[3], &cv) || !append_fits(*k, ck, pk, pos) ||
        !append_fits(*v, cv, pv, pos) || k->size(2) != v->size(2))
        Py_RETURN_NONE;
    const int64_t rows = ck.rows_b * ck.rows_h, S = k->size(2);
    int st = launch_compress(*k, rows, S, ck.cap, pos, pk, (int)ck.n_bits, ck.blocks, ck.signs, ck.norms, pk.jl_dim > 0);
    if (!st) st = launch_compress(*v, rows, S, cv.cap, pos, pv, (int)cv.n_bits, cv.blocks, cv.signs, cv.norms, false);
    if (st) return raise_status(st, "pq_compress_rows");
    if (!pos.dev) {
        const int64_t end = pos.host + S;
        if (end > ck.seq && !store_seq(args[2], end)) return nullptr;
        if (end > cv.seq && !store_seq(args[3], end)) return nullptr;
    }
    Py_RETURN_TRUE;
}

// decompress(cache, rotation, half) -> tensor or None
PyObject* decompress(PyObject*, PyObject* const* args, Py_ssize_t n) {
    Cache c;
    if (n != 3 || !read_cache(args[0], &c) || c.seq == 0 || c.seq != c.cap || c.blocks.numel() == 0 || !c.contiguous)
        Py_RETURN_NONE;
    const int dev = c.blocks.get_device();
    Plan plan;
    if (!plan_for(args[1], Py_None, dev, &plan) || plan.head_dim != c.dim || dev != c10::cuda::current_device()) Py_RETURN_NONE;
    const bool half = args[2] == Py_True;
    at::Tensor out = empty({c.rows_b, c.rows_h, c.seq, c.dim}, half ? at::kHalf : at::kFloat, dev);
    void* stream = stream_of(dev);
    const int st = launch([&] {
        return pq_dequant(c.blocks.data_ptr(), c.rows_b * c.rows_h * c.seq, (int)c.dim, (int)c.n_bits,
                          g_tables[c.n_bits].codebook, plan.rot, out.data_ptr(), half, stream);
    });
    if (st) return raise_status(st, "pq_dequant");
    return THPVariable_Wrap(out);
}

// ------------------------------------------------------------------ scratch of the attention calls
// One buffer per (device, stream) and, while the stream is being captured, one per capture (allocated from the graph's
// own pool, so it lives as long as the graph does).  The counters at its start must read zero when a launch starts; a
// launch leaves its own at zero, and with pq_decode_attn_counter_bytes() more than a call needs no record lies below
// that, so one clear when the buffer is new serves all later calls whose counters fit there.  The bridge's attention lays
// its workspace out the same way and shares the buffer.
static_assert(POLARQUANT_ATTENTION_COUNTER_BYTES == 65536, "the counter region of both kinds of attention");
struct Scratch {
    int device;
    void* stream;
    unsigned long long capture;              // 0: not captured
    at::Tensor buf;
    size_t cleared;
};
std::deque<Scratch> g_scratch;               // bounded: the least recently made entry goes
constexpr size_t kScratchLimit = 32;

// Undefined on a CUDA error.
at::Tensor attention_scratch(int device, void* stream, size_t* bytes_io, size_t counters) {
    const size_t kept = pq_decode_attn_counter_bytes(), need = *bytes_io += kept;
    cudaStreamCaptureStatus status;
    unsigned long long id = 0;
    if (cudaStreamGetCaptureInfo((cudaStream_t)stream, &status, &id) != cudaSuccess) return {};
    if (status != cudaStreamCaptureStatusActive) id = 0;
    // A stream is in one capture at a time: buffers of its earlier ones go back to their graphs' pools, which keep them for
    // as long as the graphs live and no longer.
    for (auto it = g_scratch.begin(); it != g_scratch.end();)
        it = it->device == device && it->stream == stream && it->capture && it->capture != id ? g_scratch.erase(it) : it + 1;
    Scratch* s = nullptr;
    for (Scratch& e : g_scratch)
        if (e.device == device && e.stream == stream && e.capture == id) s = &e;
    if (s && (size_t)s->buf.numel() < need) {
        s->buf = empty({(int64_t)need}, at::kByte, device);
        s->cleared = 0;
    }
    if (!s) {
        if (g_scratch.size() >= kScratchLimit) g_scratch.pop_front();
        const size_t bytes = id ? need : (need < (1u << 20) ? (1u << 20) : need);
        g_scratch.push_back({device, stream, id, empty({(int64_t)bytes}, at::kByte, device), 0});
        s = &g_scratch.back();
    }
    const size_t clear = id ? counters : kept;              // a graph replays its clear: no more of it than needed
    if (counters > kept || s->cleared < clear) {
        const size_t bytes = counters > clear ? counters : clear;
        if (cudaMemsetAsync(s->buf.data_ptr(), 0, bytes, (cudaStream_t)stream) != cudaSuccess) return {};
        if (counters <= kept) s->cleared = bytes;
    }
    return s->buf;
}

// ------------------------------------------------------------------ attention
struct Attend {                               // what decode and prefill read from their common arguments
    const at::Tensor* q;
    Cache ck, cv;
    Plan plan;
    int device;
    float scale;
    int64_t B, Hq, Hkv, Sq, D;
};
// args: query, ck, cv, rotation, jl_matrix, scale
bool read_attend(PyObject* const* args, Attend* a) {
    a->q = tensor(args[0]);
    if (!a->q || !half_contiguous(*a->q) || !read_cache(args[1], &a->ck) || !read_cache(args[2], &a->cv)) return false;
    const at::Tensor& q = *a->q;
    a->device = q.get_device();
    if (q.dim() < 3 || q.dim() > 4 || q.numel() == 0) return false;
    a->B = q.size(0);
    a->Hq = q.size(1);
    a->Sq = q.dim() == 4 ? q.size(2) : 1;
    a->D = q.size(-1);
    a->Hkv = a->ck.rows_h;
    const Cache &k = a->ck, &v = a->cv;
    if (!k.contiguous || !v.contiguous || k.blocks.get_device() != a->device || v.blocks.get_device() != a->device ||
        k.rows_b != a->B || v.rows_b != a->B || v.rows_h != a->Hkv || k.cap != v.cap || v.seq < k.seq || k.dim != a->D ||
        v.dim != a->D || a->Hkv == 0 || a->Hq % a->Hkv)
        return false;
    if (!plan_for(args[3], args[4], a->device, &a->plan) || a->plan.head_dim != a->D) return false;
    if (args[5] == Py_None) {
        a->scale = (float)(1.0 / std::sqrt((double)a->D));
    } else {
        const double s = PyFloat_AsDouble(args[5]);
        if (PyErr_Occurred()) { PyErr_Clear(); return false; }
        a->scale = (float)s;
    }
    return true;
}

// decode(query, ck, cv, rotation, jl_matrix, scale, enable_qjl, half, seq_len_tensor) -> tensor of the query's shape or None
PyObject* decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
    Attend a;
    if (n != 9 || !read_attend(args, &a) || a.Sq != 1) Py_RETURN_NONE;
    const bool qjl = args[6] == Py_True && a.plan.jl && a.ck.sketch, half = args[7] == Py_True;
    if (qjl && (!a.ck.signs.is_contiguous() || !a.ck.norms.is_contiguous() || a.ck.signs.size(-1) != a.plan.jl_dim / 8))
        Py_RETURN_NONE;
    Position len;
    int64_t S = a.ck.seq;
    if (args[8] != Py_None) {
        if (!tensor(args[8]) || !read_position(args[8], a.device, &len)) Py_RETURN_NONE;
        S = a.ck.cap;                          // the work partition and the scratch cover the capacity
    }
    void* st = stream_of(a.device);
    size_t need = pq_decode_attn_scratch_bytes((int)a.B, (int)a.Hq, (int)a.Hkv, S, (int)a.D, 0);
    const at::Tensor kept = attention_scratch(a.device, st, &need, ((size_t)a.B * a.Hq * 4 + 255) / 256 * 256);
    if (!kept.defined()) return raise_status(PQ_ERR_CUDA, "pq_decode_attn");
    void* scratch = kept.data_ptr();
    at::Tensor out = empty(a.q->sizes(), half ? at::kHalf : at::kFloat, a.device);
    const float *cbk = g_tables[a.ck.n_bits].codebook, *cbv = g_tables[a.cv.n_bits].codebook;
    const float* jl = qjl ? a.plan.jl : nullptr;
    const void *bits = qjl ? a.ck.signs.data_ptr() : nullptr, *norms = qjl ? a.ck.norms.data_ptr() : nullptr;
    const int m = qjl ? a.plan.jl_dim : 0;
    const int status = launch([&] {
        return len.dev ? pq_decode_attn_dynamic(a.q->data_ptr(), a.ck.blocks.data_ptr(), a.cv.blocks.data_ptr(), (int)a.B, (int)a.Hq,
                                         (int)a.Hkv, S, len.dev, a.ck.cap, (int)a.D, (int)a.ck.n_bits, (int)a.cv.n_bits, cbk,
                                         cbv, a.plan.rot, a.scale, jl, m, bits, norms, out.data_ptr(), half, nullptr, 0,
                                         scratch, need, st)
                       : pq_decode_attn(a.q->data_ptr(), a.ck.blocks.data_ptr(), a.cv.blocks.data_ptr(), (int)a.B, (int)a.Hq,
                                 (int)a.Hkv, S, a.ck.cap, (int)a.D, (int)a.ck.n_bits, (int)a.cv.n_bits, cbk, cbv, a.plan.rot,
                                 a.scale, jl, m, bits, norms, out.data_ptr(), half, nullptr, 0, scratch, need, st);
    });
    if (status) return raise_status(status, "pq_decode_attn");
    return THPVariable_Wrap(out);
}

// prefill(query, ck, cv, rotation, jl_matrix, scale, causal, half, workspace_limit) -> tensor or None.
// The workspace comes from torch's allocator on every call and goes back to it at once: the stream orders its reuse.
PyObject* prefill(PyObject*, PyObject* const* args, Py_ssize_t n) {
    Attend a;
    int64_t limit;
    if (n != 9 || !as_int(args[8], &limit) || !read_attend(args, &a) || a.q->dim() != 4) Py_RETURN_NONE;
    const bool half = args[7] == Py_True;
    at::Tensor out = empty(a.q->sizes(), half ? at::kHalf : at::kFloat, a.device), ws;
    const size_t need = pq_prefill_attn_workspace_bytes((int)a.B, (int)a.Hkv, a.ck.seq, (int)a.D);
    if (a.Sq * (a.Hq / a.Hkv) > 128 && need > 0 && need <= (size_t)limit) ws = empty({(int64_t)need}, at::kByte, a.device);
    const size_t parts_need = pq_prefill_attn_partial_bytes((int)a.B, (int)a.Hq, (int)a.Hkv, (int)a.Sq, a.ck.seq, (int)a.D);
    at::Tensor parts;
    if (parts_need) parts = empty({(int64_t)parts_need}, at::kByte, a.device);
    void *stream = stream_of(a.device), *wsp = ws.defined() ? ws.data_ptr() : nullptr, *pp = parts_need ? parts.data_ptr() : nullptr;
    const int status = launch([&] {
        return pq_prefill_attn_split(a.q->data_ptr(), a.ck.blocks.data_ptr(), a.cv.blocks.data_ptr(), (int)a.B, (int)a.Hq,
                                     (int)a.Hkv, (int)a.Sq, a.ck.seq, a.ck.cap, (int)a.D, (int)a.ck.n_bits, (int)a.cv.n_bits,
                                     g_tables[a.ck.n_bits].codebook, g_tables[a.cv.n_bits].codebook, a.plan.rot, a.scale,
                                     args[6] == Py_True, out.data_ptr(), half, wsp, wsp ? need : 0, pp, parts_need, stream);
    });
    if (status) return raise_status(status, "pq_prefill_attn");
    return THPVariable_Wrap(out);
}

// ------------------------------------------------------------------ prepared decode
struct Prepared {
    const void *q, *kb, *vb;
    int B, Hq, Hkv;
    int64_t cap;
    int D, kbits, vbits;
    const float *cbk, *cbv, *rot;
    float scale;
    const float* jl;
    int jl_dim;
    const void *bits, *norms;
    void* out;
    int half;
    void* partial;
    int splits;
    void* scratch;
    size_t scratch_bytes;
    const int64_t* len;
};
constexpr const char* kPreparedCapsule = "polarquant_kv.prepared";

// prepare(24 integers, scale) -> capsule; every pointer belongs to an object the caller keeps
PyObject* prepare(PyObject*, PyObject* const* args, Py_ssize_t n) {
    int64_t v[24];
    bool ok = n == 25;
    for (int i = 0; ok && i < 24; ++i) ok = as_int(args[i], &v[i]);
    const double scale = ok ? PyFloat_AsDouble(args[24]) : 0.0;
    if (!ok || PyErr_Occurred()) { PyErr_SetString(PyExc_TypeError, "prepare takes 24 integers and a float"); return nullptr; }
    Prepared* p = new Prepared{(void*)v[0], (void*)v[1], (void*)v[2], (int)v[3], (int)v[4], (int)v[5], v[6], (int)v[7], (int)v[8],
                               (int)v[9], (float*)v[10], (float*)v[11], (float*)v[12], (float)scale, (float*)v[13], (int)v[14],
                               (void*)v[15], (void*)v[16], (void*)v[17], (int)v[18], (void*)v[19], (int)v[20], (void*)v[21],
                               (size_t)v[22], (const int64_t*)v[23]};
    return PyCapsule_New(p, kPreparedCapsule, [](PyObject* c) { delete (Prepared*)PyCapsule_GetPointer(c, kPreparedCapsule); });
}
// run_prepared(capsule, ck, stream) -> status: over ck.seq_len tokens, or the device-side length
PyObject* run_prepared(PyObject*, PyObject* const* args, Py_ssize_t n) {
    int64_t stream;
    int64_t S;
    if (n != 3 || !as_int(args[2], &stream) || !attr_int(args[1], s_seq, &S)) {
        PyErr_SetString(PyExc_TypeError, "run_prepared(capsule, key cache, stream)");
        return nullptr;
    }
    const Prepared* p = (const Prepared*)PyCapsule_GetPointer(args[0], kPreparedCapsule);
    if (!p) return nullptr;
    const int st = launch([&] {
        return p->len ? pq_decode_attn_dynamic(p->q, p->kb, p->vb, p->B, p->Hq, p->Hkv, p->cap, p->len, p->cap, p->D, p->kbits,
                                                   p->vbits, p->cbk, p->cbv, p->rot, p->scale, p->jl, p->jl_dim, p->bits, p->norms,
                                                   p->out, p->half, p->partial, p->splits, p->scratch, p->scratch_bytes,
                                                   (void*)stream)
                          : pq_decode_attn(p->q, p->kb, p->vb, p->B, p->Hq, p->Hkv, S, p->cap, p->D, p->kbits, p->vbits, p->cbk,
                                           p->cbv, p->rot, p->scale, p->jl, p->jl_dim, p->bits, p->norms, p->out, p->half,
                                           p->partial, p->splits, p->scratch, p->scratch_bytes, (void*)stream);
    });
    return PyLong_FromLong(st);
}

// ------------------------------------------------------------------ the llama.cpp bridge's calls
const at::Tensor* f32(PyObject* o) {
    const at::Tensor* t = tensor(o);
    return t && t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->get_device() == c10::cuda::current_device() ? t : nullptr;
}
// bridge_compress(x, rotation, codebook) -> (radius, packed) or None (also when the call reported an error: not cleared)
PyObject* bridge_compress(PyObject*, PyObject* const* args, Py_ssize_t n) {
    const at::Tensor *x = n == 3 ? f32(args[0]) : nullptr, *R = n == 3 ? f32(args[1]) : nullptr, *cb = n == 3 ? f32(args[2]) : nullptr;
    if (!x || !R || !cb || x->dim() != 2) Py_RETURN_NONE;
    const int64_t N = x->size(0), D = x->size(1);
    if (N <= 0 || N > 0x7FFFFFFF || D <= 0 || (D & 1) || D > 1024 || cb->numel() < 1 || cb->numel() > 16 || R->numel() != D * D)
        Py_RETURN_NONE;
    const int dev = x->get_device();
    at::Tensor radius = empty({N}, at::kFloat, dev), packed = empty({N, D / 2}, at::kByte, dev);
    void* stream = stream_of(dev);
    launch([&] {
        polarquant_compress_cuda_c((const float*)x->data_ptr(), (const float*)R->data_ptr(), (const float*)cb->data_ptr(),
                                   (float*)radius.data_ptr(), (uint8_t*)packed.data_ptr(), (int)N, (int)D, (int)cb->numel(), stream);
        return 0;
    });
    PyObject *a = THPVariable_Wrap(radius), *b = THPVariable_Wrap(packed);
    PyObject* r = a && b ? PyTuple_Pack(2, a, b) : nullptr;
    Py_XDECREF(a);
    Py_XDECREF(b);
    return r;
}
// bridge_rotate(x, rotation, inverse) -> tensor or None
PyObject* bridge_rotate(PyObject*, PyObject* const* args, Py_ssize_t n) {
    const at::Tensor *x = n == 3 ? f32(args[0]) : nullptr, *R = n == 3 ? f32(args[1]) : nullptr;
    if (!x || !R || x->dim() != 2 || x->numel() == 0 || x->size(1) > 1024 || R->numel() != x->size(1) * x->size(1)) Py_RETURN_NONE;
    const int dev = x->get_device();
    at::Tensor out = empty(x->sizes(), at::kFloat, dev);
    const auto fn = args[2] == Py_True ? polarquant_inverse_rotate_cuda_c : polarquant_rotate_query_cuda_c;
    void* stream = stream_of(dev);
    launch([&] {
        fn((const float*)x->data_ptr(), (const float*)R->data_ptr(), (float*)out.data_ptr(), (int)x->size(0), (int)x->size(1), stream);
        return 0;
    });
    return THPVariable_Wrap(out);
}
// bridge_attention(q, packed_k, k_radius, packed_v, v_radius, codebook, scale, out) -> out, a new tensor for None, or None
PyObject* bridge_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 8) Py_RETURN_NONE;
    const at::Tensor *q = f32(args[0]), *kr = f32(args[2]), *vr = f32(args[4]), *cb = f32(args[5]), *pk = tensor(args[1]), *pv = tensor(args[3]);
    if (!q || !kr || !vr || !cb || !pk || !pv || q->dim() != 2 || pk->dim() != 3) Py_RETURN_NONE;
    for (const at::Tensor* t : {pk, pv})
        if (!t->is_cuda() || t->scalar_type() != at::kByte || !t->is_contiguous() || t->get_device() != q->get_device()) Py_RETURN_NONE;
    const int64_t hq = q->size(0), D = q->size(1), hkv = pk->size(0), S = pk->size(1);
    if (pv->sizes() != pk->sizes() || pk->size(2) * 2 != D || kr->dim() != 2 || vr->dim() != 2 || kr->size(0) != hkv || kr->size(1) != S ||
        vr->sizes() != kr->sizes() || hq <= 0 || hkv <= 0 || hq % hkv || S <= 0 || S > 0x7FFFFFFF || D <= 0 || (D & 1) || D > 1024 ||
        cb->numel() < 1 || cb->numel() > 16)
        Py_RETURN_NONE;
    const double scale = PyFloat_AsDouble(args[6]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    const int dev = q->get_device();
    const at::Tensor* given = f32(args[7]);
    if (args[7] != Py_None && (!given || given->sizes() != q->sizes())) Py_RETURN_NONE;
    const at::Tensor out = given ? *given : empty(q->sizes(), at::kFloat, dev);
    void* stream = stream_of(dev);
    const size_t need = polarquant_fused_attention_ws_bytes_c((int)hq, (int)hkv, (int)S, (int)D);
    at::Tensor ws;
    size_t bytes = 0;
    if (need) {
        bytes = need - POLARQUANT_ATTENTION_COUNTER_BYTES;
        ws = attention_scratch(dev, stream, &bytes, ((size_t)hq * 4 + 255) / 256 * 256);
        if (!ws.defined()) return raise_status(PQ_ERR_CUDA, "polarquant_fused_attention_ws_cuda_c");
    }
    void* wsp = need ? ws.data_ptr() : nullptr;
    launch([&] {
        polarquant_fused_attention_ws_cuda_c((const float*)q->data_ptr(), (const uint8_t*)pk->data_ptr(), (const float*)kr->data_ptr(),
                                             (const uint8_t*)pv->data_ptr(), (const float*)vr->data_ptr(), (const float*)cb->data_ptr(),
                                             (float*)out.data_ptr(), (int)hq, (int)hkv, (int)S, (int)D, (int)cb->numel(), (float)scale,
                                             wsp, bytes, stream);
        return 0;
    });
    if (given) {
        Py_INCREF(args[7]);
        return args[7];
    }
    return THPVariable_Wrap(out);
}
// bridge_error() -> code of the calling thread's last failed bridge call, cleared
PyObject* bridge_error(PyObject*, PyObject*) { return PyLong_FromLong(polarquant_last_error_c()); }

// ------------------------------------------------------------------ module
using Fast = PyObject*(PyObject*, PyObject* const*, Py_ssize_t);
// C++ exceptions (no memory, a tensor without storage) become the Python errors that torch makes of them.
template <Fast* F>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    return F(self, args, n);
    END_HANDLE_TH_ERRORS
}
#define PQ_FAST(name, doc) {#name, (PyCFunction)(void (*)(void))guarded<name>, METH_FASTCALL, doc}
PyMethodDef methods[] = {
    {"register", (PyCFunction)(void (*)(void))register_types, METH_FASTCALL, "register(CompressedKV, DevicePlan, check)"},
    PQ_FAST(plan_get, "cached plan of the matrix objects"),
    PQ_FAST(plan_put, "remember a plan"),
    PQ_FAST(plan_handle, "device constants of a plan"),
    PQ_FAST(set_tables, "codebook and thresholds of a width"),
    PQ_FAST(compress, "see quantizer.compress"),
    PQ_FAST(append, "see KVCacheManager.append"),
    PQ_FAST(decompress, "see quantizer.decompress"),
    PQ_FAST(decode, "see attention.decode_attention"),
    PQ_FAST(prefill, "see attention.prefill_attention"),
    PQ_FAST(prepare, "arguments of a prepared decode call"),
    PQ_FAST(run_prepared, "launch a prepared decode call"),
    PQ_FAST(bridge_compress, "see llama_bridge.compress"),
    PQ_FAST(bridge_rotate, "see llama_bridge.rotate_query"),
    PQ_FAST(bridge_attention, "see llama_bridge.fused_attention"),
    {"bridge_error", bridge_error, METH_NOARGS, "last error of the calling thread"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native host path of polarquant_kv.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
    struct { PyObject** at; const char* text; } names[] = {
        {&s_native, "_native"}, {&s_blocks, "blocks"}, {&s_signs, "qjl_signs"}, {&s_norms, "residual_norms"},
        {&s_bits, "n_bits"}, {&s_dim, "original_dim"}, {&s_seq, "seq_len"}, {&s_cap, "max_seq_len"}};
    for (auto& n : names)
        if (!(*n.at = PyUnicode_InternFromString(n.text))) return nullptr;
    return PyModule_Create(&module);
}
