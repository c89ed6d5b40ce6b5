// Native half of capi.py: torch tensors in, one C-ABI call, torch tensors out.
//
// A Python caller of a one-row linear spends more time on the host than the GPU spends on the
// kernel, so everything between the caller's arguments and the launch is done here: reading shapes
// and strides, filling the descriptor, allocating the result from torch's caching allocator and
// looking up the current stream.  Through ctypes the same steps took about 17 us per call (a
// descriptor object, a dozen boxed pointers, three attribute walks per tensor), which is what an
// un-captured quantizelinear + quant_dot pair cost twice: 36.5 us for 256 x 1024 x 1024.
// capi.py keeps the signatures and the documentation and passes its arguments on in order.
#include <Python.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>
#include "../../include/mgx_cuda.h"
#include <algorithm>
#include <stdexcept>

namespace {

PyObject* g_error = nullptr; // capi.MgxError

// a Python exception is set; unwinds to the entry point
struct py_error
{
};

[[noreturn]] void fail(PyObject* type, const char* text)
{
    PyErr_SetString(type, text);
    throw py_error{};
}

const at::Tensor& tensor(PyObject* o)
{
    if(not THPVariable_Check(o))
        fail(PyExc_TypeError, "expected a tensor");
    return THPVariable_Unpack(o);
}

// None or a tensor
const at::Tensor* maybe(PyObject* o) { return o == Py_None ? nullptr : &tensor(o); }

void* ptr(const at::Tensor* t) { return t == nullptr ? nullptr : t->data_ptr(); }

int64_t integer(PyObject* o)
{
    const int64_t v = PyLong_AsLongLong(o);
    if(v == -1 and PyErr_Occurred() != nullptr)
        throw py_error{};
    return v;
}

double real(PyObject* o)
{
    const double v = PyFloat_AsDouble(o);
    if(v == -1.0 and PyErr_Occurred() != nullptr)
        throw py_error{};
    return v;
}

bool truth(PyObject* o)
{
    const int v = PyObject_IsTrue(o);
    if(v < 0)
        throw py_error{};
    return v != 0;
}

at::ScalarType dtype(PyObject* o)
{
    if(not THPDtype_Check(o))
        fail(PyExc_TypeError, "expected a torch dtype");
    return reinterpret_cast<THPDtype*>(o)->scalar_type;
}

int code_of(at::ScalarType t)
{
    switch(t)
    {
    case at::kFloat: return MGX_F32;
    case at::kHalf: return MGX_F16;
    case at::kChar: return MGX_I8;
    case at::kByte: return MGX_U8;
    case at::kInt: return MGX_I32;
    case at::kFloat8_e4m3fn: return MGX_FP8_E4M3FN;
    default: fail(PyExc_KeyError, c10::toString(t));
    }
}

int index_code(const at::Tensor& t) { return t.scalar_type() == at::kLong ? MGX_I64 : MGX_I32; }

void need_dim(const at::Tensor& t, int64_t dim)
{
    if(t.dim() != dim)
        fail(PyExc_ValueError, "tensor has the wrong number of dimensions");
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType t, const at::Tensor& like)
{
    if(like.is_cuda())
        return at::detail::empty_cuda(sizes, t, like.device(), std::nullopt);
    return at::empty(sizes, like.options().dtype(t));
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// the C-ABI call, with the interpreter free meanwhile: a launch waits when the stream's queue is full
template <class F>
void call(const char* what, F f)
{
    struct released
    {
        PyThreadState* state = PyEval_SaveThread();
        ~released() { PyEval_RestoreThread(state); }
    };
    const int code = [&] {
        released r;
        return f();
    }();
    if(code == 0)
        return;
    PyObject* e = PyObject_CallFunction(g_error, "is", code, what);
    if(e != nullptr)
    {
        PyErr_SetObject(g_error, e);
        Py_DECREF(e);
    }
    throw py_error{};
}

// Strides (elements) of a tensor broadcastable to [rows, cols], as MIGraphX would pass it: 0 along
// broadcast dimensions.
struct strides2
{
    int64_t v[2] = {0, 0};
    strides2(const at::Tensor* t, int64_t cols)
    {
        if(t == nullptr or t->dim() == 0 or t->numel() == 1)
            return;
        if(t->dim() == 1)
        {
            if(t->size(0) != cols)
                fail(PyExc_ValueError, "1-D scale must have `cols` elements");
            v[1] = t->stride(0);
            return;
        }
        v[0] = t->size(0) == 1 ? 0 : t->stride(0);
        v[1] = t->size(1) == 1 ? 0 : t->stride(1);
    }
};

// rows x cols of a 2-D tensor and the element stride between rows
struct matrix
{
    int64_t rows, cols, ld;
    explicit matrix(const at::Tensor& t)
    {
        need_dim(t, 2);
        rows = t.size(0), cols = t.size(1);
        ld = rows > 1 ? t.stride(0) : cols;
    }
};

// [batch, rows, cols] of a 2-D or 3-D tensor
struct batched
{
    int64_t batch, rows, cols, ld, stride;
    explicit batched(const at::Tensor& t)
    {
        if(t.dim() == 3)
            batch = t.size(0), rows = t.size(1), cols = t.size(2), ld = t.stride(1), stride = t.stride(0);
        else
        {
            need_dim(t, 2);
            // the batch stride torch gives the unsqueezed view
            batch = 1, rows = t.size(0), cols = t.size(1), ld = t.stride(0), stride = rows * ld;
        }
    }
};

PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* wrap_or_none(const at::Tensor& t) { return t.defined() ? THPVariable_Wrap(t) : Py_NewRef(Py_None); }

// (x, scale, zp, out_dtype)
PyObject* quantizelinear(PyObject* const* a)
{
    const at::Tensor &x = tensor(a[0]), &scale = tensor(a[1]);
    const at::Tensor* zp = maybe(a[2]);
    const matrix m(x);
    const at::ScalarType t = a[3] != Py_None ? dtype(a[3]) : (zp != nullptr ? zp->scalar_type() : at::kByte);
    at::Tensor y           = empty({m.rows, m.cols}, t, x);
    const strides2 ss(&scale, m.cols), zs(zp, m.cols);
    const int xc = code_of(x.scalar_type()), yc = code_of(t);
    call("mgx_cuda_quantizelinear", [&] {
        return mgx_cuda_quantizelinear(x.data_ptr(), xc, m.ld, scale.data_ptr(), ss.v, ptr(zp), zp != nullptr ? zs.v : nullptr,
                                       y.data_ptr(), yc, m.cols, m.rows, m.cols, stream());
    });
    return wrap(std::move(y));
}

// (x, scale, zp)
PyObject* dequantizelinear(PyObject* const* a)
{
    const at::Tensor &x = tensor(a[0]), &scale = tensor(a[1]);
    const at::Tensor* zp = maybe(a[2]);
    const matrix m(x);
    at::Tensor y = empty({m.rows, m.cols}, scale.scalar_type(), x);
    const strides2 ss(&scale, m.cols), zs(zp, m.cols);
    const int xc = code_of(x.scalar_type()), sc = code_of(scale.scalar_type());
    call("mgx_cuda_dequantizelinear", [&] {
        return mgx_cuda_dequantizelinear(x.data_ptr(), xc, m.ld, scale.data_ptr(), sc, ss.v, ptr(zp),
                                         zp != nullptr ? zs.v : nullptr, y.data_ptr(), m.cols, m.rows, m.cols, stream());
    });
    return wrap(std::move(y));
}

// (a, b, b_layout, scale, scale_mode, bias, act, residual, out_dtype, out, workspace, q_out, q_scale,
//  q_zero_point, write_d, half_math, lut)
PyObject* qgemm(PyObject* const* a)
{
    const at::Tensor &A = tensor(a[0]), &B = tensor(a[1]);
    const int b_layout  = static_cast<int>(integer(a[2]));
    const at::Tensor *scale = maybe(a[3]), *bias = maybe(a[5]), *residual = maybe(a[7]), *out = maybe(a[9]),
                     *workspace = maybe(a[10]), *q_out = maybe(a[11]), *lut = maybe(a[16]);
    const int act   = static_cast<int>(integer(a[6]));
    const batched ma(A), mb(B);
    mgx_qgemm_desc d{};
    d.batch = ma.batch, d.M = ma.rows, d.K = ma.cols;
    d.N          = b_layout == MGX_B_KN ? mb.cols : mb.rows;
    d.lda        = ma.ld, d.stride_a = ma.stride;
    d.ldb        = mb.ld, d.stride_b = mb.stride;
    d.ab_type    = code_of(A.scalar_type());
    d.b_layout   = b_layout;
    d.act        = act;
    d.flags      = truth(a[15]) ? MGX_QGEMM_HALF_MATH : 0;
    if(a[4] != Py_None)
        d.scale_mode = static_cast<int>(integer(a[4]));
    else if(scale == nullptr)
        d.scale_mode = MGX_SCALE_NONE;
    else
        d.scale_mode = scale->numel() == 1 ? MGX_SCALE_PER_TENSOR
                                           : (scale->numel() == d.N ? MGX_SCALE_PER_COL : MGX_SCALE_PER_ROW);
    at::Tensor made;
    if(out == nullptr)
    {
        at::ScalarType t = at::kFloat;
        if(a[8] != Py_None)
            t = dtype(a[8]);
        else if(A.scalar_type() == at::kChar and scale == nullptr and bias == nullptr and act == MGX_ACT_NONE)
            t = at::kInt;
        made = A.dim() == 3 ? empty({d.batch, d.M, d.N}, t, A) : empty({d.M, d.N}, t, A);
    }
    const at::Tensor& D = out != nullptr ? *out : made;
    const batched md(D);
    d.ldd = md.ld, d.stride_d = md.stride;
    d.out_type = code_of(D.scalar_type());
    at::Tensor lent;
    if(b_layout == MGX_B_KN and workspace == nullptr)
    {
        // a [K,N] operand is re-laid out there; [N,K] operands take nothing
        lent      = empty({static_cast<int64_t>(mgx_cuda_qgemm_workspace(&d))}, at::kByte, A);
        workspace = &lent;
    }
    const size_t have = workspace == nullptr ? 0 : static_cast<size_t>(workspace->numel());
    mgx_qgemm_qout q{};
    if(q_out != nullptr)
    {
        const batched mq(*q_out);
        q.q = q_out->data_ptr(), q.ldq = mq.ld, q.stride_q = mq.stride;
        q.q_type     = code_of(q_out->scalar_type());
        q.scale      = static_cast<float>(real(a[12]));
        q.zero_point = static_cast<float>(real(a[13]));
        q.flags      = lut != nullptr ? MGX_QOUT_LUT : 0;
        q.lut        = ptr(lut);
    }
    void* dst = q_out == nullptr or truth(a[14]) ? D.data_ptr() : nullptr;
    const auto *sp = static_cast<const float*>(ptr(scale)), *bp = static_cast<const float*>(ptr(bias));
    call("mgx_cuda_qgemm", [&] {
        if(q_out == nullptr)
            return mgx_cuda_qgemm(&d, A.data_ptr(), B.data_ptr(), dst, sp, bp, ptr(residual), ptr(workspace), have, stream());
        return mgx_cuda_qgemm_ex(&d, A.data_ptr(), B.data_ptr(), dst, sp, bp, ptr(residual), &q, ptr(workspace), have, stream());
    });
    return out != nullptr ? Py_NewRef(a[9]) : wrap(std::move(made));
}

// (a, bp, scales, zp, zp_const, group, act, which, workspace); which: 0 auto, 1 gemv, 2 gemm
PyObject* w4a16(PyObject* const* a)
{
    const at::Tensor &A = tensor(a[0]), &Bp = tensor(a[1]), &scales = tensor(a[2]);
    const at::Tensor *zp = maybe(a[3]), *workspace = maybe(a[8]);
    need_dim(A, 2);
    mgx_w4_desc d{};
    d.M = A.size(0), d.K = A.size(1), d.N = Bp.size(0);
    d.lda = A.stride(0), d.ldd = d.N;
    d.zp_const = static_cast<int>(integer(a[4]));
    d.group    = static_cast<int>(integer(a[5]));
    d.act      = static_cast<int>(integer(a[6]));
    const int64_t which = integer(a[7]);
    at::Tensor D        = empty({d.M, d.N}, at::kHalf, A), lent;
    const size_t need   = mgx_cuda_w4a16_workspace(&d);
    if(need != 0 and workspace == nullptr)
    {
        lent      = empty({static_cast<int64_t>(need)}, at::kByte, A);
        workspace = &lent;
    }
    const size_t have = workspace == nullptr ? 0 : static_cast<size_t>(workspace->numel());
    auto* fn          = which == 0 ? mgx_cuda_w4a16 : (which == 1 ? mgx_cuda_w4a16_gemv : mgx_cuda_w4a16_gemm);
    const char* what  = which == 0 ? "mgx_cuda_w4a16[auto]" : (which == 1 ? "mgx_cuda_w4a16[gemv]" : "mgx_cuda_w4a16[gemm]");
    call(what, [&] {
        return fn(&d, A.data_ptr(), Bp.data_ptr(), scales.data_ptr(), ptr(zp), D.data_ptr(), ptr(workspace), have, stream());
    });
    return wrap(std::move(D));
}

// (x, gamma, beta, eps, q_scale, q_zero_point, write_y, dq_scale, rms)
PyObject* layernorm(PyObject* const* a)
{
    const at::Tensor& x = tensor(a[0]);
    const at::Tensor *gamma = maybe(a[1]), *beta = maybe(a[2]);
    need_dim(x, 2);
    mgx_layernorm_desc d{};
    d.rows = x.size(0), d.cols = x.size(1);
    d.ldx = x.stride(0), d.ldy = d.cols, d.ldq = d.cols;
    d.type         = code_of(x.scalar_type());
    d.eps          = static_cast<float>(real(a[3]));
    d.q_type       = MGX_I8;
    d.q_scale      = a[4] == Py_None ? 1.0f : static_cast<float>(real(a[4]));
    d.q_scale      = d.q_scale == 0.0f ? 1.0f : d.q_scale;
    d.q_zero_point = static_cast<float>(real(a[5]));
    d.flags        = truth(a[8]) ? MGX_LAYERNORM_RMS : 0;
    const bool has_dq = a[7] != Py_None;
    at::Tensor y, q, dq;
    if(truth(a[6]))
        y = empty({d.rows, d.cols}, x.scalar_type(), x);
    if(a[4] != Py_None)
        q = empty({d.rows, d.cols}, at::kChar, x);
    auto at_or_null = [](const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; };
    if(not has_dq)
    {
        call("mgx_cuda_layernorm", [&] {
            return mgx_cuda_layernorm(&d, x.data_ptr(), ptr(gamma), ptr(beta), at_or_null(y), at_or_null(q), stream());
        });
        return Py_BuildValue("NN", wrap_or_none(y), wrap_or_none(q));
    }
    dq               = empty({d.rows, d.cols}, x.scalar_type(), x);
    const float dq_s = static_cast<float>(real(a[7]));
    call("mgx_cuda_layernorm_ex", [&] {
        return mgx_cuda_layernorm_ex(&d, x.data_ptr(), ptr(gamma), ptr(beta), at_or_null(y), at_or_null(q), dq.data_ptr(),
                                     d.cols, dq_s, stream());
    });
    return Py_BuildValue("NNN", wrap_or_none(y), wrap_or_none(q), wrap_or_none(dq));
}

// (q, k, v, batch, seq, heads, scale, q_scale, q_zero_point, write_o, flags)
PyObject* attention(PyObject* const* a)
{
    const at::Tensor &q = tensor(a[0]), &k = tensor(a[1]), &v = tensor(a[2]);
    mgx_attention_desc d{};
    d.batch = integer(a[3]), d.seq = integer(a[4]), d.heads = integer(a[5]);
    d.head_dim = 64;
    d.ldq = q.stride(0), d.ldk = k.stride(0), d.ldv = v.stride(0);
    const int64_t width = d.heads * 64;
    d.ldo = width, d.ldoq = width;
    d.scale        = static_cast<float>(real(a[6]));
    d.q_scale      = a[7] == Py_None ? 1.0f : static_cast<float>(real(a[7]));
    d.q_scale      = d.q_scale == 0.0f ? 1.0f : d.q_scale;
    d.q_zero_point = static_cast<float>(real(a[8]));
    d.flags        = static_cast<int>(integer(a[10]));
    at::Tensor o, oq;
    if(truth(a[9]))
        o = empty({d.batch * d.seq, width}, at::kHalf, q);
    if(a[7] != Py_None)
        oq = empty({d.batch * d.seq, width}, at::kChar, q);
    call("mgx_cuda_attention", [&] {
        return mgx_cuda_attention(&d, q.data_ptr(), k.data_ptr(), v.data_ptr(), o.defined() ? o.data_ptr() : nullptr,
                                  oq.defined() ? oq.data_ptr() : nullptr, stream());
    });
    return Py_BuildValue("NN", wrap_or_none(o), wrap_or_none(oq));
}

// (present, seqlens, past)
PyObject* concat_past_present(PyObject* const* a)
{
    const at::Tensor &present = tensor(a[0]), &seqlens = tensor(a[1]), &past = tensor(a[2]);
    need_dim(present, 4);
    const int64_t es         = present.element_size();
    const int64_t strides[3] = {present.stride(0) * es, present.stride(1) * es, present.stride(2) * es};
    call("mgx_cuda_concat_past_present", [&] {
        return mgx_cuda_concat_past_present(present.data_ptr(), strides, present.size(0), present.size(1), present.size(2),
                                            present.size(3) * es, seqlens.data_ptr(), index_code(seqlens), past.data_ptr(),
                                            past.size(2), stream());
    });
    return Py_NewRef(a[2]);
}

// (x, positions, cos_cache, sin_cache)
PyObject* rotary_embedding(PyObject* const* a)
{
    const at::Tensor &x = tensor(a[0]), &pos = tensor(a[1]), &cosc = tensor(a[2]), &sinc = tensor(a[3]);
    need_dim(x, 4);
    const int64_t strides[3] = {x.stride(0), x.stride(1), x.stride(2)};
    at::Tensor out           = empty(x.sizes(), x.scalar_type(), x);
    const int xc             = code_of(x.scalar_type());
    call("mgx_cuda_rotary_embedding", [&] {
        return mgx_cuda_rotary_embedding(x.data_ptr(), xc, strides, x.size(0), x.size(1), x.size(2), x.size(3), pos.data_ptr(),
                                         index_code(pos), cosc.data_ptr(), sinc.data_ptr(), cosc.size(0), out.data_ptr(),
                                         stream());
    });
    return wrap(std::move(out));
}

// (q, k_cache, v_cache, seqlens, scale)
PyObject* gqa_decode_attention(PyObject* const* a)
{
    const at::Tensor &q = tensor(a[0]), &kc = tensor(a[1]), &vc = tensor(a[2]), &seqlens = tensor(a[3]);
    need_dim(q, 3);
    need_dim(kc, 4);
    mgx_gqa_decode_desc d{};
    d.batch = q.size(0), d.heads = q.size(1), d.head = q.size(2);
    d.kv_heads = kc.size(1), d.cache_seq = kc.size(2);
    d.q_batch_stride = q.stride(0), d.q_head_stride = q.stride(1);
    d.scale        = static_cast<float>(real(a[4]));
    d.seqlens_type = index_code(seqlens);
    at::Tensor out = empty({d.batch, d.heads * d.head}, at::kHalf, q);
    call("mgx_cuda_gqa_decode_attention", [&] {
        return mgx_cuda_gqa_decode_attention(&d, q.data_ptr(), kc.data_ptr(), vc.data_ptr(), seqlens.data_ptr(), out.data_ptr(),
                                             stream());
    });
    return wrap(std::move(out));
}

// A snapshot of any iterable as a tuple.  It owns its items, so that those of a sequence that makes them on
// the fly (an array, a range) live as long as the call, and a list that another thread changes meanwhile
// does not matter.
struct items
{
    PyObject* tuple;
    explicit items(PyObject* o) : tuple(PySequence_Tuple(o))
    {
        if(tuple == nullptr)
            throw py_error{};
    }
    items(const items&) = delete;
    items& operator=(const items&) = delete;
    ~items() { Py_DECREF(tuple); }
    Py_ssize_t size() const { return PyTuple_GET_SIZE(tuple); }
    PyObject* operator[](Py_ssize_t i) const { return PyTuple_GET_ITEM(tuple, i); }
};

// (inputs, program, lens, op codes by name)
PyObject* pointwise(PyObject* const* a)
{
    const items ins(a[0]), prog(a[1]), lens(a[2]);
    PyObject* ops = a[3];
    const auto ni = ins.size(), np = prog.size(), nd = lens.size();
    if(ni < 1 or np < 1)
        fail(PyExc_IndexError, "at least one input and one instruction");
    if(ni > MGX_PW_MAXIN or np > MGX_PW_MAXINSN or nd > MGX_PW_MAXDIMS)
        fail(PyExc_IndexError, "too many inputs, instructions or dimensions");
    mgx_pw_desc d{};
    d.ndim = static_cast<int>(nd), d.ninputs = static_cast<int>(ni), d.ninsns = static_cast<int>(np);
    for(Py_ssize_t k = 0; k < nd; ++k)
        d.lens[k] = integer(lens[k]);
    const at::IntArrayRef sizes(d.lens, static_cast<size_t>(nd));
    const void* in[MGX_PW_MAXIN];
    for(Py_ssize_t i = 0; i < ni; ++i)
    {
        const at::Tensor& t = tensor(ins[i]);
        if(t.sizes() != sizes)
            fail(PyExc_AssertionError, "an input does not have the shape of the result");
        d.in_type[i] = code_of(t.scalar_type());
        for(Py_ssize_t k = 0; k < nd; ++k)
            d.in_strides[i][k] = t.stride(k);
        in[i] = t.data_ptr();
    }
    for(Py_ssize_t n = 0; n < np; ++n)
    {
        const items t(prog[n]);
        if(t.size() != 4)
            fail(PyExc_ValueError, "an instruction is (op, type, operands, immediate)");
        PyObject* op = PyDict_GetItemWithError(ops, t[0]);
        if(op == nullptr)
            fail(PyExc_ValueError, "unknown element-wise operator");
        const items src(t[2]);
        d.insn[n].op   = static_cast<int>(integer(op));
        d.insn[n].type = static_cast<int>(integer(t[1]));
        d.insn[n].imm  = static_cast<float>(real(t[3]));
        const auto ns  = std::min<Py_ssize_t>(3, src.size());
        for(Py_ssize_t j = 0; j < ns; ++j)
            d.insn[n].src[j] = static_cast<int>(integer(src[j]));
    }
    at::ScalarType t = at::kFloat;
    switch(d.insn[np - 1].type)
    {
    case MGX_F32: break;
    case MGX_F16: t = at::kHalf; break;
    case MGX_I8: t = at::kChar; break;
    case MGX_U8: t = at::kByte; break;
    case MGX_I32: t = at::kInt; break;
    default: fail(PyExc_KeyError, "result type of the last instruction");
    }
    at::Tensor out = empty(sizes, t, tensor(ins[0]));
    call("mgx_cuda_pointwise", [&] { return mgx_cuda_pointwise(&d, in, out.data_ptr(), stream()); });
    return wrap(std::move(out));
}

// (x)
PyObject* softmax(PyObject* const* a)
{
    const at::Tensor& x = tensor(a[0]);
    if(x.dim() != 2 or x.stride(1) != 1)
        fail(PyExc_AssertionError, "softmax takes a 2-D tensor with contiguous rows");
    at::Tensor out = empty(x.sizes(), x.scalar_type(), x);
    const int xc   = code_of(x.scalar_type());
    call("mgx_cuda_softmax", [&] {
        return mgx_cuda_softmax(x.data_ptr(), xc, x.stride(0), out.data_ptr(), out.stride(0), x.size(0), x.size(1), stream());
    });
    return wrap(std::move(out));
}

// One entry per function: the argument count is fixed, capi.py passes every argument.
template <PyObject* (*F)(PyObject* const*), Py_ssize_t N>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    if(nargs != N)
    {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", N, nargs);
        return nullptr;
    }
    try
    {
        return F(args);
    }
    catch(const py_error&)
    {
    }
    catch(const std::exception& e)
    {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

PyObject* set_error(PyObject* const* a)
{
    Py_XSETREF(g_error, Py_NewRef(a[0]));
    Py_RETURN_NONE;
}

#define MGX_ENTRY(name, n)                                                                          \
    {                                                                                               \
        #name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<name, n>)), METH_FASTCALL, nullptr \
    }

PyMethodDef methods[] = {MGX_ENTRY(quantizelinear, 4),
                         MGX_ENTRY(dequantizelinear, 3),
                         MGX_ENTRY(qgemm, 17),
                         MGX_ENTRY(w4a16, 9),
                         MGX_ENTRY(layernorm, 9),
                         MGX_ENTRY(attention, 11),
                         MGX_ENTRY(concat_past_present, 3),
                         MGX_ENTRY(rotary_embedding, 4),
                         MGX_ENTRY(gqa_decode_attention, 5),
                         MGX_ENTRY(pointwise, 4),
                         MGX_ENTRY(softmax, 1),
                         MGX_ENTRY(set_error, 1),
                         {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "mgx_torch_ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit_mgx_torch_ops(void) { return PyModule_Create(&module); }
