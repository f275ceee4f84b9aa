// Host path of the public API calls, as a CPython extension on torch's C++ tensors.
//
// A decode step on a small batch is bound by the host: the same checks, allocations and launches written in Python
// (ctypes structures of 40 fields, one torch.empty per buffer, context managers) took 41 us for a call whose kernels run
// for 20.  Here the host's share is 7 us for a prefill call, 9-10 for a decode step and 16 for one that makes its schedule:
// arguments are checked on the C++ tensors, the split-KV scratch is one allocation, and the kernels are launched through the
// C ABI of libflashmla_b200.so, whose functions are bound by address (_capi.py loads the library; bind() checks its version).
//
// Checks and messages are those of the reference's host glue: csrc/api/dense_decode.h:13-225, csrc/api/sparse_decode.h:183-495,
// csrc/api/sparse_fwd.h:101-243.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/from_blob.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <initializer_list>
#include <mutex>
#include <stdexcept>
#include <string>

#include "../../include/flashmla_b200.h"

namespace {

// ---- the C ABI, bound by address ---------------------------------------------------------------------------
struct Api {
    decltype(&mla_abi_version) abi_version;
    decltype(&mla_last_error) last_error;
    decltype(&mla_num_sm_parts) num_sm_parts;
    decltype(&mla_num_sm_parts_uniform) num_sm_parts_uniform;
    decltype(&mla_get_sched_meta) get_sched_meta;
    decltype(&mla_dense_decode_fwd) dense_decode_fwd;
    decltype(&mla_sparse_decode_fwd) sparse_decode_fwd;
    decltype(&mla_combine) combine;
    decltype(&mla_sparse_prefill_fwd) sparse_prefill_fwd;
    decltype(&mla_quantize_fp8_kvcache_padded) quantize;
} api;

// tile-scheduler arguments (csrc/api/dense_decode.h:104-105, csrc/api/sparse_decode.h:92-99)
constexpr int BLOCK_SIZE_N = 64;
constexpr int FIXED_OVERHEAD_NUM_BLOCKS = 5;
constexpr int META_INTS = 8;

struct Refused : std::runtime_error { using std::runtime_error::runtime_error; };   // -> RuntimeError with the message as it is

[[noreturn]] void refuse(const std::string& msg) { throw Refused(msg); }
inline void require(bool ok, const char* msg) { if (__builtin_expect(!ok, 0)) refuse(msg); }

void check(int rc, const char* what) {
    if (rc) refuse(std::string(what) + " failed (code " + std::to_string(rc) + "): " + api.last_error());
}

// ---- Python arguments -----------------------------------------------------------------------------------------
const at::Tensor& tensor(PyObject* o, const char* name) {
    if (!THPVariable_Check(o)) throw py::type_error(std::string(name) + " must be a tensor");
    return THPVariable_Unpack(o);
}
const at::Tensor* optional(PyObject* o, const char* name) { return o == Py_None ? nullptr : &tensor(o, name); }

int64_t integer(PyObject* o) {
    const int64_t v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}
double real(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return v;
}
bool truth(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw python_error();
    return v != 0;
}

void require_cuda(const char* name, const at::Tensor& t, const at::Device* device = nullptr) {
    if (!t.is_cuda()) refuse(std::string(name) + " must be a CUDA tensor (this library has no CPU path)");
    if (device && t.device() != *device) refuse(std::string(name) + " must be on " + device->str() + ", got " + t.device().str());
}
void require_cuda(const char* name, const at::Tensor* t, const at::Device* device) { if (t) require_cuda(name, *t, device); }

template <typename T = void>
T* ptr(const at::Tensor& t) { return static_cast<T*>(t.data_ptr()); }
template <typename T = void>
T* ptr(const at::Tensor* t) { return t ? static_cast<T*>(t->data_ptr()) : nullptr; }

bool has_shape(const at::Tensor& t, std::initializer_list<int64_t> shape) { return t.sizes() == at::IntArrayRef(shape); }

at::Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, const at::Device& device) {
    return at::empty(shape, at::TensorOptions().dtype(dtype).device(device));
}

// Launches run without the GIL: a launch into a full queue waits for the device.
template <typename F>
void launch(PyObject* timer, const char* name, F&& f) {
    auto tell = [&](const char* method) {
        PyObject* r = PyObject_CallMethod(timer, method, "s", name);
        if (!r) throw python_error();
        Py_DECREF(r);
    };
    if (timer != Py_None) tell("start");
    int rc;
    PyThreadState* ts = PyEval_SaveThread();
    rc = f();
    PyEval_RestoreThread(ts);
    check(rc, name);
    if (timer != Py_None) tell("stop");
}

// ---- per-device status words written by kernels whose bounded waits ran out: [first code, count, -, -] --------
at::Tensor status_words[64];

// Kernels on any stream write these words, so they are zero before the first of them is launched: a fill queued on the
// first caller's stream would run behind that stream's work, over the report of another stream's kernel, or be captured
// and run with every replay.  For the same reason the memory is none of a capture's: it is allocated once per device,
// zeroed on a stream of its own, and lives as long as the process.
at::Tensor make_status_words(const at::Device& device) {
    const c10::cuda::CUDAGuard guard(device);
    const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);      // another stream may be capturing
    constexpr size_t bytes = 4 * sizeof(int32_t);
    void* words = nullptr;
    if (cudaMalloc(&words, bytes) != cudaSuccess) {                        // all memory is in the caching allocator's hands
        (void)cudaGetLastError();
        c10::cuda::CUDACachingAllocator::emptyCache();
        C10_CUDA_CHECK(cudaMalloc(&words, bytes));
    }
    cudaStream_t stream;
    C10_CUDA_CHECK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    C10_CUDA_CHECK(cudaMemsetAsync(words, 0, bytes, stream));
    C10_CUDA_CHECK(cudaStreamSynchronize(stream));
    C10_CUDA_CHECK(cudaStreamDestroy(stream));
    return at::from_blob(words, {4}, at::TensorOptions().dtype(at::kInt).device(device));
}

const at::Tensor& status(const at::Device& device) {
    const int i = device.index();
    require(i >= 0 && i < 64, "device index out of range");
    if (!status_words[i].defined()) status_words[i] = make_status_words(device);          // under the GIL
    return status_words[i];
}

// ---- pieces shared by the decode calls ----------------------------------------------------------------------------
struct Sched { at::Tensor meta, num_splits; int parts = 0; bool made = false; };

void check_sched(const Sched& s, int num_sm_parts, int64_t b, const at::Device& device) {
    require(s.meta.scalar_type() == at::kInt && s.num_splits.scalar_type() == at::kInt,
            "tile_scheduler_metadata and num_splits must have dtype int32");
    if (!has_shape(s.meta, {num_sm_parts, META_INTS}) || !has_shape(s.num_splits, {b + 1})) {
        auto text = [](const at::Tensor& t) {
            std::string r = "(";
            for (int64_t i = 0; i < t.dim(); ++i) r += std::to_string(t.size(i)) + (i + 1 < t.dim() ? ", " : t.dim() == 1 ? ",)" : ")");
            return r;
        };
        refuse("tile_scheduler_metadata must have shape (" + std::to_string(num_sm_parts) + ", " + std::to_string(META_INTS) +
               ") and num_splits (" + std::to_string(b + 1) + ",); got " + text(s.meta) + " and " + text(s.num_splits));
    }
    require(s.meta.is_contiguous() && s.num_splits.is_contiguous(), "tile_scheduler_metadata and num_splits must be contiguous");
    require_cuda("tile_scheduler_metadata", s.meta, &device);
    require_cuda("num_splits", s.num_splits, &device);
}

// The stored schedule, or a new one.  A stored one may also have `pair_parts` or `whole_parts` partitions: a schedule made when every
// shape ran on pairs of SMs, or when fewer requests were cut, stays usable (the kernels take any number of partitions).
// `new_with_pair_parts`: a new one has that many.
Sched schedule(PyObject* meta, PyObject* num_splits, mla_sched_meta_args_t a, int pair_parts, int whole_parts, bool new_with_pair_parts, const at::Device& device) {
    Sched s;
    if (meta != Py_None) {
        s.meta = tensor(meta, "tile_scheduler_metadata");
        s.num_splits = tensor(num_splits, "num_splits");
        for (int n : {pair_parts, whole_parts})
            if (has_shape(s.meta, {n, META_INTS})) a.num_sm_parts = n;
        check_sched(s, a.num_sm_parts, a.b, device);
        s.parts = a.num_sm_parts;
        return s;
    }
    if (new_with_pair_parts) a.num_sm_parts = pair_parts;
    s.parts = a.num_sm_parts;
    s.made = true;
    s.meta = empty({a.num_sm_parts, META_INTS}, at::kInt, device);
    s.num_splits = empty({a.b + 1}, at::kInt, device);
    a.block_size_n = BLOCK_SIZE_N;
    a.fixed_overhead_num_blocks = FIXED_OVERHEAD_NUM_BLOCKS;
    a.meta = ptr<mla_sched_meta_t>(s.meta);
    a.num_splits = ptr<int32_t>(s.num_splits);
    launch(Py_None, "mla_get_sched_meta", [&] { return api.get_sched_meta(&a); });
    return s;
}

// Split-KV scratch of one launch: fp32 partial outputs, then their log-sum-exps (256-byte aligned), in one allocation.
struct Scratch {
    at::Tensor bytes;
    float *o_accum, *lse_accum;
    Scratch(int64_t splits, int64_t rows, int64_t d_v, const at::Device& device) {
        const int64_t n = splits * rows, o_floats = (n * d_v + 63) / 64 * 64;
        bytes = empty({o_floats + n}, at::kFloat, device);
        o_accum = ptr<float>(bytes);
        lse_accum = o_accum + o_floats;
    }
};

PyObject* answer(std::initializer_list<at::Tensor> ts) {
    PyObject* r = PyTuple_New((Py_ssize_t)ts.size());
    if (!r) throw python_error();
    Py_ssize_t i = 0;
    for (const at::Tensor& t : ts) PyTuple_SET_ITEM(r, i++, THPVariable_Wrap(t));
    return r;
}

#define HOST_TRY HANDLE_TH_ERRORS try {
#define HOST_END } catch (const Refused& e) { PyErr_SetString(PyExc_RuntimeError, e.what()); return nullptr; } END_HANDLE_TH_ERRORS

// ---- dense decode ---------------------------------------------------------------------------------------------------
// dense_decode(q, kcache, d_v, seqlens_k, block_table, softmax_scale, causal, meta, num_splits, impl, timer)
//   -> (out, lse, meta, num_splits)
PyObject* dense_decode(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HOST_TRY
    require(nargs == 11, "dense_decode takes 11 arguments");
    const at::Tensor& q = tensor(args[0], "q");
    const at::Tensor& k = tensor(args[1], "kcache");
    const int64_t d_v = integer(args[2]);
    const at::Tensor& seqlens = tensor(args[3], "seqlens_k");
    const at::Tensor& table = tensor(args[4], "block_table");
    const double scale = real(args[5]);
    bool causal = truth(args[6]);
    const int impl = (int)integer(args[9]);
    PyObject* timer = args[10];

    require(q.scalar_type() == at::kBFloat16 || q.scalar_type() == at::kHalf, "q must have dtype bfloat16 or float16");
    require(k.scalar_type() == q.scalar_type(), "query and key must have the same dtype");
    require(seqlens.scalar_type() == at::kInt, "seqlens_k must have dtype int32");
    require(table.scalar_type() == at::kInt, "block_table must have dtype torch.int32");
    const at::Device device = q.device();
    require_cuda("q", q);
    require_cuda("kcache", k, &device);
    require_cuda("seqlens_k", seqlens, &device);
    require_cuda("block_table", table, &device);
    require(q.dim() == 4 && k.dim() == 4 && table.dim() == 2, "q and kcache must be 4-D, block_table 2-D");
    require(q.stride(3) == 1, "q must have contiguous last dimension");
    require(k.stride(3) == 1, "kcache must have contiguous last dimension");
    require(seqlens.is_contiguous(), "seqlens_k must be contiguous");
    require(table.stride(1) == 1, "block_table must have contiguous last dimension");
    const int64_t b = q.size(0), s_q = q.size(1), h_q = q.size(2), d = q.size(3), h_kv = k.size(2);
    require(d == 576 && k.size(3) == d, "Only head_size_k == 576 is supported");
    require(d_v == 512, "Only head_size_v == 512 is supported");
    require(k.size(1) == 64, "Currently page_block_size must be 64");
    require(b > 0, "batch size must be positive");
    require(h_kv > 0 && h_q % h_kv == 0, "Number of heads in key/value must divide number of heads in query");
    require(has_shape(seqlens, {b}) && table.size(0) == b,
            "seqlens_k must have shape (batch_size,) and block_table (batch_size, max_num_blocks_per_seq)");
    if (s_q == 1) causal = false;

    const c10::cuda::CUDAGuard guard(device);
    void* stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    mla_sched_meta_args_t sa = {};
    sa.b = (int32_t)b; sa.s_q = (int32_t)s_q; sa.topk = -1;
    sa.num_sm_parts = api.num_sm_parts(device.index(), MLA_MODE_DENSE_DECODE, (int)h_q, (int)h_kv, (int)s_q);
    if (sa.num_sm_parts <= 0) check(1, "mla_num_sm_parts");
    sa.seqlens_k = ptr<int32_t>(seqlens); sa.stream = stream;
    const int pair_parts = s_q * (h_q / h_kv) <= MLA_SINGLE_SM_ROWS ? api.num_sm_parts(device.index(), MLA_MODE_DENSE_DECODE, (int)h_kv * 128, (int)h_kv, 1) : sa.num_sm_parts;
    // A table of two blocks a request: as many partitions as there are SMs cut requests of two blocks in two when b of them cost
    // less than that many (two blocks and the overhead each), half as many leave them whole from half that cost on, and nothing is
    // left to combine.  us, 15 requests of 68 / 100 tokens: 33 to 64 rows 16.6 / 15.9 -> 15.7 / 14.9; up to 32 rows lose nothing.
    const int64_t cost = b * (2 + FIXED_OVERHEAD_NUM_BLOCKS);
    const bool whole = s_q * (h_q / h_kv) > 32 && table.size(1) == 2 && pair_parts <= cost && cost < sa.num_sm_parts;
    // 33 to 64 rows: a pair of SMs per partition (csrc/attn_pair.cu, half of its rows empty), which takes a tile about as fast as two single
    // SMs two of them, with half the partials and a shorter first tile, but more power.  us, 64 heads, single SMs / pairs: 1 x 9000 tokens
    // 23.7 / 19.6, 4 x 1000 15.5 / 14.1, 56 x 190 17.4 / 13.1, 4 x 30000 46.4 / 39.5; alone behind a cold L2 the same up to 37 x 4000 (65.5 / 65.5),
    // then 64 x 3000 73.7 / 80: up to 3000 blocks of the table.
    //   How long the requests are is known on the device only, and the table may be wider.  So pairs are taken for the batch sizes at which they
    // hardly lose whatever the lengths are: the two ways to cut a batch differ in how evenly they divide, which follows from the requests per
    // pair.  Pairs / single SMs over 89 batch sizes x lengths of 30 to 30000 tokens (equal, 1 : 3, lognormal), mean and worst with a stored schedule,
    // worst with the schedule's time: 1 to 34 requests (74 pairs) 0.87, 1.07, 1.02; 50 to 62 0.83, 1.08, 1.01; 160 to 192 0.93, 1.03, 0.96.
    // 35 to 49: 0.84, but 1.15 and 1.04 with equal requests of 500 to 1500 tokens, hence tables of up to seven blocks (0.73, 0.91, 0.85).  63 to
    // 74: 0.88, but 1.36 and 1.22 with requests of one or two blocks; 75 to 148: 1.00, 1.40, 1.20; 193 to 375: 0.98, 1.31, 1.16.
    //   (Tables of up to three blocks keep the rule above, and more requests than pairs theirs up to seven.  Several kv heads have not been
    // measured here.)
    const int64_t width = table.size(1), load = 100 * b / pair_parts;
    const bool even = load < 47 || (load < 67 && width <= 7) || (load >= 67 && load < 84) || (load >= 216 && load < 260);
    const bool on_pairs = h_kv == 1 && s_q * h_q > 32 && s_q * h_q <= MLA_SINGLE_SM_ROWS && even && width >= (b <= pair_parts ? 4 : 8) && b * width <= 3000;
    const Sched sched = schedule(args[7], args[8], sa, pair_parts, pair_parts, whole || on_pairs, device);
    const int parts = sched.parts;

    const at::Tensor out = empty({b, s_q, h_q, d_v}, q.scalar_type(), device);
    const at::Tensor lse = empty({b, h_q, s_q}, at::kFloat, device);
    const Scratch scratch(b + parts, s_q * h_q, d_v, device);
    mla_dense_decode_args_t a = {};
    a.b = (int32_t)b; a.s_q = (int32_t)s_q; a.h_q = (int32_t)h_q; a.h_kv = (int32_t)h_kv; a.d_qk = (int32_t)d; a.d_v = (int32_t)d_v;
    a.num_blocks = (int32_t)k.size(0); a.page_block_size = (int32_t)k.size(1);
    a.is_causal = causal; a.softmax_scale = (float)scale;
    a.q = ptr(q); a.q_stride_b = q.stride(0); a.q_stride_s = q.stride(1); a.q_stride_h = q.stride(2);
    a.k_cache = ptr(k); a.k_stride_block = k.stride(0); a.k_stride_row = k.stride(1); a.k_stride_head = k.stride(2);
    a.block_table = ptr<int32_t>(table); a.block_table_stride_b = table.stride(0); a.max_blocks_per_seq = (int32_t)table.size(1);
    a.seqlens_k = ptr<int32_t>(seqlens);
    a.out = ptr(out); a.o_stride_b = out.stride(0); a.o_stride_s = out.stride(1); a.o_stride_h = out.stride(2);
    a.lse = ptr<float>(lse); a.lse_stride_b = lse.stride(0); a.lse_stride_s = lse.stride(2); a.lse_stride_h = lse.stride(1);
    a.meta = ptr<mla_sched_meta_t>(sched.meta); a.num_splits = ptr<int32_t>(sched.num_splits); a.num_sm_parts = parts;
    a.lse_accum = scratch.lse_accum; a.o_accum = scratch.o_accum;
    a.status = ptr<int32_t>(status(device)); a.impl = impl;
    a.dtype = q.scalar_type() == at::kHalf ? MLA_DTYPE_FP16 : MLA_DTYPE_BF16; a.stream = stream;
    launch(timer, "mla_dense_decode_fwd", [&] { return api.dense_decode_fwd(&a); });
    mla_combine_args_t c = {};
    c.b = a.b; c.s_q = a.s_q; c.h_q = a.h_q; c.d_v = a.d_v;
    c.lse = a.lse; c.lse_stride_b = a.lse_stride_b; c.lse_stride_s = a.lse_stride_s; c.lse_stride_h = a.lse_stride_h;
    c.out = a.out; c.o_stride_b = a.o_stride_b; c.o_stride_s = a.o_stride_s; c.o_stride_h = a.o_stride_h;
    c.lse_accum = a.lse_accum; c.o_accum = a.o_accum; c.num_splits = a.num_splits; c.dtype = a.dtype; c.stream = stream;
    launch(timer, "mla_combine", [&] { return api.combine(&c); });
    return answer({out, lse, sched.meta, sched.num_splits});
    HOST_END
}

// ---- sparse FP8 decode ------------------------------------------------------------------------------------------------
void check_fp8_cache(const char* name, const at::Tensor& kv, int64_t d_qk) {
    const auto refuse_as = [&](const std::string& text) { refuse(name + text); };
    const at::ScalarType t = kv.scalar_type();
    if (t != at::kFloat8_e4m3fn && t != at::kChar && t != at::kByte) refuse_as(" must have dtype fp8_e4m3fn, int8 or uint8");
    if (kv.dim() != 4) refuse_as(" must be 4-D (num_blocks, page_block_size, 1, bytes_per_token)");
    if (kv.stride(3) != 1) refuse_as(" must have contiguous last dimension");
    require(kv.size(2) == 1, "Currently only MQA (i.e. h_kv == 1) is supported for sparse decoding");
    // bytes per token as the reference computes them (csrc/api/sparse_decode.h:289-299)
    const int64_t bytes = d_qk == 576 ? 512 + 64 * 2 + (512 / 128) * 4 : 448 + 64 * 2 + (448 / 64) * 1 + 1;
    if (kv.size(3) != bytes)
        refuse_as(": each token must take " + std::to_string(bytes) + " bytes (" +
                  (d_qk == 576 ? "512 fp8 + 4 fp32 scales + 64 bf16" : "448 fp8 + 64 bf16 + 7 e8m0 scales + 1 pad") +
                  "), got " + std::to_string(kv.size(3)));
    require(kv.stride(1) == bytes, "The whole block must be contiguous when is_fp8_cache is True for kv cache");
}

// sparse_decode(q, kv, indices, topk_length, attn_sink, meta, num_splits, extra_kv, extra_indices, extra_topk_length,
//               d_v, sm_scale, impl, timer) -> (out, lse, meta, num_splits)
PyObject* sparse_decode(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HOST_TRY
    require(nargs == 14, "sparse_decode takes 14 arguments");
    const at::Tensor& q = tensor(args[0], "q");
    const at::Tensor& kv = tensor(args[1], "kv");
    const at::Tensor& indices = tensor(args[2], "indices");
    const at::Tensor* topk_length = optional(args[3], "topk_length");
    const at::Tensor* sink = optional(args[4], "attn_sink");
    const at::Tensor* extra_kv = optional(args[7], "extra_kv");
    const at::Tensor* extra_indices = optional(args[8], "extra_indices");
    const at::Tensor* extra_topk_length = optional(args[9], "extra_topk_length");
    const int64_t d_v = integer(args[10]);
    const double scale = real(args[11]);
    const int impl = (int)integer(args[12]);
    PyObject* timer = args[13];

    require(q.dim() == 4 && indices.dim() == 3, "q must be 4-D and indices 3-D");
    const at::Device device = q.device();
    const int64_t b = q.size(0), s_q = q.size(1), h_q = q.size(2), d_qk = q.size(3), topk = indices.size(2);
    require(q.scalar_type() == at::kBFloat16, "q must have dtype bfloat16");
    require(d_qk == 576 || d_qk == 512, "Only head_size_k == 576 or 512 is supported for sparse decoding");
    require(d_v == 512, "Only head_size_v == 512 is supported for sparse decoding");
    require(topk > 0, "topk must be positive");
    check_fp8_cache("key", kv, d_qk);
    if (extra_kv) {
        require(extra_indices, "extra_indices_in_kvcache must be provided when extra_kcache is provided for sparse attention");
        check_fp8_cache("extra k cache", *extra_kv, d_qk);
    } else {
        require(!extra_indices, "extra_indices_in_kvcache must not be provided when extra_k_cache is not provided");
        require(!extra_topk_length, "extra_topk_length must not be provided when extra_k_cache is not provided");
    }
    const struct { const char* name; const at::Tensor* t; } all[] = {
        {"q", &q}, {"kv", &kv}, {"indices", &indices}, {"topk_length", topk_length}, {"attn_sink", sink},
        {"extra_kv", extra_kv}, {"extra_indices", extra_indices}, {"extra_topk_length", extra_topk_length}};
    for (const auto& x : all) require_cuda(x.name, x.t, &device);
    for (int i : {2, 6, 3, 7})
        if (all[i].t && all[i].t->scalar_type() != at::kInt) refuse(std::string(all[i].name) + " must have dtype int32");
    require(!sink || (sink->scalar_type() == at::kFloat && has_shape(*sink, {h_q}) && sink->is_contiguous()),
            "attn_sink must be a contiguous float32 tensor of shape (h_q,)");
    // (the list is the last dimension; one more in front of it, as prefill's lists have for the kv head, is accepted.  A missing
    // dimension is not: with several query tokens their rows would be read as one.)
    require(!extra_indices || extra_indices->dim() >= (s_q > 1 ? 3 : 2), "extra_indices must have shape (b, s_q, extra_topk)");
    require(q.stride(3) == 1 && indices.stride(2) == 1 && (!extra_indices || extra_indices->stride(-1) == 1),
            "q and indices must have contiguous last dimension");
    require(indices.size(0) == b && indices.size(1) == s_q, "indices must have shape (b, s_q, topk)");
    for (int i : {3, 7})
        if (all[i].t && !(has_shape(*all[i].t, {b}) && all[i].t->is_contiguous())) refuse(std::string(all[i].name) + " must be contiguous with shape (b,)");
    const int64_t extra_topk = extra_indices ? extra_indices->size(-1) : 0;
    require(!extra_indices || (extra_indices->size(0) == b && extra_indices->size(1) == s_q), "extra_indices must have shape (b, s_q, extra_topk)");

    const c10::cuda::CUDAGuard guard(device);
    void* stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    const bool uniform = !topk_length && !extra_topk_length;
    // (every request costs the same number of KV blocks: the partition count follows the batch size)
    const int64_t blocks = (topk + 63) / 64 + (extra_topk + 63) / 64;
    const auto general_parts = [&](int64_t heads) {
        const int n = api.num_sm_parts(device.index(), MLA_MODE_SPARSE_DECODE, (int)heads, 1, (int)s_q);
        if (n <= 0) check(1, "mla_num_sm_parts");
        return n;
    };
    // the count that stored schedules may have: one partition per request where that adds less than eight blocks to each
    const auto whole_parts = [&](int n) { return uniform && b <= n && (double)blocks - (double)blocks * b / n < 8.0 ? (int)b : n; };
    mla_sched_meta_args_t sa = {};
    sa.b = (int32_t)b; sa.s_q = (int32_t)s_q; sa.topk = (int32_t)topk; sa.extra_topk = (int32_t)extra_topk;
    sa.topk_length = ptr<int32_t>(topk_length); sa.extra_topk_length = ptr<int32_t>(extra_topk_length);
    const int general = general_parts(h_q);
    sa.num_sm_parts = uniform ? api.num_sm_parts_uniform(device.index(), MLA_MODE_SPARSE_DECODE, (int)h_q, 1, (int)s_q, (int)b, (int)blocks) : general;
    if (sa.num_sm_parts <= 0) check(1, "mla_num_sm_parts");
    sa.stream = stream;
    const Sched sched = schedule(args[5], args[6], sa, whole_parts(h_q <= MLA_SINGLE_SM_ROWS ? general_parts(128) : general), whole_parts(general), false, device);
    const int parts = sched.parts;

    const at::Tensor out = empty({b, s_q, h_q, d_v}, q.scalar_type(), device);
    const at::Tensor lse = empty({b, s_q, h_q}, at::kFloat, device);
    const Scratch scratch(b + parts, s_q * h_q, d_v, device);
    mla_sparse_decode_args_t a = {};
    a.b = (int32_t)b; a.s_q = (int32_t)s_q; a.h_q = (int32_t)h_q; a.d_qk = (int32_t)d_qk; a.d_v = (int32_t)d_v; a.sm_scale = (float)scale;
    a.q = ptr(q); a.q_stride_b = q.stride(0); a.q_stride_s = q.stride(1); a.q_stride_h = q.stride(2);
    a.kv = ptr(kv); a.kv_stride_block_bytes = kv.stride(0); a.num_blocks = (int32_t)kv.size(0); a.page_block_size = (int32_t)kv.size(1);
    a.indices = ptr<int32_t>(indices); a.indices_stride_b = indices.stride(0); a.indices_stride_s = indices.stride(1); a.topk = (int32_t)topk;
    a.topk_length = ptr<int32_t>(topk_length);
    if (extra_kv) {
        a.extra_kv = ptr(extra_kv); a.extra_kv_stride_block_bytes = extra_kv->stride(0);
        a.extra_num_blocks = (int32_t)extra_kv->size(0); a.extra_page_block_size = (int32_t)extra_kv->size(1);
        a.extra_indices = ptr<int32_t>(extra_indices);
        a.extra_indices_stride_b = extra_indices->stride(0); a.extra_indices_stride_s = extra_indices->stride(1);
        a.extra_topk = (int32_t)extra_topk; a.extra_topk_length = ptr<int32_t>(extra_topk_length);
    }
    a.attn_sink = ptr<float>(sink);
    a.out = ptr(out); a.o_stride_b = out.stride(0); a.o_stride_s = out.stride(1); a.o_stride_h = out.stride(2);
    a.lse = ptr<float>(lse); a.lse_stride_b = lse.stride(0); a.lse_stride_s = lse.stride(1); a.lse_stride_h = lse.stride(2);
    a.meta = ptr<mla_sched_meta_t>(sched.meta); a.num_splits = ptr<int32_t>(sched.num_splits); a.num_sm_parts = parts;
    a.lse_accum = scratch.lse_accum; a.o_accum = scratch.o_accum;
    a.status = ptr<int32_t>(status(device)); a.impl = impl; a.stream = stream;
    launch(timer, "mla_sparse_decode_fwd", [&] { return api.sparse_decode_fwd(&a); });
    // (equal costs and one partition per request: the scheduler cuts at every request boundary, no request is split and
    // the decode kernel has already written `out` and `lse`)
    if (!(uniform && parts == b)) {
        mla_combine_args_t c = {};
        c.b = a.b; c.s_q = a.s_q; c.h_q = a.h_q; c.d_v = a.d_v;
        c.lse = a.lse; c.lse_stride_b = a.lse_stride_b; c.lse_stride_s = a.lse_stride_s; c.lse_stride_h = a.lse_stride_h;
        c.out = a.out; c.o_stride_b = a.o_stride_b; c.o_stride_s = a.o_stride_s; c.o_stride_h = a.o_stride_h;
        c.lse_accum = a.lse_accum; c.o_accum = a.o_accum; c.num_splits = a.num_splits; c.attn_sink = a.attn_sink; c.stream = stream;
        launch(timer, "mla_combine", [&] { return api.combine(&c); });
    }
    return answer({out, lse.transpose(1, 2), sched.meta, sched.num_splits});
    HOST_END
}

// ---- sparse prefill -----------------------------------------------------------------------------------------------------
// sparse_prefill(q, kv, indices, sm_scale, d_v, attn_sink, topk_length, impl, timer) -> (out, max_logits, lse)
PyObject* sparse_prefill(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HOST_TRY
    require(nargs == 9, "sparse_prefill takes 9 arguments");
    const at::Tensor& q = tensor(args[0], "q");
    const at::Tensor& kv = tensor(args[1], "kv");
    const at::Tensor& indices = tensor(args[2], "indices");
    const double scale = real(args[3]);
    const int64_t d_v = integer(args[4]);
    const at::Tensor* sink = optional(args[5], "attn_sink");
    const at::Tensor* topk_length = optional(args[6], "topk_length");
    const int impl = (int)integer(args[7]);
    PyObject* timer = args[8];

    require(q.dim() == 3 && kv.dim() == 3 && indices.dim() == 3, "q, kv and indices must be 3-D");
    const at::Device device = q.device();
    require_cuda("q", q);
    require_cuda("kv", kv, &device);
    require_cuda("indices", indices, &device);
    require_cuda("attn_sink", sink, &device);
    require_cuda("topk_length", topk_length, &device);
    const int64_t s_q = q.size(0), h_q = q.size(1), d_qk = q.size(2), s_kv = kv.size(0), h_kv = kv.size(1), topk = indices.size(2);
    require(q.scalar_type() == at::kBFloat16 && kv.scalar_type() == at::kBFloat16, "q and kv must have dtype bfloat16");
    require(indices.scalar_type() == at::kInt, "indices must have dtype int32");
    require((d_qk == 576 || d_qk == 512) && kv.size(2) == d_qk, "Only d_qk == 576 or 512 is supported");
    require(d_v == 512, "Only d_v == 512 is supported");
    require(h_kv == 1, "Only h_kv == 1 is supported");
    require(indices.size(0) == s_q && indices.size(1) == h_kv, "indices must have shape (s_q, h_kv, topk)");
    require(q.stride(2) == 1 && kv.stride(2) == 1 && indices.stride(2) == 1, "q, kv and indices must have contiguous last dimension");
    require(!sink || (sink->scalar_type() == at::kFloat && has_shape(*sink, {h_q}) && sink->is_contiguous()),
            "attn_sink must be a contiguous float32 tensor of shape (h_q,)");
    require(!topk_length || (topk_length->scalar_type() == at::kInt && has_shape(*topk_length, {s_q}) && topk_length->is_contiguous()),
            "topk_length must be a contiguous int32 tensor of shape (s_q,)");

    const c10::cuda::CUDAGuard guard(device);
    const at::Tensor out = empty({s_q, h_q, d_v}, q.scalar_type(), device);
    const at::Tensor max_logits = empty({s_q, h_q}, at::kFloat, device);
    const at::Tensor lse = empty({s_q, h_q}, at::kFloat, device);
    mla_sparse_prefill_args_t a = {};
    a.s_q = (int32_t)s_q; a.s_kv = (int32_t)s_kv; a.h_q = (int32_t)h_q; a.h_kv = (int32_t)h_kv;
    a.d_qk = (int32_t)d_qk; a.d_v = (int32_t)d_v; a.topk = (int32_t)topk; a.sm_scale = (float)scale;
    a.q = ptr(q); a.q_stride_s = q.stride(0); a.q_stride_h = q.stride(1);
    a.kv = ptr(kv); a.kv_stride_s = kv.stride(0); a.kv_stride_h = kv.stride(1);
    a.indices = ptr<int32_t>(indices); a.indices_stride_s = indices.stride(0); a.indices_stride_h = indices.stride(1);
    a.attn_sink = ptr<float>(sink); a.topk_length = ptr<int32_t>(topk_length);
    a.out = ptr(out); a.max_logits = ptr<float>(max_logits); a.lse = ptr<float>(lse);
    a.status = ptr<int32_t>(status(device)); a.impl = impl;
    a.stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    launch(timer, "mla_sparse_prefill_fwd", [&] { return api.sparse_prefill_fwd(&a); });
    return answer({out, max_logits, lse});
    HOST_END
}

// ---- FP8 cache writer -----------------------------------------------------------------------------------------------------
// quantize(x [blocks, block_size, d], out, out_stride_block_bytes, pow2_scale, layout): `out` is the writer's own buffer
PyObject* quantize(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HOST_TRY
    require(nargs == 5, "quantize takes 5 arguments");
    const at::Tensor& x = tensor(args[0], "x");
    const at::Tensor& out = tensor(args[1], "out");
    const at::Device device = x.device();
    require_cuda("x", x);
    require_cuda("out", out, &device);
    require(x.dim() == 3, "x must be 3-D");
    const c10::cuda::CUDAGuard guard(device);
    mla_quantize_args_t a = {};
    a.x = ptr(x); a.x_stride_block = x.stride(0); a.x_stride_row = x.stride(1);
    a.num_blocks = (int32_t)x.size(0); a.block_size = (int32_t)x.size(1);
    a.out = ptr(out); a.out_stride_block_bytes = integer(args[2]);
    a.pow2_scale = truth(args[3]); a.layout = (int32_t)integer(args[4]);
    a.stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    launch(Py_None, "mla_quantize_fp8_kvcache", [&] { return api.quantize(&a); });
    Py_RETURN_NONE;
    HOST_END
}

// status(device_index) -> the device's status words;  known_status() -> those of every device that has some
PyObject* status_of(PyObject*, PyObject* arg) {
    HOST_TRY
    return THPVariable_Wrap(status(at::Device(at::kCUDA, (c10::DeviceIndex)integer(arg))));
    HOST_END
}
PyObject* known_status(PyObject*, PyObject*) {
    HOST_TRY
    PyObject* r = PyList_New(0);
    if (!r) throw python_error();
    for (const at::Tensor& t : status_words) {
        if (!t.defined()) continue;
        PyObject* o = THPVariable_Wrap(t);
        const int rc = PyList_Append(r, o);
        Py_DECREF(o);
        if (rc) { Py_DECREF(r); throw python_error(); }
    }
    return r;
    HOST_END
}

// bind(addresses of the C functions in the order of Api's members): refuses a library whose structures are not the ones this
// file was compiled with
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HOST_TRY
    require(nargs == (Py_ssize_t)(sizeof(Api) / sizeof(void*)), "bind: one address for every function is needed");
    Api given;
    for (Py_ssize_t i = 0; i < nargs; ++i) reinterpret_cast<void**>(&given)[i] = PyLong_AsVoidPtr(args[i]);
    if (PyErr_Occurred()) throw python_error();
    const int version = given.abi_version();
    if (version != MLA_ABI_VERSION)
        refuse("the host extension was compiled for ABI version " + std::to_string(MLA_ABI_VERSION) + " of the library, which has " +
               std::to_string(version) + ": rebuild both with `python -m flashmla_b200.build --force`");
    api = given;
    Py_RETURN_NONE;
    HOST_END
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f))
PyMethodDef methods[] = {
    {"bind", FAST(bind), METH_FASTCALL, nullptr},
    {"dense_decode", FAST(dense_decode), METH_FASTCALL, nullptr},
    {"sparse_decode", FAST(sparse_decode), METH_FASTCALL, nullptr},
    {"sparse_prefill", FAST(sparse_prefill), METH_FASTCALL, nullptr},
    {"quantize", FAST(quantize), METH_FASTCALL, nullptr},
    {"status", status_of, METH_O, nullptr},
    {"known_status", known_status, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

#define TEXT_(x) #x
#define TEXT(x) TEXT_(x)
PyMODINIT_FUNC PyInit__host() {
    PyObject* m = PyModule_Create(&module_def);
    // the tile scheduler's arguments, for callers that make a schedule through the C ABI
    if (m && (PyModule_AddIntConstant(m, "BLOCK_SIZE_N", BLOCK_SIZE_N) || PyModule_AddIntConstant(m, "META_INTS", META_INTS) ||
              PyModule_AddIntConstant(m, "FIXED_OVERHEAD_NUM_BLOCKS", FIXED_OVERHEAD_NUM_BLOCKS)))
        Py_CLEAR(m);
    // what the file was compiled against; _capi.py compares it with what is running
    if (m && PyModule_AddStringConstant(m, "built_for", "torch " FLASHMLA_TORCH_VERSION ", Python " TEXT(PY_MAJOR_VERSION) "." TEXT(PY_MINOR_VERSION)))
        Py_CLEAR(m);
    return m;
}
