// What the two tcgen05 attention kernels (attn_pair.cu: up to 128 query rows on a pair of SMs; attn_rows64.cu: up to 64 on
// one) have in common: their parameters, the walk over a partition's work, bounded waits, conversions, the host's
// tensor map over Q.
#pragma once
#include "common.cuh"
#include "sm100_ptx.cuh"
#include "wait_limit.h"
#include <cuda_fp16.h>
#include <string.h>
#include <algorithm>
#include <stdlib.h>
#include <mutex>

namespace mla {
namespace sm100 {

using namespace ptx;

constexpr int PAGE = 64;              // tokens per page
constexpr int D_V = 512;             // value columns = the first 512 of the 576 key columns
constexpr float RESCALE_THRESHOLD = 6.0f;         // log2 units
constexpr long long DRAIN_LIMIT = 4000000LL;              // wind-down after an expired wait: per tracked operation

enum { MODE_DENSE = 0, MODE_PREFILL = 1, MODE_SPARSE_DECODE = 2 };

struct Params {
    int b, s_q, h_q, h_kv, g, rows, causal, num_blocks;
    int head_chunks;                       // dense mode: 64-column chunks between two kv heads of a cache row
    int max_blocks;                        // dense mode: width of the block table
    float scale_log2;
    uint32_t wait_limit;                   // units of 2^WAIT_UNIT_LOG2 SM cycles after which a barrier wait gives up
    const __nv_bfloat16* q; int64_t q_sb, q_ss, q_sh;
    int q_tma, q_box_bytes;                // a request's Q comes as TMA boxes of q_box_bytes: pairs of SMs: six through the ring on their way to tensor memory, the others into a buffer of their own, which takes all of them on one SM
    __nv_bfloat16* out; int64_t o_sb, o_ss, o_sh;
    float* lse; int64_t l_sb, l_ss, l_sh;
    const int* block_table; int64_t bt_sb; const int* seqlens;
    const mla_sched_meta_t* meta; const int* num_splits;
    float* lse_accum; float* o_accum;
    int* status;
    int row_blocks;
    int q_unit;                            // pairs of SMs: rows of Q a box brings (64 rows per CTA)
    // token-sparse prefill: one "request" is one query token, its keys are gathered by index
    const int* indices; int64_t idx_ss; int topk; const int* topk_len; int s_kv;
    const __nv_bfloat16* kv; int64_t kv_ss;
    // sparse FP8 decode: two index scopes (main cache, optional extra cache) of 656-byte token records
    const uint8_t* kvb[2]; int64_t kvb_sblock[2]; int pbs[2]; uint32_t pbs_mul[2]; int pbs_shift[2];      // (a token's page: times mul, shifted)
    uint32_t tokens[2];                    // of the cache: indices below are valid
    const int* sidx[2]; int64_t sidx_sb[2], sidx_ss[2]; int stopk[2]; const int* stopk_len[2];
    const float* attn_sink; float* max_logits;
};

// The page of token `id` of scope `scope` (id < p.tokens[scope]) and its place there.
__device__ __forceinline__ uint32_t page_of_token(const Params& p, int scope, uint32_t id, uint32_t& off) {
    const uint32_t page = (uint32_t)(((uint64_t)id * p.pbs_mul[scope]) >> p.pbs_shift[scope]);
    off = id - page * (uint32_t)p.pbs[scope];
    return page;
}

// One unit of work of a partition: a request and the range of its 64-token blocks walked here.
struct Work {
    int req, blk_begin, blk_end, ntiles, seqlen, is_split, slot;
    int len0, len1, nblk0;      // sparse decode: valid positions of the two index scopes, blocks of the first scope
};

template <int MODE>
struct Walker;

// dense decode: the requests and block range of one SM partition, from the tile-scheduler metadata
template <>
struct Walker<MODE_DENSE> {
    mla_sched_meta_t m;
    const Params& p;
    int req;
    __device__ Walker(const Params& p_, int part) : p(p_) { m = p_.meta[part]; req = m.begin_req_idx; }
    __device__ bool valid() const { return m.begin_req_idx < p.b && req <= m.end_req_idx; }
    __device__ Work get() const {
        Work w;
        w.req = req;
        w.seqlen = p.seqlens[req];
        w.blk_begin = req == m.begin_req_idx ? m.begin_block_idx : 0;
        w.blk_end = req == m.end_req_idx ? m.end_block_idx : (w.seqlen + PAGE - 1) / PAGE;
        if (w.blk_end < w.blk_begin) w.blk_end = w.blk_begin;
        w.ntiles = (w.blk_end - w.blk_begin + 1) / 2;
        w.is_split = req == m.begin_req_idx ? m.is_first_req_splitted : (req == m.end_req_idx ? m.is_last_req_splitted : 0);
        w.slot = p.num_splits[req] + (req == m.begin_req_idx ? m.begin_split_idx : 0);
        return w;
    }
    __device__ void next() { ++req; }
};

// sparse FP8 decode: like dense decode, but a request's "sequence" is its top-k list: blocks [0, nblk0) index the
// main cache, the following blocks the optional extra cache (block counts as in the tile scheduler)
template <>
struct Walker<MODE_SPARSE_DECODE> {
    mla_sched_meta_t m;
    const Params& p;
    int req;
    __device__ Walker(const Params& p_, int part) : p(p_) { m = p_.meta[part]; req = m.begin_req_idx; }
    __device__ bool valid() const { return m.begin_req_idx < p.b && req <= m.end_req_idx; }
    __device__ Work get() const {
        Work w;
        w.req = req;
        const int l0 = p.stopk_len[0] ? p.stopk_len[0][req] : p.stopk[0];
        const int l1 = p.stopk[1] ? (p.stopk_len[1] ? p.stopk_len[1][req] : p.stopk[1]) : 0;
        w.len0 = min(max(l0, 0), p.stopk[0]);
        w.len1 = min(max(l1, 0), p.stopk[1]);
        w.nblk0 = max((l0 + PAGE - 1) / PAGE, 1);
        const int total = w.nblk0 + (l1 + PAGE - 1) / PAGE;
        w.seqlen = total * PAGE;
        w.blk_begin = req == m.begin_req_idx ? m.begin_block_idx : 0;
        w.blk_end = req == m.end_req_idx ? m.end_block_idx : total;
        if (w.blk_end < w.blk_begin) w.blk_end = w.blk_begin;
        w.ntiles = (w.blk_end - w.blk_begin + 1) / 2;
        w.is_split = req == m.begin_req_idx ? m.is_first_req_splitted : (req == m.end_req_idx ? m.is_last_req_splitted : 0);
        w.slot = p.num_splits[req] + (req == m.begin_req_idx ? m.begin_split_idx : 0);
        return w;
    }
    __device__ void next() { ++req; }
};

// sparse prefill: CTA pair `part` takes query tokens part, part + gridDim.z, ... ; "seqlen" is the number of
// top-k positions that may be valid
template <>
struct Walker<MODE_PREFILL> {
    const Params& p;
    int req;
    __device__ Walker(const Params& p_, int part) : p(p_), req(part) {}
    __device__ bool valid() const { return req < p.b; }
    __device__ Work get() const {
        Work w;
        w.req = req;
        w.seqlen = p.topk_len ? min(max(p.topk_len[req], 0), p.topk) : p.topk;
        w.blk_begin = 0;
        w.blk_end = (w.seqlen + PAGE - 1) / PAGE;
        w.ntiles = (w.blk_end + 1) / 2;
        w.is_split = 0;
        w.slot = 0;
        return w;
    }
    __device__ void next() { req += gridDim.z; }
};

template <int N> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

// ---- bounded waits -------------------------------------------------------------------------------------------
// A wait is a loop of probes (the hardware holds a thread for a while before it answers one) and clock reads, compared in 32
// bits and units of 2^8 cycles.  All roles of a CTA share one instruction cache, and there are some thirty wait sites in
// their loops.  Measured with the kernel of score and value CTAs that was here before attn_pair.cu (back to back, otherwise equal):
// with 64-bit comparisons and the report at every site, 4096-token prefill took 2870 us in the place of 2800, FP8 decode of 64
// requests 95.7 (94.4), of 512-wide records 84.7 (81.6), dense decode the same.  Counted in cycles, prefill (2774 against 2790) and
// dense decode (192.2 against 193.1 for the serving batch) were 0.5 % faster, but limits above 2^32 cycles are lost; waiting for
// those in several 32-bit spans cost every site a few instructions more: 2920, and FP8 decode 93.6 -> 105.2.
// A thread whose wait ran out only keeps the site's code; it reports when it has left its role.
//
// wait() / wait_warp() return false when the wait ran out now or earlier: the caller leaves its role.  Arrivals of the other CTA of a
// pair are waited for at CTA scope too: what they announce is not read by the waiting thread (mbar_arrive_remote_cta, sm100_ptx.cuh).
struct Waiter {
    uint32_t limit;                      // units of 2^WAIT_UNIT_LOG2 SM cycles
    int code = 0;
    __device__ explicit Waiter(uint32_t limit_) : limit(limit_) {}
    __device__ __forceinline__ bool expired() const { return code != 0; }
    __device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity, int site) {
        if (expired()) return false;
        if (mbar_try_wait(smem_addr(bar), parity)) return true;
        const uint32_t t0 = clock_units<WAIT_UNIT_LOG2>();
#pragma unroll 1
        while (!mbar_try_wait(smem_addr(bar), parity))
            if (clock_units<WAIT_UNIT_LOG2>() - t0 > limit) { code = site; break; }
        return !expired();
    }
    // whole warps (all 32 lanes execute this): the same answer for every lane
    __device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, int site) {
        wait(bar, parity, site);
        return !__any_sync(0xffffffffu, expired());
    }
};
// First code and a count in the global status words, the `aborted` flag of this CTA and of its peer.
static __device__ __noinline__ void report_expired_wait(int* status, uint32_t* flag, uint32_t peer_flag, int code) {
    *reinterpret_cast<volatile uint32_t*>(flag) = 1;
    if (peer_flag) st_cluster_u32(peer_flag, 1u);
    if (status) { atomicCAS(status, 0, code); atomicAdd(status + 1, 1); }
}

// single-thread roles: leave at once
#define WAIT_OR_LEAVE(W, bar, par, code) do { if (!(W).wait(bar, par, code)) goto wind_down; } while (0)
// whole warps (all 32 lanes execute this): leave together, tcgen05.ld/st and shuffles are warp-collective
#define WAIT_WARP_OR_LEAVE(W, bar, par, code) do { if (!(W).wait_warp(bar, par, code)) goto wind_down; } while (0)

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// two fp32 -> one 32-bit word of the 16-bit input type (bf16 or fp16), `lo` in the low half
template <bool FP16>
__device__ __forceinline__ uint32_t pack16(float lo, float hi) {
    uint32_t r;
    if (FP16) asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    else asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) { return pack16<false>(lo, hi); }

// e8m0 scale byte `k` of a word -> fp32: 2^(e - 127), 255 is NaN (as the format defines it).  Through bf16, which has all of these values, the
// subnormal 2^-127 of byte 0 included.
__device__ __forceinline__ float e8m0_of(uint32_t word, int k) {
    uint32_t r;
    asm("{\n\t.reg .b16 x, y;\n\tmov.b32 {x, y}, %1;\n\tcvt.rn.bf16x2.ue8m0x2 %0, x;\n\t}" : "=r"(r) : "r"(__byte_perm(word, 0, 0x4440 | k)));
    return __uint_as_float(r << 16);
}

// two fp32 products in one instruction
__device__ __forceinline__ float2 mul_f32x2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
// 16 e4m3 values (one uint4) times an fp32 scale -> 16 bf16 (two uint4), one rounding: bf16(fp32(e4m3) * scale).
// (A conversion-free variant that places the e4m3 magnitude bits into an fp32 word and multiplies by scale * 2^120 is
// bit-identical but needs more instructions per value and measured slower.)
__device__ __forceinline__ void dequant16(const uint4& raw, float scale, uint4& lo, uint4& hi) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
    uint32_t o[8];
    const float2 scale2 = make_float2(scale, scale);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        __half2_raw h0 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[i] & 0xffffu), __NV_E4M3);
        __half2_raw h1 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[i] >> 16), __NV_E4M3);
        const float2 f0 = mul_f32x2(__half22float2(*reinterpret_cast<__half2*>(&h0)), scale2);
        const float2 f1 = mul_f32x2(__half22float2(*reinterpret_cast<__half2*>(&h1)), scale2);
        o[2 * i] = pack_bf16(f0.x, f0.y);
        o[2 * i + 1] = pack_bf16(f1.x, f1.y);
    }
    lo = make_uint4(o[0], o[1], o[2], o[3]);
    hi = make_uint4(o[4], o[5], o[6], o[7]);
}
__device__ __forceinline__ const uint8_t* shfl_ptr(const uint8_t* ptr, int src_lane) {
    const unsigned long long v = reinterpret_cast<unsigned long long>(ptr);
    const uint32_t lo = __shfl_sync(0xffffffffu, (uint32_t)v, src_lane);
    const uint32_t hi = __shfl_sync(0xffffffffu, (uint32_t)(v >> 32), src_lane);
    return reinterpret_cast<const uint8_t*>(((unsigned long long)hi << 32) | lo);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)f;
    }
    return fn;
}

// Barrier-wait limit of the attention kernels (MLA_WAIT_LIMIT_CYCLES is read once).
static uint32_t wait_limit() {
    static const uint32_t v = wait_units_from(getenv("MLA_WAIT_LIMIT_CYCLES"));
    return v;
}

// cudaFuncSetAttribute(max dynamic shared memory) once per kernel instance and device
template <typename K>
static int configure_once(K kernel, bool (&done)[64], size_t smem_bytes) {
    static std::mutex mu;
    int dev = 0;
    MLA_CHECK_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 0 || dev >= 64 || !done[dev]) {
        MLA_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes));
        if (dev >= 0 && dev < 64) done[dev] = true;
    }
    return MLA_OK;
}

// Tensor map over Q as (576 columns, heads, query tokens, requests) with boxes of 64 columns x box_h heads x box_t
// tokens.  Returns false (the kernels then load every Q with their own threads) when Q's base or strides do not meet
// TMA's 16-byte rules or the driver rejects the map.
static bool encode_q_map(CUtensorMap* qmap, const void* q, int b, int s_q, int h_q, int64_t sb, int64_t ss, int64_t sh,
                         int box_h, int box_t, int* box_bytes, bool fp16 = false, int d_qk = 576) {
    static const bool enabled = [] { const char* e = getenv("MLA_Q_TMA"); return !(e && e[0] == '0'); }();
    EncodeTiledFn encode = get_encode_fn();
    if (!enabled || !encode || !q) return false;
    if (h_q <= 1) sh = 576;                         // a dimension of extent 1 never strides: give it a legal value
    if (s_q <= 1) ss = sh * h_q;
    if (b <= 1) sb = ss * s_q;
    if ((reinterpret_cast<uintptr_t>(q) & 15) || sb <= 0 || ss <= 0 || sh <= 0 || (sb % 8) || (ss % 8) || (sh % 8)) return false;
    if (sb * 2 >= (1ll << 40) || ss * 2 >= (1ll << 40) || sh * 2 >= (1ll << 40)) return false;
    if (box_h < 1 || box_h > 256 || box_t < 1 || box_t > 256 || box_h * box_t > 128) return false;
    // (512-wide rows: the ninth box of a request lies wholly outside the tensor and arrives as zeros)
    cuuint64_t dims[4] = {(cuuint64_t)d_qk, (cuuint64_t)h_q, (cuuint64_t)s_q, (cuuint64_t)b};
    cuuint64_t strides[3] = {(cuuint64_t)sh * 2, (cuuint64_t)ss * 2, (cuuint64_t)sb * 2};
    cuuint32_t box[4] = {64, (cuuint32_t)box_h, (cuuint32_t)box_t, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = encode(qmap, fp16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(q),
                              dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return false;
    *box_bytes = 128 * box_h * box_t;
    return true;
}

// Tensor map over the prefill's keys as rows (d_qk columns, s_kv rows) for gathers of four rows by index, 64 columns at a time.  Returns false
// where the driver makes none; driver 580 does for all keys that get here, padded rows and rows that overlap among them.
static bool encode_kv_rows_map(CUtensorMap* kmap, const mla_sparse_prefill_args_t& a) {
    EncodeTiledFn encode = get_encode_fn();
    if (!encode) return false;
    cuuint64_t dims[2] = {(cuuint64_t)a.d_qk, (cuuint64_t)a.s_kv}, strides[1] = {(cuuint64_t)(a.s_kv > 1 ? a.kv_stride_s : 576) * 2};
    cuuint32_t box[2] = {64, 1}, estr[2] = {1, 1};
    return encode(kmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(a.kv), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ---- the kernels' parameters from a call's arguments -----------------------------------------------------------
static Params dense_params(const mla_dense_decode_args_t& a, int head_chunks) {
    Params p = {};
    p.b = a.b; p.s_q = a.s_q; p.h_q = a.h_q; p.h_kv = a.h_kv; p.g = a.h_q / a.h_kv;
    p.rows = a.s_q * p.g;
    p.causal = (a.is_causal && a.s_q > 1) ? 1 : 0;
    p.scale_log2 = a.softmax_scale * kLog2e;
    p.wait_limit = wait_limit();
    p.q = (const __nv_bfloat16*)a.q; p.q_sb = a.q_stride_b; p.q_ss = a.q_stride_s; p.q_sh = a.q_stride_h;
    p.out = (__nv_bfloat16*)a.out; p.o_sb = a.o_stride_b; p.o_ss = a.o_stride_s; p.o_sh = a.o_stride_h;
    p.lse = a.lse; p.l_sb = a.lse_stride_b; p.l_ss = a.lse_stride_s; p.l_sh = a.lse_stride_h;
    p.block_table = a.block_table; p.bt_sb = a.block_table_stride_b; p.seqlens = a.seqlens_k;
    p.max_blocks = a.max_blocks_per_seq;
    p.meta = a.meta; p.num_splits = a.num_splits; p.lse_accum = a.lse_accum; p.o_accum = a.o_accum;
    p.status = a.status;
    p.num_blocks = a.num_blocks;
    p.head_chunks = head_chunks;
    return p;
}

static Params prefill_params(const mla_sparse_prefill_args_t& a) {
    Params p = {};
    p.b = a.s_q; p.s_q = 1; p.h_q = a.h_q; p.h_kv = 1; p.g = a.h_q; p.rows = a.h_q;
    p.causal = 0;
    p.scale_log2 = a.sm_scale * kLog2e;
    p.wait_limit = wait_limit();
    p.q = (const __nv_bfloat16*)a.q; p.q_ss = a.q_stride_s; p.q_sh = a.q_stride_h;
    p.out = (__nv_bfloat16*)a.out; p.lse = a.lse; p.max_logits = a.max_logits;
    p.attn_sink = a.attn_sink;
    p.indices = a.indices; p.idx_ss = a.indices_stride_s; p.topk = a.topk; p.topk_len = a.topk_length; p.s_kv = a.s_kv;
    p.kv = (const __nv_bfloat16*)a.kv; p.kv_ss = a.kv_stride_s;
    p.status = a.status;
    return p;
}

// n / d = n * mul >> shift for 0 <= n < 2^31, d >= 1: with 2^l >= d, mul = floor(2^(31 + l) / d) + 1 is off by at most d / 2^(31 + l), so the
// product by less than 1 / d of the quotient (T. Granlund, P. L. Montgomery, "Division by invariant integers using multiplication",
// PLDI 1994).
static void reciprocal(int d, uint32_t& mul, int& shift) {
    int l = 0;
    while (((int64_t)1 << l) < d) ++l;
    mul = (uint32_t)(((uint64_t)1 << (31 + l)) / (uint64_t)d + 1);
    shift = 31 + l;
}

static Params sparse_decode_params(const mla_sparse_decode_args_t& a) {
    Params p = {};
    p.b = a.b; p.s_q = a.s_q; p.h_q = a.h_q; p.h_kv = 1; p.g = a.h_q; p.rows = a.h_q;
    p.causal = 0;
    p.scale_log2 = a.sm_scale * kLog2e;
    p.wait_limit = wait_limit();
    p.q = (const __nv_bfloat16*)a.q; p.q_sb = a.q_stride_b; p.q_ss = a.q_stride_s; p.q_sh = a.q_stride_h;
    p.out = (__nv_bfloat16*)a.out; p.o_sb = a.o_stride_b; p.o_ss = a.o_stride_s; p.o_sh = a.o_stride_h;
    p.lse = a.lse; p.l_sb = a.lse_stride_b; p.l_ss = a.lse_stride_s; p.l_sh = a.lse_stride_h;
    p.attn_sink = a.attn_sink;
    p.meta = a.meta; p.num_splits = a.num_splits; p.lse_accum = a.lse_accum; p.o_accum = a.o_accum;
    p.status = a.status;
    p.kvb[0] = (const uint8_t*)a.kv; p.kvb_sblock[0] = a.kv_stride_block_bytes; p.pbs[0] = a.page_block_size;
    p.sidx[0] = a.indices; p.sidx_sb[0] = a.indices_stride_b; p.sidx_ss[0] = a.indices_stride_s; p.stopk[0] = a.topk;
    p.stopk_len[0] = a.topk_length;
    p.kvb[1] = (const uint8_t*)a.extra_kv; p.kvb_sblock[1] = a.extra_kv_stride_block_bytes;
    p.pbs[1] = a.extra_page_block_size > 0 ? a.extra_page_block_size : 1;
    p.sidx[1] = a.extra_indices; p.sidx_sb[1] = a.extra_indices_stride_b; p.sidx_ss[1] = a.extra_indices_stride_s;
    p.stopk[1] = a.extra_kv ? a.extra_topk : 0; p.stopk_len[1] = a.extra_topk_length;
    const int nblocks[2] = {a.num_blocks, a.extra_num_blocks};
    for (int i = 0; i < 2; ++i) {
        p.tokens[i] = (uint32_t)std::min((int64_t)std::max(nblocks[i], 0) * p.pbs[i], (int64_t)1 << 31);
        reciprocal(p.pbs[i], p.pbs_mul[i], p.pbs_shift[i]);
    }
    return p;
}

}  // namespace sm100
}  // namespace mla
