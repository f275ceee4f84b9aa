// Split-KV combine: for every request whose KV range was split over several SM partitions, merge
// the per-split fp32 partial outputs O_s (each already normalised by its own row sum) and base-2
// log-sum-exps lse2_s into the final bf16 output and natural-log LSE:
//     g = log2 sum_s 2^{lse2_s},  out = sum_s 2^{lse2_s - g'} O_s,  lse = g * ln 2
// where g' additionally absorbs the attention sink: g' = g + log2(1 + 2^{sink*log2e - g}).
// Semantics follow csrc/smxx/decode/combine/combine.cu:72-160 of the reference.
//
// Per (request, query token, head) it reads n_splits * 2 KiB and writes 1 KiB: HBM-bound where there are many rows, bound
// by its chain of memory latencies (split counts -> log-sum-exps -> partials -> output) where there are few.  A row is served
// by WPR warps of a CTA, each taking every WPR-th split with 16 output columns per lane (4 x float4 per split: 512 coalesced
// bytes per warp instruction); with WPR > 1 their sums meet in shared memory.  Where there are hardly any rows, PARTS CTAs share
// a row's columns.  The first partials are requested together
// with the log-sum-exps, so that a row of up to WPR * UNROLL splits costs two round trips instead of three.  There is no
// limit on the number of splits.
#include "common.cuh"
#include <cuda_fp16.h>
#include <algorithm>

namespace mla {

constexpr int COMBINE_WARPS = 8;

template <int WPR, int PARTS>
__global__ void __launch_bounds__(COMBINE_WARPS * 32, WPR == 8 ? 2 : WPR == 1 ? 4 : 3)
combine_kernel(const mla_combine_args_t a) {
    // launched with programmatic stream serialization: the decode kernel before it may still be running.  (Letting the next
    // kernel set itself up from here on costs more than it hides: its CTAs take whole SMs while this grid still needs them;
    // dense decode with 2 query tokens 346 -> 351 us a step.  Every CTA does so when it has its sums: 16 heads, 1, 4, 8, 16
    // requests of 100 tokens 11.05, 11.12, 11.19, 11.39 -> 10.77, 10.79, 10.86, 10.95 us a step, of 8000 15.5, 18.6, 24.6, 38.6 -> 15.3, 18.3, 24.2, 38.0;
    // 16 of 900 tokens, 64 heads 16.7 -> 17.0; the full batches nothing.  With eight warps a row when they are in shared memory: one request of 100003
    // tokens, with its schedule, takes 44.8 as without, 45.1 otherwise.)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int ROWS = COMBINE_WARPS / WPR;            // heads per CTA
    constexpr int NV = 4 / PARTS;                        // float4s of a split per lane
    constexpr int UNROLL = (WPR == 8 ? 4 : 2) * PARTS;   // splits in flight per warp
    __shared__ float part[WPR > 1 ? COMBINE_WARPS * 512 / PARTS : 1];
    const int col0 = PARTS > 1 ? (int)blockIdx.z * (512 / PARTS) : 0;      // this CTA's columns
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = warp % WPR;
    const int bs_idx = blockIdx.x;                       // request * s_q + query token
    const int req = bs_idx / a.s_q, t = bs_idx - req * a.s_q;
    const int head = min((int)blockIdx.y * ROWS + warp / WPR, a.h_q - 1);
    const bool head_ok = blockIdx.y * ROWS + warp / WPR < a.h_q;
    const int s0 = a.num_splits[req], s1 = a.num_splits[req + 1];
    const int n = s1 - s0;
    if (n <= 1) return;                                  // the decode kernel wrote the final result (whole CTA)

    const int64_t row_stride = (int64_t)a.s_q * a.h_q;   // rows per split slot
    const float* lse_acc = a.lse_accum + (int64_t)s0 * row_stride + (int64_t)t * a.h_q + head;
    const float4* o_acc = reinterpret_cast<const float4*>(a.o_accum + ((int64_t)s0 * row_stride + (int64_t)t * a.h_q + head) * 512 + col0) + lane;
    const int64_t o_step = row_stride * 128;             // float4s from one split to the next

    // the first partials of this warp; their weights are not known yet
    float4 v[UNROLL][NV];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
        const int s = sub + u * WPR;
        if (s < n) {
#pragma unroll
            for (int i = 0; i < NV; ++i) v[u][i] = __ldcs(o_acc + s * o_step + i * 32);
        }
    }

    // pass 1: global log-sum-exp over the splits
    const float l_first = lane < n ? lse_acc[lane * row_stride] : -INFINITY;
    float mx = l_first;
#pragma unroll 1
    for (int s = lane + 32; s < n; s += 32) mx = fmaxf(mx, lse_acc[(int64_t)s * row_stride]);
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (mx == -INFINITY) mx = 0.f;
    float sum = exp2f(l_first - mx);
#pragma unroll 1
    for (int s = lane + 32; s < n; s += 32) sum += exp2f(lse_acc[(int64_t)s * row_stride] - mx);
#pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    float g = (sum == 0.f || sum != sum) ? INFINITY : log2f(sum) + mx;
    if (lane == 0 && sub == 0 && head_ok && col0 == 0)
        a.lse[req * a.lse_stride_b + t * a.lse_stride_s + head * a.lse_stride_h] = g * kLn2;
    if (a.attn_sink) {
        const float sink = a.attn_sink[head];
        if (g != INFINITY) g += log2f(1.f + exp2f(sink * kLog2e - g));
        else g = sink == -INFINITY ? INFINITY : sink * kLog2e;
    }

    // pass 2: weighted sum of this warp's splits.  Lane l holds columns 4 l .. 4 l + 3 of every 128.
    float4 acc[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    float w_block = exp2f(l_first - g);                  // weights of splits block .. block + 31, one per lane
    int block = 0;
#pragma unroll 1
    for (int base = sub; base < n; base += UNROLL * WPR) {
        if (base >= UNROLL * WPR) {
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                const int s = base + u * WPR;
                if (s < n) {
#pragma unroll
                    for (int i = 0; i < NV; ++i) v[u][i] = __ldcs(o_acc + s * o_step + i * 32);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int s = base + u * WPR;
            if (s < n) {
                if ((s & ~31) != block) {                // (splits of a warp ascend)
                    block = s & ~31;
                    w_block = block + lane < n ? exp2f(lse_acc[(int64_t)(block + lane) * row_stride] - g) : 0.f;
                }
                const float w = __shfl_sync(0xffffffffu, w_block, s & 31);
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    acc[i].x += w * v[u][i].x; acc[i].y += w * v[u][i].y; acc[i].z += w * v[u][i].z; acc[i].w += w * v[u][i].w;
                }
            }
        }
    }
    if (WPR < 8) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // out is bf16 or fp16: both are 2 bytes wide
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(a.out) + req * a.o_stride_b + t * a.o_stride_s + head * a.o_stride_h + col0;
    auto store4 = [&](int col, float4 x) {
        uint2 packed;
        if (a.dtype == MLA_DTYPE_FP16) {
            __half2 lo = __floats2half2_rn(x.x, x.y);
            __half2 hi = __floats2half2_rn(x.z, x.w);
            packed.x = *reinterpret_cast<uint32_t*>(&lo);
            packed.y = *reinterpret_cast<uint32_t*>(&hi);
        } else {
            __nv_bfloat162 lo = __floats2bfloat162_rn(x.x, x.y);
            __nv_bfloat162 hi = __floats2bfloat162_rn(x.z, x.w);
            packed.x = *reinterpret_cast<uint32_t*>(&lo);
            packed.y = *reinterpret_cast<uint32_t*>(&hi);
        }
        *reinterpret_cast<uint2*>(o + col) = packed;
    };
    if (WPR == 1) {
        if (!head_ok) return;
#pragma unroll
        for (int i = 0; i < NV; ++i) store4((lane + i * 32) * 4, acc[i]);
    } else {
        constexpr int ROW = 128 / PARTS;                  // float4s of a row
        float4* mine = reinterpret_cast<float4*>(part) + warp * ROW + lane;
#pragma unroll
        for (int i = 0; i < NV; ++i) mine[i * 32] = acc[i];
        __syncthreads();
        if (WPR == 8) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        // every warp of the row adds up and writes 512 / WPR columns
        if (!head_ok) return;
        const float4* row = reinterpret_cast<const float4*>(part) + (warp - sub) * ROW;
        for (int c = sub * (ROW / WPR) + lane; c < (sub + 1) * (ROW / WPR); c += 32) {
            float4 x = row[c];
#pragma unroll
            for (int k = 1; k < WPR; ++k) {
                const float4 y = row[k * ROW + c];
                x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
            }
            store4(c * 4, x);
        }
    }
}

int launch_combine(const mla_combine_args_t& a) {
    MLA_CHECK_ARG(a.b > 0 && a.s_q > 0 && a.h_q > 0, "combine: b, s_q, h_q must be positive");
    MLA_CHECK_ARG(a.d_v == 512, "combine: only d_v == 512 is supported (got %d)", a.d_v);
    MLA_CHECK_ARG(a.dtype == MLA_DTYPE_BF16 || a.dtype == MLA_DTYPE_FP16, "combine: dtype must be MLA_DTYPE_BF16 or MLA_DTYPE_FP16 (got %d)", a.dtype);
    MLA_CHECK_ARG(a.lse && a.out && a.lse_accum && a.o_accum && a.num_splits, "combine: null pointer");
    MLA_CHECK_ARG(is_aligned16(a.o_accum), "combine: o_accum must be 16-byte aligned");
    MLA_CHECK_ARG(((uintptr_t)a.out & 7u) == 0 && a.o_stride_b % 4 == 0 && a.o_stride_s % 4 == 0 && a.o_stride_h % 4 == 0,
                  "combine: out must be 8-byte aligned with strides that are multiples of 4 elements");
    // Warps per row, from an estimate of the splits a request has: the SM pairs shared out over row blocks of 128 and the batch
    // (up to 64 rows: the SMs over the batch).
    // This kernel knows neither the partition count nor h_kv: the estimate is high for several kv heads and low, in sparse decode,
    // for several query tokens of at most 64 heads (3 x 64, one request: 38, of 49 partitions).  The bounds on the rows (all CTAs in one wave: 2 per SM with the deeper
    // unrolling of WPR = 8, else 3) keep that harmless.  us alone, behind a 256 MB scrub, with
    // 1 / 2 / 4 / 8 warps per row, and the rule's choice (event resolution 2 us):
    //    rows  splits                            rows  splits
    //     128    74    35 / 23 / 16 / 14   8      1024    10    12 / 12 / 12 / 14   2
    //     128    16    12 / 10 /  8 /  8   8      1536     7    12 / 12 / 12 / 16   2
    //     256    37    23 / 16 / 12 / 12   8      1536     2     8 /  8 / 10 / 16   2
    //     512    19    14 / 12 / 12 / 12   4       976     2     8 /  8 / 10 / 12   1
    //     768    13    14 / 12 / 12 / 14   4     16384     2    20 / 27 / 45 /100   1
    const int64_t rows = (int64_t)a.b * a.s_q * a.h_q;
    const int sms = current_device_num_sms() > 0 ? current_device_num_sms() : 148;
    const int rows_each = a.s_q * a.h_q;
    const int splits = 1 + (rows_each <= MLA_SINGLE_SM_ROWS ? sms : sms / 2) / std::max(1, (rows_each + 127) / 128) / a.b;
    const int64_t wave = (int64_t)sms * 3 * COMBINE_WARPS;         // warps
    const int wpr = splits >= 16 && rows <= 2 * sms ? 8 : splits >= 8 && rows * 4 <= wave ? 4 : splits >= 4 && rows * 2 <= wave ? 2 : 1;
    const int rows_per_cta = COMBINE_WARPS / wpr;
    // Up to a row per SM and 48 splits or more by the estimate (on 148 SMs one to three requests with 148 rows together, of more than 64 rows each
    // one): a row's columns in two CTAs, twice as many splits in flight each.  us a step, one CTA / two, one request: 20000 tokens, 128 heads 20.2 /
    // 18.9, 64 heads 20.0 / 18.8, 16 heads 18.7 / 17.1; two requests of 2048 keys, 64 heads 16.7 / 16.1; 2000 tokens, 1, 2, 3 requests of 16 heads 12.8,
    // 12.8, 13.1 / 12.3, 12.4, 12.6.  The estimate knows no lengths.  Short requests have fewer splits and lose: 2 splits (100 tokens), 1, 2, 3 requests of 16
    // heads 10.85, 10.77, 10.94 / 10.94, 10.94, 11.03, of 48 heads 13.85, 14.01, 14.02 / 14.02, 14.18, 14.21; 5 splits 0.1 or less; from 10 on both are equal or
    // two CTAs ahead.  Four requests of 64..512 tokens lose (12.3 / 12.45) and stay with one.
    //   Left to the device - up to 8 or 16 splits the first CTA takes all columns, the second leaves - 2 splits are as fast as with one CTA, but rows of other
    // calls are slower by the longer code: 15 splits 12.3 -> 12.7, 105 splits 17.3 -> 17.7, four requests of 100 tokens 10.8 -> 11.1 (one source for both forms).
    const int parts = wpr == 8 && splits >= 48 && rows <= sms ? 2 : 1;
    const dim3 grid(a.b * a.s_q, (a.h_q + rows_per_cta - 1) / rows_per_cta, parts), block(COMBINE_WARPS * 32);
    const cudaStream_t stream = (cudaStream_t)a.stream;
    MLA_CHECK_CUDA(parts == 2 ? launch_dependent(combine_kernel<8, 2>, grid, block, 0, stream, a)
                   : wpr == 8 ? launch_dependent(combine_kernel<8, 1>, grid, block, 0, stream, a)
                   : wpr == 4 ? launch_dependent(combine_kernel<4, 1>, grid, block, 0, stream, a)
                   : wpr == 2 ? launch_dependent(combine_kernel<2, 1>, grid, block, 0, stream, a)
                              : launch_dependent(combine_kernel<1, 1>, grid, block, 0, stream, a));
    return MLA_OK;
}

}  // namespace mla
