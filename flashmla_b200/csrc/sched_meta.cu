// Tile-scheduler metadata kernel: splits the 64-token KV blocks of a decode batch over the SM
// partitions of the decode kernels and records, per request, how many partial results (splits)
// the combine kernel has to merge.
//
// The greedy rule and every output value follow the reference kernel
// csrc/smxx/decode/get_decoding_sched_meta/get_decoding_sched_meta.cu:28-106 bit for bit for equal
// (num_sm_parts, block_size_n, fixed_overhead): each partition gets a budget of
// ceil(total/num_sm_parts) + fixed_overhead blocks, where every request costs its blocks plus
// fixed_overhead; whole requests are taken while they fit, otherwise the remaining budget minus the
// overhead is taken from the next request and the partition ends.
//
// One CTA.  In terms of the prefix sums C[i] = cost of requests 0 .. i - 1 (blocks plus overhead each), a partition that
// starts at cost position x (request r, block x - C[r]) may spend up to X = x + budget: it finishes every request e' with
// C[e' + 1] <= X, and cuts the next one, e, if blocks are left after that request's overhead (X - F > C[e]).  So the next
// partition starts at X - F or at C[e], and only this position is serial: one warp walks the partitions, comparing 32
// prefix sums at a time (a vote instead of a walk over the requests).  Nothing else stands in that chain: lane l keeps the
// start of partition l, and 32 metadata rows are finished and written side by side, each ending where the next one starts.
// What bounds it is the chain, about 130 cycles a partition.  us a schedule, one after the other in a graph: one thread that
// walks requests and partitions / rows written and cuts counted by one lane inside the chain / now:
//    b 1, 74 partitions  9 / 13 / 5.3;   b 32  12 / 15.5 / 6.6;   b 128  17 / 16 / 6.9;   b 1000  60 / 20 / 10.6
#include "common.cuh"

#include <limits.h>

namespace mla {

constexpr int SCHED_THREADS = 256;

// Inclusive scan of one value per thread; `carry` (shared by all threads) is added and moved on.
__device__ __forceinline__ int block_scan(int v, int* warp_sums, int& carry) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += x;
    }
    if (lane == 31) warp_sums[warp] = v;
    __syncthreads();
    int before = carry, total = 0;
#pragma unroll
    for (int w = 0; w < SCHED_THREADS / 32; ++w) {
        const int x = warp_sums[w];
        if (w < warp) before += x;
        total += x;
    }
    __syncthreads();
    carry += total;
    return v + before;
}

__global__ void __launch_bounds__(SCHED_THREADS, 1)
sched_meta_kernel(const mla_sched_meta_args_t a) {
    // the decode kernel that follows is launched with programmatic stream serialization: let its prologue (barrier and
    // tensor-memory set-up) start now; it waits for this kernel's completion before it reads the metadata
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    extern __shared__ int smem_i[];
    const int b = a.b, bs = a.block_size_n, F = a.fixed_overhead_num_blocks, P = a.num_sm_parts;
    int* C = smem_i;                              // [b + 1]  prefix sums of the requests' costs
    int* cuts = C + b + 1;                        // [b]      partitions that end inside a request
    uint32_t* zero_len = reinterpret_cast<uint32_t*>(cuts + b);      // a bit per request without keys
    __shared__ int warp_sums[SCHED_THREADS / 32];

    int carry = 0;
    for (int i0 = 0; i0 < b; i0 += SCHED_THREADS) {
        const int i = i0 + threadIdx.x;
        int cost = 0;
        bool zero = false;
        if (i < b) {
            int s;
            if (a.topk == -1) {
                s = a.seqlens_k[i];
            } else {
                s = a.topk_length ? a.topk_length[i] : a.topk;
                if (s == 0) s = 1;
                if (a.extra_topk) {
                    s = (s + bs - 1) / bs * bs;
                    s += a.extra_topk_length ? a.extra_topk_length[i] : a.extra_topk;
                }
            }
            zero = s == 0;
            cost = max(s - 1, 0) / bs + 1 + F;    // a zero-length request still costs one block
            cuts[i] = 0;
        }
        const uint32_t zeros = __ballot_sync(0xffffffffu, zero);
        if ((threadIdx.x & 31) == 0 && i < b) zero_len[i >> 5] = zeros;
        const int end = block_scan(cost, warp_sums, carry);
        if (i < b) C[i + 1] = end;
    }
    if (threadIdx.x == 0) C[0] = 0;
    __syncthreads();

    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const int budget = (C[b] + P - 1) / P + F;
        auto blocks = [&](int r) { const int n = C[r + 1] - C[r] - F; return (zero_len[r >> 5] >> (r & 31)) & 1u ? -1 : n; };
        // window: lane l holds C[base + l + 1] (past the end: never reached)
        int base = 0, window = lane < b ? C[lane + 1] : INT_MAX;
        int x = 0, r = 0, split = 0, at_r = 0;                      // at_r = C[r]
        for (int p0 = 0; p0 < P; p0 += 32) {
            // lane l keeps where partition p0 + l begins: request, block, split
            int begin_r = r, begin_block = x - at_r, begin_split = split;
            const int n_parts = min(32, P - p0);
#pragma unroll 1
            for (int i = 1; i <= n_parts && r < b; ++i) {          // (behind the last request every partition begins where this one ends)
                const int X = x + budget;
                int n = __popc(__ballot_sync(0xffffffffu, window <= X));
                int at_e = __shfl_sync(0xffffffffu, window, n - 1);
                while (n == 32) {                                  // the window lies wholly inside the budget: the next one
                    base += 32;
                    at_r = at_e;
                    window = base + lane < b ? C[base + lane + 1] : INT_MAX;
                    n = __popc(__ballot_sync(0xffffffffu, window <= X));
                    at_e = __shfl_sync(0xffffffffu, window, n - 1);
                }
                const int e = base + n;
                at_e = n ? at_e : at_r;
                const bool cut = e < b && X - F > at_e;
                split = cut ? (e == r ? split + 1 : 1) : 0;
                x = cut ? X - F : at_e;
                r = e;
                at_r = at_e;
                if (lane >= i) { begin_r = r; begin_block = x - at_r; begin_split = split; }
            }
            // ... and ends where the next one begins
            mla_sched_meta_t m;
            m.end_req_idx = __shfl_down_sync(0xffffffffu, begin_r, 1);
            m.end_block_idx = __shfl_down_sync(0xffffffffu, begin_block, 1);
            if (lane == n_parts - 1) { m.end_req_idx = r; m.end_block_idx = x - at_r; }
            if (lane < n_parts) {
                m.begin_req_idx = begin_r;
                // A partition that starts after the last request reports the last block index of request 0
                // here: the reference reads one element past its first-block array, which is the first
                // element of its last-block array.  Consumers skip such partitions (begin_req_idx >= b).
                m.begin_block_idx = begin_r < b ? begin_block : abs(blocks(0)) - 1;
                m.begin_split_idx = begin_split;
                m.is_first_req_splitted = begin_block != 0;
                if (m.end_block_idx == 0) {
                    --m.end_req_idx;
                    m.end_block_idx = max(blocks(m.end_req_idx), 0);
                } else {
                    atomicAdd(&cuts[m.end_req_idx], 1);
                }
                const int n_end = blocks(m.end_req_idx);
                m.is_last_req_splitted = n_end > 0 && m.end_block_idx != n_end;
                if (m.begin_req_idx == m.end_req_idx)
                    m.is_first_req_splitted = m.is_last_req_splitted = (m.is_first_req_splitted || m.is_last_req_splitted);
                m._pad = 0;
                a.meta[p0 + lane] = m;
            }
        }
    }
    __syncthreads();

    // a request has one piece more than cuts
    carry = 0;
    if (threadIdx.x == 0) a.num_splits[0] = 0;
    for (int i0 = 0; i0 < b; i0 += SCHED_THREADS) {
        const int i = i0 + threadIdx.x;
        const int end = block_scan(i < b ? cuts[i] + 1 : 0, warp_sums, carry);
        if (i < b) a.num_splits[i + 1] = end;
    }
}

int launch_sched_meta(const mla_sched_meta_args_t& a) {
    MLA_CHECK_ARG(a.b > 0, "sched_meta: batch size must be positive (got %d)", a.b);
    MLA_CHECK_ARG(a.num_sm_parts > 0, "sched_meta: num_sm_parts must be positive (got %d)", a.num_sm_parts);
    MLA_CHECK_ARG(a.block_size_n > 0 && a.fixed_overhead_num_blocks >= 0, "sched_meta: bad block size / overhead");
    MLA_CHECK_ARG(a.meta && a.num_splits, "sched_meta: output pointers must not be null");
    MLA_CHECK_ARG(a.topk != -1 || a.seqlens_k, "sched_meta: seqlens_k is required for dense attention");
    MLA_CHECK_ARG(sizeof(int) * (2 * (size_t)a.b + 1) <= 200 * 1024, "sched_meta: batch size %d too large (max 25000)", a.b);
    const size_t smem = sizeof(int) * (2 * (size_t)a.b + 1 + ((size_t)a.b + 31) / 32);
    if (smem > 48 * 1024)
        MLA_CHECK_CUDA(cudaFuncSetAttribute(sched_meta_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    MLA_CHECK_CUDA(launch_dependent(sched_meta_kernel, dim3(1), dim3(SCHED_THREADS), smem, (cudaStream_t)a.stream, a));
    return MLA_OK;
}

}  // namespace mla
