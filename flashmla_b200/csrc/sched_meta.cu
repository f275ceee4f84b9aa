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
// partition starts at the larger of X - F and C[e] (at the end of all costs if X reaches that), and only this position is
// serial: one warp walks the partitions, 32 prefix sums at a time, whose largest one within X is one reduction.  Everything
// else follows from two neighbouring positions - requests by binary search, splits because starts inside a request lie
// budget - F apart - and is done with a thread per partition afterwards.
// What bounds it is the chain, about 78 cycles a partition; up to 64 query rows have a partition per SM, and with votes and
// shuffles in the chain (118 cycles) their schedules took 4 to 5 us longer than with one per pair of SMs.  us a schedule of
// lengths up to 8000, one after the other in a graph, votes and shuffles / now:
//                     b 4          b 32         b 64         b 128        b 1000
//    74 partitions    6.6 / 5.3    7.0 / 5.8    7.0 / 5.9    7.2 / 6.1    10.8 / 9.3
//   148 partitions   11.1 / 8.2   11.4 / 8.7   11.8 / 9.0   12.1 / 9.3    15.7 / 12.6
// Where requests span more than eight partitions each on average, their ends alone are walked, 400 cycles a request, in loops that are
// not unrolled (a launch fetches its instructions anew: unrolled the walk takes 0.1 to 0.5 us more, and the chain 0.05).  us, the chain / now, requests
// of one length:              1 x 30     1 x 400    1 x 8000   4 x 1000   4 x 8000   9 x 200    9 x 8000   16 x 1000
//    74 partitions           2.2 / 2.2  2.4 / 2.5  4.8 / 2.4  3.6 / 3.7  5.0 / 3.5  3.2 / 3.2  5.4 / 5.5  5.1 / 5.2
//   148 partitions           2.4 / 2.4  2.6 / 2.7  7.6 / 2.5  5.1 / 3.7  7.8 / 3.5  4.0 / 4.1  8.6 / 5.2  6.6 / 6.7
// (The test that chooses costs every schedule 0.03 to 0.07.)  One of 100003 tokens decoded with 128 heads, schedule included, 48.9 -> 46.3.
// (A serial walk over the requests by one thread: 6.9, 8.4, 9.8, 12.2, 32 with 148 partitions.  A branch that steps inside a
// request without the reduction: 6.4, 7.7, 8.8, 10.2, 15.4, but slower than votes and shuffles where requests are short.)
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
    __shared__ int warp_sums[SCHED_THREADS / 32], starts[SCHED_THREADS + 1];

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

    const int total = C[b], budget = (total + P - 1) / P + F, own = budget - F;
    const int lane = threadIdx.x & 31;
    // (first warp) window: lane l holds C[base + l + 1] (past the end: never reached); floor and top: C[base], C[base + 32]
    int base = 0, window = lane < b ? C[lane + 1] : INT_MAX, floor = 0, top = b >= 32 ? C[32] : INT_MAX;
    int x = 0;
    auto blocks = [&](int r) { const int n = C[r + 1] - C[r] - F; return (zero_len[r >> 5] >> (r & 31)) & 1u ? -1 : n; };
    auto request_at = [&](int pos, int lo) {                        // the request a position lies in (b: behind the last one), lo or a later one
        int hi = b;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (C[mid + 1] <= pos) lo = mid + 1; else hi = mid;
        }
        return lo;
    };
    for (int p0 = 0; p0 < P; p0 += SCHED_THREADS) {
        // the serial chain: where partitions p0 .. begin, and where the last of them ends
        if (threadIdx.x < 32) {
            const int n_all = min(SCHED_THREADS, P - p0);
            // (either way finds the same starts: the line between them may be rounded)
            if (P <= SCHED_THREADS && (float)(total - b * F) > 8.f * (float)b * (float)own) {
                // Requests of more than eight partitions each: as long as no request ends inside the budget the starts lie budget - F
                // apart, so all of these are written at once and only the requests' ends stand in the chain.
                int p = 0, r = 0;
#pragma unroll 1
                while (p < P && x < total) {
#pragma unroll 1
                    while (C[r + 1] <= x) ++r;
                    const int gap = C[r + 1] - budget - x, n = gap > 0 ? min((gap + own - 1) / own, P - p) : 0;
#pragma unroll 1
                    for (int j = lane; j <= n; j += 32) starts[p + j] = x + j * own;
                    p += n;
                    x += n * own;
                    if (p < P) {
#pragma unroll 1
                        while (r < b && C[r + 1] <= x + budget) ++r;
                        x = min(max(C[r], x + own), total);
                        ++p;
                    }
                }
#pragma unroll 1
                for (int j = p + lane; j <= P; j += 32) starts[j] = x;
            } else
            for (int g0 = 0; g0 < n_all; g0 += 32) {
                int begin = x;                                      // lane l: where partition p0 + g0 + l begins
                const int n = min(32, n_all - g0);
#pragma unroll 1
                for (int i = 1; i <= n && x < total; ++i) {         // (behind the last request every partition begins where this one ends)
                    const int X = x + budget;
                    while (X >= top) {                              // the window lies wholly inside the budget: the next one
                        base += 32;
                        floor = top;
                        window = base + lane < b ? C[base + lane + 1] : INT_MAX;
                        top = base + 32 <= b ? C[base + 32] : INT_MAX;
                    }
                    x = min(max(__reduce_max_sync(0xffffffffu, window <= X ? window : floor), x + own), total);
                    if (lane >= i) begin = x;
                }
                if (g0 + lane < n_all) starts[g0 + lane] = begin;
            }
            if (lane == 0) starts[n_all] = x;
        }
        __syncthreads();
        // the rows, a thread each: every partition ends where the next one begins
        if (p0 + threadIdx.x < P) {
            const int begin = starts[threadIdx.x], end = starts[threadIdx.x + 1];
            mla_sched_meta_t m;
            m.begin_req_idx = request_at(begin, 0);
            m.end_req_idx = request_at(end, m.begin_req_idx);
            const int begin_block = begin - C[m.begin_req_idx];
            m.end_block_idx = end - C[m.end_req_idx];
            // A partition that starts after the last request reports the last block index of request 0
            // here: the reference reads one element past its first-block array, which is the first
            // element of its last-block array.  Consumers skip such partitions (begin_req_idx >= b).
            m.begin_block_idx = m.begin_req_idx < b ? begin_block : abs(blocks(0)) - 1;
            // Inside a request the starts lie budget - F apart, the first at most that far from the request's beginning.
            m.begin_split_idx = (begin_block + own - 1) / own;
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
            a.meta[p0 + threadIdx.x] = m;
        }
        __syncthreads();
    }

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
