// MLA attention for sm_100a: tcgen05 MMAs with TMEM accumulators.  One kernel template serves
//   MODE_DENSE          dense BF16 / FP16 paged decode, fed by TMA loads of 64-token KV pages through the block table
//   MODE_PREFILL        token-sparse prefill, KV rows gathered by index with cp.async
//   MODE_SPARSE_DECODE  sparse FP8 decode, 656-byte records gathered by index and de-quantised in shared memory
//
// Problem shape per (request, kv head): 128 query rows (query token x head, padded with zero rows)
// against a stream of 576-wide K rows whose first 512 columns are also V.  The fp32 output
// accumulator O[128 x 512] fills all 512 columns of one SM's tensor memory, so the work of one row
// block is split over a CLUSTER OF TWO CTAs on two SMs that walk the same KV range in tiles of 128
// tokens (two pages):
//
//   CTA 0 ("score" CTA)  S = Q K^T: 36 MMAs 128x128x16 per tile (N = 128 runs the tensor pipe at full
//       rate, N = 64 does not).  Q is the A operand and lives in tensor memory (packed bf16).  K arrives
//       through a ring of 48 KB groups; a group is three 64-dim chunks of a tile (each [128 tokens][64 dims],
//       K-major, 128-byte swizzle) and is refilled as soon as its twelve MMAs have retired.
//         dense mode:   all 576 dims of Q in tensor memory (288 columns) next to ONE S accumulator (128 columns);
//                       the shared memory this frees makes the ring FOUR groups deep (192 KB): the time a tile
//                       takes is the refill latency of a ring slot divided by the slots that can be in flight.
//         gather modes: dims 0..447 of Q in tensor memory, dims 448..575 in shared memory, two S accumulators,
//                       a ring of three groups.
//       Two softmax warpgroups (one per page of the tile, one thread per row and page) exchange row
//       maxima through shared memory, write P (bf16) in MMA operand layout to a staging buffer and
//       push it to CTA 1 with bulk shared-to-shared copies that complete on CTA 1's barriers.
//   CTA 1 ("value" CTA)  O += P V: per page 2 x 4 MMAs 128x256x16 (A = P from shared memory, B = the
//       first 512 dims of the page viewed MN-major; 5-slot ring of [64 tokens][256 dims]),
//       the rare O rescale, and the epilogue (normalise; bf16 output or fp32 split partials).
//
// The tensor work divides 576 : 512 between the two SMs; each KV page is fetched from HBM by whichever
// CTA asks first and from L2 by the other.  No TMA multicast is used.  (MMAs that span the CTA pair,
// cta_group::2, were considered and not used: with 64 of the 128 rows per CTA each CTA still has to stage its
// half of the tokens for Q K^T and ALL tokens of its half of the columns for P V - 136 KB per tile and CTA
// against 144 + 128 KB here - so neither the bytes that enter the SMs nor the ring depth improve.)
//
// Softmax uses the running maximum lazily: O is rescaled only when a row's maximum grew by more than 2^6
// since the value in use; P, the row sum and O always refer to the same maximum, so results are exact
// up to rounding.
//
// Every mbarrier wait is bounded (Params::wait_limit SM cycles, about a second by default).  A thread whose
// wait ran out LEAVES its role - it issues no further arrival, MMA or copy -, records a code in the status words and raises
// the `aborted` flag of both CTAs.  Single-thread roles leave at once; warps leave together (a vote
// after every wait, because tcgen05.ld/st are warp-collective); the two softmax warpgroups, which meet at a
// named barrier every tile, carry the flag through that barrier (bar.red.or) and leave together behind it.
// Threads that depend on the one that left run into their own limit.  The wind-down then waits - again
// bounded - for this CTA's own MMAs and TMA loads, meets the peer CTA, gives copies between the two CTAs time
// to land, and only then frees tensor memory; both CTAs leave together.
//
// Behavioural reference: csrc/sm90/decode/dense/splitkv_mla.cuh:959-1272 (masking, split / direct
// epilogue, empty rows), csrc/sm100/decode/head64/kernel.cuh:19-849 (FP8 records, validity, attn_sink) and
// csrc/sm100/prefill/sparse/fwd/head128/phase1.cuh:65-614 (prefill outputs) of deepseek-ai/FlashMLA.
#include "attn_shared.cuh"

namespace mla {
namespace sm100 {

constexpr int ROWS = 128;
constexpr int BOX_BYTES = 8192;       // 64 tokens x 64 bf16, 128-byte swizzled rows
constexpr int K_CHUNK_BYTES = 2 * BOX_BYTES;  // one 64-dim chunk of a tile: [128 tokens][64 dims]
constexpr int K_GROUP_BYTES = 3 * K_CHUNK_BYTES;   // the K ring moves in groups of 3 chunks (one barrier pair per group)
constexpr int V_SLOT_BYTES = 4 * BOX_BYTES;   // half a page of V: [64 tokens][256 dims] as 4 boxes
constexpr int NVS = 5;                        // V ring slots
constexpr int P_SUB_BYTES = ROWS * PAGE * 2;  // P of one page: [128 rows][64 tokens] bf16
constexpr int NPB = 4;                        // P buffers in the value CTA: (tile parity, page of the tile)
constexpr int NRING = 5;                      // ring barriers: K groups (score CTA, 3 or 4) / V slots (value CTA, 5)
constexpr int SIDE_BYTES = 144;               // per warp and tile: 32 rescale factors + flag (+ pad)
constexpr int NTHREADS = 384;                 // dense mode: control warpgroup + two softmax / correction warpgroups
constexpr long long SETTLE_CYCLES = 400000LL;             // ... and for copies between the two CTAs
#ifndef MLA_TAIL_BULK
#define MLA_TAIL_BULK 1
#endif

// Warps behind the control warpgroup and the two softmax / correction warpgroups: GATHER warps copy KV rows by index,
// CONVERT warps de-quantise FP8 records.  A kernel starts with its registers shared out evenly (launch bound) and every
// warpgroup re-sizes its share as the first thing in its branch; the shares add up to no more than the launch had.
//   prefill     640 threads x 96 registers: control 96, softmax 136, gather 56.  EIGHT gather warps: an SM's copy rate is
//               bound by what its warps can issue, 77 GB/s with four warps, 102 with eight (stand-alone probe).  The control
//               warps' share is what the issuing thread of the MMAs needs: with less it spills the descriptors of its unrolled
//               loop (4096 tokens: 2526 us with control 64, 2428 with 80, 2421 with 96 in short runs; 2894, 2812 and 2800
//               back to back under the power limit).  Warps 8-11 of the value CTA have no work in the gather modes, and
//               their registers none either: the shares are the same in both CTAs.
//   FP8 decode  768 threads x 80 registers: control 48, softmax 112, gather 80, convert 64.  The conversion has warps of its
//               own: on the softmax warps it was serial with the softmax (5.2 us a tile).
template <int MODE>
struct Warps {
    static constexpr int GATHER = MODE == MODE_DENSE ? 0 : MODE == MODE_PREFILL ? 8 : 4;
    static constexpr int CONVERT = MODE == MODE_SPARSE_DECODE ? 8 : 0;
    static constexpr int FIRST_GATHER = 12, FIRST_CONVERT = 12 + GATHER;
    static constexpr int THREADS = (12 + GATHER + CONVERT) * 32;
};

// Shared-memory and tensor-memory plan of the score CTA, per mode (byte offsets inside Smem::data).
template <int MODE>
struct Lay {
    static constexpr bool DENSE = MODE == MODE_DENSE;
    // WIDE plan (dense decode): all 576 dims of Q in tensor memory (288 columns) next to ONE S accumulator, which frees
    // the shared memory for a K ring of FOUR groups.  The gather modes keep the narrow plan (dims 0..447 of Q in tensor
    // memory, 448..575 in shared memory, two S accumulators, three groups): prefill is paced by the copy instructions of
    // its gather warps, not by the ring (the wide plan, measured when four warps copied: 3.49 against 3.41 ms), and FP8 decode
    // needs 4 KB for the tokens' scales.
    static constexpr bool WIDE = MODE == MODE_DENSE;
    static constexpr int NKS = WIDE ? 4 : 3;              // K ring slots; group j of tile g is fill 3 g + j and uses slot (3 g + j) mod NKS
    static constexpr int S_BUFS = WIDE ? 1 : 2;           // S accumulators in tensor memory
    static constexpr int Q_TMEM_CHUNKS = WIDE ? 9 : 7;    // 64-dim chunks of Q kept in tensor memory (the rest in SC_Q78)
    static constexpr int Q_SPLIT = WIDE ? 5 : 4;          // chunks [0, Q_SPLIT) are moved there by softmax warpgroup 0, the others by 1
    static constexpr uint32_t TM_S = 0, TM_Q = 128 * S_BUFS;
    static constexpr int SC_Q78 = 0;                                    // narrow plan: Q dims 448..575, 2 x [128][64]
    static constexpr int SC_KRING = WIDE ? 0 : 2 * 16384;
    static constexpr int SC_STAGE = SC_KRING + NKS * K_GROUP_BYTES;     // 8 warps x 4 KB P staging
    static constexpr int SC_SIDE = SC_STAGE + 8 * 4096;                 // 4 warps x 144 B factor/flag staging
    static constexpr int SC_XMAX = SC_SIDE + 4 * SIDE_BYTES;            // [2][2][128] floats
    static constexpr int SC_END = SC_XMAX + 2 * 2 * ROWS * 4;
    // gather modes only
    static constexpr int SC_MASK = SC_END;                // validity bits of the last 4 tiles, [4][4] words
    static constexpr int SC_LSUM = SC_MASK + 64;          // narrow plan: row sums of softmax warpgroup 1, handed to warpgroup 0 at the end of a request
    static constexpr int SC_SCALES = SC_LSUM + ROWS * 4;  // FP8 decode: the 4 scales of every token of the last two tiles, [2][128] float4
    static constexpr int SC_TOTAL = DENSE ? SC_END : (WIDE ? SC_MASK + 64 : SC_SCALES + 2 * ROWS * 16);
    static_assert(TM_Q + Q_TMEM_CHUNKS * 32 <= 512, "tensor-memory columns of the score CTA");
};
// value CTA (all modes)
constexpr int VA_VRING = 0;
constexpr int VA_P = VA_VRING + NVS * V_SLOT_BYTES;
constexpr int VA_SIDE = VA_P + NPB * P_SUB_BYTES;         // factors + flag received with the first page of tile parity 0 / 1: [2][4][SIDE_BYTES]
constexpr int VA_FIN = VA_SIDE + 2 * 4 * SIDE_BYTES;      // final row sum / running maximum / true maximum of the request: 3 x [128] floats
constexpr int VA_END = VA_FIN + 3 * ROWS * 4;
constexpr int cmax(int a, int b) { return a > b ? a : b; }
constexpr int DATA_BYTES = cmax(cmax(VA_END, Lay<MODE_DENSE>::SC_TOTAL), cmax(Lay<MODE_PREFILL>::SC_TOTAL, Lay<MODE_SPARSE_DECODE>::SC_TOTAL));

struct Smem {
    uint8_t data[DATA_BYTES];
    uint64_t kv_full[NRING], kv_empty[NRING];     // K groups (score CTA) / V slots (value CTA)
    uint64_t s_full[2], s_empty[2], q_ready, stage_full[2];
    uint64_t p_empty[NPB], stage_free[2], fin_empty;              // live in the score CTA, arrived by the value CTA
    uint64_t p_full[NPB], pv_done[NPB], corr_done[NPB], fin_full; // live in the value CTA
    uint64_t q_landed, ring_released;    // score CTA: a request's Q boxes have landed / have been copied out of the K ring
    uint64_t raw_full[NRING];            // FP8 decode: the raw records of a K group (score CTA) / V slot (value CTA) have landed
    uint64_t drain;                      // wind-down after an expired wait: this CTA's MMAs have retired
    uint32_t tmem_base;
    uint32_t aborted;                    // a bounded wait ran out in this CTA or in its peer
};
static_assert(sizeof(Smem) <= 232448, "shared memory budget");

// the two softmax warpgroups of the score CTA: their named barrier carries the flag
#define BAR_OR_LEAVE(flag) do { if (named_bar_red_or(1, 256, flag)) goto wind_down; } while (0)

// Rare paths of the value CTA's correction warpgroup, kept out of line so that the loop around them stays small.
// O rows times their rescale factor (each thread its own row = tensor-memory lane).
__device__ __noinline__ void rescale_o_rows(uint32_t tlane, float f) {
#pragma unroll 1
    for (int c = 0; c < D_V / 32; ++c) {
        uint32_t v[32];
        tmem_ld32(tlane + c * 32, v);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 32; ++k) v[k] = __float_as_uint(__uint_as_float(v[k]) * f);
        tmem_st32(tlane + c * 32, v);
    }
    tmem_wait_st();
}
// Rows [first, 64) of a dense V slot ([8-token group][chunk][8 rows x 128 B]) set to zero by threads 128..255.
__device__ __noinline__ void zero_v_rows(uint8_t* vst, int first) {
    const int nz = (PAGE - first) * 4 * 8;              // rows x boxes x 16-byte chunks
    for (int k = threadIdx.x - 128; k < nz; k += 128) {
        const int chunk = k & 7, box = (k >> 3) & 3, rr = first + (k >> 5);
        *reinterpret_cast<uint4*>(vst + (rr >> 3) * 4096 + box * 1024 + (rr & 7) * 128 + chunk * 16) = make_uint4(0, 0, 0, 0);
    }
}

// A request's Q row moved by the softmax threads themselves, one thread per row: the path for Q tensors whose base or
// strides do not fit a TMA box (several times slower than the boxes; kept out of line, it is rarely taken).
// Warpgroup `half` takes its share of the chunks: to tensor memory, in the gather modes chunks 7 / 8 to shared memory.
template <int MODE>
__device__ __noinline__ void load_q_by_threads(Smem& sm, const __nv_bfloat16* qrow, bool row_ok, int half, int r, uint32_t tlane, bool no_chunk8) {
    using L = Lay<MODE>;
    const int c_begin = half ? L::Q_SPLIT : 0, c_end = half ? L::Q_TMEM_CHUNKS : L::Q_SPLIT, c_smem = half ? 8 : 7;
#pragma unroll 1
    for (int c = c_begin; c < c_end + (L::WIDE ? 0 : 1); ++c) {
        const int chunk = c < c_end ? c : c_smem;
        uint32_t v[32];
        if (row_ok && !(no_chunk8 && chunk == 8)) {
            const uint4* src = reinterpret_cast<const uint4*>(qrow + chunk * 64);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint4 x = __ldg(src + i);
                v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
        }
        if (c < c_end) {
            tmem_st32(tlane + L::TM_Q + chunk * 32, v);
        } else {
            uint8_t* qdst = sm.data + L::SC_Q78 + (chunk - L::Q_TMEM_CHUNKS) * 16384 + (r >> 3) * 1024 + (r & 7) * 128;
#pragma unroll
            for (int ch = 0; ch < 8; ++ch)
                *reinterpret_cast<uint4*>(qdst + ((ch ^ (r & 7)) << 4)) = make_uint4(v[4 * ch], v[4 * ch + 1], v[4 * ch + 2], v[4 * ch + 3]);
        }
    }
}

// ALT selects the second data format of a mode.  Dense mode: q, the cache and out are fp16 instead of bf16 (accumulation
// is fp32 either way).  Sparse FP8 decode: the 512-wide record form (448 e4m3 + 64 bf16 RoPE per token, seven e8m0 scales
// per token stored behind the block's tokens, V = all 512 dims): chunk 7 of a tile is the RoPE part, chunk 8 is zeros.
// Sparse prefill: 512-wide rows; the ninth 64-column chunk of Q and K is zeros.  (A compile-time switch in every mode: the
// same choice read from the parameters inside the gather loop cost the 576-wide prefill 8 %.)
template <int MODE, bool ALT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Warps<MODE>::THREADS, 1)
attn_sm100_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                  const __grid_constant__ CUtensorMap qmap, const Params p) {
    using WalkerT = Walker<MODE>;
    using L = Lay<MODE>;
    using W = Warps<MODE>;
    constexpr int NKS = L::NKS;
    constexpr bool DENSE = MODE == MODE_DENSE;
    constexpr bool FP16 = ALT && MODE == MODE_DENSE;
    constexpr bool M1 = ALT && MODE == MODE_SPARSE_DECODE;
    // How far the MMA issue loops are unrolled (turns of one loop body).  Unrolled, an MMA's descriptor is a compile-time
    // offset and issuing is fastest; rolled, the roles of an SM share less code.  FP8 decode has issue time to spare and six
    // roles per SM (64 requests: unrolled 102.2 us, rolled by groups 94.4); prefill and dense decode have not (4096 tokens:
    // 2800 unrolled, 3393 rolled; the serving batch 196.3 and 202.5).  The pages of P V stay rolled everywhere (unrolled:
    // prefill 2918, FP8 decode 99.2, dense decode the same).  All back to back.
    constexpr int MMA_GROUPS = MODE == MODE_SPARSE_DECODE ? 1 : 3;
    constexpr bool NO_CHUNK8 = ALT && MODE != MODE_DENSE;  // 512-wide rows
    constexpr int REC_BYTES = M1 ? 576 : 656;              // bytes between two tokens' values inside a block
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    const uint32_t cta_rank = cluster_ctarank();          // 0 = score CTA, 1 = value CTA
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row_blk = MODE == MODE_SPARSE_DECODE ? 0 : blockIdx.y % p.row_blocks;
    const int hk = MODE == MODE_SPARSE_DECODE ? 0 : blockIdx.y / p.row_blocks;
    const int part = blockIdx.z;

    if ((smem_addr(smem_raw) & 1023u) != 0) {              // the swizzled tiles need a 1024-byte aligned base
        if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, 900);
        return;                                            // both CTAs of the pair take this branch
    }

    if (threadIdx.x == 0) {
        // a ring slot is filled by TMA (one arrive.expect_tx + bytes) in dense mode, by the gather threads in prefill, and
        // handed over by the converting threads in FP8 decode
        const uint32_t full_count = DENSE ? 1 : 32 * (MODE == MODE_SPARSE_DECODE ? W::CONVERT : W::GATHER);
        for (int i = 0; i < NRING; ++i) { mbar_init(smem_addr(&sm.kv_full[i]), full_count); mbar_init(smem_addr(&sm.kv_empty[i]), 1); }
        for (int i = 0; i < NRING; ++i) mbar_init(smem_addr(&sm.raw_full[i]), DENSE ? 1 : 32 * W::GATHER);
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_addr(&sm.s_full[i]), 1);
            mbar_init(smem_addr(&sm.s_empty[i]), 256);
            mbar_init(smem_addr(&sm.stage_free[i]), 1);
            mbar_init(smem_addr(&sm.stage_full[i]), 128);
        }
        for (int i = 0; i < NPB; ++i) {
            mbar_init(smem_addr(&sm.p_empty[i]), 1);
            mbar_init(smem_addr(&sm.p_full[i]), 1);        // one arrive.expect_tx by the sending thread
            mbar_init(smem_addr(&sm.pv_done[i]), 1);
            mbar_init(smem_addr(&sm.corr_done[i]), 128);
        }
        mbar_init(smem_addr(&sm.q_ready), 256);
        mbar_init(smem_addr(&sm.q_landed), 1);
        mbar_init(smem_addr(&sm.ring_released), 256);
        mbar_init(smem_addr(&sm.fin_empty), 128);
        mbar_init(smem_addr(&sm.fin_full), 128);
        mbar_init(smem_addr(&sm.drain), 1);
        sm.aborted = 0;
        // first use of every P buffer: its arrival and expected byte count are armed here (matters in the value CTA)
        for (int i = 0; i < NPB; ++i)
            mbar_arrive_expect_tx(smem_addr(&sm.p_full[i]), P_SUB_BYTES + ((i & 1) == 0 ? 4 * SIDE_BYTES : 0));
        fence_mbar_init();
        if (DENSE) prefetch_tensormap(cta_rank == 0 ? &kmap : &vmap);
        if (p.q_tma && cta_rank == 0) prefetch_tensormap(&qmap);
    }
    if (warp == 1) { tmem_alloc(smem_addr(&sm.tmem_base), 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    cluster_sync();                                        // the peer's barriers exist before anyone arrives remotely
    // Programmatic dependent launch: everything above ran while the previous kernel of the stream (the tile scheduler,
    // or whatever produced q) was still draining; from here on its results are read.  The kernel after this one (the
    // split-KV combine) may be scheduled as SMs become free: it waits for this grid's completion itself.
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t tmem = sm.tmem_base;
    Waiter wt(p.wait_limit);
    const int oob_page = p.num_blocks;                     // a page coordinate outside the cache: TMA fills zeros
    // what the wind-down has to wait for after an expired wait (thread 0: ring fills and Q boxes it armed)
    uint32_t fills_armed = 0, q_armed = 0;

    // A request's Q (score CTA): nine [rows][64 columns] boxes into the K ring once the previous request's tiles
    // have left it (the softmax warpgroups move them on to tensor memory and release the ring); in the gather modes
    // chunks 7 and 8 go to their final place in shared memory instead.  Large boxes stream several times faster into
    // one SM than per-thread loads, and the request boundary - where the MMA warp idles - is what this shortens.
    auto issue_q = [&](const Work& w) {
        const uint32_t bar = smem_addr(&sm.q_landed);
        mbar_arrive_expect_tx(bar, 9u * (uint32_t)p.q_box_bytes);
        ++q_armed;
        // coordinates: (column, head, query token, request); prefill: a "request" is a query token of the only batch
        const int c1 = MODE == MODE_SPARSE_DECODE ? 0 : MODE == MODE_PREFILL ? row_blk * ROWS : hk * p.g;
        const int c2 = MODE == MODE_SPARSE_DECODE ? (int)blockIdx.y : MODE == MODE_PREFILL ? w.req : row_blk * (ROWS / p.g);
        const int c3 = MODE == MODE_PREFILL ? 0 : w.req;
#pragma unroll 1
        for (int c = 0; c < 9; ++c) {
            const uint32_t dst = c < L::Q_TMEM_CHUNKS ? smem_addr(sm.data + L::SC_KRING + c * 16384)
                                                      : smem_addr(sm.data + L::SC_Q78 + (c - L::Q_TMEM_CHUNKS) * 16384);
            tma_load_4d(dst, &qmap, bar, c * 64, c1, c2, c3);
        }
    };

    // =====================================================================================================
    // (the compiler budgets registers per branch from the share each takes first)
    if (warp < 4) {
    // (prefill: keeps the 96 it started with)
    if (MODE == MODE_SPARSE_DECODE) regs_dec<48>();
    if (warp == 0) {
        // ---------------- TMA producer (both CTAs) ---------------------------------------------------------
        if (!DENSE) {
            // sparse modes: the gather warpgroup fills the rings
            if (p.q_tma && cta_rank == 0 && lane == 0) {
                uint32_t ks = 0, nreq = 0;
                for (WalkerT wk(p, part); wk.valid(); wk.next(), ++nreq) {
                    const Work w = wk.get();
                    issue_q(w);
                    WAIT_OR_LEAVE(wt, false, &sm.ring_released, nreq & 1, 11);     // (a request without tiles must not be overtaken)
                    // The next request's boxes may go out once every MMA of this one has finished with the ring and with
                    // Q.  A parity wait only means what it says to a thread that has seen every earlier phase of the
                    // barrier, so this thread follows the ring fill by fill.
                    for (int i = 0; i < 3 * w.ntiles; ++i, ++ks)
                        WAIT_OR_LEAVE(wt, false, &sm.kv_empty[ks % NKS], (ks / NKS) & 1, 13);
                }
            }
        } else if (lane == 0) {
            uint32_t ks = 0;                               // ring fill counter (K groups or V half-pages)
            uint32_t nreq = 0;
            const int chunk0 = hk * p.head_chunks;         // the kv head's first 64-column chunk in the tensor maps
            for (WalkerT wk(p, part); wk.valid(); wk.next(), ++nreq) {
                const Work w = wk.get();
                const int* bt = p.block_table + (int64_t)w.req * p.bt_sb;
                // a block index beyond the table's width reads no table entry: its keys are zeros
                auto page_of = [&](int blk) -> int { return (blk < w.blk_end && blk < p.max_blocks) ? __ldg(bt + blk) : oob_page; };
                // page ids are fetched one tile ahead so the block-table latency stays off the TMA issue path
                int nxt0 = oob_page, nxt1 = oob_page;
                if (w.ntiles > 0) { nxt0 = page_of(w.blk_begin); nxt1 = page_of(w.blk_begin + 1); }
                if (p.q_tma && cta_rank == 0) {
                    // the K ring stages this request's Q first: wait until the previous request's groups (and every MMA
                    // that read its Q) are done - slot s is free for its next fill -, send the boxes, and take the ring
                    // back once they have been copied out
                    for (uint32_t s = 0; s < (uint32_t)NKS; ++s) {
                        const uint32_t nf = ks + (uint32_t)(((int)s - (int)(ks % NKS) + NKS) % NKS);      // the next fill that uses slot s
                        WAIT_OR_LEAVE(wt, false, &sm.kv_empty[s], ((nf / NKS) & 1) ^ 1, 13);
                    }
                    issue_q(w);
                    WAIT_OR_LEAVE(wt, false, &sm.ring_released, nreq & 1, 11);
                }
                for (int i = 0; i < w.ntiles; ++i) {
                    const int page0 = nxt0, page1 = nxt1;
                    if (i + 1 < w.ntiles) {
                        const int nb = w.blk_begin + 2 * (i + 1);
                        nxt0 = page_of(nb);
                        nxt1 = page_of(nb + 1);
                    }
                    if (cta_rank == 0) {
                        for (int grp = 0; grp < 3; ++grp, ++ks) {
                            const uint32_t slot = ks % NKS;
                            WAIT_OR_LEAVE(wt, false, &sm.kv_empty[slot], ((ks / NKS) & 1) ^ 1, 1);
                            const uint32_t bar = smem_addr(&sm.kv_full[slot]);
                            mbar_arrive_expect_tx(bar, K_GROUP_BYTES);
                            fills_armed = ks + 1;
                            const uint32_t dst = smem_addr(sm.data + L::SC_KRING + slot * K_GROUP_BYTES);
                            // one box per page: 3 chunks x 64 tokens land as [8-token group][chunk][8 x 128 B]
                            tma_load_5d(dst, &kmap, bar, 0, 0, chunk0 + grp * 3, 0, page0);
                            tma_load_5d(dst + K_GROUP_BYTES / 2, &kmap, bar, 0, 0, chunk0 + grp * 3, 0, page1);
                        }
                    } else {
                        for (int h = 0; h < 2; ++h) {
                            const int page = h ? page1 : page0;
                            for (int nh = 0; nh < 2; ++nh, ++ks) {
                                const uint32_t slot = ks % NVS;
                                WAIT_OR_LEAVE(wt, false, &sm.kv_empty[slot], ((ks / NVS) & 1) ^ 1, 101);
                                const uint32_t bar = smem_addr(&sm.kv_full[slot]);
                                mbar_arrive_expect_tx(bar, V_SLOT_BYTES);
                                fills_armed = ks + 1;
                                const uint32_t dst = smem_addr(sm.data + VA_VRING + slot * V_SLOT_BYTES);
                                // one box: 4 chunks x 64 tokens as [8-token group][chunk][8 x 128 B]
                                tma_load_5d(dst, &vmap, bar, 0, 0, chunk0 + nh * 4, 0, page);
                            }
                        }
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer -----------------------------------------------------------------------
        if (elect_one()) {
            uint32_t g = 0, ks = 0, nreq = 0;
            if (cta_rank == 0) {
                constexpr uint32_t idesc = make_idesc_16(ROWS, 128, false, FP16);
                const uint32_t q78_lo = sw128_desc_lo(smem_addr(sm.data + L::SC_Q78), 16);
                const uint32_t kring_lo = sw128_desc_lo(smem_addr(sm.data + L::SC_KRING), 16);
                const uint32_t kv_empty0 = smem_addr(&sm.kv_empty[0]);
                const uint32_t kv_full0 = smem_addr(&sm.kv_full[0]);
                uint32_t slot = 0, par = 0;                 // ring position of the next group: slot = ks mod NKS, par = (ks / NKS) & 1
                for (WalkerT wk(p, part); wk.valid(); wk.next(), ++nreq) {
                    const Work w = wk.get();
                    WAIT_OR_LEAVE(wt, false, &sm.q_ready, nreq & 1, 2);
                    for (int i = 0; i < w.ntiles; ++i, ++g) {
                        const uint32_t sb = L::S_BUFS == 2 ? (g & 1) : 0;
                        const uint32_t s_par = L::S_BUFS == 2 ? ((g >> 1) & 1) : (g & 1);
                        WAIT_OR_LEAVE(wt, false, &sm.s_empty[sb], s_par ^ 1, 4);
                        tc_fence_after();
                        const uint32_t d_tmem = tmem + L::TM_S + sb * 128;
                        // Descriptors advance by 32-bit adds only and the loop is fully unrolled: one thread issues
                        // everything, so its instruction latency is the issue rate.
                        constexpr uint32_t hi = sw128_desc_hi(1024);
                        // K operand: the gather modes store a tile as 9 chunks of [128 tokens][128 B]; the dense mode's
                        // TMA boxes interleave the 3 chunks of a ring group inside every 8-token group.
                        constexpr uint32_t hi_k = sw128_desc_hi(DENSE ? 3 * 1024 : 1024);
                        // The probe of the next group's barrier is issued before this group's MMAs so that its
                        // latency hides behind them (the MMA queue is shallow: time the issuing thread spends
                        // waiting is time the tensor pipe idles).
                        // (narrow plan: three slots, so group j of every tile sits in slot j with the tile's parity and
                        // every address below is a compile-time offset)
                        if (!L::WIDE) { slot = 0; par = g & 1; }
                        bool ready = mbar_try_wait(kv_full0 + slot * 8, par);
#pragma unroll MMA_GROUPS
                        for (int grp = 0; grp < 3; ++grp) {
                            const uint32_t cur = L::WIDE ? slot : (uint32_t)grp;
                            if (!ready) WAIT_OR_LEAVE(wt, false, &sm.kv_full[cur], par, 3);
                            tc_fence_after();
                            if (L::WIDE) { if (++slot == (uint32_t)NKS) { slot = 0; par ^= 1; } }
                            if (grp < 2) ready = mbar_try_wait(kv_full0 + (L::WIDE ? slot : (uint32_t)(grp + 1)) * 8, par);
                            const uint32_t grp_lo = kring_lo + cur * (K_GROUP_BYTES >> 4);
#pragma unroll
                            for (int c = 0; c < 3; ++c) {
                                const int j = grp * 3 + c;
                                const uint32_t b_lo = DENSE ? grp_lo + c * (1024 >> 4) : grp_lo + c * (K_CHUNK_BYTES >> 4);
#pragma unroll
                                for (int k4 = 0; k4 < 4; ++k4) {
                                    const uint32_t acc = (j > 0 || k4 > 0) ? 1u : 0u;
                                    if (j < L::Q_TMEM_CHUNKS) mma_ts_lohi(d_tmem, tmem + L::TM_Q + j * 32 + k4 * 8, b_lo + k4 * 2, hi_k, idesc, acc);
                                    else mma_ss_lohi(d_tmem, q78_lo + (j - L::Q_TMEM_CHUNKS) * (16384 >> 4) + k4 * 2, hi, b_lo + k4 * 2, hi_k, idesc, acc);
                                }
                            }
                            tc_commit(kv_empty0 + cur * 8);
                        }
                        tc_commit(smem_addr(&sm.s_full[sb]));
                    }
                }
            } else {
                constexpr uint32_t idesc = make_idesc_16(ROWS, 256, true, FP16);
                // V operand (MN-major): LBO = stride between 64-dim chunks, SBO = stride between 8-token groups.  Gather
                // modes: 4 chunks of [64 tokens][128 B]; dense mode: chunks interleaved inside every 8-token group.
                constexpr uint32_t hi_a = sw128_desc_hi(1024), hi_b = sw128_desc_hi(DENSE ? 4 * 1024 : 1024);
                constexpr uint32_t v_kstep = (DENSE ? 2 * 4096 : 2 * 1024) >> 4;      // 16 tokens
                const uint32_t p_lo = sw128_desc_lo(smem_addr(sm.data + VA_P), 16);
                const uint32_t vring_lo = sw128_desc_lo(smem_addr(sm.data + VA_VRING), DENSE ? 1024 : BOX_BYTES);
                for (WalkerT wk(p, part); wk.valid(); wk.next(), ++nreq) {
                    const Work w = wk.get();
                    for (int i = 0; i < w.ntiles; ++i, ++g) {
#pragma unroll 1
                        for (int h = 0; h < 2; ++h) {
                            const uint32_t pb = (g & 1) * 2 + h, pph = (g >> 1) & 1;
                            WAIT_OR_LEAVE(wt, true, &sm.p_full[pb], pph, 104);
                            WAIT_OR_LEAVE(wt, false, &sm.corr_done[pb], pph, 105);
                            const uint32_t a_lo = p_lo + pb * (P_SUB_BYTES >> 4);
#pragma unroll
                            for (int nh = 0; nh < 2; ++nh, ++ks) {
                                const uint32_t slot = ks % NVS;
                                WAIT_OR_LEAVE(wt, false, &sm.kv_full[slot], (ks / NVS) & 1, 103);
                                if (nh == 0) fence_proxy_async_smem();
                                tc_fence_after();
                                const uint32_t b_lo = vring_lo + slot * (V_SLOT_BYTES >> 4);
#pragma unroll
                                for (int kt = 0; kt < PAGE / 16; ++kt)
                                    mma_ss_lohi(tmem + nh * 256, a_lo + kt * 2, hi_a, b_lo + kt * v_kstep, hi_b, idesc,
                                                (i > 0 || h > 0 || kt > 0) ? 1u : 0u);
                                tc_commit(smem_addr(&sm.kv_empty[slot]));
                            }
                            tc_commit(smem_addr(&sm.pv_done[pb]));
                        }
                    }
                }
            }
        }
    } else if (warp == 2 || warp == 3) {
        // ---------------- score CTA: push finished P pages (and, with page 0, the rescale factors) to the value CTA
        if (cta_rank == 0 && lane == 0) {
            const int half = warp - 2;
            uint32_t g = 0;
            const uint32_t src_p = smem_addr(sm.data + L::SC_STAGE + half * 4 * 4096);
            const uint32_t src_side = smem_addr(sm.data + L::SC_SIDE);
            const uint32_t remote_p = map_to_cta(smem_addr(sm.data + VA_P), 1);
            const uint32_t remote_side = map_to_cta(smem_addr(sm.data + VA_SIDE), 1);
            uint32_t remote_p_full[NPB];
            for (int i = 0; i < NPB; ++i) remote_p_full[i] = map_to_cta(smem_addr(&sm.p_full[i]), 1);
            for (WalkerT wk(p, part); wk.valid(); wk.next()) {
                const Work w = wk.get();
                for (int i = 0; i < w.ntiles; ++i, ++g) {
                    const uint32_t pb = (g & 1) * 2 + half;
                    WAIT_OR_LEAVE(wt, false, &sm.stage_full[half], g & 1, 9);
                    WAIT_OR_LEAVE(wt, true, &sm.p_empty[pb], ((g >> 1) & 1) ^ 1, 6);   // that P buffer of the value CTA has been consumed
                    // p_full[pb] is armed (arrival + expected bytes) by the value CTA itself: a remote arrive with
                    // release semantics costs over a microsecond, the copies below only count bytes.
                    bulk_copy_to_cluster(remote_p + pb * P_SUB_BYTES, src_p, P_SUB_BYTES, remote_p_full[pb]);
                    if (half == 0)
                        bulk_copy_to_cluster(remote_side + (g & 1) * 4 * SIDE_BYTES, src_side, 4 * SIDE_BYTES, remote_p_full[pb]);
                }
            }
        }
        // ---------------- value CTA: tell the score CTA when a P buffer has been consumed ------------------
        if (cta_rank == 1 && warp == 2 && lane == 0) {
            uint32_t g = 0;
            uint32_t remote_p_empty[NPB];
            for (int i = 0; i < NPB; ++i) remote_p_empty[i] = map_to_cta(smem_addr(&sm.p_empty[i]), 0);
            for (WalkerT wk(p, part); wk.valid(); wk.next()) {
                const Work w = wk.get();
                for (int i = 0; i < w.ntiles; ++i, ++g) {
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t pb = (g & 1) * 2 + h;
                        WAIT_OR_LEAVE(wt, false, &sm.pv_done[pb], (g >> 1) & 1, 106);
                        // arm the buffer's barrier for its next use, then let the score CTA refill it
                        mbar_arrive_expect_tx(smem_addr(&sm.p_full[pb]), P_SUB_BYTES + (h == 0 ? 4 * SIDE_BYTES : 0));
                        mbar_arrive_remote_relaxed(remote_p_empty[pb]);
                    }
                }
            }
        }
    }
    } else if (!DENSE && warp >= W::FIRST_GATHER && warp < W::FIRST_CONVERT) {
        if (MODE == MODE_PREFILL) regs_dec<56>();          // (FP8 decode: keeps the 80 it started with)
        // ---------------- gather warpgroup (sparse modes): fills the K ring (score CTA) / V ring (value CTA) by index ----
        // Every warp owns a block of tokens; one cp.async instruction of the warp copies consecutive 16-byte pieces of
        // ONE token row (coalesced 128-byte lines, no registers held, as many copies in flight as the ring has room
        // for) into the 128-byte-swizzled operand layout; invalid tokens get zeros (zero-size source).  The ring
        // barrier counts one arrival per thread, made by the copy engine when that thread's copies have landed.
        const int gw = warp - W::FIRST_GATHER;
        constexpr int TPW = 128 / (W::GATHER ? W::GATHER : 1), VPW = TPW / 2;      // tokens per warp: of a tile (score CTA) / of a page (value CTA)
        uint32_t ks = 0, g = 0, nreq_p = 0;
        uint32_t* kmask = reinterpret_cast<uint32_t*>(sm.data + L::SC_MASK);
        if (MODE == MODE_SPARSE_DECODE) {
            // FP8 records: index -> (page, offset) -> 656-byte record = 512 e4m3 | 4 fp32 scales | 64 bf16 RoPE.
            // A "piece" is 16 e4m3 values (16 bytes) that de-quantise (one rounding: bf16(fp32(e4m3) * scale)) into two
            // 16-byte slots of a 128-byte operand row.  Two decoupled steps per ring element (a K group of 3 chunks in
            // the score CTA, a V slot of 4 chunks in the value CTA):
            //   copy:    this warpgroup brings every raw piece with cp.async straight into the UPPER of its own two
            //            destination slots (lanes = pieces of two token rows: coalesced, no registers held), RoPE pieces
            //            into their final place, and counts the landing on the element's raw_full barrier;
            //   convert: eight warps of its own expand the pieces of their token row in place (a thread reads
            //            a slot only it will overwrite; 16-byte accesses, conflict-free thanks to the swizzle) and hand
            //            the element to the MMA warp.
            // Copying and converting run side by side on different warps; record pointers (and, in the score CTA, the
            // scales the converting threads read from shared memory) are fetched one tile ahead.  The conversion loops
            // are deliberately left rolled: with every instance unrolled the conversion code was several times the
            // instruction cache and the warps waited for instructions more than they computed.
            const int tq = blockIdx.y;
            bool ring_lent = false;                                       // the K ring first stages every request's Q
            uint32_t nreq_g = 0;
            float4 sc_cur = make_float4(0.f, 0.f, 0.f, 0.f);
            const uint32_t kring = smem_addr(sm.data + L::SC_KRING);
            const uint32_t vring = smem_addr(sm.data + VA_VRING);
            for (WalkerT wk(p, part); wk.valid(); wk.next(), ++nreq_g) {
                const Work w = wk.get();
                ring_lent = p.q_tma && cta_rank == 0;
                if (ring_lent && w.ntiles == 0) WAIT_WARP_OR_LEAVE(wt, false, &sm.ring_released, nreq_g & 1, 211);   // follow every phase
                const int* idx0 = p.sidx[0] + (int64_t)w.req * p.sidx_sb[0] + (int64_t)tq * p.sidx_ss[0];
                const int* idx1 = p.stopk[1] ? p.sidx[1] + (int64_t)w.req * p.sidx_sb[1] + (int64_t)tq * p.sidx_ss[1] : nullptr;
                // index -> record address in two steps, so that the index of a tile can be loaded two tiles ahead and
                // turned into an address (and a scale load) one tile ahead without waiting on memory
                auto load_id = [&](int blk, int off) -> int {
                    if (blk >= w.blk_end) return -1;
                    const int scope = blk >= w.nblk0 ? 1 : 0;
                    const int pos = (scope ? blk - w.nblk0 : blk) * PAGE + off;
                    if (pos >= (scope ? w.len1 : w.len0)) return -1;
                    return __ldg((scope ? idx1 : idx0) + pos);
                };
                auto rec_of = [&](int blk, int id) -> const uint8_t* {
                    const int scope = blk >= w.nblk0 ? 1 : 0;
                    const int pbs = p.pbs[scope];
                    if (id < 0 || (int64_t)id >= (int64_t)p.nblocks[scope] * pbs) return nullptr;
                    return p.kvb[scope] + (int64_t)(id / pbs) * p.kvb_sblock[scope] + (int64_t)(id % pbs) * REC_BYTES;
                };
                // the token's scales as they are stored: four fp32 inside the record, or (512-wide form) eight bytes -
                // seven e8m0 exponents and a pad - behind the block's tokens, carried in the first two words
                auto scales_of = [&](int blk, int id, const uint8_t* rec) {
                    if (!rec) return make_float4(0.f, 0.f, 0.f, 0.f);
                    if (!M1) return __ldg(reinterpret_cast<const float4*>(rec + 512));
                    const int scope = blk >= w.nblk0 ? 1 : 0;
                    const int pbs = p.pbs[scope];
                    const uint2 e = __ldg(reinterpret_cast<const uint2*>(p.kvb[scope] + (int64_t)(id / pbs) * p.kvb_sblock[scope] +
                                                                         (int64_t)pbs * 576 + (int64_t)(id % pbs) * 8));
                    return make_float4(__uint_as_float(e.x), __uint_as_float(e.y), 0.f, 0.f);
                };
                if (cta_rank == 0) {
                    // warp gw owns tokens 32*gw .. 32*gw+31 of the tile; lane l looks up token 32*gw + l
                    const int tok = gw * 32 + lane;
                    const int myblk = w.blk_begin + (tok >> 6);              // this lane's block of tile 0
                    const int id_first = load_id(myblk, tok & 63);
                    const uint8_t* rec_next = rec_of(myblk, id_first);
                    float4 sc_next = scales_of(myblk, id_first, rec_next);
                    int id_next = load_id(myblk + 2, tok & 63);              // tile 1
                    for (int i = 0; i < w.ntiles; ++i, ++g) {
                        const uint8_t* rec = rec_next;
                        sc_cur = sc_next;
                        // validity bits and scales of this tile's tokens for the threads that convert / mask it (the fence
                        // comes before the prefetch loads are issued: it would wait for them)
                        const uint32_t bal = __ballot_sync(0xffffffffu, rec != nullptr);
                        if (lane == 0) kmask[(g & 3) * 4 + gw] = bal;
                        reinterpret_cast<float4*>(sm.data + L::SC_SCALES)[(g & 1) * ROWS + tok] = sc_cur;
                        __threadfence_block();
                        rec_next = rec_of(myblk + 2 * (i + 1), id_next);
                        sc_next = scales_of(myblk + 2 * (i + 1), id_next, rec_next);
                        id_next = load_id(myblk + 2 * (i + 2), tok & 63);
                        if (ring_lent) { WAIT_WARP_OR_LEAVE(wt, false, &sm.ring_released, nreq_g & 1, 211); ring_lent = false; }
#pragma unroll 1
                        for (int grp = 0; grp < 3; ++grp, ++ks) {
                            WAIT_WARP_OR_LEAVE(wt, false, &sm.kv_empty[grp], ((ks / NKS) & 1) ^ 1, 201);
                            // copy: groups 0, 1: 12 raw pieces per row; group 2: 8 raw pieces + 8 RoPE pieces per row.  A copy
                            // instruction costs the warp the same whatever its active lanes: each one serves two rows.
                            // (512-wide form: every group has 12 pieces per row; group 2 is chunk 6 - 4 raw pieces - and the 8 RoPE
                            // pieces, which are chunk 7; chunk 8 is zeroed by the converting threads)
                            const int per_row = (grp < 2 || M1) ? 12 : 16;
                            const int sub = (grp < 2 || M1) ? (lane >= 12) + (lane >= 24) : lane >> 4, ql = lane - sub * per_row;
                            const bool active = sub < 2;
                            constexpr int N_RAW2 = M1 ? 4 : 8;               // raw pieces of group 2
                            const bool is_rope = grp == 2 && ql >= N_RAW2;
                            const int q = grp * 12 + ql;                      // raw piece index in the row
                            const int srcoff = is_rope ? (M1 ? 448 : 528) + (ql - N_RAW2) * 16 : q * 16;
                            const int dslot = is_rope ? ql - N_RAW2 : 2 * (q & 3) + 1;
                            const uint32_t dst0 = kring + (is_rope ? (M1 ? 7 : 8) : (q >> 2)) * K_CHUNK_BYTES + gw * 32 * 128;
#pragma unroll 4
                            for (int u = 0; u < 16; ++u) {
                                const int rr = 2 * u + (active ? sub : 0);
                                const uint8_t* r = shfl_ptr(rec, rr);
                                if (active)
                                    cp_async16_zfill(dst0 + rr * 128 + ((dslot ^ (rr & 7)) << 4), (r ? r : p.kvb[0]) + srcoff, r ? 16u : 0u);
                            }
                            // the converting warps expand the pieces in place once they have landed
                            cp_async_arrive_noinc(smem_addr(&sm.raw_full[grp]));
                        }
                    }
                } else {
                    // value CTA: warp gw owns tokens 16*gw .. 16*gw+15 of each page; lanes l and l + 16 look up the same token
                    const int tok = gw * 16 + (lane & 15);
                    const uint8_t* rec_next = rec_of(w.blk_begin, load_id(w.blk_begin, tok));
                    int id_next = load_id(w.blk_begin + 1, tok);
                    for (int i = 0; i < w.ntiles; ++i, ++g) {
#pragma unroll 1
                        for (int h = 0; h < 2; ++h) {
                            const uint8_t* rec = rec_next;
                            const int nblk = w.blk_begin + 2 * i + h + 1;
                            rec_next = rec_of(nblk, id_next);
                            id_next = load_id(nblk + 1, tok);
#pragma unroll 1
                            for (int nh = 0; nh < 2; ++nh, ++ks) {
                                const uint32_t slot = ks % NVS;
                                WAIT_WARP_OR_LEAVE(wt, false, &sm.kv_empty[slot], ((ks / NVS) & 1) ^ 1, 202);
                                // copy: 16 raw pieces per row (dims nh*256 .. nh*256+255); one instruction serves two rows
                                const int ql = lane & 15, sub = lane >> 4;
                                const int q = nh * 16 + ql;
                                const uint32_t dst0 = vring + slot * V_SLOT_BYTES + (ql >> 2) * BOX_BYTES + gw * 16 * 128;
                                const int dslot = 2 * (ql & 3) + 1;
                                // (512-wide form, second half: 12 raw pieces - chunks 4, 5, 6 - and, below, the RoPE part as chunk 7)
                                const bool piece_ok = !M1 || nh == 0 || ql < 12;
#pragma unroll 4
                                for (int u = 0; u < 8; ++u) {
                                    const int rr = 2 * u + sub;
                                    const uint8_t* r = shfl_ptr(rec, rr);
                                    if (piece_ok)
                                        cp_async16_zfill(dst0 + rr * 128 + ((dslot ^ (rr & 7)) << 4), (r ? r : p.kvb[0]) + q * 16, r ? 16u : 0u);
                                }
                                if (M1 && nh == 1) {
                                    const int piece = lane & 7;
                                    const uint32_t dst7 = vring + slot * V_SLOT_BYTES + 3 * BOX_BYTES + gw * 16 * 128;
#pragma unroll
                                    for (int u = 0; u < 4; ++u) {
                                        const int rr = 4 * u + (lane >> 3);
                                        const uint8_t* r = shfl_ptr(rec, rr);
                                        cp_async16_zfill(dst7 + rr * 128 + ((piece ^ (rr & 7)) << 4), (r ? r : p.kvb[0]) + 448 + piece * 16, r ? 16u : 0u);
                                    }
                                }
                                cp_async_arrive_noinc(smem_addr(&sm.raw_full[slot]));      // the converting warps expand the pieces
                            }
                        }
                    }
                }
            }
        } else
        for (WalkerT wk(p, part); wk.valid(); wk.next(), ++nreq_p) {
            const Work w = wk.get();
            bool ring_lent = p.q_tma && cta_rank == 0;          // the K ring first stages this query token's Q
            if (ring_lent && w.ntiles == 0) WAIT_WARP_OR_LEAVE(wt, false, &sm.ring_released, nreq_p & 1, 211);        // follow every phase
            const int* idx = p.indices + (int64_t)w.req * p.idx_ss;
            // the index of a tile's token is loaded one tile ahead (a load that is used at once costs its latency)
            int id_next = -1;
            const int tok = gw * TPW + lane % TPW, vtok = gw * VPW + lane % VPW;      // token this lane looks up
            if (cta_rank == 0) id_next = tok < w.seqlen ? __ldg(idx + tok) : -1;
            int vid_next = -1;                       // value CTA: index of this lane's token of the next page
            if (cta_rank == 1) vid_next = vtok < w.seqlen ? __ldg(idx + vtok) : -1;
            for (int i = 0; i < w.ntiles; ++i, ++g) {
                if (cta_rank == 0) {
                    // warp gw owns tokens TPW*gw .. TPW*gw + TPW-1 of the tile
                    const int id = id_next;
                    const bool ok = id >= 0 && id < p.s_kv;
                    const uint32_t bal = __ballot_sync(0xffffffffu, ok);
                    // token 32w + l of the tile is bit l of word w; a warp of 16 tokens writes half a word
                    if (lane == 0) { reinterpret_cast<uint16_t*>(kmask)[(g & 3) * 8 + gw] = (uint16_t)bal; __threadfence_block(); }
                    // (issued after the fence, which would otherwise wait for it)
                    { const int posn = (i + 1) * 128 + tok; id_next = posn < w.seqlen ? __ldg(idx + posn) : -1; }
                    const int row_id = ok ? id : -1;
                    // A copy instruction costs the warp the same whatever its active lanes, so a token row (72 pieces of
                    // 16 bytes) is copied by two full-warp instructions (chunks 0-3, chunks 4-7) and the RoPE chunk of
                    // four rows by a third: 36 instructions per 16 rows.  The ring barriers still count per group of 3
                    // chunks: every group's arrival is issued once all copies that touch it have been issued.
                    // the tile's three groups are fills ks, ks + 1, ks + 2 of the ring; chunk c of the tile lives in the slot of
                    // group c / 3, at chunk position c % 3
                    const uint32_t ring0 = smem_addr(sm.data + L::SC_KRING) + gw * TPW * 128;
                    // (three slots: group j sits in slot j and every address below is a compile-time offset)
                    const uint32_t slot0 = L::WIDE ? ks % NKS : 0u, slot1 = L::WIDE ? (ks + 1) % NKS : 1u, slot2 = L::WIDE ? (ks + 2) % NKS : 2u;
                    const int c = lane & 7;
                    if (ring_lent) { WAIT_WARP_OR_LEAVE(wt, false, &sm.ring_released, nreq_p & 1, 211); ring_lent = false; }
                    WAIT_WARP_OR_LEAVE(wt, false, &sm.kv_empty[slot0], ((ks / NKS) & 1) ^ 1, 201);
                    WAIT_WARP_OR_LEAVE(wt, false, &sm.kv_empty[slot1], (((ks + 1) / NKS) & 1) ^ 1, 201);
                    {
                        const int ch = lane >> 3;                     // chunks 0-3: 0, 1, 2 in group 0, chunk 3 in group 1
                        const uint32_t dst0 = ring0 + (ch < 3 ? slot0 * K_GROUP_BYTES + ch * K_CHUNK_BYTES : slot1 * K_GROUP_BYTES);
#pragma unroll 8
                        for (int rr = 0; rr < TPW; ++rr) {
                            const int rid = __shfl_sync(0xffffffffu, row_id, rr);
                            const __nv_bfloat16* src = p.kv + (int64_t)(rid < 0 ? 0 : rid) * p.kv_ss + lane * 8;
                            cp_async16_zfill(dst0 + rr * 128 + ((c ^ (rr & 7)) << 4), src, rid < 0 ? 0u : 16u);
                        }
                    }
                    cp_async_arrive_noinc(smem_addr(&sm.kv_full[slot0]));
                    WAIT_WARP_OR_LEAVE(wt, false, &sm.kv_empty[slot2], (((ks + 2) / NKS) & 1) ^ 1, 201);
                    {
                        const int ch = 4 + (lane >> 3);               // chunks 4-7: 4, 5 in group 1, chunks 6, 7 in group 2
                        const uint32_t dst0 = ring0 + (ch < 6 ? slot1 * K_GROUP_BYTES + (ch - 3) * K_CHUNK_BYTES
                                                              : slot2 * K_GROUP_BYTES + (ch - 6) * K_CHUNK_BYTES);
#pragma unroll 8
                        for (int rr = 0; rr < TPW; ++rr) {
                            const int rid = __shfl_sync(0xffffffffu, row_id, rr);
                            const __nv_bfloat16* src = p.kv + (int64_t)(rid < 0 ? 0 : rid) * p.kv_ss + (32 + lane) * 8;
                            cp_async16_zfill(dst0 + rr * 128 + ((c ^ (rr & 7)) << 4), src, rid < 0 ? 0u : 16u);
                        }
                    }
                    cp_async_arrive_noinc(smem_addr(&sm.kv_full[slot1]));
                    {
                        const uint32_t dst0 = ring0 + slot2 * K_GROUP_BYTES + 2 * K_CHUNK_BYTES;      // chunk 8
#pragma unroll
                        for (int q4 = 0; q4 < TPW / 4; ++q4) {
                            const int rr = 4 * q4 + (lane >> 3);
                            const int rid = __shfl_sync(0xffffffffu, row_id, rr);
                            // (rows of 512 columns have no ninth chunk: zeros, as for an invalid token)
                            const __nv_bfloat16* src = p.kv + (int64_t)(rid < 0 ? 0 : rid) * p.kv_ss + (NO_CHUNK8 ? 0 : (64 + c) * 8);
                            cp_async16_zfill(dst0 + rr * 128 + ((c ^ (rr & 7)) << 4), src, (rid < 0 || NO_CHUNK8) ? 0u : 16u);
                        }
                    }
                    cp_async_arrive_noinc(smem_addr(&sm.kv_full[slot2]));
                    ks += 3;
                } else {
                    // warp gw owns tokens VPW*gw .. VPW*gw + VPW-1 of each page; one instruction copies 512 bytes of one row
                    for (int h = 0; h < 2; ++h) {
                        const int id = vid_next;
                        { const int posn = i * 128 + (h + 1) * 64 + vtok; vid_next = posn < w.seqlen ? __ldg(idx + posn) : -1; }
                        const int row_id = (id >= 0 && id < p.s_kv) ? id : -1;
                        for (int nh = 0; nh < 2; ++nh, ++ks) {
                            const uint32_t slot = ks % NVS;
                            WAIT_WARP_OR_LEAVE(wt, false, &sm.kv_empty[slot], ((ks / NVS) & 1) ^ 1, 202);
                            const int box = lane >> 3, c = lane & 7;
                            const uint32_t dst0 = smem_addr(sm.data + VA_VRING + slot * V_SLOT_BYTES) + box * BOX_BYTES + gw * VPW * 128;
#pragma unroll 8
                            for (int rr = 0; rr < VPW; ++rr) {
                                const int rid = __shfl_sync(0xffffffffu, row_id, rr);
                                const __nv_bfloat16* src = p.kv + (int64_t)(rid < 0 ? 0 : rid) * p.kv_ss + (nh * 32 + lane) * 8;
                                cp_async16_zfill(dst0 + rr * 128 + ((c ^ (rr & 7)) << 4), src, rid < 0 ? 0u : 16u);
                            }
                            cp_async_arrive_noinc(smem_addr(&sm.kv_full[slot]));
                        }
                    }
                }
            }
        }
    } else if (MODE == MODE_SPARSE_DECODE && warp >= W::FIRST_CONVERT) {
        regs_dec<64>();
        // ---------------- FP8 decode: these 256 threads de-quantise the raw records in place ---------------------------
        const int ct = threadIdx.x - W::FIRST_CONVERT * 32;
        uint32_t g = 0, ks = 0;
        if (cta_rank == 0) {
            // K groups: two threads per token row, every other 16-value piece each
            const int r = ct & 127, half = ct >> 7, sw = r & 7;
            for (WalkerT wk(p, part); wk.valid(); wk.next()) {
                const Work w = wk.get();
                for (int i = 0; i < w.ntiles; ++i, ++g) {
                    float4 sc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
                    for (int grp = 0; grp < 3; ++grp) {
                        WAIT_WARP_OR_LEAVE(wt, false, &sm.raw_full[grp], g & 1, 205);
                        // the tile's scales were stored (and fenced) by the gather warps before they issued its first copies
                        if (grp == 0) sc = reinterpret_cast<const float4*>(sm.data + L::SC_SCALES)[(g & 1) * ROWS + r];
                        // group 2: chunks 6, 7 and the RoPE chunk (copied as it is); 512-wide form: chunk 6, the RoPE chunk and zeros
                        const int nconv = grp < 2 ? 3 : (M1 ? 1 : 2);
#pragma unroll 1
                        for (int cj = 0; cj < nconv; ++cj) {
                            const int j = grp * 3 + cj, sg = j >> 1;
                            uint8_t* rowp = sm.data + L::SC_KRING + j * K_CHUNK_BYTES + r * 128;
                            // one fp32 scale per two chunks, or one e8m0 exponent byte per chunk (byte j of the first two words)
                            const float scale = M1 ? e8m0_to_float((__float_as_uint(j < 4 ? sc.x : sc.y) >> (8 * (j & 3))) & 0xffu)
                                                   : (sg == 0 ? sc.x : sg == 1 ? sc.y : sg == 2 ? sc.z : sc.w);
                            uint4 raw[2];
#pragma unroll
                            for (int k2 = 0; k2 < 2; ++k2) raw[k2] = *reinterpret_cast<const uint4*>(rowp + (((2 * (half + 2 * k2) + 1) ^ sw) << 4));
#pragma unroll
                            for (int k2 = 0; k2 < 2; ++k2) {
                                const int k = half + 2 * k2;
                                uint4 lo, hi;
                                dequant16(raw[k2], scale, lo, hi);
                                *reinterpret_cast<uint4*>(rowp + (((2 * k) ^ sw) << 4)) = lo;
                                *reinterpret_cast<uint4*>(rowp + (((2 * k + 1) ^ sw) << 4)) = hi;
                            }
                        }
                        if (M1 && grp == 2) {
                            // the ninth chunk of a 512-wide row does not exist: zeros (this thread's half of the token's row)
                            uint8_t* row8 = sm.data + L::SC_KRING + 8 * K_CHUNK_BYTES + r * 128;
#pragma unroll
                            for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(row8 + (((half * 4 + k) ^ sw) << 4)) = make_uint4(0, 0, 0, 0);
                        }
                        fence_proxy_async_smem();          // generic-proxy stores -> visible to the tensor core's reads
                        mbar_arrive(smem_addr(&sm.kv_full[grp]));
                    }
                }
            }
        } else {
            // V slots: thread = (token row of the page, chunk of the slot).  It looks up its token's record by itself, one
            // page ahead, for the scales it needs; the raw pieces were copied by the gather warpgroup.
            const int trow = ct & 63, box = ct >> 6, sw = trow & 7;
            const int tq = blockIdx.y;
            for (WalkerT wk(p, part); wk.valid(); wk.next()) {
                const Work w = wk.get();
                const int* idx0 = p.sidx[0] + (int64_t)w.req * p.sidx_sb[0] + (int64_t)tq * p.sidx_ss[0];
                const int* idx1 = p.stopk[1] ? p.sidx[1] + (int64_t)w.req * p.sidx_sb[1] + (int64_t)tq * p.sidx_ss[1] : nullptr;
                auto load_id = [&](int blk) -> int {
                    if (blk >= w.blk_end) return -1;
                    const int scope = blk >= w.nblk0 ? 1 : 0;
                    const int pos = (scope ? blk - w.nblk0 : blk) * PAGE + trow;
                    if (pos >= (scope ? w.len1 : w.len0)) return -1;
                    return __ldg((scope ? idx1 : idx0) + pos);
                };
                // the scales of this thread's chunk in the two halves of the page: x of dims 0..255, y of dims 256..511 (512-wide
                // form: the record's eight exponent bytes)
                auto scales_of_id = [&](int blk, int id) -> float2 {
                    const int scope = blk >= w.nblk0 ? 1 : 0;
                    const int pbs = p.pbs[scope];
                    if (id < 0 || (int64_t)id >= (int64_t)p.nblocks[scope] * pbs) return make_float2(0.f, 0.f);
                    const uint8_t* block = p.kvb[scope] + (int64_t)(id / pbs) * p.kvb_sblock[scope];
                    if (M1) return __ldg(reinterpret_cast<const float2*>(block + (int64_t)pbs * 576 + (int64_t)(id % pbs) * 8));
                    const float* sc = reinterpret_cast<const float*>(block + (int64_t)(id % pbs) * 656 + 512);
                    return make_float2(__ldg(sc + (box >> 1)), __ldg(sc + 2 + (box >> 1)));
                };
                float2 sc_next = scales_of_id(w.blk_begin, load_id(w.blk_begin));
                int id_next = load_id(w.blk_begin + 1);
                for (int i = 0; i < w.ntiles; ++i) {
#pragma unroll 1
                    for (int h = 0; h < 2; ++h) {
                        const float2 sc = sc_next;
                        const int nblk = w.blk_begin + 2 * i + h + 1;
                        sc_next = scales_of_id(nblk, id_next);
                        id_next = load_id(nblk + 1);
#pragma unroll 1
                        for (int nh = 0; nh < 2; ++nh, ++ks) {
                            const uint32_t slot = ks % NVS;
                            WAIT_WARP_OR_LEAVE(wt, false, &sm.raw_full[slot], (ks / NVS) & 1, 206);
                            // (512-wide form: one exponent byte per chunk; chunk 7 is the RoPE part, copied as it is)
                            if (!(M1 && nh == 1 && box == 3)) {
                                const float scale = M1 ? e8m0_to_float((__float_as_uint(nh ? sc.y : sc.x) >> (8 * box)) & 0xffu) : (nh ? sc.y : sc.x);
                                uint8_t* rowp = sm.data + VA_VRING + slot * V_SLOT_BYTES + box * BOX_BYTES + trow * 128;
                                uint4 raw[4];
#pragma unroll
                                for (int k = 0; k < 4; ++k) raw[k] = *reinterpret_cast<const uint4*>(rowp + (((2 * k + 1) ^ sw) << 4));
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    uint4 lo, hi;
                                    dequant16(raw[k], scale, lo, hi);
                                    *reinterpret_cast<uint4*>(rowp + (((2 * k) ^ sw) << 4)) = lo;
                                    *reinterpret_cast<uint4*>(rowp + (((2 * k + 1) ^ sw) << 4)) = hi;
                                }
                            }
                            fence_proxy_async_smem();              // generic-proxy stores -> visible to the tensor core's reads
                            mbar_arrive(smem_addr(&sm.kv_full[slot]));
                        }
                    }
                }
            }
        }
    } else {
        if (MODE == MODE_PREFILL) regs_inc<136>();
        if (MODE == MODE_SPARSE_DECODE) regs_inc<112>();
        const int wq = warp & 3;                                  // TMEM lane quarter of this warp
        const int half = (warp - 4) >> 2;                         // score CTA: page of the tile this warpgroup owns
        const int r = wq * 32 + lane;                             // row inside the block = TMEM lane
        const uint32_t tlane = tmem + ((uint32_t)(wq * 32) << 16);
        const int row = row_blk * ROWS + r;                       // row inside the (request, kv head) group
        const bool row_ok = row < p.rows;
        // dense: rows are (query token, head of the kv group); sparse decode: the CTA pair serves one query token
        const int t = MODE == MODE_SPARSE_DECODE ? (int)blockIdx.y : (row_ok ? row / p.g : 0);
        const int hd = MODE == MODE_SPARSE_DECODE ? (row_ok ? row : 0) : hk * p.g + (row_ok ? row - t * p.g : 0);
        uint32_t g = 0, nreq = 0;

        if (cta_rank == 0) {
            // ---------------- softmax warpgroups of the score CTA --------------------------------------------
            // These 256 threads meet at a named barrier every tile, so none of them may leave alone: a thread whose
            // wait ran out keeps walking (its later waits return at once, it arrives nowhere and stores nothing
            // outside its own staging) until the next such barrier, which carries the flag to everyone (bar.red.or);
            // behind it all 256 leave together.
            uint8_t* stage = sm.data + L::SC_STAGE + (half * 4 + wq) * 4096;
            float* side_src = reinterpret_cast<float*>(sm.data + L::SC_SIDE + wq * SIDE_BYTES);
            float* xmax = reinterpret_cast<float*>(sm.data + L::SC_XMAX);
            const uint32_t remote_fin = map_to_cta(smem_addr(sm.data + VA_FIN), 1) + (uint32_t)r * 4u;
            const uint32_t remote_fin_full = map_to_cta(smem_addr(&sm.fin_full), 1);
            for (WalkerT wk(p, part); wk.valid(); wk.next(), ++nreq) {
                const Work w = wk.get();
                // ---- Q row -> A operand: chunks [0, Q_TMEM_CHUNKS) to tensor memory (2 x 16 bit per 32-bit column), in the
                // gather modes chunks 7, 8 to shared memory (K-major, 128-byte swizzle).  Warpgroup 0 takes chunks
                // [0, Q_SPLIT) (and 7), warpgroup 1 the others (and 8).
                // Every MMA that read the previous request's Q has completed: this thread saw s_full of its last tile.
                {
                    const __nv_bfloat16* qrow = MODE == MODE_PREFILL
                        ? p.q + (int64_t)w.req * p.q_ss + (int64_t)hd * p.q_sh
                        : p.q + (int64_t)w.req * p.q_sb + (int64_t)t * p.q_ss + (int64_t)hd * p.q_sh;
                    const int c_begin = half ? L::Q_SPLIT : 0, c_end = half ? L::Q_TMEM_CHUNKS : L::Q_SPLIT;
                    if (p.q_tma) {
                        // Q arrived as TMA boxes: in the gather modes chunks 7 and 8 are in place; the others wait in the K
                        // ring as [row][128 B] with the 128-byte swizzle
                        wt.template wait<false>(&sm.q_landed, nreq & 1, 12);
#pragma unroll 1
                        for (int c = c_begin; c < c_end; ++c) {
                            const uint8_t* qsrc = sm.data + L::SC_KRING + c * 16384 + r * 128;
                            uint32_t v[32];
#pragma unroll
                            for (int ch = 0; ch < 8; ++ch) {
                                const uint4 x = *reinterpret_cast<const uint4*>(qsrc + ((ch ^ (r & 7)) << 4));
                                v[4 * ch] = x.x; v[4 * ch + 1] = x.y; v[4 * ch + 2] = x.z; v[4 * ch + 3] = x.w;
                            }
                            tmem_st32(tlane + L::TM_Q + c * 32, v);
                        }
                        tmem_wait_st();
                        if (!wt.expired()) mbar_arrive(smem_addr(&sm.ring_released));        // the producers may fill the ring with K now
                    } else {
                        load_q_by_threads<MODE>(sm, qrow, row_ok, half, r, tlane, NO_CHUNK8);
                    }
                    tmem_wait_st();
                    fence_proxy_async_smem();
                    tc_fence_before();
                    if (!wt.expired()) mbar_arrive(smem_addr(&sm.q_ready));
                }
                // first key position this row must NOT see (causal limit, and the end of this partition's range)
                const int limit = min(p.causal ? w.seqlen - (p.s_q - 1 - t) : w.seqlen, w.blk_end * PAGE);
                float m_run = -INFINITY, l_run = 0.f, m_true = -INFINITY;
                for (int i = 0; i < w.ntiles; ++i, ++g) {
                    const uint32_t sb = L::S_BUFS == 2 ? (g & 1) : 0;
                    const uint32_t ph = L::S_BUFS == 2 ? ((g >> 1) & 1) : (g & 1);
                    wt.template wait<false>(&sm.s_full[sb], ph, 5);
                    tc_fence_after();
                    uint32_t s[64];
                    {
                        uint32_t (&lo)[32] = *reinterpret_cast<uint32_t (*)[32]>(&s[0]);
                        uint32_t (&hi)[32] = *reinterpret_cast<uint32_t (*)[32]>(&s[32]);
                        tmem_ld32(tlane + L::TM_S + sb * 128 + half * 64, lo);
                        tmem_ld32(tlane + L::TM_S + sb * 128 + half * 64 + 32, hi);
                    }
                    // Validity bits of the gathered tokens: token 32w + l of the tile is bit l of word w.  They are read before the
                    // arrival below: through the MMAs of tile g + 2, which wait for it, it is all that keeps the copy warps
                    // from writing tile g + 4's bits over these.
                    uint32_t m0 = 0xffffffffu, m1 = 0xffffffffu;
                    if (!DENSE) {
                        const uint32_t* km = reinterpret_cast<const uint32_t*>(sm.data + L::SC_MASK) + (g & 3) * 4 + half * 2;
                        m0 = km[0];
                        m1 = km[1];
                    }
                    tmem_wait_ld();
                    tc_fence_before();
                    if (!wt.expired()) mbar_arrive(smem_addr(&sm.s_empty[sb]));            // the MMA warp may overwrite this S accumulator

                    if (!DENSE) {
                        if ((m0 & m1) != 0xffffffffu) {
#pragma unroll
                            for (int c = 0; c < 64; ++c)
                                if (!(((c < 32 ? m0 : m1) >> (c & 31)) & 1u)) s[c] = 0xff800000u;      // -inf
                        }
                    } else {
                        const int nvalid = limit - (w.blk_begin + 2 * i + half) * PAGE;   // columns [0, nvalid) are visible
                        if (nvalid < PAGE) {
#pragma unroll
                            for (int c = 0; c < 64; ++c)
                                if (c >= nvalid) s[c] = 0xff800000u;          // -inf
                        }
                    }
                    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
                    for (int c = 0; c < 64; c += 2) {
                        mx0 = fmaxf(mx0, __uint_as_float(s[c]));
                        mx1 = fmaxf(mx1, __uint_as_float(s[c + 1]));
                    }
                    float mx = fmaxf(mx0, mx1);
                    // the row maximum over both pages of the tile; the barrier also carries the abort flag
                    xmax[((g & 1) * 2 + half) * ROWS + r] = mx;
                    BAR_OR_LEAVE(wt.expired());
                    mx = fmaxf(mx, xmax[((g & 1) * 2 + (half ^ 1)) * ROWS + r]);
                    mx *= p.scale_log2;                                // scale > 0: max commutes with scaling
                    m_true = fmaxf(m_true, mx);
                    float factor = 1.f;
                    bool resc = false;
                    if (i == 0) {
                        m_run = mx;
                    } else if (mx > m_run + RESCALE_THRESHOLD) {
                        factor = ex2(m_run - mx);                      // m_run = -inf -> 0
                        l_run *= factor;
                        m_run = mx;
                        resc = true;
                    }
                    const float neg_m = m_run == -INFINITY ? 0.f : -m_run;
                    uint32_t pk[32];
                    float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
                    for (int c = 0; c < 64; c += 2) {
                        const float e0 = ex2(fmaf(__uint_as_float(s[c]), p.scale_log2, neg_m));
                        const float e1 = ex2(fmaf(__uint_as_float(s[c + 1]), p.scale_log2, neg_m));
                        sum0 += e0; sum1 += e1;
                        pk[c >> 1] = pack16<FP16>(e0, e1);
                    }
                    l_run += sum0 + sum1;
                    const bool any_resc = __any_sync(0xffffffffu, resc);

                    // staging of this warp is free once the previous tile's copy has landed in the value CTA
                    wt.template wait<true>(&sm.stage_free[half], (g & 1) ^ 1, 8);
                    if (!wt.expired()) {
                        uint8_t* prow = stage + (lane >> 3) * 1024 + (lane & 7) * 128;
#pragma unroll
                        for (int ch = 0; ch < 8; ++ch)
                            *reinterpret_cast<uint4*>(prow + ((ch ^ (lane & 7)) << 4)) = make_uint4(pk[4 * ch], pk[4 * ch + 1], pk[4 * ch + 2], pk[4 * ch + 3]);
                        if (half == 0) {
                            side_src[lane] = factor;
                            if (lane == 0) reinterpret_cast<uint32_t*>(side_src)[32] = any_resc ? 1u : 0u;
                        }
                        fence_proxy_async_smem();                          // staging is read by the bulk-copy engine
                        mbar_arrive(smem_addr(&sm.stage_full[half]));      // the sender warp pushes it to the value CTA
                    }
                }
                // final statistics of this request for the epilogue in the value CTA: warpgroup 1 hands its row sums to
                // warpgroup 0, which sends sum, running maximum and true maximum.  (The wide plan has no spare shared memory:
                // the hand-over uses the row-maximum slots of the tile parity that is not in use.)
                {
                    float* lsum = L::WIDE ? xmax + ((g & 1) * 2) * ROWS : reinterpret_cast<float*>(sm.data + L::SC_LSUM);
                    if (half == 1) lsum[r] = l_run;
                    BAR_OR_LEAVE(wt.expired());
                    if (half == 0) l_run += lsum[r];
                    BAR_OR_LEAVE(wt.expired());
                }
                if (half == 0) {
                    wt.template wait<true>(&sm.fin_empty, (nreq & 1) ^ 1, 7);
                    if (!wt.expired()) {
                        st_cluster_f32(remote_fin, l_run);
                        st_cluster_f32(remote_fin + ROWS * 4, m_run);
                        st_cluster_f32(remote_fin + 2 * ROWS * 4, m_true);
                        mbar_arrive_remote(remote_fin_full);
                    }
                }
            }
        } else if (warp < 8) {
            // ---------------- correction / epilogue warpgroup of the value CTA ---------------------------------
            const uint32_t remote_fin_empty = map_to_cta(smem_addr(&sm.fin_empty), 0);
            const uint32_t remote_stage_free0 = map_to_cta(smem_addr(&sm.stage_free[0]), 0);
            const uint32_t remote_stage_free1 = map_to_cta(smem_addr(&sm.stage_free[1]), 0);
            const float* fin = reinterpret_cast<const float*>(sm.data + VA_FIN);
            uint32_t vs = 0;                                          // V ring slot counter
            // 16-bit output rows start on 32-byte boundaries: 256-bit stores may be used (decode modes; measured in one run
            // against 16-byte stores: dense 0.2134 -> 0.2088 ms, FP8 decode 0.1107 -> 0.1090 ms, prefill 3.348 -> 3.379 ms,
            // so prefill keeps the 16-byte stores)
            const bool wide_out = MODE != MODE_PREFILL && (reinterpret_cast<uintptr_t>(p.out) & 31) == 0 &&
                                  ((p.o_sb | p.o_ss | p.o_sh) & 15) == 0;
            for (WalkerT wk(p, part); wk.valid(); wk.next(), ++nreq) {
                const Work w = wk.get();
                for (int i = 0; i < w.ntiles; ++i, ++g) {
                    for (int h = 0; h < 2; ++h, vs += 2) {
                        const uint32_t pb = (g & 1) * 2 + h, ph = (g >> 1) & 1;
                        WAIT_WARP_OR_LEAVE(wt, true, &sm.p_full[pb], ph, 107);
                        if (threadIdx.x == 128) {
                            mbar_arrive_remote_relaxed(h ? remote_stage_free1 : remote_stage_free0);   // the copy has landed
                        }
                        if (h == 0 && i > 0) {
                            const float* side = reinterpret_cast<const float*>(sm.data + VA_SIDE + ((g & 1) * 4 + wq) * SIDE_BYTES);
                            const bool need = reinterpret_cast<const uint32_t*>(side)[32] != 0;    // warp-uniform
                            if (need) {
                                // every earlier PV MMA has finished before O is touched
                                WAIT_WARP_OR_LEAVE(wt, false, &sm.pv_done[((g - 1) & 1) * 2 + 1], ((g - 1) >> 1) & 1, 108);
                                tc_fence_after();
                                rescale_o_rows(tlane, side[lane]);
                            }
                        }
                        // Tokens at or beyond the sequence length may hold anything (NaN included) in a real page:
                        // their probabilities are zero, so their V rows are zeroed to keep 0 * NaN out of O.
                        const int blk = w.blk_begin + 2 * i + h;
                        const int nvalid = w.seqlen - blk * PAGE;
                        if (DENSE && blk < w.blk_end && nvalid < PAGE) {
                            const int first = max(nvalid, 0);
                            for (int nh = 0; nh < 2; ++nh) {
                                const uint32_t slot = (vs + nh) % NVS;
                                WAIT_WARP_OR_LEAVE(wt, false, &sm.kv_full[slot], ((vs + nh) / NVS) & 1, 109);
                                zero_v_rows(sm.data + VA_VRING + slot * V_SLOT_BYTES, first);
                            }
                            fence_proxy_async_smem();
                        }
                        tc_fence_before();
                        mbar_arrive(smem_addr(&sm.corr_done[pb]));
                    }
                }
                // ---- epilogue -----------------------------------------------------------------------------------
                const bool has_tiles = w.ntiles > 0;
                if (has_tiles) WAIT_WARP_OR_LEAVE(wt, false, &sm.pv_done[((g - 1) & 1) * 2 + 1], ((g - 1) >> 1) & 1, 110);
                WAIT_WARP_OR_LEAVE(wt, true, &sm.fin_full, nreq & 1, 111);
                tc_fence_after();
                const float Lsum = fin[r], M = fin[ROWS + r];
                const bool empty = !(Lsum > 0.f) || !has_tiles;          // also catches NaN
                float scale = empty ? 0.f : 1.f / Lsum;
                if (!DENSE && !w.is_split && p.attn_sink && !empty && row_ok)
                    scale = 1.f / (Lsum + exp2f(p.attn_sink[hd] * kLog2e - M));
                if (!w.is_split) {
                    __nv_bfloat16* orow = MODE == MODE_PREFILL
                        ? p.out + ((int64_t)w.req * p.h_q + hd) * D_V
                        : p.out + (int64_t)w.req * p.o_sb + (int64_t)t * p.o_ss + (int64_t)hd * p.o_sh;
#pragma unroll 1
                    for (int c = 0; c < D_V / 32; ++c) {
                        uint32_t v[32];
                        if (has_tiles) { tmem_ld32(tlane + c * 32, v); tmem_wait_ld(); }
                        if (row_ok) {
                            uint32_t o[16];
#pragma unroll
                            for (int e = 0; e < 16; ++e)
                                o[e] = empty ? 0u : pack16<FP16>(__uint_as_float(v[2 * e]) * scale, __uint_as_float(v[2 * e + 1]) * scale);
                            if (wide_out) {                   // whole 32-byte sectors per store
                                st_global_v8(orow + c * 32, o[0], o[1], o[2], o[3], o[4], o[5], o[6], o[7]);
                                st_global_v8(orow + c * 32 + 16, o[8], o[9], o[10], o[11], o[12], o[13], o[14], o[15]);
                            } else {
#pragma unroll
                                for (int k = 0; k < 4; ++k)
                                    *reinterpret_cast<uint4*>(orow + c * 32 + k * 8) = make_uint4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
                            }
                        }
                    }
                    if (row_ok) {
                        const float lse_nat = empty ? INFINITY : (log2f(Lsum) + M) * kLn2;
                        if (MODE == MODE_PREFILL) {
                            p.lse[(int64_t)w.req * p.h_q + hd] = lse_nat;
                            p.max_logits[(int64_t)w.req * p.h_q + hd] = empty ? -INFINITY : fin[2 * ROWS + r] * kLn2;
                        } else {
                            p.lse[w.req * p.l_sb + t * p.l_ss + hd * p.l_sh] = lse_nat;
                        }
                    }
                } else if (DENSE && MLA_TAIL_BULK && w.last && has_tiles) {
                    // The partition's last partial: the V ring is idle by now, so every thread stages its row there, half a
                    // row (1 KiB) at a time, and hands it to the bulk-copy engine as one piece.  Stores by the thread itself
                    // (one lane per row, 32 bytes per instruction) keep the load/store unit busy for 8 us per 256 KiB.
                    const int64_t arow = ((int64_t)w.slot * p.s_q + t) * p.h_q + hd;
                    float* orow = p.o_accum + arow * D_V;
                    uint8_t* rowbuf = sm.data + VA_VRING + r * 1040;          // 1040: rows 16 bytes apart in the banks
#pragma unroll 1
                    for (int hf = 0; hf < 2; ++hf) {
                        if (hf) bulk_wait_group_read0();
#pragma unroll 1
                        for (int c = 0; c < 8; ++c) {
                            uint32_t v[32];
                            tmem_ld32(tlane + hf * 256 + c * 32, v);
                            tmem_wait_ld();
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                *reinterpret_cast<uint4*>(rowbuf + c * 128 + k * 16) =
                                    make_uint4(empty ? 0u : __float_as_uint(__uint_as_float(v[4 * k]) * scale),
                                               empty ? 0u : __float_as_uint(__uint_as_float(v[4 * k + 1]) * scale),
                                               empty ? 0u : __float_as_uint(__uint_as_float(v[4 * k + 2]) * scale),
                                               empty ? 0u : __float_as_uint(__uint_as_float(v[4 * k + 3]) * scale));
                        }
                        fence_proxy_async_smem();
                        if (row_ok) bulk_store_to_global(orow + hf * 256, smem_addr(rowbuf), 1024);
                        bulk_commit_group();
                    }
                    if (row_ok) p.lse_accum[arow] = empty ? -INFINITY : log2f(Lsum) + M;
                    bulk_wait_group0();
                } else {
                    const int64_t arow = ((int64_t)w.slot * p.s_q + t) * p.h_q + hd;
                    float* orow = p.o_accum + arow * D_V;
#pragma unroll 1
                    for (int c = 0; c < D_V / 32; ++c) {
                        uint32_t v[32];
                        if (has_tiles) { tmem_ld32(tlane + c * 32, v); tmem_wait_ld(); }
                        if (row_ok) {
                            // whole 32-byte sectors per store: each thread writes its own row, so a 16-byte store would
                            // send half-filled sectors and twice the instructions through the load/store unit
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                uint32_t o[8];
#pragma unroll
                                for (int e = 0; e < 8; ++e) o[e] = empty ? 0u : __float_as_uint(__uint_as_float(v[8 * k + e]) * scale);
                                st_global_v8(orow + c * 32 + k * 8, o[0], o[1], o[2], o[3], o[4], o[5], o[6], o[7]);
                            }
                        }
                    }
                    if (row_ok) p.lse_accum[arow] = empty ? -INFINITY : log2f(Lsum) + M;
                }
                tc_fence_before();
                mbar_arrive_remote(remote_fin_empty);        // the final statistics may be rewritten
            }
        }
    }

wind_down:
    if (wt.expired()) report_expired_wait(p.status, &sm.aborted, map_to_cta(smem_addr(&sm.aborted), cta_rank ^ 1u), wt.code);
    // ---- wind down: both CTAs leave together, tensor memory is released -----------------------------------
    if (!DENSE && warp >= 12) cp_async_wait_all();          // this thread's own row copies have landed
    tc_fence_before();
    if (__syncthreads_or((int)*reinterpret_cast<volatile uint32_t*>(&sm.aborted))) {
        // A bounded wait ran out in this CTA or in its peer; every thread of this CTA has left its role and issues
        // nothing more.  Wait - bounded again - for what this CTA still has in flight: its MMAs (they read shared memory
        // and write tensor memory) and the TMA loads into its rings.
        if (warp == 1 && elect_one()) {
            tc_commit(smem_addr(&sm.drain));
            mbar_wait_bounded(smem_addr(&sm.drain), 0, DRAIN_LIMIT);
        }
        if (threadIdx.x == 0) {
            if (DENSE) {
                const uint32_t nslots = cta_rank == 0 ? (uint32_t)NKS : (uint32_t)NVS;
                for (uint32_t back = 1; back <= nslots && back <= fills_armed; ++back) {
                    const uint32_t f = fills_armed - back;     // one of the last fills this thread armed: its slot has seen no later phase
                    mbar_wait_bounded(smem_addr(&sm.kv_full[f % nslots]), (f / nslots) & 1, DRAIN_LIMIT);
                }
            }
            if (q_armed) mbar_wait_bounded(smem_addr(&sm.q_landed), (q_armed - 1) & 1, DRAIN_LIMIT);
        }
    }
    cluster_sync();                                            // from here on neither CTA starts anything
    if (__syncthreads_or((int)*reinterpret_cast<volatile uint32_t*>(&sm.aborted))) {
        // copies from the peer's shared memory into this one (P pages, final statistics) that were still under way
        const long long t0 = clock64();
        while (clock64() - t0 < SETTLE_CYCLES) { }
    }
    cluster_sync();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// ---- self-test of the bounded wait: one CTA, one barrier nobody arrives on ---------------------------------
// Uses the same Waiter and the same reporting as the attention kernels, with nothing in flight (no TMA, no MMA, no
// cluster): the wait runs into its limit, the status words are written, the kernel returns normally.
__global__ void bounded_wait_selftest_kernel(int* status, uint32_t limit, int code, int* flag_out) {
    __shared__ uint64_t bar;
    __shared__ uint32_t flag;
    if (threadIdx.x == 0) { mbar_init(smem_addr(&bar), 1); flag = 0; fence_mbar_init(); }
    __syncthreads();
    Waiter w(limit);
    bool ok = threadIdx.x < 32 ? w.wait<false>(&bar, 0, code) : w.wait_warp<false>(&bar, 0, code);
    // a second wait by the same thread returns at once
    if (threadIdx.x < 32) ok = w.wait<false>(&bar, 0, code + 1) || ok;
    if (w.expired()) report_expired_wait(status, &flag, 0u, w.code);
    __syncthreads();
    if (threadIdx.x == 0 && flag_out) { flag_out[0] = (int)flag; flag_out[1] = ok ? 1 : 0; }
}

}  // namespace sm100

int launch_bounded_wait_selftest(long long limit_cycles, int code, int* status, int* flag_out, void* stream) {
    MLA_CHECK_ARG(limit_cycles > 0 && limit_cycles <= 2000000000LL, "mla_selftest_bounded_wait: limit_cycles must be in (0, 2e9]");
    MLA_CHECK_ARG(status != nullptr, "mla_selftest_bounded_wait: status must not be null");
    sm100::bounded_wait_selftest_kernel<<<1, 64, 0, (cudaStream_t)stream>>>(status, wait_units(limit_cycles), code, flag_out);
    MLA_CHECK_CUDA(cudaGetLastError());
    return MLA_OK;
}

bool dense_decode_sm100_supports(const mla_dense_decode_args_t& a) {
    if (a.d_qk != 576 || a.d_v != 512 || a.page_block_size != 64) return false;
    if (a.h_kv <= 0 || a.h_q % a.h_kv != 0) return false;
    // TMA: strides in bytes must be multiples of 16 and below 2^40
    const int64_t lim = (int64_t)1 << 39;
    if (a.k_stride_block <= 0 || a.k_stride_row <= 0 || a.k_stride_head <= 0) return false;
    if (a.k_stride_block >= lim || a.k_stride_row >= lim || a.k_stride_head >= lim) return false;
    if (a.k_stride_block % 8 || a.k_stride_row % 8 || a.k_stride_head % 8) return false;
    // the kv heads of a row are addressed as 64-column chunks of one tensor-map dimension
    if (a.h_kv > 1 && a.k_stride_head % 64) return false;
    const int rows = a.s_q * (a.h_q / a.h_kv);
    const int64_t row_blocks = (rows + 127) / 128;
    if (row_blocks * a.h_kv > 65535 || a.num_sm_parts > 65535) return false;
    if (!(a.softmax_scale > 0.f)) return false;       // the row maximum is taken before scaling
    if (reinterpret_cast<uintptr_t>(a.o_accum) & 31) return false;      // split partials leave with 256-bit stores
    return true;
}

// The two cache tensor maps of a dense launch depend only on the cache tensor (pointer, strides, pages, heads, type):
// a decode loop calls with the same cache every step, so the last encoding is kept per host thread.
struct CacheMaps {
    const void* k_cache = nullptr;
    int64_t sb = 0, sr = 0, sh = 0;
    int num_blocks = 0, h_kv = 0, fp16 = 0;
    CUtensorMap kmap, vmap;
};

int launch_dense_decode_sm100(const mla_dense_decode_args_t& a) {
    using namespace sm100;
    EncodeTiledFn encode = get_encode_fn();
    if (!encode) return set_error(MLA_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const bool fp16 = a.dtype == MLA_DTYPE_FP16;

    // The cache as a 5-D tensor (64 columns of a chunk, 8 tokens, chunks, 8 token groups, pages): one box brings
    // all 64 tokens of a page for 3 (K) or 4 (V) chunks in a single instruction, and lands as
    // [token group][chunk][8 rows x 128 B] - 1 KiB swizzle atoms that the MMA descriptors walk with a stride of
    // 3 or 4 KiB between token groups.  (The per-instruction cost of TMA is what limits one SM's fill rate: 8 KiB
    // boxes stream at 35-45 GB/s per SM, 24 KiB boxes at about 90.)
    const int head_chunks = a.h_kv > 1 ? (int)(a.k_stride_head / 64) : 9;
    static thread_local CacheMaps cm;
    if (cm.k_cache != a.k_cache || cm.sb != a.k_stride_block || cm.sr != a.k_stride_row || cm.sh != a.k_stride_head ||
        cm.num_blocks != a.num_blocks || cm.h_kv != a.h_kv || cm.fp16 != (int)fp16) {
        cm.k_cache = nullptr;
        const CUtensorMapDataType dt = fp16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
        cuuint64_t dims[5] = {64, 8, (cuuint64_t)((a.h_kv - 1) * head_chunks + 9), 8, (cuuint64_t)a.num_blocks};
        cuuint64_t strides[4] = {(cuuint64_t)a.k_stride_row * 2, 128, (cuuint64_t)a.k_stride_row * 16, (cuuint64_t)a.k_stride_block * 2};
        cuuint32_t estr[5] = {1, 1, 1, 1, 1};
        cuuint32_t kbox[5] = {64, 8, 3, 8, 1};
        cuuint32_t vbox[5] = {64, 8, 4, 8, 1};
        CUresult r = encode(&cm.kmap, dt, 5, const_cast<void*>(a.k_cache), dims, strides, kbox, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r == CUDA_SUCCESS)
            r = encode(&cm.vmap, dt, 5, const_cast<void*>(a.k_cache), dims, strides, vbox, estr,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return set_error(MLA_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
        cm.k_cache = a.k_cache; cm.sb = a.k_stride_block; cm.sr = a.k_stride_row; cm.sh = a.k_stride_head;
        cm.num_blocks = a.num_blocks; cm.h_kv = a.h_kv; cm.fp16 = (int)fp16;
    }

    Params p = dense_params(a, head_chunks);
    p.row_blocks = (p.rows + ROWS - 1) / ROWS;
    CUtensorMap qmap;
    memset(&qmap, 0, sizeof(qmap));
    if (p.row_blocks == 1 || ROWS % p.g == 0)
        p.q_tma = encode_q_map(&qmap, a.q, a.b, a.s_q, a.h_q, a.q_stride_b, a.q_stride_s, a.q_stride_h, p.g,
                               p.row_blocks == 1 ? a.s_q : ROWS / p.g, &p.q_box_bytes, fp16) ? 1 : 0;

    dim3 grid(2, p.row_blocks * a.h_kv, a.num_sm_parts);
    if (fp16) {
        static bool configured[64] = {};
        if (int rc = configure_once(attn_sm100_kernel<MODE_DENSE, true>, configured, sizeof(Smem))) return rc;
        MLA_CHECK_CUDA(launch_dependent(attn_sm100_kernel<MODE_DENSE, true>, grid, dim3(NTHREADS), sizeof(Smem), (cudaStream_t)a.stream, cm.kmap, cm.vmap, qmap, p));
    } else {
        static bool configured[64] = {};
        if (int rc = configure_once(attn_sm100_kernel<MODE_DENSE, false>, configured, sizeof(Smem))) return rc;
        MLA_CHECK_CUDA(launch_dependent(attn_sm100_kernel<MODE_DENSE, false>, grid, dim3(NTHREADS), sizeof(Smem), (cudaStream_t)a.stream, cm.kmap, cm.vmap, qmap, p));
    }
    MLA_CHECK_CUDA(cudaGetLastError());
    return MLA_OK;
}

bool sparse_prefill_sm100_supports(const mla_sparse_prefill_args_t& a) {
    if ((a.d_qk != 576 && a.d_qk != 512) || a.d_v != 512 || a.h_kv != 1) return false;
    if (a.kv_stride_s <= 0 || a.kv_stride_s % 8 || a.kv_stride_s >= ((int64_t)1 << 39)) return false;
    if (!(a.sm_scale > 0.f)) return false;
    if (a.h_q > 128 * 65535) return false;
    return true;
}

int launch_sparse_prefill_sm100(const mla_sparse_prefill_args_t& a) {
    using namespace sm100;
    CUtensorMap kmap;
    memset(&kmap, 0, sizeof(kmap));     // rows are gathered with cp.async by the kernel's own threads, no TMA descriptor

    Params p = prefill_params(a);
    p.row_blocks = (p.rows + ROWS - 1) / ROWS;

    const bool d512 = a.d_qk == 512;
    static bool configured[64] = {}, configured_512[64] = {};
    if (int rc = d512 ? configure_once(attn_sm100_kernel<MODE_PREFILL, true>, configured_512, sizeof(Smem))
                      : configure_once(attn_sm100_kernel<MODE_PREFILL, false>, configured, sizeof(Smem))) return rc;
    const int sms = current_device_num_sms();
    int pairs = sms / 2 / p.row_blocks;
    if (pairs < 1) pairs = 1;
    if (pairs > a.s_q) pairs = a.s_q;
    dim3 grid(2, p.row_blocks, pairs);
    CUtensorMap qmap;
    memset(&qmap, 0, sizeof(qmap));
    p.q_tma = encode_q_map(&qmap, a.q, 1, a.s_q, a.h_q, 0, a.q_stride_s, a.q_stride_h, a.h_q < ROWS ? a.h_q : ROWS, 1,
                           &p.q_box_bytes, false, a.d_qk) ? 1 : 0;
    if (d512)
        MLA_CHECK_CUDA(launch_dependent(attn_sm100_kernel<MODE_PREFILL, true>, grid, dim3(Warps<MODE_PREFILL>::THREADS), sizeof(Smem), (cudaStream_t)a.stream, kmap, kmap, qmap, p));
    else
        MLA_CHECK_CUDA(launch_dependent(attn_sm100_kernel<MODE_PREFILL, false>, grid, dim3(Warps<MODE_PREFILL>::THREADS), sizeof(Smem), (cudaStream_t)a.stream, kmap, kmap, qmap, p));
    MLA_CHECK_CUDA(cudaGetLastError());
    return MLA_OK;
}

bool sparse_decode_sm100_supports(const mla_sparse_decode_args_t& a) {
    if ((a.d_qk != 576 && a.d_qk != 512) || a.d_v != 512) return false;
    if (a.h_q > 128 || a.s_q > 65535 || a.num_sm_parts > 65535) return false;
    if (!(a.sm_scale > 0.f)) return false;
    if (reinterpret_cast<uintptr_t>(a.o_accum) & 31) return false;      // split partials leave with 256-bit stores
    return true;
}

int launch_sparse_decode_sm100(const mla_sparse_decode_args_t& a) {
    using namespace sm100;
    Params p = sparse_decode_params(a);
    p.row_blocks = 1;

    const bool m1 = a.d_qk == 512;                  // the 512-wide record form: the ninth chunk of Q and K is zeros
    static bool configured[64] = {}, configured_m1[64] = {};
    if (int rc = m1 ? configure_once(attn_sm100_kernel<MODE_SPARSE_DECODE, true>, configured_m1, sizeof(Smem))
                    : configure_once(attn_sm100_kernel<MODE_SPARSE_DECODE, false>, configured, sizeof(Smem))) return rc;
    CUtensorMap unused_map, qmap;
    memset(&unused_map, 0, sizeof(unused_map));     // this mode gathers K and V with its own threads
    memset(&qmap, 0, sizeof(qmap));
    p.q_tma = encode_q_map(&qmap, a.q, a.b, a.s_q, a.h_q, a.q_stride_b, a.q_stride_s, a.q_stride_h,
                           a.h_q < ROWS ? a.h_q : ROWS, 1, &p.q_box_bytes, false, a.d_qk) ? 1 : 0;
    dim3 grid(2, a.s_q, a.num_sm_parts);
    if (m1)
        MLA_CHECK_CUDA(launch_dependent(attn_sm100_kernel<MODE_SPARSE_DECODE, true>, grid, dim3(Warps<MODE_SPARSE_DECODE>::THREADS), sizeof(Smem), (cudaStream_t)a.stream, unused_map, unused_map, qmap, p));
    else
        MLA_CHECK_CUDA(launch_dependent(attn_sm100_kernel<MODE_SPARSE_DECODE, false>, grid, dim3(Warps<MODE_SPARSE_DECODE>::THREADS), sizeof(Smem), (cudaStream_t)a.stream, unused_map, unused_map, qmap, p));
    MLA_CHECK_CUDA(cudaGetLastError());
    return MLA_OK;
}

}  // namespace mla
