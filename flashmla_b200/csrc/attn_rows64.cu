// MLA attention for up to 64 query rows on ONE SM (sm_100a, tcgen05).  One kernel template serves
//   MODE_DENSE          dense BF16 / FP16 paged decode with at most 64 rows (query token x head) per kv head
//   MODE_PREFILL        token-sparse prefill with at most 64 heads
//   MODE_SPARSE_DECODE  sparse FP8 decode, a CTA per 64 heads
//
// With NH <= 64 rows everything about a request fits one SM when the products are taken TRANSPOSED:
//   S^T = K Q^T   [128 tokens x NH]   A = the tile's K rows (K-major),            B = Q (K-major)
//   O^T = V^T P^T [512 dims x NH]     A = the same bytes read along the dims      B = P (one row of NH values per token,
//                                     (MN-major), 4 blocks of 128 dims            MN-major)
// Both keep M = 128, O^T takes 4 x NH columns of tensor memory, and a KV tile enters the SM once and serves both products.
// The kernel for 128 rows (attn_pair.cu) needs a pair of SMs, because O[128 x 512] fills one SM's tensor memory, and brings
// 1.44 times a tile's bytes into the two of them.
//
// A tile is 128 tokens (two pages): four PAIRS of 64-dim chunks (dims 128 p .. 128 p + 127) in a ring of NP slots, and the
// RoPE chunk (576-wide rows) in a slot of its own.  Layout of a pair: [8-token group][chunk][8 rows x 128 B], 128-byte swizzle.
// Order of the MMAs: Q K^T over the pairs as they arrive, then P V block by block; block m reads pair m only, so the next
// tile's pairs move in while P V still runs.
//
// Where the ring holds more than a tile (dense, up to 32 rows), the next tile's first pair is multiplied during the softmax.
//
// Softmax: warps 4..11, a thread = one token (tensor-memory lane) and NH / 2 rows (columns).  A row's running maximum is shared
// by all threads and only has to bound the scores: it moves when a score exceeds it by 2^6 (always on a request's first
// tile), which is what the threads vote on once per tile; P, the row sums and O always refer to the same maximum, so results
// are exact up to rounding.  Sums stay per thread until the end of a request.
//
// What bounds it: one tile is in flight, so a tile's period is the chain  fill -> Q K^T (36 MMAs) -> softmax -> P V (32 MMAs); an
// MMA of 128 x NH x 16 takes what its operands take to be read, 40 SM cycles (NH = 16) to 49 (64).
// us a tile on all SMs at once (148 lists of two lengths, short runs of one input): dense, 16 / 32 / 64 rows 3.2 / 3.2 / 3.5, of which
// DRAM's rate asks for 3.3 (the fills come behind P V; the next tile's pages are prefetched into L2 while this one is worked on: a
// third longer with 64 rows without); prefill, 64 heads 3.35 (576-wide) and 2.95, copies and P V slowed by them; FP8, 64 heads 6.0 and
// 4.9, 16 heads 4.8 and 3.6, conversion and its loads two thirds of them.
// us a call, pairs of SMs for every shape (score and value CTAs, no longer here) -> now, inputs changing from call to call, clocks settled:
//   dense, 4 requests of 64..512, 16 heads     18.3 ->  13.1    dense fp16, 61 x 4096, 16 heads     95.9 ->  64.4
//   FP8, 2 x 2 x 2048, 64 heads, schedule too  26.2 ->  21.7    prefill 512-wide, 117 tokens, ragged 38.8 ->  30.6
// and with the issuing thread elected (elect_one, sm100_ptx.cuh) 13.4 -> 12.6, 63.8 -> 62.1, 22.1 -> 21.7 and
// 30.6 -> 24.4,
// and one input in short runs:
//   dense, 30 x 2048, 8 heads                  32.8 ->  23.7    dense, 61 x 4096, 32 / 64 heads     77 / 79.3 -> 68.7 / 78.0
//   FP8, 64 x 2048, 16 heads                   93.3 ->  54.7    FP8, 74 x 2048, 64 heads            95.9 ->  82.2
//   (these two since: 52.5 and 75.9)
//   prefill, 512 x 2048, 64 heads               333 ->   308    prefill, 2000 x 1024, 64 heads       677 ->   564
// Dense decode with 33 to 64 rows runs on pairs of SMs (attn_pair.cu) for batch sizes at which that hardly loses whatever the lengths are, where the block
// table says that few tokens are to be read: see csrc/host.cpp.
// Registers: at the launch bound of the FP8 variants 12 to 68 bytes are spilled (576-wide 64 / 16 heads 68 / 40, 512-wide 44 / 12);
// where they are reloaded has not been established.  Dense and prefill: none.
// FP8 decode with 128 heads as two CTAs of 64 is slower than a pair of SMs (64 x 2048: 101, pairs 56), since both CTAs convert
// every record.
//
// Bounded waits and the wind-down are those of attn_pair.cu (attn_shared.cuh).
//
// Behavioural reference: csrc/sm90/decode/dense/splitkv_mla.cuh:959-1272 (masking, split / direct epilogue, empty rows),
// csrc/sm100/decode/head64/kernel.cuh:19-849 (FP8 records, validity, attn_sink) and
// csrc/sm100/prefill/sparse/fwd/head64/phase1.cuh (prefill with 64 heads) of deepseek-ai/FlashMLA.
#include "attn_shared.cuh"
#include <float.h>

namespace mla {
namespace sm100 {
namespace rows64 {

constexpr int TILE = 128;                         // tokens
constexpr int PAIR_BYTES = 2 * TILE * 128;        // two 64-dim chunks of a tile
constexpr int ROPE_BYTES = TILE * 128;
constexpr int P_BYTES = TILE * 128;               // P: a 128-byte row per token (NH <= 64 values)
constexpr int NP_MAX = 5;

// Warps behind the control warpgroup (0..3) and the softmax warps (4..11) that bring KV rows in: prefill copies them by index
// with cp.async (eight warps), FP8 decode loads, converts and stores them (sixteen).
template <int MODE>
struct Warps {
    static constexpr int FEED = MODE == MODE_DENSE ? 0 : MODE == MODE_PREFILL ? 8 : 16;
    static constexpr int FIRST_FEED = 12;
    static constexpr int THREADS = (12 + FEED) * 32;
    // Registers per thread: what a launch gets (LAUNCH, the launch bound's), and each role's share after it has been re-sized.  A
    // larger share waits until the others have given theirs up: together no more than the launch had.
    static constexpr int LAUNCH = MODE == MODE_DENSE ? 168 : MODE == MODE_PREFILL ? 96 : 72;
    static constexpr int CONTROL = MODE == MODE_PREFILL ? 56 : 40, SOFTMAX = MODE == MODE_PREFILL ? 136 : 104, FEEDING = MODE == MODE_PREFILL ? 56 : 64;
    static_assert(MODE == MODE_DENSE || 128 * CONTROL + 256 * SOFTMAX + FEED * 32 * FEEDING <= THREADS * LAUNCH, "register shares");
};

// Shared memory (byte offsets inside Smem::data).  WIDE: 576-wide rows (a RoPE chunk).
template <int NH, bool WIDE>
struct Lay {
    static constexpr int CHUNKS = WIDE ? 9 : 8;
    static constexpr int Q_CHUNK = NH * 128;
    // 64 rows of 576: Q, four pairs, RoPE and P together are 5 KB more than there is.  P moves into the RoPE slot, which Q K^T has
    // read by then (the next tile's RoPE chunk waits for P V, like its last pair).
    // (With 32 rows the same buys a fifth pair.)
    static constexpr bool P_IN_ROPE = NH >= 32 && WIDE;
    static constexpr int NP = NH <= 32 ? 5 : 4;
    static constexpr int Q = 0;
    static constexpr int RING = Q + CHUNKS * Q_CHUNK;
    static constexpr int ROPE = RING + NP * PAIR_BYTES;
    static constexpr int P = WIDE && !P_IN_ROPE ? ROPE + ROPE_BYTES : ROPE;
    static constexpr int END = P + P_BYTES;
    static_assert(RING % 1024 == 0, "swizzle atoms");
};
constexpr int DATA_BYTES = Lay<64, true>::END > Lay<16, true>::END ? Lay<64, true>::END : Lay<16, true>::END;
static_assert(Lay<32, true>::END <= DATA_BYTES && Lay<32, false>::END <= DATA_BYTES && Lay<64, false>::END <= DATA_BYTES, "shared memory plan");

struct Smem {
    uint8_t data[DATA_BYTES];
    uint64_t k_full[NP_MAX], k_empty[NP_MAX], r_full, r_empty, q_full, q_empty, s_full, p_full, o_full, drain;
    uint32_t tmem_base, aborted;
    uint64_t optr[64];                            // where a row's results go
    __align__(16) float mref[64], bound[64], fac[64], inv[64];    // maximum in use, score that moves it, rescale factor, 1 / row sum
    float cmax[4][64], csum[4][64], ctrue[4][64]; // per quarter of a tile's tokens
    __align__(16) uint32_t mask[2][4];            // validity bits of a tile's tokens, two tiles
};
static_assert(sizeof(Smem) <= 232448, "shared memory budget");

// position in a ring of N slots, fill by fill
template <int N>
struct RingPos {
    uint32_t slot = 0, par = 0;
    __device__ __forceinline__ void next() { if (++slot == (uint32_t)N) { slot = 0; par ^= 1; } }
};

__device__ __forceinline__ int ordered(uint32_t f) { return (int)f ^ (((int)f >> 31) & 0x7fffffff); }      // floats as integers of the same order
__device__ __forceinline__ float from_ordered(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

// v[c] of 32 lanes -> on lane l, column l % HC combined over the warp
template <int HC, typename F>
__device__ __forceinline__ float combine_columns(float (&v)[HC], int lane, F f) {
#pragma unroll
    for (int n = HC / 2; n >= 1; n >>= 1) {
        const bool up = lane & n;
#pragma unroll
        for (int k = 0; k < n; ++k) {
            const float other = __shfl_xor_sync(0xffffffffu, up ? v[k] : v[k + n], n);
            v[k] = f(up ? v[k + n] : v[k], other);
        }
    }
#pragma unroll
    for (int n = HC; n < 32; n <<= 1) v[0] = f(v[0], __shfl_xor_sync(0xffffffffu, v[0], n));
    return v[0];
}

// O^T columns times their rows' factors: this warp's 32 dims of blocks m0 and m0 + 1.  (Rare: eight columns at a time.)
template <int NH>
__device__ __forceinline__ void rescale_o(uint32_t tlane, int m0, const float* fac) {
#pragma unroll 1
    for (int c0 = 0; c0 < 2 * NH; c0 += 8) {
        uint32_t v[8];
        tmem_ld8(tlane + m0 * NH + c0, v);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) * fac[c0 % NH + c]);
        tmem_st8(tlane + m0 * NH + c0, v);
    }
    tmem_wait_st();
}

// FP8 decode of 576-wide records: the record and the scales of list entries that are no token (loads without a condition: 74 x 2048 keys, 64 heads
// 79.9 -> 77.0 us, 64 x 2048, 16 heads 54.4 -> 53.2; 512-wide records lose, 46.1 -> 48.6)
__device__ __align__(128) uint8_t no_record[656];

// ALT: the second data format of a mode - fp16 in the place of bf16 (dense), 512-wide rows / records (gather modes).
template <int MODE, bool ALT, int NH>
__global__ void __launch_bounds__(Warps<MODE>::THREADS, 1)
attn_rows64_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap rmap,
                   const __grid_constant__ CUtensorMap qmap, const Params p) {
    constexpr bool DENSE = MODE == MODE_DENSE, PREFILL = MODE == MODE_PREFILL, SPARSE = MODE == MODE_SPARSE_DECODE;
    constexpr bool FP16 = ALT && DENSE;
    constexpr bool WIDE = DENSE || !ALT;                   // 576-wide rows
    constexpr bool M1 = ALT && SPARSE;                     // 512-wide records
    using L = Lay<NH, WIDE>;
    using W = Warps<MODE>;
    using WalkerT = Walker<MODE>;
    constexpr int NP = L::NP, HC = NH / 2;
    constexpr bool EARLY = DENSE && NP > 4;                // Q K^T of the next tile begins before P V of this one
    constexpr uint32_t TM_O = 0, TM_S = 4 * NH;            // tensor memory: O^T, S^T (EARLY: of two tiles)
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = DENSE ? 0 : blockIdx.x * NH;          // gather modes: the first head of this CTA
    const int hk = DENSE ? blockIdx.y : 0;
    const int rows = DENSE ? p.rows : min(NH, p.h_q - row0);
    const int part = blockIdx.z;

    if ((smem_addr(smem_raw) & 1023u) != 0) {              // the swizzled tiles need a 1024-byte aligned base
        if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, 900);
        return;
    }
    if (threadIdx.x == 0) {
        // a pair is filled by TMA (one arrival and bytes), by 256 threads' copies, or by sixteen warps' stores
        const uint32_t full = DENSE ? 1 : PREFILL ? 256 : 16;
        for (int i = 0; i < NP_MAX; ++i) { mbar_init(smem_addr(&sm.k_full[i]), full); mbar_init(smem_addr(&sm.k_empty[i]), 1); }
        mbar_init(smem_addr(&sm.r_full), full);
        mbar_init(smem_addr(&sm.r_empty), 1);
        mbar_init(smem_addr(&sm.q_full), p.q_tma ? 1 : 64);
        mbar_init(smem_addr(&sm.q_empty), 1);
        mbar_init(smem_addr(&sm.s_full), 1);
        mbar_init(smem_addr(&sm.p_full), 256);
        mbar_init(smem_addr(&sm.o_full), 1);
        mbar_init(smem_addr(&sm.drain), 1);
        sm.aborted = 0;
        fence_mbar_init();
        if (DENSE) { prefetch_tensormap(&kmap); prefetch_tensormap(&rmap); }
        if (p.q_tma) prefetch_tensormap(&qmap);
    }
    if (warp == 1) { tmem_alloc(smem_addr(&sm.tmem_base), 512); tmem_relinquish(); }
    {
        // rows of Q that no load ever writes: zeros, so that their scores are
        const int first = p.q_tma ? p.q_box_bytes >> 7 : rows;
        const int n = (NH - first) * L::CHUNKS * 8;
        for (int k = threadIdx.x; k < n; k += W::THREADS) {
            const int c = k / ((NH - first) * 8), r = first + (k >> 3) % (NH - first);
            *reinterpret_cast<uint4*>(sm.data + L::Q + c * L::Q_CHUNK + r * 128 + (k & 7) * 16) = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // (programmatic dependent launch: from here on results of the previous kernel of the stream are read)
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t tmem = sm.tmem_base;
    Waiter wt(p.wait_limit);
    // what the wind-down has to wait for after an expired wait (thread 0: loads it armed)
    uint32_t fills_armed = 0, ropes_armed = 0, q_armed = 0;

    if (warp < 4) {
    if (!DENSE) regs_dec<W::CONTROL>();
    if (warp == 0) {
        // ---------------- TMA producer: Q, in dense mode the tiles too ---------------------------------------
        if (lane == 0) {
            RingPos<NP> ring;
            uint32_t nq = 0, nr = 0;
            const int chunk0 = hk * p.head_chunks;
            for (WalkerT wk(p, part); wk.valid(); wk.next()) {
                const Work w = wk.get();
                if (w.ntiles == 0) continue;
                if (p.q_tma) {
                    // coordinates: (column, head, query token, request); prefill: a "request" is a query token of the only batch
                    const int c1 = DENSE ? hk * p.g : row0, c2 = DENSE ? 0 : PREFILL ? w.req : (int)blockIdx.y, c3 = PREFILL ? 0 : w.req;
                    if (nq > 0) WAIT_OR_LEAVE(wt, &sm.q_empty, (nq - 1) & 1, 13);
                    const uint32_t bar = smem_addr(&sm.q_full);
                    mbar_arrive_expect_tx(bar, L::CHUNKS * (uint32_t)p.q_box_bytes);
                    q_armed = ++nq;
#pragma unroll 1
                    for (int c = 0; c < L::CHUNKS; ++c) tma_load_4d(smem_addr(sm.data + L::Q + c * L::Q_CHUNK), &qmap, bar, c * 64, c1, c2, c3);
                }
                if (DENSE) {
                    const int* bt = p.block_table + (int64_t)w.req * p.bt_sb;
                    // a block index beyond the table's width reads no table entry: its keys are zeros
                    auto page_of = [&](int blk) -> int { return (blk < w.blk_end && blk < p.max_blocks) ? __ldg(bt + blk) : p.num_blocks; };
                    int nxt0 = page_of(w.blk_begin), nxt1 = page_of(w.blk_begin + 1);
                    for (int i = 0; i < w.ntiles; ++i) {
                        const int page0 = nxt0, page1 = nxt1;
                        if (i + 1 < w.ntiles) {
                            const int nb = w.blk_begin + 2 * (i + 1);
                            nxt0 = page_of(nb);
                            nxt1 = page_of(nb + 1);
                        }
#pragma unroll 1
                        for (int q = 0; q < 4; ++q, ring.next()) {
                            WAIT_OR_LEAVE(wt, &sm.k_empty[ring.slot], ring.par ^ 1, 1);
                            const uint32_t bar = smem_addr(&sm.k_full[ring.slot]);
                            mbar_arrive_expect_tx(bar, PAIR_BYTES);
                            ++fills_armed;
                            const uint32_t dst = smem_addr(sm.data + L::RING) + ring.slot * PAIR_BYTES;
                            tma_load_5d(dst, &kmap, bar, 0, 0, chunk0 + 2 * q, 0, page0);
                            tma_load_5d(dst + PAIR_BYTES / 2, &kmap, bar, 0, 0, chunk0 + 2 * q, 0, page1);
                        }
                        WAIT_OR_LEAVE(wt, &sm.r_empty, (nr & 1) ^ 1, 2);
                        const uint32_t bar = smem_addr(&sm.r_full);
                        mbar_arrive_expect_tx(bar, ROPE_BYTES);
                        ropes_armed = ++nr;
                        const uint32_t dst = smem_addr(sm.data + L::ROPE);
                        tma_load_5d(dst, &rmap, bar, 0, 0, chunk0 + 8, 0, page0);
                        tma_load_5d(dst + ROPE_BYTES / 2, &rmap, bar, 0, 0, chunk0 + 8, 0, page1);
                        if (i + 1 < w.ntiles) {                       // the next tile into L2
#pragma unroll 1
                            for (int q = 0; q < 4; ++q) {
                                tma_prefetch_5d(&kmap, 0, 0, chunk0 + 2 * q, 0, nxt0);
                                tma_prefetch_5d(&kmap, 0, 0, chunk0 + 2 * q, 0, nxt1);
                            }
                            tma_prefetch_5d(&rmap, 0, 0, chunk0 + 8, 0, nxt0);
                            tma_prefetch_5d(&rmap, 0, 0, chunk0 + 8, 0, nxt1);
                        }
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer -----------------------------------------------------------------------
        if (elect_one()) {
            constexpr uint32_t idesc_s = make_idesc_ab(128, NH, false, false, FP16), idesc_o = make_idesc_ab(128, NH, true, true, FP16);
            // pairs: 64-dim chunks interleaved in every 8-token group (2 KB); RoPE and P: plain rows of 128 bytes
            constexpr uint32_t hi_pair = sw128_desc_hi(2048), hi_row = sw128_desc_hi(1024);
            const uint32_t ring_k = sw128_desc_lo(smem_addr(sm.data + L::RING), 16), ring_v = sw128_desc_lo(smem_addr(sm.data + L::RING), 1024);
            const uint32_t rope_lo = sw128_desc_lo(smem_addr(sm.data + L::ROPE), 16);
            const uint32_t q_lo = sw128_desc_lo(smem_addr(sm.data + L::Q), 16), p_lo = sw128_desc_lo(smem_addr(sm.data + L::P), 1024);
            RingPos<NP> ring;
            uint32_t g = 0, nq = 0;
            // Q K^T over pair q of a tile, which is in `slot`
            auto scores_of_pair = [&](uint32_t d_tmem, int q, uint32_t slot) {
                if (!DENSE) fence_proxy_async_smem();      // the feeding warps' stores and copies -> visible to the tensor core
                tc_fence_after();
                const uint32_t a_lo = ring_k + slot * (PAIR_BYTES >> 4), b_lo = q_lo + q * (2 * L::Q_CHUNK >> 4);
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int k4 = 0; k4 < 4; ++k4)
                        mma_ss_lohi(d_tmem, a_lo + c * (1024 >> 4) + k4 * 2, hi_pair, b_lo + c * (L::Q_CHUNK >> 4) + k4 * 2, hi_row,
                                    idesc_s, (q | c | k4) ? 1u : 0u);
            };
            for (WalkerT wk(p, part); wk.valid(); wk.next()) {
                const Work w = wk.get();
                if (w.ntiles == 0) continue;
                WAIT_OR_LEAVE(wt, &sm.q_full, nq & 1, 3);
                ++nq;
                bool begun = false;                        // the tile's first pair has been done already
                for (int i = 0; i < w.ntiles; ++i, ++g) {
                    const uint32_t s_tmem = tmem + TM_S + (EARLY ? (g & 1) * NH : 0);
                    RingPos<NP> pv = ring;
                    if (begun) ring.next();
#pragma unroll 1
                    for (int q = begun ? 1 : 0; q < 4; ++q, ring.next()) {
                        WAIT_OR_LEAVE(wt, &sm.k_full[ring.slot], ring.par, 4);
                        scores_of_pair(s_tmem, q, ring.slot);
                    }
                    if (WIDE) {
                        WAIT_OR_LEAVE(wt, &sm.r_full, g & 1, 5);
                        if (!DENSE) fence_proxy_async_smem();      // the feeding warps' stores and copies -> visible to the tensor core
                        tc_fence_after();
#pragma unroll
                        for (int k4 = 0; k4 < 4; ++k4)
                            mma_ss_lohi(s_tmem, rope_lo + k4 * 2, hi_row, q_lo + 8 * (L::Q_CHUNK >> 4) + k4 * 2, hi_row, idesc_s, 1u);
                        if (!L::P_IN_ROPE) tc_commit(smem_addr(&sm.r_empty));
                    }
                    if (i + 1 == w.ntiles) tc_commit(smem_addr(&sm.q_empty));
                    tc_commit(smem_addr(&sm.s_full));
                    // While the softmax runs: the next tile's first pair, where the ring holds one more than a tile and it is there.
                    begun = EARLY && i + 1 < w.ntiles && mbar_try_wait(smem_addr(&sm.k_full[ring.slot]), ring.par);
                    if (begun) scores_of_pair(tmem + TM_S + ((g + 1) & 1) * NH, 0, ring.slot);
                    WAIT_OR_LEAVE(wt, &sm.p_full, g & 1, 6);
                    tc_fence_after();
#pragma unroll 1
                    for (int m = 0; m < 4; ++m, pv.next()) {
                        const uint32_t a_lo = ring_v + pv.slot * (PAIR_BYTES >> 4);
#pragma unroll
                        for (int kt = 0; kt < TILE / 16; ++kt)
                            mma_ss_lohi(tmem + TM_O + m * NH, a_lo + kt * (4096 >> 4), hi_pair, p_lo + kt * (2048 >> 4), hi_row, idesc_o,
                                        (i > 0 || kt > 0) ? 1u : 0u);
                        tc_commit(smem_addr(&sm.k_empty[pv.slot]));
                    }
                    if (L::P_IN_ROPE) tc_commit(smem_addr(&sm.r_empty));
                    if (i + 1 == w.ntiles) tc_commit(smem_addr(&sm.o_full));
                }
            }
        }
    } else if (!p.q_tma) {
        // ---------------- Q rows that TMA cannot address: 64 threads copy them ----------------------------------
        uint32_t nq = 0;
        for (WalkerT wk(p, part); wk.valid(); wk.next()) {
            const Work w = wk.get();
            if (w.ntiles == 0) continue;
            if (nq > 0) WAIT_OR_LEAVE(wt, &sm.q_empty, (nq - 1) & 1, 14);
            ++nq;
            for (int k = threadIdx.x - 64; k < rows * L::CHUNKS * 8; k += 64) {
                const int r = k / (L::CHUNKS * 8), piece = k - r * (L::CHUNKS * 8), c = piece >> 3, u = piece & 7;
                const int t = DENSE ? r / p.g : SPARSE ? (int)blockIdx.y : 0, hd = DENSE ? hk * p.g + r - t * p.g : row0 + r;
                const __nv_bfloat16* src = PREFILL ? p.q + (int64_t)w.req * p.q_ss + (int64_t)hd * p.q_sh
                                                   : p.q + (int64_t)w.req * p.q_sb + (int64_t)t * p.q_ss + (int64_t)hd * p.q_sh;
                *reinterpret_cast<uint4*>(sm.data + L::Q + c * L::Q_CHUNK + r * 128 + ((u ^ (r & 7)) << 4)) =
                    __ldg(reinterpret_cast<const uint4*>(src + piece * 8));
            }
            fence_proxy_async_smem();
            mbar_arrive(smem_addr(&sm.q_full));
        }
    }
    } else if (!DENSE && warp >= W::FIRST_FEED) {
        regs_dec<W::FEEDING>();
        const int fw = warp - W::FIRST_FEED;
        RingPos<NP> ring;
        uint32_t g = 0;
        if (PREFILL) {
            // ---------------- prefill: rows by index, 16 tokens of the tile per warp --------------------------------
            // One cp.async instruction of the warp copies 256 bytes of two rows (a pair's share); invalid tokens get zeros.
            const int tok0 = fw * 16;
            const uint32_t ring0 = smem_addr(sm.data + L::RING) + (tok0 >> 3) * 2048 + ((lane >> 3) & 1) * 1024;
            for (WalkerT wk(p, part); wk.valid(); wk.next()) {
                const Work w = wk.get();
                const int* idx = p.indices + (int64_t)w.req * p.idx_ss;
                const int tok = tok0 + (lane & 15);
                int id_next = tok < w.seqlen ? __ldg(idx + tok) : -1;          // (a tile ahead)
                for (int i = 0; i < w.ntiles; ++i, ++g) {
                    const int id = id_next;
                    const int row_id = id >= 0 && id < p.s_kv ? id : -1;
                    const uint32_t bal = __ballot_sync(0xffffffffu, row_id >= 0);
                    { const int posn = (i + 1) * TILE + tok; id_next = posn < w.seqlen ? __ldg(idx + posn) : -1; }
#pragma unroll 1
                    for (int q = 0; q < 4; ++q, ring.next()) {
                        WAIT_WARP_OR_LEAVE(wt, &sm.k_empty[ring.slot], ring.par ^ 1, 201);
                        if (q == 0 && lane == 0) { reinterpret_cast<uint16_t*>(sm.mask[g & 1])[fw] = (uint16_t)bal; __threadfence_block(); }
                        const uint32_t dst0 = ring0 + ring.slot * PAIR_BYTES;
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            const int tk = 2 * u + (lane >> 4);
                            const int rid = __shfl_sync(0xffffffffu, row_id, tk);
                            const __nv_bfloat16* src = p.kv + (int64_t)(rid < 0 ? 0 : rid) * p.kv_ss + q * 128 + (lane & 15) * 8;
                            cp_async16_zfill(dst0 + (tk >> 3) * 2048 + (tk & 7) * 128 + (((lane & 7) ^ (tk & 7)) << 4), src, rid < 0 ? 0u : 16u);
                        }
                        cp_async_arrive_noinc(smem_addr(&sm.k_full[ring.slot]));
                    }
                    if (WIDE) {
                        WAIT_WARP_OR_LEAVE(wt, &sm.r_empty, (g & 1) ^ 1, 202);
                        const uint32_t dst0 = smem_addr(sm.data + L::ROPE) + tok0 * 128;
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int tk = 4 * u + (lane >> 3);
                            const int rid = __shfl_sync(0xffffffffu, row_id, tk);
                            const __nv_bfloat16* src = p.kv + (int64_t)(rid < 0 ? 0 : rid) * p.kv_ss + 512 + (lane & 7) * 8;
                            cp_async16_zfill(dst0 + tk * 128 + (((lane & 7) ^ (tk & 7)) << 4), src, rid < 0 ? 0u : 16u);
                        }
                        cp_async_arrive_noinc(smem_addr(&sm.r_full));
                    }
                }
            }
        } else {
            // ---------------- FP8 decode: records by index, 8 tokens of the tile per warp -----------------------------
            // index -> (page, offset) -> 656-byte record = 512 e4m3 | 4 fp32 scales | 64 bf16 RoPE (512-wide form: 448 e4m3 | 64
            // bf16 RoPE, seven e8m0 scale bytes per token behind the block's tokens).  The warp loads its raw bytes straight into
            // registers, a tile ahead (four lanes per token, 16 bytes a lane), converts them (one rounding:
            // bf16(fp32(e4m3) * scale)) when the pair's slot is free, and stores 16 bytes at a time: the two tokens of eight lanes
            // are an even and an odd row, whose swizzle sends them to eight different 16-byte banks.
            const int tl = lane >> 2, piece = lane & 3;               // this lane's token of the warp's eight, its piece of every chunk
            const int tok = fw * 8 + tl;
            const uint32_t ring0 = smem_addr(sm.data + L::RING) + fw * 2048 + tl * 128;
            const int tq = blockIdx.y;
            for (WalkerT wk(p, part); wk.valid(); wk.next()) {
                const Work w = wk.get();
                const int* idx0 = p.sidx[0] + (int64_t)w.req * p.sidx_sb[0] + (int64_t)tq * p.sidx_ss[0];
                const int* idx1 = p.stopk[1] ? p.sidx[1] + (int64_t)w.req * p.sidx_sb[1] + (int64_t)tq * p.sidx_ss[1] : nullptr;
                auto load_id = [&](int blk) -> int {
                    if (blk >= w.blk_end) return -1;
                    const int scope = blk >= w.nblk0 ? 1 : 0;
                    const int pos = (scope ? blk - w.nblk0 : blk) * PAGE + (tok & 63);
                    if (pos >= (scope ? w.len1 : w.len0)) return -1;
                    return __ldg((scope ? idx1 : idx0) + pos);
                };
                const uint8_t* const none = M1 ? nullptr : no_record;
                // the token's record and its scales as they are stored: four fp32, or eight bytes in the first two words
                auto look_up = [&](int blk, int id, uint4& sc) -> const uint8_t* {
                    const int scope = blk >= w.nblk0 ? 1 : 0;
                    const int pbs = p.pbs[scope];
                    sc = make_uint4(0, 0, 0, 0);
                    if ((uint32_t)id >= p.tokens[scope]) return none;
                    const uint8_t* block = p.kvb[scope] + (int64_t)(id / pbs) * p.kvb_sblock[scope];
                    const int off = id % pbs;
                    if (M1) {
                        const uint2 e = __ldg(reinterpret_cast<const uint2*>(block + (int64_t)pbs * 576 + (int64_t)off * 8));
                        sc.x = e.x; sc.y = e.y;
                        return block + (int64_t)off * 576;
                    }
                    sc = __ldg(reinterpret_cast<const uint4*>(block + (int64_t)off * 656 + 512));
                    return block + (int64_t)off * 656;
                };
                uint4 raw[4][2], rope[2];
                auto load16 = [&](const uint8_t* rec, int off) { return !M1 || rec ? __ldg(reinterpret_cast<const uint4*>(rec + off)) : make_uint4(0, 0, 0, 0); };
                auto load_pair = [&](const uint8_t* r, int q) {
                    raw[q][0] = load16(r, q * 128 + piece * 16);
                    // (512-wide form, chunk 7: RoPE, copied as it is, 32 bytes per lane)
                    raw[q][1] = load16(r, M1 && q == 3 ? 448 + piece * 32 : q * 128 + 64 + piece * 16);
                    if (M1 && q == 3) rope[0] = load16(r, 448 + piece * 32 + 16);
                };
                auto load_rope = [&](const uint8_t* r) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) rope[u] = load16(r, 528 + piece * 32 + u * 16);
                };
                const int blk0 = w.blk_begin + (tok >> 6);
                uint4 sc, sc_next;
                const uint8_t* rec = look_up(blk0, load_id(blk0), sc);
                int id_next = load_id(blk0 + 2);
#pragma unroll
                for (int q = 0; q < 4; ++q) load_pair(rec, q);
                if (WIDE) load_rope(rec);
                for (int i = 0; i < w.ntiles; ++i, ++g) {
                    const uint32_t bal = __ballot_sync(0xffffffffu, rec != none);      // four lanes a token
                    rec = look_up(blk0 + 2 * (i + 1), id_next, sc_next);
                    id_next = load_id(blk0 + 2 * (i + 2));
#pragma unroll
                    for (int q = 0; q < 4; ++q, ring.next()) {
                        WAIT_WARP_OR_LEAVE(wt, &sm.k_empty[ring.slot], ring.par ^ 1, 201);
                        if (q == 0 && lane == 0) {
                            uint32_t bits = 0;
#pragma unroll
                            for (int t = 0; t < 8; ++t) bits |= (bal >> (4 * t) & 1u) << t;
                            reinterpret_cast<uint8_t*>(sm.mask[g & 1])[fw] = (uint8_t)bits;
                        }
                        const uint32_t dst0 = ring0 + ring.slot * PAIR_BYTES;
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const uint32_t word = M1 ? (q < 2 ? sc.x : sc.y) : q == 0 ? sc.x : q == 1 ? sc.y : q == 2 ? sc.z : sc.w;
                            const float scale = M1 ? e8m0_of(word, (2 * q + u) & 3) : __uint_as_float(word);
                            uint4 lo = raw[q][u], hi = rope[0];
                            if (!(M1 && q == 3 && u == 1)) dequant16(raw[q][u], scale, lo, hi);
                            st_shared_v4(dst0 + u * 1024 + (((2 * piece) ^ tl) << 4), lo);
                            st_shared_v4(dst0 + u * 1024 + (((2 * piece + 1) ^ tl) << 4), hi);
                        }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(smem_addr(&sm.k_full[ring.slot]));
                        load_pair(rec, q);
                    }
                    if (WIDE) {
                        WAIT_WARP_OR_LEAVE(wt, &sm.r_empty, (g & 1) ^ 1, 202);
#pragma unroll
                        for (int u = 0; u < 2; ++u)
                            st_shared_v4(smem_addr(sm.data + L::ROPE) + tok * 128 + (((2 * piece + u) ^ tl) << 4), rope[u]);
                        __syncwarp();
                        if (lane == 0) mbar_arrive(smem_addr(&sm.r_full));
                        load_rope(rec);
                    }
                    sc = sc_next;
                }
            }
        }
    } else {
        // ---------------- softmax, rescale and epilogue: thread = token of the tile (lane) x HC rows --------------------
        if (!DENSE) regs_inc<W::SOFTMAX>();
        const int wq = warp & 3, half = (warp - 4) >> 2;
        const int tok = wq * 32 + lane;                               // = tensor-memory lane
        const int tid = threadIdx.x - 128;                            // 0..255
        const uint32_t tlane = tmem + ((uint32_t)(wq * 32) << 16);
        const int col0 = half * HC;
        const bool active = col0 < rows;                              // (warp-uniform) this half has rows at all
        const uint32_t prow = smem_addr(sm.data + L::P) + tok * 128;
        constexpr int CW = DENSE || HC < 16 ? HC : 16;
        const float inv_scale = 1.f / p.scale_log2;
        uint32_t g = 0, nreq = 0;
        RingPos<NP> ring;
        // These 256 threads meet at a named barrier every tile, so none of them may leave alone: a thread whose wait ran out keeps
        // walking (it arrives nowhere and stores nothing) until the next such barrier, which carries the flag to everyone.
        for (WalkerT wk(p, part); wk.valid(); wk.next()) {
            const Work w = wk.get();
            const int limit = min(w.seqlen, w.blk_end * PAGE);
            float l[HC], top[PREFILL ? HC : 1];                       // row sums (and true maxima) over this thread's tokens
#pragma unroll
            for (int c = 0; c < HC; ++c) { l[c] = 0.f; if (PREFILL) top[c] = -INFINITY; }
            for (int i = 0; i < w.ntiles; ++i, ++g) {
                wt.wait(&sm.s_full, g & 1, 7);
                tc_fence_after();
                const int blk = w.blk_begin + 2 * i + (tok >> 6), pos = blk * PAGE + (tok & 63);
                const bool ok = DENSE ? pos < limit : (sm.mask[g & 1][wq] >> lane) & 1u;
                const bool causal = DENSE && p.causal && pos + p.s_q > w.seqlen;     // rows of earlier query tokens do not see the last keys
                // Scores of CW rows at a time, -inf where masked.  Dense mode keeps all of them in registers; the gather modes, whose
                // registers hold the sums and little else, read tensor memory again for every pass.
                auto scores = [&](int c0, uint32_t (&s)[CW]) {
                    tmem_ld(tlane + TM_S + (EARLY ? (g & 1) * NH : 0) + col0 + c0, s);
                    tmem_wait_ld();
                    if (!ok) {
#pragma unroll
                        for (int c = 0; c < CW; ++c) s[c] = 0xff800000u;
                    }
                    if (causal) {
                        int t = (col0 + c0) / p.g, h = col0 + c0 - t * p.g;
#pragma unroll
                        for (int c = 0; c < CW; ++c) {
                            if (pos >= w.seqlen - (p.s_q - 1 - t)) s[c] = 0xff800000u;
                            if (++h == p.g) { h = 0; ++t; }
                        }
                    }
                };
                uint32_t kept[DENSE ? HC : 1];
                if constexpr (DENSE) { if (active) scores(0, kept); }
                auto each = [&](auto&& f) {
                    if constexpr (DENSE) {
                        f(0, kept);
                    } else {
#pragma unroll
                        for (int c0 = 0; c0 < HC; c0 += CW) {
                            uint32_t s[CW];
                            scores(c0, s);
                            f(c0, s);
                        }
                    }
                };
                // does any score exceed the maximum in use by more than the threshold?
                bool grow = wt.expired();
                if (active) {
                    if (i > 0 || PREFILL) {
each([&](int c0, uint32_t (&s)[CW]) {
#pragma unroll
                            for (int c = 0; c < CW; c += 4) {
                                const float4 t = *reinterpret_cast<const float4*>(&sm.bound[col0 + c0 + c]);
                                grow |= __uint_as_float(s[c]) > t.x;
                                grow |= __uint_as_float(s[c + 1]) > t.y;
                                grow |= __uint_as_float(s[c + 2]) > t.z;
                                grow |= __uint_as_float(s[c + 3]) > t.w;
                            }
                            if (PREFILL) {
#pragma unroll
                                for (int c = 0; c < CW; ++c) top[c0 + c] = fmaxf(top[c0 + c], __uint_as_float(s[c]));
                            }
                        });
                    }
                }
                if (i > 0) grow = named_bar_red_or(1, 256, grow);
                if (i == 0 || grow) {
                    if (active) {
                        int mine = 0;
each([&](int c0, uint32_t (&s)[CW]) {
#pragma unroll
                            for (int c = 0; c < CW; ++c) {
                                const int k = __reduce_max_sync(0xffffffffu, ordered(s[c]));
                                if (lane == c0 + c) mine = k;
                            }
                        });
                        if (lane < HC) sm.cmax[wq][col0 + lane] = from_ordered(mine);
                    }
                    if (named_bar_red_or(1, 256, wt.expired())) goto wind_down;
                    if (tid < NH) {
                        // (before a row's first finite score its maximum is the lowest finite value: any finite score, scaled,
                        // is at least that, and no difference below is infinity minus infinity.  Rows that do not exist: zeros.)
                        const float mx = fmaxf(fmaxf(sm.cmax[0][tid], sm.cmax[1][tid]), fmaxf(sm.cmax[2][tid], sm.cmax[3][tid])) * p.scale_log2;
                        const float old = i == 0 ? -FLT_MAX : sm.mref[tid];
                        const bool up = mx > old + RESCALE_THRESHOLD;
                        const float m = tid >= rows ? 0.f : up ? mx : old;
                        sm.mref[tid] = m;
                        sm.bound[tid] = (m + RESCALE_THRESHOLD) * inv_scale;
                        sm.fac[tid] = tid < rows && up ? ex2(old - mx) : 1.f;
                    }
                    named_bar_sync(1, 256);
                    if (i > 0) {
                        if (active) {
#pragma unroll
                            for (int c = 0; c < HC; ++c) l[c] *= sm.fac[col0 + c];
                        }
                        rescale_o<NH>(tlane + TM_O, 2 * half, sm.fac);      // (s_full: every earlier P V has finished)
                    }
                }
                if (active) {
each([&](int c0, uint32_t (&s)[CW]) {
#pragma unroll
                        for (int c = 0; c < CW; c += 8) {
                            uint32_t pk[4];
#pragma unroll
                            for (int k = 0; k < 8; k += 4) {
                                const float4 m = *reinterpret_cast<const float4*>(&sm.mref[col0 + c0 + c + k]);
                                const float e0 = ex2(fmaf(__uint_as_float(s[c + k]), p.scale_log2, -m.x));
                                const float e1 = ex2(fmaf(__uint_as_float(s[c + k + 1]), p.scale_log2, -m.y));
                                const float e2 = ex2(fmaf(__uint_as_float(s[c + k + 2]), p.scale_log2, -m.z));
                                const float e3 = ex2(fmaf(__uint_as_float(s[c + k + 3]), p.scale_log2, -m.w));
                                float* lk = &l[c0 + c + k];
                                lk[0] += e0; lk[1] += e1; lk[2] += e2; lk[3] += e3;
                                pk[k / 2] = pack16<FP16>(e0, e1);
                                pk[k / 2 + 1] = pack16<FP16>(e2, e3);
                            }
                            if (!wt.expired()) st_shared_v4(prow + ((((col0 + c0 + c) >> 3) ^ (tok & 7)) << 4), make_uint4(pk[0], pk[1], pk[2], pk[3]));
                        }
                    });
                }
                if (DENSE) {
                    // Tokens at or beyond the sequence length may hold anything (NaN included) in a real page: their probabilities
                    // are zero, so their rows are zeroed to keep 0 * NaN out of O (Q K^T has read them).
                    if (blk < w.blk_end && pos >= w.seqlen && !wt.expired()) {
                        RingPos<NP> slot = ring;
#pragma unroll 1
                        for (int q = 0; q < 4; ++q, slot.next()) {
                            if ((q >> 1) != half) continue;
                            const uint32_t row = smem_addr(sm.data + L::RING) + slot.slot * PAIR_BYTES + (tok >> 3) * 2048 + (tok & 7) * 128;
#pragma unroll 1
                            for (int k = 0; k < 16; ++k) st_shared_v4(row + (k >> 3) * 1024 + (k & 7) * 16, make_uint4(0, 0, 0, 0));
                        }
                    }
                    for (int q = 0; q < 4; ++q) ring.next();
                }
                fence_proxy_async_smem();
                tc_fence_before();
                if (!wt.expired()) mbar_arrive(smem_addr(&sm.p_full));
            }
            // ---- epilogue: a row's sum over all tokens, then O^T / sum, a lane per dim ------------------------------------
            if (active) {
                const float x = combine_columns<HC>(l, lane, [](float a, float b) { return a + b; });
                if (lane < HC) sm.csum[wq][col0 + lane] = x;
                if (PREFILL) {
                    const float y = combine_columns<PREFILL ? HC : 1>(top, lane, [](float a, float b) { return fmaxf(a, b); });
                    if (lane < HC) sm.ctrue[wq][col0 + lane] = y;
                }
            }
            const bool has_tiles = w.ntiles > 0;
            if (has_tiles) { wt.wait(&sm.o_full, nreq & 1, 8); ++nreq; }
            if (named_bar_red_or(1, 256, wt.expired())) goto wind_down;
            tc_fence_after();
            if (tid < rows) {
                const int t = DENSE ? tid / p.g : SPARSE ? (int)blockIdx.y : 0, hd = DENSE ? hk * p.g + tid - t * p.g : row0 + tid;
                const float sum = sm.csum[0][tid] + sm.csum[1][tid] + sm.csum[2][tid] + sm.csum[3][tid];
                const float m = sm.mref[tid];
                const bool empty = !has_tiles || !(sum > 0.f);        // also catches NaN
                float scale = 1.f / sum;
                if (!DENSE && !w.is_split && p.attn_sink) scale = 1.f / (sum + exp2f(p.attn_sink[hd] * kLog2e - m));
                sm.inv[tid] = empty ? -1.f : scale;                   // (a sign that no sum has)
                if (w.is_split) {
                    const int64_t arow = ((int64_t)w.slot * p.s_q + t) * p.h_q + hd;
                    sm.optr[tid] = reinterpret_cast<uint64_t>(p.o_accum + arow * D_V);
                    p.lse_accum[arow] = empty ? -INFINITY : log2f(sum) + m;
                } else {
                    const float lse_nat = empty ? INFINITY : (log2f(sum) + m) * kLn2;
                    if (PREFILL) {
                        const int64_t arow = (int64_t)w.req * p.h_q + hd;
                        sm.optr[tid] = reinterpret_cast<uint64_t>(p.out + arow * D_V);
                        p.lse[arow] = lse_nat;
                        p.max_logits[arow] = empty ? -INFINITY
                            : fmaxf(fmaxf(sm.ctrue[0][tid], sm.ctrue[1][tid]), fmaxf(sm.ctrue[2][tid], sm.ctrue[3][tid])) * p.scale_log2 * kLn2;
                    } else {
                        sm.optr[tid] = reinterpret_cast<uint64_t>(p.out + (int64_t)w.req * p.o_sb + (int64_t)t * p.o_ss + (int64_t)hd * p.o_sh);
                        p.lse[w.req * p.l_sb + t * p.l_ss + hd * p.l_sh] = lse_nat;
                    }
                }
            }
            named_bar_sync(1, 256);
            // (Short loops: a kernel runs this once or twice, and the time of an unrolled body is that of fetching its instructions.
            // Prefill, 700 x 640 keys, 512-wide: 142.3 us with 32 rows at a time and a branch per two rows, 136.5 with 16 and none.
            // Partials of 64 rows, 128 KB a CTA, are bound by the stores: FP8, 74 x 2048: 81.4 us with 32, 83 with 16.)
            constexpr int WC = PREFILL || NH < 32 || (DENSE && NH == 32) ? 16 : 32;
#pragma unroll 1
            for (int c0 = 0; c0 < 2 * NH; c0 += WC) {                 // this half's two blocks of dims, WC rows at a time
                const int d = (2 * half + c0 / NH) * 128 + tok, r0 = c0 % NH;
                uint32_t v[WC];
                if (has_tiles) { tmem_ld(tlane + TM_O + 2 * half * NH + c0, v); tmem_wait_ld(); }
                if (w.is_split) {
#pragma unroll
                    for (int c = 0; c < WC; ++c) {
                        if (r0 + c < rows) {
                            const float f = sm.inv[r0 + c];
                            reinterpret_cast<float*>(sm.optr[r0 + c])[d] = f < 0.f ? 0.f : __uint_as_float(v[c]) * f;
                        }
                    }
                } else {
                    // two rows at a time: the even lane of a pair takes both dims of the first row, the odd lane those of the second
#pragma unroll
                    for (int c = 0; c < WC; c += 2) {
                        const float f0 = sm.inv[r0 + c], f1 = sm.inv[r0 + c + 1];
                        const float x0 = f0 < 0.f ? 0.f : __uint_as_float(v[c]) * f0, x1 = f1 < 0.f ? 0.f : __uint_as_float(v[c + 1]) * f1;
                        const bool odd = lane & 1;
                        const float other = __shfl_xor_sync(0xffffffffu, odd ? x0 : x1, 1);
                        const int r = r0 + c + odd;
                        if (r < rows)
                            *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(sm.optr[r]) + (d & ~1)) =
                                odd ? pack16<FP16>(other, x1) : pack16<FP16>(x0, other);
                    }
                }
            }
            tc_fence_before();
        }
    }

wind_down:
    if (wt.expired()) report_expired_wait(p.status, &sm.aborted, 0u, wt.code);
    if (PREFILL && warp >= W::FIRST_FEED) cp_async_wait_all();
    tc_fence_before();
    if (__syncthreads_or((int)*reinterpret_cast<volatile uint32_t*>(&sm.aborted))) {
        // A bounded wait ran out; every thread has left its role and issues nothing more.  Wait - bounded again - for what is
        // still in flight: the MMAs and the TMA loads.
        if (warp == 1 && elect_one()) {
            tc_commit(smem_addr(&sm.drain));
            mbar_wait_bounded(smem_addr(&sm.drain), 0, DRAIN_LIMIT);
        }
        if (threadIdx.x == 0) {
            for (uint32_t back = 1; back <= (uint32_t)NP && back <= fills_armed; ++back) {
                const uint32_t f = fills_armed - back;         // one of the last fills this thread armed: its slot has seen no later phase
                mbar_wait_bounded(smem_addr(&sm.k_full[f % NP]), (f / NP) & 1, DRAIN_LIMIT);
            }
            if (ropes_armed) mbar_wait_bounded(smem_addr(&sm.r_full), (ropes_armed - 1) & 1, DRAIN_LIMIT);
            if (q_armed) mbar_wait_bounded(smem_addr(&sm.q_full), (q_armed - 1) & 1, DRAIN_LIMIT);
        }
        __syncthreads();
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

template <int MODE, bool ALT, int NH>
static int launch(dim3 grid, const CUtensorMap& kmap, const CUtensorMap& rmap, const CUtensorMap& qmap, const Params& p, void* stream) {
    static bool configured[64] = {};
    if (int rc = configure_once(attn_rows64_kernel<MODE, ALT, NH>, configured, sizeof(Smem))) return rc;
    MLA_CHECK_CUDA(launch_dependent(attn_rows64_kernel<MODE, ALT, NH>, grid, dim3(Warps<MODE>::THREADS), sizeof(Smem), (cudaStream_t)stream, kmap, rmap, qmap, p));
    MLA_CHECK_CUDA(cudaGetLastError());
    return MLA_OK;
}

}  // namespace rows64

// The two cache tensor maps of a dense launch depend only on the cache tensor: a decode loop calls with the same cache every
// step, so the last encoding is kept per host thread.
struct Rows64Maps {
    const void* k_cache = nullptr;
    int64_t sb = 0, sr = 0, sh = 0;
    int num_blocks = 0, h_kv = 0, fp16 = 0;
    CUtensorMap kmap, rmap;
};

}  // namespace sm100

int launch_dense_decode_rows64(const mla_dense_decode_args_t& a) {
    using namespace sm100;
    EncodeTiledFn encode = get_encode_fn();
    if (!encode) return set_error(MLA_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const bool fp16 = a.dtype == MLA_DTYPE_FP16;
    // The cache as a 5-D tensor (64 columns of a chunk, 8 tokens, chunks, 8 token groups, pages): one box brings all 64 tokens
    // of a page for a pair of chunks (or the RoPE chunk) and lands as [token group][chunk][8 rows x 128 B].
    const int head_chunks = a.h_kv > 1 ? (int)(a.k_stride_head / 64) : 9;
    static thread_local Rows64Maps cm;
    if (cm.k_cache != a.k_cache || cm.sb != a.k_stride_block || cm.sr != a.k_stride_row || cm.sh != a.k_stride_head ||
        cm.num_blocks != a.num_blocks || cm.h_kv != a.h_kv || cm.fp16 != (int)fp16) {
        cm.k_cache = nullptr;
        const CUtensorMapDataType dt = fp16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
        cuuint64_t dims[5] = {64, 8, (cuuint64_t)((a.h_kv - 1) * head_chunks + 9), 8, (cuuint64_t)a.num_blocks};
        cuuint64_t strides[4] = {(cuuint64_t)a.k_stride_row * 2, 128, (cuuint64_t)a.k_stride_row * 16, (cuuint64_t)a.k_stride_block * 2};
        cuuint32_t estr[5] = {1, 1, 1, 1, 1};
        cuuint32_t kbox[5] = {64, 8, 2, 8, 1}, rbox[5] = {64, 8, 1, 8, 1};
        CUresult r = encode(&cm.kmap, dt, 5, const_cast<void*>(a.k_cache), dims, strides, kbox, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r == CUDA_SUCCESS)
            r = encode(&cm.rmap, dt, 5, const_cast<void*>(a.k_cache), dims, strides, rbox, estr,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return set_error(MLA_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
        cm.k_cache = a.k_cache; cm.sb = a.k_stride_block; cm.sr = a.k_stride_row; cm.sh = a.k_stride_head;
        cm.num_blocks = a.num_blocks; cm.h_kv = a.h_kv; cm.fp16 = (int)fp16;
    }
    CUtensorMap qmap;
    Params p = dense_params(a, head_chunks);
    memset(&qmap, 0, sizeof(qmap));
    p.q_tma = encode_q_map(&qmap, a.q, a.b, a.s_q, a.h_q, a.q_stride_b, a.q_stride_s, a.q_stride_h, p.g, a.s_q, &p.q_box_bytes, fp16) ? 1 : 0;
    const dim3 grid(1, a.h_kv, a.num_sm_parts);
#define MLA_DENSE(NH) (fp16 ? rows64::launch<MODE_DENSE, true, NH>(grid, cm.kmap, cm.rmap, qmap, p, a.stream) \
                            : rows64::launch<MODE_DENSE, false, NH>(grid, cm.kmap, cm.rmap, qmap, p, a.stream))
    return p.rows <= 16 ? MLA_DENSE(16) : p.rows <= 32 ? MLA_DENSE(32) : MLA_DENSE(64);
#undef MLA_DENSE
}

int launch_sparse_prefill_rows64(const mla_sparse_prefill_args_t& a) {
    using namespace sm100;
    Params p = prefill_params(a);
    CUtensorMap unused, qmap;
    memset(&unused, 0, sizeof(unused));
    memset(&qmap, 0, sizeof(qmap));
    p.q_tma = encode_q_map(&qmap, a.q, 1, a.s_q, a.h_q, 0, a.q_stride_s, a.q_stride_h, a.h_q < 64 ? a.h_q : 64, 1, &p.q_box_bytes, false, a.d_qk) ? 1 : 0;
    const int blocks = (a.h_q + 63) / 64, sms = current_device_num_sms();
    int ctas = sms / blocks;
    if (ctas < 1) ctas = 1;
    if (ctas > a.s_q) ctas = a.s_q;
    const dim3 grid(blocks, 1, ctas);
    return a.d_qk == 512 ? rows64::launch<MODE_PREFILL, true, 64>(grid, unused, unused, qmap, p, a.stream)
                         : rows64::launch<MODE_PREFILL, false, 64>(grid, unused, unused, qmap, p, a.stream);
}

int launch_sparse_decode_rows64(const mla_sparse_decode_args_t& a) {
    using namespace sm100;
    Params p = sparse_decode_params(a);
    CUtensorMap unused, qmap;
    memset(&unused, 0, sizeof(unused));
    memset(&qmap, 0, sizeof(qmap));
    p.q_tma = encode_q_map(&qmap, a.q, a.b, a.s_q, a.h_q, a.q_stride_b, a.q_stride_s, a.q_stride_h, a.h_q < 64 ? a.h_q : 64, 1,
                           &p.q_box_bytes, false, a.d_qk) ? 1 : 0;
    const dim3 grid((a.h_q + 63) / 64, a.s_q, a.num_sm_parts);
#define MLA_SPARSE(NH) (a.d_qk == 512 ? rows64::launch<MODE_SPARSE_DECODE, true, NH>(grid, unused, unused, qmap, p, a.stream) \
                                      : rows64::launch<MODE_SPARSE_DECODE, false, NH>(grid, unused, unused, qmap, p, a.stream))
    // (17 to 32 heads: a variant of 32, with a fifth pair as in dense decode, has not been measured)
    return a.h_q <= 16 ? MLA_SPARSE(16) : MLA_SPARSE(64);
#undef MLA_SPARSE
}

}  // namespace mla
