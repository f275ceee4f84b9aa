// MLA attention for up to 128 query rows on a PAIR of SMs whose MMAs span both (sm_100a, tcgen05 with cta_group::2).  One kernel template:
//   MODE_DENSE          dense BF16 / FP16 paged decode, fed by TMA loads of 64-token KV pages through the block table
//   MODE_PREFILL        token-sparse prefill, KV rows gathered by index: the own page's with cp.async, the other page's with TMA
//   MODE_SPARSE_DECODE  sparse FP8 decode, token records gathered by address, converted in registers
// Up to 64 rows: attn_rows64.cu (on one SM), or, for short prefills and dense batches of few tokens, this one.
//
// Each CTA holds 64 of the 128 rows.  With M = 128 over two CTAs both score and output accumulators split by rows:
//   S = Q K^T   64 x 128 per CTA in 64 columns    A = Q (chunks 0..5 in tensor memory, the others in shared memory)
//                                                 B = K, 128 tokens split by N: every CTA brings ITS page of the tile, 576 dims
//   O += P V    64 x 512 per CTA in 256 columns   A = P of the CTA's own rows (never leaves the SM)
//                                                 B = V, the dims split by N: every CTA brings BOTH pages, 256 dims
// so 64 x 576 + 64 x 256 values enter an SM per tile of 128 tokens; softmax, P and epilogue are divided evenly, and no CTA waits for the
// other's P.  (The kernel before this one split the products: a score CTA took 128 x 576 values a tile, a value CTA 128 x 512, P went from
// one to the other, and one of them ran each epilogue.  Its times are the left-hand figures below.)
//
// One instruction's descriptors name the same offsets in both CTAs.  A tile takes four slots of a ring, slot q holding chunks 2 q and
// 2 q + 1 of the CTA's own page.  CTA 0 serves the dims of slots 0 and 1, CTA 1 those of 2 and 3.  P V of page h reads slots 2 h and
// 2 h + 1: in CTA h that is its own page's half of the dims, in place since Q K^T; in the other CTA those slots held dims it does
// not serve, which Q K^T alone needed - behind it they are filled again with page h's dims that it serves.  CTA 1's are in Q K^T's first
// half (k_half), CTA 0's in the second (k_done), and P V is issued page by page: page 0, whose other part is there first, gives the
// slots back that the tile after next waits for while page 1 is still on its way.
//
// The RoPE chunks have two buffers of their own, and nobody waits for those: a tile's last two slots are given back by P V of page 0 of
// the tile before last or later, or by the hand-over of a Q behind that tile, and its Q K^T is older than either.
//
// Softmax: warps 4..11, a thread = one row, one page, half of the page's tokens.  P is made with the maximum in use on the guess that no
// row has outgrown it by 2^6.  The warps vote on that before they make P, on an mbarrier, so that the answer is there when P is; every warp
// hands its part of P over by itself.  Where the guess was wrong (and on a request's first tile) all meet, the maxima are exchanged, O is
// rescaled and P is made again.  P, the row sums and O always refer to the same maximum, so results are exact up to rounding.
//
// CTA 0's issuing thread takes whatever is ready: Q K^T of the next tile slot by slot, or P V of the last one.  It is chosen with
// elect_one (sm100_ptx.cuh).  A chain of these MMAs takes 33 cycles per 128 x 128 x 16 and 65 per 128 x 256 x 16.  Arrivals on CTA 0's
// barriers order inside the arriving CTA only (mbar_arrive_remote_cta): what they announce is read by that CTA's own tensor core.
// With cluster-wide releases a tile of dense decode took 5350 cycles in the place of 4110.
//
// What bounds it.  Dense decode, 128 requests of about 4096 tokens: 2700 to 3300 cycles a tile, of which the tensor core works 2250 (60 % of
// the launch); DRAM at 4.9 TB/s in a launch by itself (136 us at 1.63 GHz), back to back the power limit (1.32 to 1.39 GHz).  A tile's loads wait for
// P V two tiles before, 2000 to 2900 cycles before they have landed.  Prefill: 3700 cycles a tile, the tensor core 2250, the own page's copies
// (144 instructions an SM, 14.5 cycles each at best) and the other page's row gathers (64 of TMA, 20 each) beside each other; back to back the
// power limit (1.6 GHz).  FP8 decode: 4300 to 4800 cycles a tile; 64 x 2048
// keys take 54 us, without the records' loads 47, without their conversion 52, without both 43 (512-wide 48.5, 46.6, 41.6, 38.9; shares of
// other values in their place): the chain conversion -> Q K^T -> softmax -> P V behind a ring of two and a half tiles, the loads' way
// through the little that is left of L1, and the conversion.  One copy of every converted value would save a third of the conversion but the
// exchange costs more: by 16-byte asynchronous stores into the other SM 93 us, by bulk copies 75.5, converting the half of the
// other page again 57.0 (first line below).  us a call, back to back, score and value CTAs -> now:
//   one input per call                                          inputs changing from call to call, clocks settled
//   FP8, 64 x 2048 keys, 128 heads              91.2 -> 56.2      92.4 -> 60.8
//   FP8, 74 x (512 + 1024) ragged, 512-wide     78.2 -> 51.0      77.8 -> 50.6
//   prefill, 4096 x 2048 keys, 128 heads        2740 -> 2284      2809 -> 2339
//   prefill, 1 x 64 keys, 128 heads             16.3 ->  9.9
//   dense, 128 x ~4096 tokens                    185 ->  172       189 ->  173
//   dense, two query tokens                      314 ->  294       325 ->  300
//   dense, one request of 100003 tokens                           54.9 -> 47.8
// (914 calls of dense and FP8 decode and prefill with 64 to 128 heads: between 1.04 and 2.0 times as fast, none slower.)  From that state on, with
// P V page by page, the vote on an mbarrier and no wait for the RoPE buffers (the table's calls with inputs changing, both in turn): FP8 60.5 -> 57.7,
// prefill 2338 -> 2252; dense and two query tokens nothing to 1 % (181.7 -> 179.9, 309.0 -> 307.2), 128 requests of lognormal lengths nothing (534 ->
// 533); 512-wide records, whose exponent bytes are converted by the instruction for them, whose loads have no condition and are preceded by L2
// prefetches, 50.8 -> 47.5.
// Registers: both FP8 forms spill 4 bytes a thread, the others none.
//
// Every mbarrier wait is bounded (Params::wait_limit SM cycles, about a second by default).  A thread whose wait ran out LEAVES its role -
// it issues no further arrival, MMA or copy -, records a code in the status words and raises the `aborted` flag of both CTAs.
// Single-thread roles leave at once; warps leave together (a vote after every wait, because tcgen05.ld/st are warp-collective); the softmax
// warpgroups vote against the guess, meet at a named barrier that carries the flag (bar.red.or) and leave behind it.  Threads that
// depend on the one that left run into their own limit.  The wind-down then waits - again bounded - for the MMAs, meets the peer
// CTA, gives loads still under way time to land, and only then frees tensor memory; both CTAs leave together.
//
// Behavioural reference: csrc/sm90/decode/dense/splitkv_mla.cuh:959-1272 (masking, split / direct epilogue, empty rows),
// csrc/sm100/decode/head64/kernel.cuh:19-849 (FP8 records, validity, attn_sink) and
// csrc/sm100/prefill/sparse/fwd/head128/phase1.cuh:65-614 (prefill outputs) of deepseek-ai/FlashMLA.
#include "attn_shared.cuh"

namespace mla {
namespace sm100 {
namespace pair {

constexpr int ROWS = 128, HALF = 64;              // query rows of the pair / of a CTA
constexpr int CHUNK = 8192;                       // 64 rows x 64 16-bit values, 128-byte swizzled rows
constexpr int SLOT = 2 * CHUNK;                   // two chunks of a page: [8-token group][chunk][8 rows x 128 B]
constexpr int NSLOT = 10, NROPE = 2;              // ring of slots: a tile takes four, a request's Q three before its first tile; of RoPE chunks
constexpr int QT = 6;                             // 64-dim chunks of Q in tensor memory, the others in shared memory
constexpr int Q_SLOTS = QT / 2;                   // ring slots that a request's Q takes on its way there
constexpr uint32_t TM_O = 0, TM_S = 256, TM_Q = 320;
static_assert(TM_Q + QT * 32 <= 512, "tensor-memory columns");

// Warps behind the control warpgroup (0..3) and the softmax warps (4..11): FP8 decode has sixteen that load records, convert and
// store them.  Registers per thread: what a launch gets (LAUNCH, the launch bound's), and each role's share after it has been
// re-sized; a larger share waits until the others have given theirs up.
template <int MODE>
struct Warps {
    static constexpr int FEED = MODE == MODE_DENSE ? 0 : MODE == MODE_PREFILL ? 8 : 16;
    static constexpr int FIRST_FEED = 12;
    static constexpr int THREADS = (12 + FEED) * 32;
    static constexpr int LAUNCH = MODE == MODE_DENSE ? 168 : MODE == MODE_PREFILL ? 96 : 72;
    static constexpr int SOFTMAX = MODE == MODE_PREFILL ? 112 : 88, FEEDING = MODE == MODE_PREFILL ? 80 : 64;
    static_assert(MODE == MODE_DENSE || 128 * LAUNCH + 256 * SOFTMAX + FEED * 32 * FEEDING <= THREADS * LAUNCH, "register shares");
};

constexpr int AT_ROPE = NSLOT * SLOT;
constexpr int AT_Q = AT_ROPE + NROPE * CHUNK;
constexpr int AT_P = AT_Q + (9 - QT) * CHUNK;     // P: per page of the tile [64 rows][64 tokens]
constexpr int AT_XMAX = AT_P + 2 * CHUNK;         // [2][4][64] floats: a row's maximum / sum in the four quarters of its tiles
constexpr int NTAB = 4;                           // gather modes: tiles whose tokens' addresses are looked up ahead
constexpr int AT_TAB = AT_XMAX + 2 * 4 * HALF * 4;   // FP8 decode: per tile [128 tokens] addresses of the record and of its scales
constexpr int DATA_BYTES = AT_TAB + NTAB * ROWS * 16;

struct Smem {
    uint8_t data[DATA_BYTES];
    // (those that only the issuing thread waits on live in CTA 0)  full[s]: the two slots from s on, behind a tile's second two its RoPE chunk too
    uint64_t full[NSLOT], empty[NSLOT], p_full[2][2], k_done[2], k_half[2], f_tail, q_staged, q_taken, q_next, q_free, q_full, q_ready, s_full, s_empty,
        pv_done, o_empty, vote[2], drain;
    uint32_t tmem_base, aborted, outgrown[2];
    uint64_t tab_full[NTAB], tab_empty[NTAB];
    uint64_t l_full[NSLOT];                       // prefill: this CTA's copies (as full) have landed
    uint32_t mask[2 * NTAB][4];                   // gather modes: validity bits of a tile's tokens
};
static_assert(sizeof(Smem) <= 232448, "shared memory budget");

// position in a ring of N slots, fill by fill
template <int N>
struct RingPos {
    uint32_t slot = 0, par = 0;
    __device__ __forceinline__ void skip(uint32_t n) { slot += n; while (slot >= (uint32_t)N) { slot -= N; par ^= 1; } }
    __device__ __forceinline__ void skip_many(uint32_t n) { slot += n; par ^= slot / N & 1; slot %= N; }
    __device__ __forceinline__ void next() { if (++slot == (uint32_t)N) { slot = 0; par ^= 1; } }
};

// (a barrier that is ready costs a probe and a vote)
#define READY_OR_WAIT(W, bar, par, code) do { if (!__all_sync(0xffffffffu, mbar_try_wait(smem_addr(bar), par))) WAIT_WARP_OR_LEAVE(W, bar, par, code); } while (0)
// the softmax warpgroups' named barrier carries the flag of an expired wait
#define BAR_OR_LEAVE(flag) do { if (named_bar_red_or(1, 256, flag)) goto wind_down; } while (0)

// O rows times their factor: this warp's lanes, 128 columns.  (Rare: eight columns at a time.)
__device__ __forceinline__ void rescale_o(uint32_t taddr, float f) {
#pragma unroll 1
    for (int c = 0; c < 128; c += 8) {
        uint32_t v[8];
        tmem_ld8(taddr + c, v);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = __float_as_uint(__uint_as_float(v[k]) * f);
        tmem_st8(taddr + c, v);
    }
    tmem_wait_st();
}
// Rows [first, 64) of a slot set to zero by the 256 softmax threads.
__device__ __noinline__ void zero_rows(uint8_t* slot, int first) {
    const int n = (PAGE - first) * 16;                  // 16-byte pieces
    for (int k = threadIdx.x - 128; k < n; k += 256) {
        const int piece = k & 7, c = (k >> 3) & 1, r = first + (k >> 4);
        *reinterpret_cast<uint4*>(slot + (r >> 3) * 2048 + c * 1024 + (r & 7) * 128 + piece * 16) = make_uint4(0, 0, 0, 0);
    }
}
// Stores 32 words of every lane's row (`to`: where the row's part starts, 0 where the lane has none) `off` bytes behind it.  Four
// lanes exchange their rows' quarters first, so that they write the 128-byte lines of four rows one after the other: a lane that
// writes its own row touches a line of its own in every instruction.
__device__ __forceinline__ void store_rows(uint32_t (&v)[32], unsigned long long to, int off, bool wide, int lane) {
#pragma unroll
    for (int bit = 1; bit <= 2; bit <<= 1) {
        const bool up = lane & bit;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            if (b & bit) continue;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                uint32_t &lo = v[8 * b + k], &hi = v[8 * (b + bit) + k];
                const uint32_t x = __shfl_xor_sync(0xffffffffu, up ? lo : hi, bit);
                if (up) lo = x; else hi = x;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint8_t* at = const_cast<uint8_t*>(shfl_ptr(reinterpret_cast<const uint8_t*>(to), (lane & ~3) + j));
        if (!at) continue;
        at += off + (lane & 3) * 32;
        const uint32_t* x = &v[8 * j];
        if (wide) {
            st_global_v8(at, x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7]);
        } else {
            *reinterpret_cast<uint4*>(at) = make_uint4(x[0], x[1], x[2], x[3]);
            *reinterpret_cast<uint4*>(at + 16) = make_uint4(x[4], x[5], x[6], x[7]);
        }
    }
}
// Q moved by the softmax threads themselves, for tensors that no box of a tensor map fits: row r of this CTA, the chunks of
// warpgroup wg (0: 0, 1, 2 and 6; 1: 3, 4, 5 and 7, 8).  `first`: this thread's lane half writes the chunks in shared memory.
__device__ __noinline__ void load_q_by_threads(Smem& sm, const __nv_bfloat16* qrow, bool row_ok, int wg, int r, uint32_t tlane, bool first, bool no_chunk8) {
#pragma unroll 1
    for (int k = 0; k < (wg ? 5 : 4); ++k) {
        const int c = k < 3 ? wg * 3 + k : wg ? 4 + k : 6;
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint4 x = row_ok && !(no_chunk8 && c == 8) ? __ldg(reinterpret_cast<const uint4*>(qrow + c * 64) + i) : make_uint4(0, 0, 0, 0);
            v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
        }
        if (c < QT) {
            tmem_st32(tlane + TM_Q + c * 32, v);
        } else if (first) {
            uint8_t* dst = sm.data + AT_Q + (c - QT) * CHUNK + r * 128;
#pragma unroll
            for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(dst + ((i ^ (r & 7)) << 4)) = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
    }
}

// FP8 decode of 512-wide records: the record and the scales of list entries that are no token (loads without a condition: 49.1 -> 47.4 us for
// 74 x (512 + 1024), 128 heads; 576-wide records lose, 52.9 -> 54.8 for 64 x 2048)
__device__ __align__(128) uint8_t no_record[576];

template <int MODE, bool ALT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Warps<MODE>::THREADS, 1)
attn_pair_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap rmap,
                 const __grid_constant__ CUtensorMap qmap, const Params p) {
    constexpr bool DENSE = MODE == MODE_DENSE, PREFILL = MODE == MODE_PREFILL, SPARSE = MODE == MODE_SPARSE_DECODE;
    constexpr bool FP16 = ALT && DENSE;
    constexpr bool WIDE = DENSE || !ALT;                   // 576-wide rows (a RoPE chunk behind the eight)
    constexpr bool M1 = ALT && SPARSE;                     // 512-wide records
    constexpr int CHUNKS = WIDE ? 9 : 8;
    using W = Warps<MODE>;
    using WalkerT = Walker<MODE>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    const uint32_t rank = cluster_ctarank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row_blk = SPARSE ? 0 : blockIdx.y % p.row_blocks;
    const int hk = SPARSE ? 0 : blockIdx.y / p.row_blocks;
    const int part = blockIdx.z;
    const int row0 = row_blk * ROWS + (int)rank * HALF;    // this CTA's first row

    if ((smem_addr(smem_raw) & 1023u) != 0) {              // the swizzled tiles need a 1024-byte aligned base
        if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, 900);
        return;                                            // both CTAs of the pair take this branch
    }
    if (threadIdx.x == 0) {
        // a slot is filled by TMA (one arrival and bytes), by both CTAs' copies (one relaying thread each), or by both CTAs' feeding warps
        const uint32_t fill = DENSE ? 1 : PREFILL ? 2 : 2 * W::FEED;
        for (int i = 0; i < NSLOT; ++i) { mbar_init(smem_addr(&sm.full[i]), fill); mbar_init(smem_addr(&sm.empty[i]), 1); }
        for (int i = 0; i < 4; ++i) mbar_init(smem_addr(&sm.p_full[i >> 1][i & 1]), SPARSE ? 8 + W::FEED : PREFILL ? 8 : 9);
        for (int i = 0; i < 2; ++i) mbar_init(smem_addr(&sm.vote[i]), 8);
        for (int i = 0; i < 2; ++i) { mbar_init(smem_addr(&sm.k_done[i]), 1); mbar_init(smem_addr(&sm.k_half[i]), 1); }
        mbar_init(smem_addr(&sm.f_tail), 1);
        if (PREFILL) {
            for (int i = 0; i < NSLOT; ++i) mbar_init(smem_addr(&sm.l_full[i]), 32 * W::FEED);
        }
        for (int i = 0; i < NTAB; ++i) { mbar_init(smem_addr(&sm.tab_full[i]), 32); mbar_init(smem_addr(&sm.tab_empty[i]), W::FEED > 0 ? W::FEED : 1); }
        mbar_init(smem_addr(&sm.q_staged), 1);
        mbar_init(smem_addr(&sm.q_taken), 1);
        mbar_init(smem_addr(&sm.q_next), 1);
        mbar_init(smem_addr(&sm.q_free), 1);
        mbar_init(smem_addr(&sm.q_full), 1);
        mbar_init(smem_addr(&sm.q_ready), 2);              // one thread of each CTA
        mbar_init(smem_addr(&sm.s_full), 1);
        mbar_init(smem_addr(&sm.s_empty), 16);             // the softmax warps of both CTAs
        mbar_init(smem_addr(&sm.pv_done), 1);
        mbar_init(smem_addr(&sm.o_empty), 16);
        mbar_init(smem_addr(&sm.drain), 1);
        sm.aborted = 0;
        sm.outgrown[0] = sm.outgrown[1] = 0;
        fence_mbar_init();
        if (!SPARSE) prefetch_tensormap(&kmap);
        if (DENSE) prefetch_tensormap(&rmap);
        if (p.q_tma) prefetch_tensormap(&qmap);
    }
    if (warp == 1) { tmem_alloc2(smem_addr(&sm.tmem_base), 512); tmem_relinquish2(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    cluster_sync();                                        // the peer's barriers exist, its tensor memory is allocated
    // (programmatic dependent launch: from here on results of the previous kernel of the stream are read)
    griddep_wait();
    griddep_launch_dependents();
    constexpr uint32_t tmem = 0;                           // (an allocation of all 512 columns begins at column 0)
    Waiter wt(p.wait_limit);
    auto lead = [&](uint64_t& bar) { return map_to_cta(smem_addr(&bar), 0); };    // the barrier of CTA 0

    if (warp < 4) {
    if (warp == 0) {
        // ---------------- own page of every tile (and Q's chunks for tensor memory, through the ring) ----------------
        if (elect_one()) {
            RingPos<NSLOT> ring;
            RingPos<NROPE> rope;
            uint32_t nq = 0, n_next = 0;
            int tiles_before = 0;
            const int chunk0 = hk * p.head_chunks;
            const uint32_t full0 = lead(sm.full[0]);
            for (WalkerT wk(p, part); wk.valid(); wk.next()) {
                const Work w = wk.get();
                if (w.ntiles == 0) continue;
                if (p.q_tma) {
                    // A parity wait only means what it says to a thread for which the barrier's phase before is known to be over, and which
                    // the phase behind waits for.  In the gather modes this thread does not see the ring's fills: the last Q K^T but one of
                    // the request before (where it has a single tile, q_taken) says that all but the last releases of these slots are past.
                    if (!DENSE && tiles_before > 1) { WAIT_OR_LEAVE(wt, &sm.q_next, n_next & 1, 12); ++n_next; }
                    tiles_before = w.ntiles;
                    if (nq > 0) WAIT_OR_LEAVE(wt, &sm.q_taken, (nq - 1) & 1, 13);      // q_staged's previous phase is over
                    ++nq;
                    const uint32_t bar = smem_addr(&sm.q_staged);
                    uint32_t slots[Q_SLOTS];
#pragma unroll
                    for (int k = 0; k < Q_SLOTS; ++k) {
                        WAIT_OR_LEAVE(wt, &sm.empty[ring.slot], ring.par ^ 1, 11);
                        slots[k] = ring.slot;
                        ring.next();
                    }
                    mbar_arrive_expect_tx(bar, QT * CHUNK);
#pragma unroll
                    for (int c = 0; c < QT; ++c) {
                        const uint32_t dst = smem_addr(sm.data) + slots[c / 2] * SLOT + (c & 1) * CHUNK;
#pragma unroll 1
                        for (int r = 0; r < HALF; r += p.q_unit) {
                            const int row = row0 + r;
                            tma_load_4d(dst + r * 128, &qmap, bar, c * 64, DENSE ? hk * p.g + row % p.g : row,
                                        SPARSE ? (int)blockIdx.y : PREFILL ? w.req : row / p.g, PREFILL ? 0 : w.req);
                        }
                    }
                }
                if (DENSE) {
                    const int* bt = p.block_table + (int64_t)w.req * p.bt_sb;
                    // a block index beyond the table's width reads no table entry: its keys are zeros
                    auto page_of = [&](int blk) -> int { return (blk < w.blk_end && blk < p.max_blocks) ? __ldg(bt + blk) : p.num_blocks; };
                    int nxt = page_of(w.blk_begin + rank);
                    for (int i = 0; i < w.ntiles; ++i) {
                        const int page = nxt;
                        if (i + 1 < w.ntiles) nxt = page_of(w.blk_begin + 2 * (i + 1) + rank);
                        uint32_t bar = 0;
#pragma unroll 1
                        for (int q = 0; q < 4; ++q, ring.next()) {
                            WAIT_OR_LEAVE(wt, &sm.empty[ring.slot], ring.par ^ 1, 1);
                            if (!(q & 1)) {
                                bar = ring.slot;
                                if (rank == 0) mbar_arrive_expect_tx(smem_addr(&sm.full[bar]), 4 * SLOT + (q ? 2 * CHUNK : 0));
                            }
                            tma2_load_5d(smem_addr(sm.data) + ring.slot * SLOT, &kmap, full0 + bar * 8, 0, 0, chunk0 + 2 * q, 0, page);
                        }
                        tma2_load_5d(smem_addr(sm.data) + AT_ROPE + rope.slot * CHUNK, &rmap, full0 + bar * 8, 0, 0, chunk0 + 8, 0, page);
                        rope.next();
                    }
                } else {
                    ring.skip_many(4 * w.ntiles);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (CTA 0, for both) -------------------------------------------------------
        if (rank == 0 && elect_one()) {
            constexpr uint32_t idesc_s = make_idesc_16(ROWS, 128, false, FP16), idesc_o = make_idesc_16(ROWS, 256, true, FP16);
            constexpr uint32_t hi_slot = sw128_desc_hi(2048), hi_row = sw128_desc_hi(1024);
            const uint32_t k_lo = sw128_desc_lo(smem_addr(sm.data), 16), v_lo = sw128_desc_lo(smem_addr(sm.data), 1024);
            const uint32_t r_lo = sw128_desc_lo(smem_addr(sm.data) + AT_ROPE, 16), q_lo = sw128_desc_lo(smem_addr(sm.data) + AT_Q, 16);
            const uint32_t p_lo = sw128_desc_lo(smem_addr(sm.data) + AT_P, 16);
            constexpr uint32_t d_s = tmem + TM_S, d_o = tmem + TM_O, a_q = tmem + TM_Q;
            const uint32_t full0 = smem_addr(&sm.full[0]), empty0 = smem_addr(&sm.empty[0]);
            const uint32_t p_full0 = smem_addr(&sm.p_full[0][0]), s_empty = smem_addr(&sm.s_empty), o_empty = smem_addr(&sm.o_empty);
            RingPos<NSLOT> ring;
            RingPos<NROPE> rope;
            uint32_t g = 0, nq = 0, full_par = 0;          // full_par: bit s is the parity of slot s's next fill with K
            for (WalkerT wk(p, part); wk.valid(); wk.next()) {
                const Work w = wk.get();
                if (w.ntiles == 0) continue;
                if (p.q_tma) {
                    ring.skip(Q_SLOTS);
                    WAIT_OR_LEAVE(wt, &sm.q_full, nq & 1, 3);
                }
                WAIT_OR_LEAVE(wt, &sm.q_ready, nq & 1, 4);
                // Two streams of work: Q K^T of tile qi in two stages (two slots each, the second with the RoPE chunk) as they are filled, and
                // where the next stage is not there, P V of tile pi.  A probe of a barrier costs this thread 150 to 300 cycles beside the
                // other roles' traffic, eight MMAs of Q K^T 270 of the tensor core: with few probes it keeps ahead.  (4096 tokens, 576-wide
                // prefill: all barriers probed at every step 2620 us, one stage per slot 2320.)
                RingPos<NSLOT> pv = ring;
                int qi = 0, pi = 0, stage = 0, half = 0;
                auto is = [&](uint32_t bar, uint32_t par) { return mbar_test_wait(bar, par & 1); };
                uint32_t t0 = clock_units<WAIT_UNIT_LOG2>();
#pragma unroll 1
                while (pi < w.ntiles) {
                    const uint32_t gp = g + pi, gq = g + qi;
                    if (qi < w.ntiles && qi <= pi + 1 && (stage > 0 || is(s_empty, gq + 1)) && is(full0 + ring.slot * 8, full_par >> ring.slot)) {
                        full_par ^= 1u << ring.slot;
                        tc_fence_after();
                        uint32_t b_lo = k_lo + ring.slot * (SLOT >> 4);
                        ring.next();
                        // (the first two 64-dim chunks of the stage)
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            mma2_ts_lohi(d_s, a_q + stage * 128 + k * 8, b_lo + (k >> 2) * (1024 >> 4) + (k & 3) * 2, hi_slot, idesc_s, (stage | k) ? 1u : 0u);
                        b_lo = k_lo + ring.slot * (SLOT >> 4);
                        ring.next();
                        if (stage == 0) {
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                mma2_ts_lohi(d_s, a_q + 64 + k * 8, b_lo + (k >> 2) * (1024 >> 4) + (k & 3) * 2, hi_slot, idesc_s, 1u);
                            tc_commit2(smem_addr(&sm.k_half[gq & 1]));
                            stage = 1;
                        } else {
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                mma2_ss_lohi(d_s, q_lo + (k >> 2) * (CHUNK >> 4) + (k & 3) * 2, hi_row, b_lo + (k >> 2) * (1024 >> 4) + (k & 3) * 2, hi_slot, idesc_s, 1u);
                            if (WIDE) {
#pragma unroll
                                for (int k = 0; k < 4; ++k)
                                    mma2_ss_lohi(d_s, q_lo + 2 * (CHUNK >> 4) + k * 2, hi_row, r_lo + rope.slot * (CHUNK >> 4) + k * 2, hi_row, idesc_s, 1u);
                            }
                            tc_commit2(smem_addr(&sm.s_full));
                            tc_commit2(smem_addr(&sm.k_done[gq & 1]));
                            if (!DENSE && qi + 2 == w.ntiles) tc_commit2(smem_addr(&sm.q_next));
                            if (qi + 1 == w.ntiles) tc_commit2(smem_addr(&sm.q_free));
                            if (WIDE) rope.next();
                            stage = 0;
                            ++qi;
                        }
                    } else if (pi < qi && is(p_full0 + (gp & 1) * 16 + half * 8, gp >> 1) && (pi > 0 || half > 0 || is(o_empty, nq + 1))) {
                        tc_fence_after();
#pragma unroll
                        for (int n = 0; n < 2; ++n, pv.next()) {
                            const uint32_t b_lo = v_lo + pv.slot * (SLOT >> 4), a_lo = p_lo + half * (CHUNK >> 4);
#pragma unroll
                            for (int kt = 0; kt < 4; ++kt)
                                mma2_ss_lohi(d_o + n * 128, a_lo + kt * 2, hi_row, b_lo + kt * (4096 >> 4), hi_slot, idesc_o,
                                             (pi > 0 || half > 0 || kt > 0) ? 1u : 0u);
                            tc_commit2(empty0 + pv.slot * 8);
                        }
                        if (half) { tc_commit2(smem_addr(&sm.pv_done)); ++pi; }
                        half ^= 1;
                    } else {
                        if (clock_units<WAIT_UNIT_LOG2>() - t0 > wt.limit) { wt.code = 6; goto wind_down; }
                        continue;
                    }
                    t0 = clock_units<WAIT_UNIT_LOG2>();
                }
                g += w.ntiles;
                ++nq;
            }
        }
    } else if (warp == 2) {
        // ---------------- this CTA's half of the dims of the other CTA's page, over chunks that Q K^T has read ----------
        if ((DENSE || p.q_tma) && elect_one()) {
            RingPos<NSLOT> ring;
            uint32_t g = 0, nq = 0;
            const int chunk0 = hk * p.head_chunks;
            const uint32_t p_full0 = lead(sm.p_full[0][0]), q_full = lead(sm.q_full);
            for (WalkerT wk(p, part); wk.valid(); wk.next()) {
                const Work w = wk.get();
                if (w.ntiles == 0) continue;
                if (p.q_tma) {
                    ring.skip(Q_SLOTS);
                    // nothing reads the previous request's Q any more (in the gather modes this thread follows no tile, in CTA 1 only the first half of
                    // each tile's Q K^T)
                    if (nq++ > 0) WAIT_OR_LEAVE(wt, &sm.q_free, nq & 1, 23);
                    if (rank == 0) mbar_arrive_expect_tx(smem_addr(&sm.q_full), 2 * (CHUNKS - QT) * CHUNK);
#pragma unroll 1
                    for (int c = QT; c < CHUNKS; ++c)
                        for (int r = 0; r < HALF; r += p.q_unit) {
                            const int row = row0 + r;
                            tma2_load_4d(smem_addr(sm.data) + AT_Q + (c - QT) * CHUNK + r * 128, &qmap, q_full, c * 64, DENSE ? hk * p.g + row % p.g : row,
                                         SPARSE ? (int)blockIdx.y : PREFILL ? w.req : row / p.g, PREFILL ? 0 : w.req);
                        }
                }
                if (!DENSE) continue;
                const int* bt = p.block_table + (int64_t)w.req * p.bt_sb;
                auto page_of = [&](int blk) -> int { return (blk < w.blk_end && blk < p.max_blocks) ? __ldg(bt + blk) : p.num_blocks; };
                int nxt = page_of(w.blk_begin + (1 - (int)rank));
                for (int i = 0; i < w.ntiles; ++i, ++g) {
                    const int page = nxt, blk0 = w.blk_begin + 2 * i;
                    if (i + 1 < w.ntiles) nxt = page_of(blk0 + 2 + (1 - (int)rank));
                    WAIT_OR_LEAVE(wt, rank == 0 ? &sm.k_done[g & 1] : &sm.k_half[g & 1], (g >> 1) & 1, 21);
                    // a page that the sequence ends in: its rows beyond the end are zeroed by the softmax warps when it has landed
                    auto ends_in = [&](int blk) { return blk < w.blk_end && w.seqlen < (blk + 1) * PAGE; };
                    if (rank == 0) {
                        mbar_arrive_expect_tx(smem_addr(&sm.p_full[g & 1][0]), ends_in(blk0) ? 0 : 2 * SLOT);
                        mbar_arrive_expect_tx(smem_addr(&sm.p_full[g & 1][1]), ends_in(blk0 + 1) ? 0 : 2 * SLOT);
                    }
                    const bool tail = ends_in(blk0 + (1 - (int)rank));
                    if (tail) mbar_arrive_expect_tx(smem_addr(&sm.f_tail), 2 * SLOT);
#pragma unroll 1
                    for (int q = 0; q < 4; ++q, ring.next()) {
                        if ((q >> 1) == (int)rank) continue;           // (slots of this CTA's own half)
                        const uint32_t dst = smem_addr(sm.data) + ring.slot * SLOT;
                        if (tail) tma_load_5d(dst, &kmap, smem_addr(&sm.f_tail), 0, 0, chunk0 + 4 * rank + 2 * (q & 1), 0, page);
                        else tma2_load_5d(dst, &kmap, p_full0 + (g & 1) * 16 + (1 - rank) * 8, 0, 0, chunk0 + 4 * rank + 2 * (q & 1), 0, page);
                    }
                }
            }
        }
    } else if (SPARSE) {
        // ---------------- FP8 decode: index -> (page, offset) -> address of the record and of its scales, tiles ahead ----------
        uint32_t g = 0;
        const int tq = blockIdx.y;
        for (WalkerT wk(p, part); wk.valid(); wk.next()) {
            const Work w = wk.get();
            const int* idx0 = p.sidx[0] + (int64_t)w.req * p.sidx_sb[0] + (int64_t)tq * p.sidx_ss[0];
            const int* idx1 = p.stopk[1] ? p.sidx[1] + (int64_t)w.req * p.sidx_sb[1] + (int64_t)tq * p.sidx_ss[1] : nullptr;
            auto load_id = [&](int blk, int tok) -> int {
                if (blk >= w.blk_end) return -1;
                const int scope = blk >= w.nblk0 ? 1 : 0;
                const int pos = (scope ? blk - w.nblk0 : blk) * PAGE + tok;
                if (pos >= (scope ? w.len1 : w.len0)) return -1;
                return __ldg((scope ? idx1 : idx0) + pos);
            };
            int id[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) id[k] = w.ntiles > 0 ? load_id(w.blk_begin + (k >> 1), (k & 1) * 32 + lane) : -1;
#pragma unroll 1
            for (int i = 0; i < w.ntiles; ++i, ++g) {
                WAIT_WARP_OR_LEAVE(wt, &sm.tab_empty[g % NTAB], ((g / NTAB) & 1) ^ 1, 205);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int blk = w.blk_begin + 2 * i + (k >> 1), scope = blk >= w.nblk0 ? 1 : 0;
                    const bool ok = (uint32_t)id[k] < p.tokens[scope];
                    ulonglong2 e = make_ulonglong2(0, 0);
                    if (M1) e.x = e.y = reinterpret_cast<unsigned long long>(no_record);
                    if (ok) {
                        uint32_t off;
                        const uint8_t* block = p.kvb[scope] + page_of_token(p, scope, id[k], off) * p.kvb_sblock[scope];
                        e.x = reinterpret_cast<unsigned long long>(block + (uint64_t)off * (M1 ? 576 : 656));
                        e.y = M1 ? reinterpret_cast<unsigned long long>(block + (int64_t)p.pbs[scope] * 576 + (uint64_t)off * 8) : e.x + 512;
                    }
                    // the own page's records into L2, tiles ahead of the loads, which keep L1's few free lines (what is left of 256 KB) busy as
                    // long as they are under way (512-wide records only: of 576-wide ones, 64 x 2048, 53.2 -> 57.9 us)
                    if (M1 && ok && (k >> 1) == (int)rank) {
#pragma unroll
                        for (int at = 0; at < 576; at += 128) prefetch_l2(e.x + at);
                        prefetch_l2(e.y);
                    }
                    reinterpret_cast<ulonglong2*>(sm.data + AT_TAB)[g % NTAB * ROWS + k * 32 + lane] = e;
                    const uint32_t bits = __ballot_sync(0xffffffffu, ok);
                    if (lane == 0) sm.mask[g % (2 * NTAB)][k] = bits;
                    id[k] = load_id(blk + 2, (k & 1) * 32 + lane);
                }
                mbar_arrive(smem_addr(&sm.tab_full[g % NTAB]));
            }
        }
    } else if (PREFILL && elect_one()) {
        // ---------------- prefill: copies have landed -> CTA 0's barriers -----------------------------------------------
        RingPos<NSLOT> ring;
        uint32_t par = 0;                                  // bit s is the parity of barrier s's next phase
        const uint32_t full0 = lead(sm.full[0]);
        for (WalkerT wk(p, part); wk.valid(); wk.next()) {
            const int ntiles = wk.get().ntiles;
            if (ntiles == 0) continue;
            if (p.q_tma) ring.skip(Q_SLOTS);
            for (int i = 0; i < 2 * ntiles; ++i, ring.skip(2)) {
                WAIT_OR_LEAVE(wt, &sm.l_full[ring.slot], (par >> ring.slot) & 1, 24);
                par ^= 1u << ring.slot;
                fence_proxy_async_smem();
                mbar_arrive_remote_cta(full0 + ring.slot * 8);
            }
        }
    }
    } else if (PREFILL && warp >= W::FIRST_FEED) {
        regs_dec<W::FEEDING>();
        // ---------------- prefill: rows by index, eight tokens of a page per warp -----------------------------------------
        // One cp.async instruction of the warp copies 256 bytes of two rows (a slot's share); invalid tokens get zeros.  A barrier of this
        // CTA counts one arrival per thread, made by the copy engine when that thread's copies have landed; a thread of warp 3 passes it on.
        const int fw = warp - W::FIRST_FEED;
        const int other = (lane >> 3) & 1, page_of_lane = other ? 1 - (int)rank : (int)rank;       // lanes 0..7 look up the own page's tokens, 8..15 the other's
        const int tok = page_of_lane * PAGE + fw * 8 + (lane & 7);
        const uint32_t group = smem_addr(sm.data) + fw * 2048 + ((lane >> 3) & 1) * 1024;
        const uint32_t p_full0 = lead(sm.p_full[0][0]);
        RingPos<NSLOT> ring;
        uint32_t g = 0;
        // this CTA's copy of slot-wide pieces (dims 128 q ..) of the eight rows that lanes l0 .. l0 + 7 looked up
        auto copy_slot = [&](uint32_t slot, int q, int row_id, int l0) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int tk = 2 * u + (lane >> 4);
                const int rid = __shfl_sync(0xffffffffu, row_id, l0 + tk);
                const __nv_bfloat16* src = p.kv + (int64_t)(rid < 0 ? 0 : rid) * p.kv_ss + q * 128 + (lane & 15) * 8;
                cp_async16_zfill(group + slot * SLOT + tk * 128 + (((lane & 7) ^ tk) << 4), src, rid < 0 ? 0u : 16u);
            }
        };
        for (WalkerT wk(p, part); wk.valid(); wk.next()) {
            const Work w = wk.get();
            if (w.ntiles == 0) continue;
            if (p.q_tma) ring.skip(Q_SLOTS);
            const int* idx = p.indices + (int64_t)w.req * p.idx_ss;
            int id_next = tok < w.seqlen ? __ldg(idx + tok) : -1;      // (a tile ahead)
            int row_id = -1;
#pragma unroll 1
            for (int i = 0; i <= w.ntiles; ++i) {
                const int before = row_id;                             // tile i - 1
                const bool here = i < w.ntiles;
                if (here) {
                    row_id = id_next >= 0 && id_next < p.s_kv ? id_next : -1;
                    const uint32_t bal = __ballot_sync(0xffffffffu, row_id >= 0);
                    // token 32 w + l of the tile is bit l of word w
                    if (lane < 2) { reinterpret_cast<uint8_t*>(sm.mask[(g + i) % (2 * NTAB)])[(lane ? 1 - rank : rank) * 8 + fw] = (uint8_t)(bal >> (8 * lane)); __threadfence_block(); }
                    // (issued after the fence, which would otherwise wait for it)
                    { const int posn = (i + 1) * 2 * PAGE + tok; id_next = posn < w.seqlen ? __ldg(idx + posn) : -1; }
                    uint32_t bar = 0;
#pragma unroll 1
                    for (int q = 0; q < 4; ++q, ring.next()) {
                        READY_OR_WAIT(wt, &sm.empty[ring.slot], ring.par ^ 1, 201);
                        copy_slot(ring.slot, q, row_id, 0);
                        if (!(q & 1)) bar = ring.slot;
                        if (q == 1 || (!WIDE && q == 3)) cp_async_arrive_noinc(smem_addr(&sm.l_full[bar]));
                    }
                    if (WIDE) {
                        const uint32_t rs = (g + i) % NROPE;
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int tk = 4 * u + (lane >> 3);
                            const int rid = __shfl_sync(0xffffffffu, row_id, tk);
                            const __nv_bfloat16* src = p.kv + (int64_t)(rid < 0 ? 0 : rid) * p.kv_ss + 512 + (lane & 7) * 8;
                            cp_async16_zfill(smem_addr(sm.data) + AT_ROPE + rs * CHUNK + fw * 1024 + tk * 128 + (((lane & 7) ^ tk) << 4), src, rid < 0 ? 0u : 16u);
                        }
                        cp_async_arrive_noinc(smem_addr(&sm.l_full[bar]));
                    }
                }
                if (i > 0) {
                    // the other page of tile i - 1, over slots that its Q K^T has read
                    const uint32_t gp = g + i - 1;
                    READY_OR_WAIT(wt, rank == 0 ? &sm.k_done[gp & 1] : &sm.k_half[gp & 1], (gp >> 1) & 1, 203);
                    const uint32_t back = (here ? 8 : 4) - (rank == 0 ? 2 : 0);
                    int rid[8];                                        // (a row behind the tensor's last one reads zeros)
#pragma unroll
                    for (int k = 0; k < 8; ++k) { rid[k] = __shfl_sync(0xffffffffu, before, 8 + k); rid[k] = rid[k] < 0 ? p.s_kv : rid[k]; }
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const uint32_t dst = smem_addr(sm.data) + (ring.slot + NSLOT - back + k) % NSLOT * SLOT + fw * 2048;
#pragma unroll
                            for (int u = 0; u < 4; ++u)
                                tma2_gather4(dst + u * 512, &kmap, p_full0 + (gp & 1) * 16 + (1 - rank) * 8, (2 * rank + k) * 128 + (u >> 1) * 64,
                                             rid[(u & 1) * 4], rid[(u & 1) * 4 + 1], rid[(u & 1) * 4 + 2], rid[(u & 1) * 4 + 3]);
                        }
                    }
                    __syncwarp();
                }
            }
            g += w.ntiles;
        }
    } else if (SPARSE && warp >= W::FIRST_FEED) {
        regs_dec<W::FEEDING>();
        // ---------------- FP8 decode: records by address, four tokens of a page per warp ------------------------------------
        // 656-byte record = 512 e4m3 | 4 fp32 scales | 64 bf16 RoPE (512-wide form: 448 e4m3 | 64 bf16 RoPE).  A warp loads its raw bytes
        // straight into registers, a tile ahead (eight lanes per token, 16 bytes a lane: a slot's two chunks), converts them (one
        // rounding: bf16(fp32(e4m3) * scale)) when the slot is free, and stores 16 bytes at a time.  After Q K^T of a tile it stores this
        // CTA's half of the other page's dims over the slots of the half that the other CTA serves.
        const int fw = warp - W::FIRST_FEED, piece = lane & 3, ch = lane >> 4;
        const int r = fw * 4 + ((lane >> 2) & 3);                     // token of the page
        // (eight lanes: an even and an odd row, whose swizzle sends them to eight different 16-byte banks)
        const uint32_t row_at = smem_addr(sm.data) + (r >> 3) * 2048 + ch * 1024 + (r & 7) * 128 + (((2 * piece) ^ (r & 7)) << 4);
        const uint32_t lead0 = lead(sm.full[0]);
        auto lead_at = [&](uint64_t& bar) { return lead0 + (smem_addr(&bar) - smem_addr(&sm.full[0])); };
        const ulonglong2* tab = reinterpret_cast<const ulonglong2*>(sm.data + AT_TAB) + r;
        RingPos<NSLOT> ring;
        RingPos<NROPE> rope;
        uint32_t g = 0;
        auto load16 = [&](unsigned long long rec, int off) { return M1 || rec ? __ldg(reinterpret_cast<const uint4*>(rec + off)) : make_uint4(0, 0, 0, 0); };
        // slot q's share of a record: 16 e4m3 (512-wide form, chunk 7: 32 bytes of RoPE, the second half in `more`)
        auto is_rope = [&](int q) { return M1 && q == 3 && ch == 1; };
        auto load_share = [&](unsigned long long rec, int q, uint4& more) {
            if (is_rope(q)) more = load16(rec, 448 + piece * 32 + 16);
            return load16(rec, is_rope(q) ? 448 + piece * 32 : q * 128 + ch * 64 + piece * 16);
        };
        // (a scale word: fp32, or four exponent bytes of the 512-wide form)
        auto store_share = [&](uint32_t slot, int q, const uint4& raw, const uint4& more, uint32_t word) {
            uint4 lo = raw, hi = more;
            const float scale = M1 ? e8m0_of(word, 2 * (q & 1) + ch) : __uint_as_float(word);
            if (!is_rope(q)) dequant16(raw, scale, lo, hi);
            st_shared_v4(row_at + slot * SLOT, lo);
            st_shared_v4((row_at + slot * SLOT) ^ 16, hi);
        };
        for (WalkerT wk(p, part); wk.valid(); wk.next()) {
            const int ntiles = wk.get().ntiles;
            if (ntiles == 0) continue;
            if (p.q_tma) ring.skip(Q_SLOTS);
            uint4 raw[4], rope_raw = make_uint4(0, 0, 0, 0), raw_o[2], rope_o = make_uint4(0, 0, 0, 0);
            uint32_t sc[4] = {}, sc_o[2] = {};
            // (one turn before the first tile, to load it, and one behind the last, for its other page)
#pragma unroll 1
            for (int i = -1; i <= ntiles; ++i, ++g) {
                // g counts the tile i + 1
                const bool here = i >= 0 && i < ntiles;
                unsigned long long own = 0, own_sc = 0;
                if (i + 1 < ntiles) {
                    WAIT_WARP_OR_LEAVE(wt, &sm.tab_full[g % NTAB], (g / NTAB) & 1, 204);
                    const ulonglong2 e = tab[g % NTAB * ROWS + rank * PAGE];
                    own = e.x; own_sc = e.y;
                }
                if (M1 && i < ntiles) {
                    // (two slots at a time: with a RoPE chunk to store, 576-wide records are faster by single slots, 53.3 us against 55.4)
#pragma unroll
                    for (int q = 0; q < 4; q += 2) {
                        if (here) {
                            const uint32_t s0 = ring.slot, par0 = ring.par ^ 1;
                            ring.next();
                            const uint32_t s1 = ring.slot, par1 = ring.par ^ 1;
                            ring.next();
                            if (!__all_sync(0xffffffffu, mbar_try_wait(smem_addr(&sm.empty[s0]), par0, smem_addr(&sm.empty[s1]), par1))) {
                                WAIT_WARP_OR_LEAVE(wt, &sm.empty[s0], par0, 201);
                                WAIT_WARP_OR_LEAVE(wt, &sm.empty[s1], par1, 201);
                            }
                            store_share(s0, q, raw[q], rope_raw, sc[q]);
                            store_share(s1, q + 1, raw[q + 1], rope_raw, sc[q]);
                            fence_proxy_async_smem();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_remote_cta(lead0 + s0 * 8);
                        }
                        if (i + 1 < ntiles) {
                            raw[q] = load_share(own, q, rope_raw);
                            raw[q + 1] = load_share(own, q + 1, rope_raw);
                        }
                    }
                } else if (here) {
                    uint32_t bar = 0;
#pragma unroll
                    for (int q = 0; q < 4; ++q, ring.next()) {
                        WAIT_WARP_OR_LEAVE(wt, &sm.empty[ring.slot], ring.par ^ 1, 201);
                        store_share(ring.slot, q, raw[q], rope_raw, sc[q]);
                        if (!(q & 1)) bar = lead0 + ring.slot * 8;
                        if (q == 1) {
                            fence_proxy_async_smem();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_remote_cta(bar);
                        }
                        raw[q] = load_share(own, q, rope_raw);
                    }
                    st_shared_v4(smem_addr(sm.data) + AT_ROPE + rope.slot * CHUNK + r * 128 + (((ch * 4 + piece) ^ (r & 7)) << 4), rope_raw);
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote_cta(bar);
                    rope.next();
                } else if (i < 0) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) raw[q] = load_share(own, q, rope_raw);
                }
                if (i + 1 < ntiles) {
                    if (WIDE) rope_raw = load16(own, 528 + (ch * 4 + piece) * 16);
                    if (M1) { const uint2 e = __ldg(reinterpret_cast<const uint2*>(own_sc)); sc[0] = e.x; sc[2] = e.y; }
                    else { const uint4 e = load16(own_sc, 0); sc[0] = e.x; sc[1] = e.y; sc[2] = e.z; sc[3] = e.w; }
                }
                if (i > 0) {
                    // the other page of tile i - 1 (= g - 2), over slots that its Q K^T has read
                    const uint32_t gp = g - 2;
                    WAIT_WARP_OR_LEAVE(wt, rank == 0 ? &sm.k_done[gp & 1] : &sm.k_half[gp & 1], (gp >> 1) & 1, 203);
                    const uint32_t back = (here ? 8 : 4) - (rank == 0 ? 2 : 0);
#pragma unroll
                    for (int k = 0; k < 2; ++k) store_share((ring.slot + NSLOT - back + k) % NSLOT, 2 * rank + k, raw_o[k], rope_o, sc_o[k]);
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote_cta(lead_at(sm.p_full[gp & 1][1 - rank]));
                }
                if (here) {
                    const uint32_t gi = g - 1;
                    const ulonglong2 e = tab[gi % NTAB * ROWS + (1 - rank) * PAGE];
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_addr(&sm.tab_empty[gi % NTAB]));
                    if (M1) { sc_o[0] = sc_o[1] = __ldg(reinterpret_cast<const uint32_t*>(e.y) + rank); }
                    else { const uint2 x = e.y ? __ldg(reinterpret_cast<const uint2*>(e.y) + rank) : make_uint2(0, 0); sc_o[0] = x.x; sc_o[1] = x.y; }
#pragma unroll
                    for (int k = 0; k < 2; ++k) raw_o[k] = load_share(e.x, 2 * rank + k, rope_o);
                }
            }
            g -= 2;
        }
    } else {
        // ---------------- softmax, rescale and epilogue ---------------------------------------------------------
        if (!DENSE) regs_inc<W::SOFTMAX>();
        // S of this CTA's 64 rows lies in 64 columns: lanes 0..63 hold the rows' scores of page 0, lanes 64..127 of page 1; a
        // thread has a row, a page and (warpgroup) one half of the page's tokens.  O: 256 columns, lanes 0..63 dims 0..255, lanes
        // 64..127 dims 256..511; a thread has half of its lane's columns.
        const int wq = warp & 3, wg = (warp - 4) >> 2, page = wq >> 1;
        const int r = (wq & 1) * 32 + lane;                           // row of this CTA
        const int quarter = page * 2 + wg;
        const uint32_t tlane = tmem + ((uint32_t)(wq * 32) << 16);
        const int row = row0 + r;                                     // row inside the (request, kv head) group
        const bool row_ok = row < p.rows;
        const int t = SPARSE ? (int)blockIdx.y : (row_ok ? row / p.g : 0);
        const int hd = SPARSE ? (row_ok ? row : 0) : hk * p.g + (row_ok ? row - t * p.g : 0);
        float* xmax = reinterpret_cast<float*>(sm.data + AT_XMAX);
        const uint32_t prow = smem_addr(sm.data) + AT_P + page * CHUNK + r * 128;
        const uint32_t s_empty = lead(sm.s_empty), p_full0 = lead(sm.p_full[0][0]), o_empty = lead(sm.o_empty), q_ready = lead(sm.q_ready);
        const bool wide_out = (reinterpret_cast<uintptr_t>(p.out) & 31) == 0 &&
                              (PREFILL || ((p.o_sb | p.o_ss | p.o_sh) & 15) == 0);
        RingPos<NSLOT> ring, q_ring;
        uint32_t g = 0, nq = 0, ntail = 0;
        bool have_q = false, pending = false;
        WalkerT qw(p, part), wk(p, part);
        Work w;
        float m_run = -INFINITY, l_run = 0.f, m_true = -INFINITY;
        // These 256 threads meet at a named barrier at every request and where the guess was wrong, so none of them may leave alone: a warp
        // with an expired wait votes against the guess, stores nothing and announces nothing more until the barrier that carries the flag.
        while (true) {
            // ---- Q of the next request that has tiles, before this one's epilogue: its first Q K^T runs meanwhile
            for (; !have_q && qw.valid(); qw.next()) {
                const Work v = qw.get();
                if (v.ntiles == 0) continue;
                // (every MMA that read the previous request's Q has completed: this thread saw s_full of its last tile)
                if (p.q_tma) {
                    wt.wait(&sm.q_staged, nq & 1, 31);
#pragma unroll 1
                    for (int c = wg * 3; c < wg * 3 + 3; ++c) {
                        const uint8_t* src = sm.data + (q_ring.slot + c / 2) % NSLOT * SLOT + (c & 1) * CHUNK + r * 128;
                        uint32_t x[32];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const uint4 y = *reinterpret_cast<const uint4*>(src + ((i ^ (r & 7)) << 4));
                            x[4 * i] = y.x; x[4 * i + 1] = y.y; x[4 * i + 2] = y.z; x[4 * i + 3] = y.w;
                        }
                        tmem_st32(tlane + TM_Q + c * 32, x);
                    }
                    tmem_wait_st();
                    tc_fence_before();
                    BAR_OR_LEAVE(wt.expired());
                    if (threadIdx.x == 128) mbar_arrive(smem_addr(&sm.q_taken));
                    if (threadIdx.x < 128 + Q_SLOTS) mbar_arrive(smem_addr(&sm.empty[(q_ring.slot + threadIdx.x - 128) % NSLOT]));
                    q_ring.slot = (q_ring.slot + Q_SLOTS + 4 * v.ntiles) % NSLOT;
                } else {
                    const __nv_bfloat16* qrow = PREFILL ? p.q + (int64_t)v.req * p.q_ss + (int64_t)hd * p.q_sh
                                                        : p.q + (int64_t)v.req * p.q_sb + (int64_t)t * p.q_ss + (int64_t)hd * p.q_sh;
                    load_q_by_threads(sm, qrow, row_ok, wg, r, tlane, page == 0, !WIDE);
                    tmem_wait_st();
                    fence_proxy_async_smem();
                    tc_fence_before();
                    BAR_OR_LEAVE(wt.expired());
                }
                if (threadIdx.x == 128) mbar_arrive_remote_cta(q_ready);
                have_q = true;
                ++nq;
            }
            if (pending) {
                // ---- epilogue -----------------------------------------------------------------------------------------
                const bool has_tiles = w.ntiles > 0;
                if (has_tiles) wt.wait(&sm.pv_done, (g - 1) & 1, 32);
                tc_fence_after();
                const bool stores = row_ok && !wt.expired();              // (the flag of an expired wait goes on to the next barrier)
                const bool empty = !(l_run > 0.f) || !has_tiles;         // also catches NaN
                float scale = empty ? 0.f : 1.f / l_run;
                if (!DENSE && !w.is_split && p.attn_sink && !empty && row_ok)
                    scale = 1.f / (l_run + exp2f(p.attn_sink[hd] * kLog2e - m_run));
                // 32 words of a row at a time: 32 fp32 values of a partial, 64 16-bit ones of the output (a request without tiles reads
                // what is there and writes zeros)
                const uint32_t o_addr = tlane + TM_O + wg * 128;
                const int dim0 = page * 256 + wg * 128;
                unsigned long long to = 0;                               // where this thread's row goes
                if (w.is_split) {
                    const int64_t arow = ((int64_t)w.slot * p.s_q + t) * p.h_q + hd;
                    if (stores) to = reinterpret_cast<unsigned long long>(p.o_accum + arow * D_V + dim0);
                    if (stores && quarter == 0) p.lse_accum[arow] = empty ? -INFINITY : log2f(l_run) + m_run;
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        uint32_t v[32];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t x[16];
                            tmem_ld16(o_addr + c * 32 + h * 16, x);
                            tmem_wait_ld();
#pragma unroll
                            for (int e = 0; e < 16; ++e) v[h * 16 + e] = empty ? 0u : __float_as_uint(__uint_as_float(x[e]) * scale);
                        }
                        store_rows(v, to, c * 128, true, lane);
                    }
                } else {
                    const int64_t orow = PREFILL ? ((int64_t)w.req * p.h_q + hd) * D_V : (int64_t)w.req * p.o_sb + (int64_t)t * p.o_ss + (int64_t)hd * p.o_sh;
                    if (stores) to = reinterpret_cast<unsigned long long>(p.out + orow + dim0);
                    if (stores && quarter == 0) {
                        const float lse_nat = empty ? INFINITY : (log2f(l_run) + m_run) * kLn2;
                        if (PREFILL) {
                            p.lse[(int64_t)w.req * p.h_q + hd] = lse_nat;
                            p.max_logits[(int64_t)w.req * p.h_q + hd] = empty ? -INFINITY : m_true * kLn2;
                        } else {
                            p.lse[w.req * p.l_sb + t * p.l_ss + hd * p.l_sh] = lse_nat;
                        }
                    }
#pragma unroll 1
                    for (int c = 0; c < 2; ++c) {
                        uint32_t v[32];
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            uint32_t x[16];
                            tmem_ld16(o_addr + c * 64 + h * 16, x);
                            tmem_wait_ld();
#pragma unroll
                            for (int e = 0; e < 8; ++e)
                                v[h * 8 + e] = empty ? 0u : pack16<FP16>(__uint_as_float(x[2 * e]) * scale, __uint_as_float(x[2 * e + 1]) * scale);
                        }
                        store_rows(v, to, c * 128, wide_out, lane);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (has_tiles && lane == 0 && !wt.expired()) mbar_arrive_remote_cta(o_empty);
            }
            if (!wk.valid()) break;
            w = wk.get();
            wk.next();
            pending = true;
            if (w.ntiles == 0) continue;
            have_q = false;
            if (p.q_tma) ring.skip(Q_SLOTS);
            // first key position this row must NOT see (causal limit, and the end of this partition's range)
            const int limit = min(p.causal ? w.seqlen - (p.s_q - 1 - t) : w.seqlen, w.blk_end * PAGE);
            m_run = -INFINITY; l_run = 0.f; m_true = -INFINITY;
            for (int i = 0; i < w.ntiles; ++i, ++g) {
                wt.wait(&sm.s_full, g & 1, 33);
                tc_fence_after();
                uint32_t s[32];
                tmem_ld32(tlane + TM_S + wg * 32, s);
                const uint32_t valid = DENSE ? 0xffffffffu : sm.mask[g % (2 * NTAB)][quarter];      // (P needs it, and P V gives the tile's slots back: that keeps the entry)
                tmem_wait_ld();
                tc_fence_before();
                if (lane == 0 && !wt.expired()) mbar_arrive_remote_cta(s_empty);          // S may be overwritten
                if (!DENSE) {
                    if (valid != 0xffffffffu) {
#pragma unroll
                        for (int c = 0; c < 32; ++c)
                            if (!((valid >> c) & 1u)) s[c] = 0xff800000u;      // -inf
                    }
                } else {
                    const int nvalid = limit - (w.blk_begin + 2 * i + page) * PAGE - wg * 32;   // columns [0, nvalid) are visible
                    if (nvalid < 32) {
#pragma unroll
                        for (int c = 0; c < 32; ++c)
                            if (c >= nvalid) s[c] = 0xff800000u;          // -inf
                    }
                }
                float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    mx0 = fmaxf(mx0, __uint_as_float(s[c]));
                    mx1 = fmaxf(mx1, __uint_as_float(s[c + 1]));
                }
                const float mx = fmaxf(mx0, mx1) * p.scale_log2;   // scale > 0: max commutes with scaling
                m_true = fmaxf(m_true, mx);
                // P with the maximum in use, on the guess that no row of this CTA outgrows it: the warps vote on it while P is made.
                // Otherwise the rows' maxima are exchanged and P is made again; on a request's first tile that is always so, and nothing is
                // made on the guess (3 x 100 tokens 14.2 -> 13.7 us; the votes are cast all the same, so that their phases follow the tiles).
                volatile uint32_t& outgrown = sm.outgrown[g & 1];
                if (__any_sync(0xffffffffu, mx > m_run + RESCALE_THRESHOLD || wt.expired()) && lane == 0) outgrown = g + 1;
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_addr(&sm.vote[g & 1]));
                uint32_t pk[16];
                float sum0, sum1;
                auto make = [&] {
                    const float neg_m = m_run == -INFINITY ? 0.f : -m_run;
                    sum0 = 0.f; sum1 = 0.f;
#pragma unroll
                    for (int c = 0; c < 32; c += 2) {
                        const float e0 = ex2(fmaf(__uint_as_float(s[c]), p.scale_log2, neg_m));
                        const float e1 = ex2(fmaf(__uint_as_float(s[c + 1]), p.scale_log2, neg_m));
                        sum0 += e0; sum1 += e1;
                        pk[c >> 1] = pack16<FP16>(e0, e1);
                    }
                };
                auto store = [&] {
#pragma unroll
                    for (int ch = 0; ch < 4; ++ch)
                        st_shared_v4(prow + (((wg * 4 + ch) ^ (r & 7)) << 4), make_uint4(pk[4 * ch], pk[4 * ch + 1], pk[4 * ch + 2], pk[4 * ch + 3]));
                };
                if (i > 0) make();
                // P's buffer is free, and O may be touched, when the previous tile's P V has finished
                if (g > 0) wt.wait(&sm.pv_done, (g - 1) & 1, 34);
                if (i > 0) wt.wait(&sm.vote[g & 1], (g >> 1) & 1, 36);
                // something of this tile that all warps have a hand in
                bool together = i == 0 || __any_sync(0xffffffffu, outgrown == g + 1 || wt.expired());
                if (together) {
                    // ---- some row has outgrown its maximum (or a wait ran out)
                    xmax[quarter * HALF + r] = mx;
                    BAR_OR_LEAVE(wt.expired());
                    const float top = fmaxf(fmaxf(xmax[r], xmax[HALF + r]), fmaxf(xmax[2 * HALF + r], xmax[3 * HALF + r]));
                    float factor = 1.f;
                    if (top > m_run + RESCALE_THRESHOLD) {
                        factor = ex2(m_run - top);                     // m_run = -inf -> 0
                        l_run *= factor;
                        m_run = top;
                    }
                    if (i > 0 && __any_sync(0xffffffffu, factor != 1.f)) {
                        tc_fence_after();
                        rescale_o(tlane + TM_O + wg * 128, factor);
                    }
                    make();
                }
                store();
                l_run += sum0 + sum1;
                if (DENSE) {
                    // Tokens at or beyond the sequence length may hold anything (NaN included) in a real page: their probabilities
                    // are zero, so their V rows are zeroed to keep 0 * NaN out of O (Q K^T has read them).
#pragma unroll 1
                    for (int h = 0; h < 2; ++h) {
                        const int blk = w.blk_begin + 2 * i + h;
                        if (blk < w.blk_end && w.seqlen < (blk + 1) * PAGE) {
                            if (h != (int)rank) { wt.wait(&sm.f_tail, ntail & 1, 35); ++ntail; }
                            if (!wt.expired())
                                for (int n = 0; n < 2; ++n) zero_rows(sm.data + (ring.slot + 2 * h + n) % NSLOT * SLOT, max(w.seqlen - blk * PAGE, 0));
                            together = true;
                        }
                    }
                }
                ring.skip(4);
                fence_proxy_async_smem();                      // P and zeroed rows are read by the tensor core
                tc_fence_before();
                if (together) BAR_OR_LEAVE(wt.expired());
                __syncwarp();
                if (lane == 0 && !wt.expired()) {              // (prefill: CTA 0 adds the bytes that complete the barrier)
                    if (PREFILL && rank == 0 && (warp == 4 || warp == 6)) mbar_arrive_expect_tx(smem_addr(&sm.p_full[g & 1][page]), 2 * SLOT);
                    else mbar_arrive_remote_cta(p_full0 + (g & 1) * 16 + page * 8);
                }
            }
            // the row's sum (and true maximum) over its four quarters (the barrier of the next request's Q comes before the next use
            // of the buffers)
            xmax[quarter * HALF + r] = l_run;
            xmax[(4 + quarter) * HALF + r] = m_true;
            BAR_OR_LEAVE(wt.expired());
            l_run = (xmax[r] + xmax[HALF + r]) + (xmax[2 * HALF + r] + xmax[3 * HALF + r]);
            m_true = fmaxf(fmaxf(xmax[4 * HALF + r], xmax[5 * HALF + r]), fmaxf(xmax[6 * HALF + r], xmax[7 * HALF + r]));
        }
    }

wind_down:
    if (PREFILL && warp >= W::FIRST_FEED) cp_async_wait_all();      // this thread's own copies have landed
    if (wt.expired()) report_expired_wait(p.status, &sm.aborted, map_to_cta(smem_addr(&sm.aborted), rank ^ 1u), wt.code);
    tc_fence_before();
    if (__syncthreads_or((int)*reinterpret_cast<volatile uint32_t*>(&sm.aborted))) {
        // A bounded wait ran out in this CTA or in its peer; every thread of this CTA has left its role and issues nothing more.
        // Wait - bounded again - for the MMAs in flight (they read and write both CTAs' memory) ...
        if (warp == 1 && rank == 0 && elect_one()) {
            tc_commit2(smem_addr(&sm.drain));
            mbar_wait_bounded(smem_addr(&sm.drain), 0, DRAIN_LIMIT);
        }
    }
    cluster_sync();                                            // from here on neither CTA starts anything
    if (__syncthreads_or((int)*reinterpret_cast<volatile uint32_t*>(&sm.aborted))) {
        // ... and for the loads into either CTA's shared memory, whose bytes count on barriers nobody watches any more
        const long long t0 = clock64();
        while (clock64() - t0 < 400000LL) { }
    }
    cluster_sync();
    if (warp == 1) tmem_dealloc2(sm.tmem_base, 512);
}

template <int MODE, bool ALT>
static int launch(dim3 grid, const CUtensorMap& kmap, const CUtensorMap& rmap, const CUtensorMap& qmap, const Params& p, void* stream) {
    static bool configured[64] = {};
    if (int rc = configure_once(attn_pair_kernel<MODE, ALT>, configured, sizeof(Smem))) return rc;
    MLA_CHECK_CUDA(launch_dependent(attn_pair_kernel<MODE, ALT>, grid, dim3(Warps<MODE>::THREADS), sizeof(Smem), (cudaStream_t)stream, kmap, rmap, qmap, p));
    MLA_CHECK_CUDA(cudaGetLastError());
    return MLA_OK;
}

}  // namespace pair

// ---- self-test of the bounded wait: one CTA, one barrier nobody arrives on ---------------------------------
// Uses the same Waiter and the same reporting as the attention kernels, with nothing in flight (no TMA, no MMA, no
// cluster): the wait runs into its limit, the status words are written, the kernel returns normally.
__global__ void bounded_wait_selftest_kernel(int* status, uint32_t limit, int code, int* flag_out) {
    __shared__ uint64_t bar;
    __shared__ uint32_t flag;
    if (threadIdx.x == 0) { mbar_init(smem_addr(&bar), 1); flag = 0; fence_mbar_init(); }
    __syncthreads();
    Waiter w(limit);
    bool ok = threadIdx.x < 32 ? w.wait(&bar, 0, code) : w.wait_warp(&bar, 0, code);
    // a second wait by the same thread returns at once
    if (threadIdx.x < 32) ok = w.wait(&bar, 0, code + 1) || ok;
    if (w.expired()) report_expired_wait(status, &flag, 0u, w.code);
    __syncthreads();
    if (threadIdx.x == 0 && flag_out) { flag_out[0] = (int)flag; flag_out[1] = ok ? 1 : 0; }
}

// The two cache tensor maps of a dense launch depend only on the cache tensor (pointer, strides, pages, heads, type): a decode loop
// calls with the same cache every step, so the last encoding is kept per host thread.
struct PairMaps {
    const void* k_cache = nullptr;
    int64_t sb = 0, sr = 0, sh = 0;
    int num_blocks = 0, h_kv = 0, fp16 = 0;
    CUtensorMap kmap, rmap;
};

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

bool sparse_prefill_sm100_supports(const mla_sparse_prefill_args_t& a) {
    if ((a.d_qk != 576 && a.d_qk != 512) || a.d_v != 512 || a.h_kv != 1) return false;
    if (a.kv_stride_s <= 0 || a.kv_stride_s % 8 || a.kv_stride_s >= ((int64_t)1 << 39)) return false;
    if (!(a.sm_scale > 0.f)) return false;
    if (a.h_q > 128 * 65535) return false;
    return true;
}

bool sparse_decode_sm100_supports(const mla_sparse_decode_args_t& a) {
    if ((a.d_qk != 576 && a.d_qk != 512) || a.d_v != 512) return false;
    if (a.h_q > 128 || a.s_q > 65535 || a.num_sm_parts > 65535) return false;
    if (!(a.sm_scale > 0.f)) return false;
    if (reinterpret_cast<uintptr_t>(a.o_accum) & 31) return false;      // split partials leave with 256-bit stores
    return true;
}

int launch_dense_decode_pair(const mla_dense_decode_args_t& a) {
    using namespace sm100;
    EncodeTiledFn encode = get_encode_fn();
    if (!encode) return set_error(MLA_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const bool fp16 = a.dtype == MLA_DTYPE_FP16;
    const int head_chunks = a.h_kv > 1 ? (int)(a.k_stride_head / 64) : 9;
    static thread_local PairMaps cm;
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
    Params p = dense_params(a, head_chunks);
    p.row_blocks = (p.rows + pair::ROWS - 1) / pair::ROWS;
    CUtensorMap qmap;
    memset(&qmap, 0, sizeof(qmap));
    // boxes of q_unit rows: all 64 of a CTA where they are heads of one token or whole tokens, otherwise pieces that divide a
    // token's heads
    int unit = 64, box_h = 64, box_t = 1;
    if (a.s_q > 1) {
        while (p.g % unit) unit >>= 1;
        box_h = unit;
        if (unit == p.g) { box_t = 64 / unit; unit = 64; }
    }
    p.q_unit = unit;
    if (unit >= 8)                                         // (a swizzle atom)
        p.q_tma = encode_q_map(&qmap, a.q, a.b, a.s_q, a.h_q, a.q_stride_b, a.q_stride_s, a.q_stride_h, box_h, box_t, &p.q_box_bytes, fp16) ? 1 : 0;
    const dim3 grid(2, p.row_blocks * a.h_kv, a.num_sm_parts);
    return fp16 ? pair::launch<MODE_DENSE, true>(grid, cm.kmap, cm.rmap, qmap, p, a.stream)
                : pair::launch<MODE_DENSE, false>(grid, cm.kmap, cm.rmap, qmap, p, a.stream);
}

int launch_sparse_decode_pair(const mla_sparse_decode_args_t& a) {
    using namespace sm100;
    Params p = sparse_decode_params(a);
    p.row_blocks = 1;
    CUtensorMap unused, qmap;
    memset(&unused, 0, sizeof(unused));
    memset(&qmap, 0, sizeof(qmap));
    p.q_unit = pair::HALF;
    p.q_tma = encode_q_map(&qmap, a.q, a.b, a.s_q, a.h_q, a.q_stride_b, a.q_stride_s, a.q_stride_h, pair::HALF, 1, &p.q_box_bytes, false, a.d_qk) ? 1 : 0;
    const dim3 grid(2, a.s_q, a.num_sm_parts);
    return a.d_qk == 512 ? pair::launch<MODE_SPARSE_DECODE, true>(grid, unused, unused, qmap, p, a.stream)
                         : pair::launch<MODE_SPARSE_DECODE, false>(grid, unused, unused, qmap, p, a.stream);
}

int launch_sparse_prefill_pair(const mla_sparse_prefill_args_t& a) {
    using namespace sm100;
    Params p = prefill_params(a);
    p.row_blocks = (p.rows + pair::ROWS - 1) / pair::ROWS;
    CUtensorMap kmap, unused, qmap;
    // (a driver that refuses rows that overlap: the kernel for all shapes)
    if (!encode_kv_rows_map(&kmap, a)) return a.impl == 2 ? set_error(MLA_ERR_UNSUPPORTED, "mla_sparse_prefill_fwd: no tensor map over these keys") : launch_sparse_prefill_portable(a);
    memset(&unused, 0, sizeof(unused));
    memset(&qmap, 0, sizeof(qmap));
    p.q_unit = pair::HALF;
    p.q_tma = encode_q_map(&qmap, a.q, 1, a.s_q, a.h_q, 0, a.q_stride_s, a.q_stride_h, pair::HALF, 1, &p.q_box_bytes, false, a.d_qk) ? 1 : 0;
    int pairs = current_device_num_sms() / 2 / p.row_blocks;
    if (pairs < 1) pairs = 1;
    if (pairs > a.s_q) pairs = a.s_q;
    const dim3 grid(2, p.row_blocks, pairs);
    return a.d_qk == 512 ? pair::launch<MODE_PREFILL, true>(grid, kmap, unused, qmap, p, a.stream)
                         : pair::launch<MODE_PREFILL, false>(grid, kmap, unused, qmap, p, a.stream);
}

}  // namespace mla
