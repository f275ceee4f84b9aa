// FP8 KV-cache writer: bf16 token rows [576] -> 656-byte records (512 e4m3 | 4 fp32 scales | 64 bf16 RoPE), the
// format the sparse decode kernels read.  Follows the reference's test quantiser value for value
// (tests/quant.py:20-53 of the reference: scale = amax / 448 per group of 128, optionally rounded up to a power of
// two; q = e4m3(x / scale), round to nearest even).
//
// A warp takes a token; lane l holds values 16l .. 16l+15 (8 lanes per scale group), so the record's e4m3 part is one coalesced
// 512-byte store.  1152 bytes read + 656 bytes written per token.  The quotients x / s only need the correctly rounded reciprocal
// of s, once per group, and three instructions each (Markstein's theorem; quotient16 below), two values per instruction.  66 K
// tokens take 23.3 us (5.1 TB/s), 256 K 87 us (5.3 TB/s), back to back on one input; with inputs that change 66 K took 26.2 (28.7 with
// two tokens per warp and scalar instructions) and take 23.7 in the launch chain below.  Registers count: with two tokens per warp (75 of them in the place of 47)
// 26.6 and 96.7 us; with the scalar instructions, two / one token per warp, 27.3 / 26.8 and 98.2 / 99.2.  A persistent grid that
// loads a token ahead is no faster (27.3).
//
// Layout 1 is the 512-wide "MODEL1" form (tests/quant.py:55-75 of the reference): 448 values in groups of 64 with
// power-of-two scales stored as e8m0 bytes, 64 bf16 RoPE values; a block is block_size x 576 value bytes followed by
// block_size x 8 scale bytes (7 scales + 1 pad).  Lanes 0-27 hold the quantised values (4 lanes per group), lanes 28-31
// the RoPE part.  A warp of a long call takes two tokens, whose loads are in flight together, with registers for 32 warps per SM
// (20 bytes of them spilled), in blocks of four warps (of eight: 45 K tokens 17.7 us, four 17.1; 66 K 25.3, 24.6; 256 K 91.5, 89.5; the 656-byte
// form loses, 23.7, 24.3).  Before that and the launch chain: 66 K tokens 27.2 us, 256 K 92.9 (one token per warp 27.2 and 101, scalar instructions 35.5 and
// 131.7).  A short call is bound by its own latency and takes one (MODEL1_TWO_FROM).  The first warps also zero
// the `pad_bytes` behind every block, where the caller owns them (one warp a block; with the last token's stores, inside the
// loop, 66 K tokens took 36.9 us instead of 34.9, on the scalar kernel).
#include "common.cuh"

#include <cuda_fp8.h>

namespace mla {

// Layout 1, more tokens than this: two per warp, up to it one.  us, one / two tokens per warp, inputs changing: 64 tokens 1.55 / 2.15, 4 K 2.5 / 3.1,
// 16 K 7.88 / 7.97, 26 K 11.26 / 11.20, 33 K 13.7 / 13.9, 40 K 16.3 / 16.6, 45 K 18.2 / 17.9, 66 K 25.7 / 25.0, 131 K 49.2 / 46.8, 256 K 94.2 / 88.6.
constexpr int64_t MODEL1_TWO_FROM = 40000;

__device__ __forceinline__ float pow2_ceil(float s) {
    // smallest power of two >= s (s > 0, normal)
    const uint32_t bits = __float_as_uint(s);
    const uint32_t mant = bits & 0x007fffffu;
    return __uint_as_float((bits & 0x7f800000u) + (mant ? 0x00800000u : 0u));
}

// two fp32 operations in one instruction
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\tfma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}

// A lane's 16 values, NEGATED (what the quotients below start from), and their largest magnitude.
__device__ __forceinline__ void unpack16(const uint4& v0, const uint4& v1, float (&f)[16], float& amax) {
    const uint32_t w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    amax = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16 ^ 0x80000000u);
        f[2 * i + 1] = __uint_as_float((w[i] & 0xffff0000u) ^ 0x80000000u);
        amax = fmaxf(amax, fmaxf(fabsf(f[2 * i]), fabsf(f[2 * i + 1])));
    }
}

// e4m3(x / s) of a lane's 16 values (f holds -x), x / s rounded to fp32 first.  With r = RN(1 / s) and q = RN(x r), q + r (x - q s)
// is RN(x / s) (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34, 1990; here checked for every bf16 significand against every fp32 significand of s).  It is computed as
// q + (-r) (q s - x): for x = -0 the remainder q s - x is -0 + 0 = +0 and the sum -0 + -0 keeps the sign, where
// x - q s = +0 would give +0 + -0 = +0.  The remainder has to be exact: the
// group's largest magnitude `amax` keeps clear of overflow and underflow, and values so far below it that the remainder
// could be subnormal (below 2^-20 amax) have quotients under 2^-11, which are zeros in e4m3 whatever their last bit.
// Groups outside that range (warp-uniform choice) divide.
__device__ __forceinline__ uint4 quotient16(const float (&f)[16], float s, float amax) {
    const bool plain = (amax >= 0x1p-60f && amax <= 0x1p100f) || amax == 0.f;
    uint32_t q[4];
    if (__all_sync(0xffffffffu, plain)) {
        const float r = -__frcp_rn(s);
        const float2 r2 = make_float2(r, r), s2 = make_float2(s, s);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float2 d[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const float2 nx = make_float2(f[4 * i + 2 * k], f[4 * i + 2 * k + 1]), q0 = mul2(nx, r2);
                d[k] = fma2(fma2(q0, s2, nx), r2, q0);
            }
            q[i] = (uint32_t)__nv_cvt_float2_to_fp8x2(d[0], __NV_SATFINITE, __NV_E4M3) |
                   (uint32_t)__nv_cvt_float2_to_fp8x2(d[1], __NV_SATFINITE, __NV_E4M3) << 16;
        }
    } else {
#pragma unroll 1
        for (int i = 0; i < 4; ++i) {
            uint32_t word = 0;
#pragma unroll
            for (int k = 0; k < 16; ++k)
                if (k >> 2 == i) word |= (uint32_t)__nv_cvt_float_to_fp8(__fdiv_rn(-f[k], s), __NV_SATFINITE, __NV_E4M3) << (8 * (k & 3));
            if (i == 0) q[0] = word; else if (i == 1) q[1] = word; else if (i == 2) q[2] = word; else q[3] = word;
        }
    }
    return make_uint4(q[0], q[1], q[2], q[3]);
}

// 32-bit division where the token count allows
__device__ __forceinline__ void block_of(int64_t tok, int64_t ntok, int block_size, int64_t& blk, int64_t& row) {
    blk = ntok <= 0x7fffffff ? (int64_t)((uint32_t)tok / (uint32_t)block_size) : tok / block_size;
    row = tok - blk * block_size;
}

// The writers are launched as dependents of what is before them in the stream, and let their own dependents start when all their CTAs
// have: back to back, the next call's CTAs are there when this one's last wave ends (66 K tokens 26.5 -> 23.7 us, inputs changing).  What a single call
// between two ordinary kernels adds to them, as a plain launch / now: 1 K tokens 3.0 / 2.2 us, 8 K 4.7 / 4.0, 66 K 23.6 / 22.75; 512-wide 2.6 / 1.9, 5.0 /
// 4.1, 26.2 / 25.0 (the blocks of four warps among it).
__device__ __forceinline__ void join_chain() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__global__ void __launch_bounds__(256)
quantize_fp8_kernel(const mla_quantize_args_t a) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t ntok = (int64_t)a.num_blocks * a.block_size;
    join_chain();
    for (int64_t tok = warp; tok < ntok; tok += nwarps) {
        int64_t blk, row;
        block_of(tok, ntok, a.block_size, blk, row);
        const __nv_bfloat16* x = (const __nv_bfloat16*)a.x + blk * a.x_stride_block + row * a.x_stride_row;
        uint8_t* out = (uint8_t*)a.out + blk * a.out_stride_block_bytes + row * 656;
        const uint4 v0 = __ldcs(reinterpret_cast<const uint4*>(x + lane * 16));
        const uint4 v1 = __ldcs(reinterpret_cast<const uint4*>(x + lane * 16 + 8));
        uint4 rope;
        if (lane < 8) rope = __ldcs(reinterpret_cast<const uint4*>(x + 512 + lane * 8));
        float f[16], amax;
        unpack16(v0, v1, f, amax);
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
        float s = __fdiv_rn(amax, 448.f);
        s = a.pow2_scale ? pow2_ceil(fmaxf(s, 1e-4f)) : fmaxf(s, 1e-30f);
        *reinterpret_cast<uint4*>(out + lane * 16) = quotient16(f, s, amax);
        const float sg = __shfl_sync(0xffffffffu, s, (lane & 3) * 8);          // lanes 0-3: scale of group `lane`
        if (lane < 4) reinterpret_cast<float*>(out + 512)[lane] = sg;
        if (lane < 8) *reinterpret_cast<uint4*>(out + 528 + lane * 16) = rope;
    }
}

// TOKENS: tokens per warp, in flight together
template <int TOKENS>
__global__ void __launch_bounds__(128, 8)
quantize_fp8_model1_kernel(const mla_quantize_args_t a, const int pad_bytes) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t ntok = (int64_t)a.num_blocks * a.block_size;
    join_chain();
    if (pad_bytes)
#pragma unroll 1
        for (int64_t blk = warp; blk < a.num_blocks; blk += nwarps)
            for (int i = lane * 8; i < pad_bytes; i += 256)
                *reinterpret_cast<uint2*>((uint8_t*)a.out + blk * a.out_stride_block_bytes + (int64_t)a.block_size * 584 + i) = make_uint2(0, 0);
    for (int64_t tok0 = warp * TOKENS; tok0 < ntok; tok0 += nwarps * TOKENS) {
        uint4 v0[TOKENS], v1[TOKENS];
        int64_t blk[TOKENS], row[TOKENS];
#pragma unroll
        for (int k = 0; k < TOKENS; ++k) {
            if (tok0 + k >= ntok) break;
            block_of(tok0 + k, ntok, a.block_size, blk[k], row[k]);
            const __nv_bfloat16* x = (const __nv_bfloat16*)a.x + blk[k] * a.x_stride_block + row[k] * a.x_stride_row;
            v0[k] = __ldcs(reinterpret_cast<const uint4*>(x + lane * 16));
            v1[k] = __ldcs(reinterpret_cast<const uint4*>(x + lane * 16 + 8));
        }
#pragma unroll
        for (int k = 0; k < TOKENS; ++k) {
            if (tok0 + k >= ntok) break;
            uint8_t* block = (uint8_t*)a.out + blk[k] * a.out_stride_block_bytes;
            uint8_t* out = block + row[k] * 576;
            float f[16], amax;
            unpack16(v0[k], v1[k], f, amax);
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
            const float s = pow2_ceil(fmaxf(__fdiv_rn(amax, 448.f), 1e-4f));
            const uint4 q = quotient16(f, s, lane < 28 ? amax : 0.f);
            if (lane < 28) {
                *reinterpret_cast<uint4*>(out + lane * 16) = q;
            } else {
                *reinterpret_cast<uint4*>(out + 448 + (lane - 28) * 32) = v0[k];
                *reinterpret_cast<uint4*>(out + 448 + (lane - 28) * 32 + 16) = v1[k];
            }
            // lane g < 7 writes the scale of group g (held by lanes 4g .. 4g+3) as its exponent byte; lane 7 the pad byte
            const float sg = __shfl_sync(0xffffffffu, s, (lane & 7) * 4);
            uint8_t* scales = block + (int64_t)a.block_size * 576;
            if (lane < 8) scales[row[k] * 8 + lane] = lane < 7 ? (uint8_t)(__float_as_uint(sg) >> 23) : 0;
        }
    }
}

int launch_quantize_fp8(const mla_quantize_args_t& a, bool zero_padding) {
    MLA_CHECK_ARG(a.x && a.out, "mla_quantize_fp8_kvcache: x and out must not be null");
    MLA_CHECK_ARG(a.num_blocks > 0 && a.block_size > 0, "mla_quantize_fp8_kvcache: num_blocks and block_size must be positive");
    MLA_CHECK_ARG(a.layout == 0 || a.layout == 1, "mla_quantize_fp8_kvcache: layout must be 0 (656-byte records) or 1 (MODEL1)");
    const int d = a.layout ? 512 : 576, rec = a.layout ? 584 : 656;
    MLA_CHECK_ARG(is_aligned16(a.x) && a.x_stride_block % 8 == 0 && a.x_stride_row % 8 == 0 && a.x_stride_row >= d,
                  "mla_quantize_fp8_kvcache: x must be 16-byte aligned with strides that are multiples of 8 elements");
    MLA_CHECK_ARG(is_aligned16(a.out) && a.out_stride_block_bytes % 16 == 0 && a.out_stride_block_bytes >= (int64_t)a.block_size * rec,
                  "mla_quantize_fp8_kvcache: out must be 16-byte aligned, block stride a multiple of 16 bytes and >= block_size * %d", rec);
    // (records and stride are multiples of 8 bytes, so the padding is too)
    const int64_t pad_bytes = zero_padding && a.layout ? a.out_stride_block_bytes - (int64_t)a.block_size * rec : 0;
    MLA_CHECK_ARG(pad_bytes <= 0x7fffff00, "mla_quantize_fp8_kvcache_padded: more than 2 GB of padding behind a block");
    const int64_t ntok = (int64_t)a.num_blocks * a.block_size;
    const int per_warp = a.layout && ntok > MODEL1_TWO_FROM ? 2 : 1, warps = a.layout ? 4 : 8, per_block = warps * per_warp;      // tokens
    const int64_t blocks = min((ntok + per_block - 1) / per_block, (int64_t)1 << 24);
    const cudaStream_t stream = (cudaStream_t)a.stream;
    const dim3 grid((unsigned)blocks), block(32 * warps);
    MLA_CHECK_CUDA(!a.layout       ? launch_dependent(quantize_fp8_kernel, grid, block, 0, stream, a)
                   : per_warp == 2 ? launch_dependent(quantize_fp8_model1_kernel<2>, grid, block, 0, stream, a, (int)pad_bytes)
                                   : launch_dependent(quantize_fp8_model1_kernel<1>, grid, block, 0, stream, a, (int)pad_bytes));
    MLA_CHECK_CUDA(cudaGetLastError());
    return MLA_OK;
}

}  // namespace mla
