// What the GEMM kernels share: element types, activations, expansion of quantised weights.
#pragma once
#include "common.cuh"
#include "sm100_ptx.cuh"

namespace ovb {

constexpr int TILE_N = 128;      // weight rows of a tile (MMA M per CTA)
constexpr int TILE_K = 64;       // bf16 elements per k-block = one 128-byte swizzle span

template <bool F16>
struct Elem {
    using type = __nv_bfloat16;
};
template <>
struct Elem<true> {
    using type = __half;
};

__device__ __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float to_float(__half v) { return __half2float(v); }
template <class E>
__device__ __forceinline__ E from_float(float v);
template <>
__device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) {
    return __float2bfloat16_rn(v);
}
template <>
__device__ __forceinline__ __half from_float<__half>(float v) {
    return __float2half_rn(v);
}

// cap * tanh(v / cap); the error is of the order of an ulp of cap.
__device__ __forceinline__ float soft_cap(float v, float cap) { return cap - __fdividef(2.0f * cap, 1.0f + __expf(__fdividef(2.0f * v, cap))); }

// Two fp32 values in a register pair: one instruction for both.
__device__ __forceinline__ uint64_t pair_of(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t pair_of(float a) { return pair_of(a, a); }
__device__ __forceinline__ void unpair(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// v * Phi(v) of two values. With x = |v| and h = Phi(-x) it is max(v, 0) - x h: no cancellation for positive v, and for negative v none
// that h does not have. h = 1/2 - x P(x^2) up to 1.6, exp(-x^2 / 2) Q(x) above (from 5.5 on, where h < 2e-8, with Q(5.5)). P and Q are
// minimax fits (Lawson's iteration on Chebyshev nodes): P - a0, of degree 6, within 3e-9 of (Phi(x) - 1/2) / x; Q, of degree 7, such that
// h is within 3e-9. Error against 64 bits, rms (largest): v in (0.01, 3) 2.9e-8 (1.1e-7) of the value, 0.5 v (1 + erff(v / sqrt 2))
// has 3.8e-8 (1.3e-7); (-1, -0.01) 4.2e-8 (1.5e-7), there 5.0e-8 (2.2e-7); (-2, -1) 1.4e-7 (6.9e-7), there 1.9e-7 (1.0e-6).
// The epilogue's instructions set the time of short products: 6144 x 4096 x 1024 in fp16, cold caches, 102 us with erff, 76 us with this (58 us
// without an activation; erfc by Abramowitz and Stegun 7.1.26, four times as far off as erff over (0.01, 3), 78 us).
__device__ __forceinline__ void gelu_erf2(float& v0, float& v1) {
    const uint64_t v = pair_of(v0, v1), s = mul2(v, v);
    const uint64_t nx = pair_of(fmaxf(-fabsf(v0), -5.5f), fmaxf(-fabsf(v1), -5.5f));      // -x
    uint64_t p = pair_of(3.88307512e-07f);
    p = fma2(p, s, pair_of(-8.56560655e-06f));
    p = fma2(p, s, pair_of(0.000113983522f));
    p = fma2(p, s, pair_of(-0.00118607341f));
    p = fma2(p, s, pair_of(0.00997303519f));
    p = fma2(p, s, pair_of(-0.0664903f));
    p = fma2(p, s, pair_of(-1.34248355e-08f));
    uint64_t q = pair_of(1.29784776e-05f);
    q = fma2(q, nx, pair_of(0.000298278086f));
    q = fma2(q, nx, pair_of(0.00303096278f));
    q = fma2(q, nx, pair_of(0.0180309042f));
    q = fma2(q, nx, pair_of(0.0701728687f));
    q = fma2(q, nx, pair_of(0.189219281f));
    q = fma2(q, nx, pair_of(0.363507748f));
    q = fma2(q, nx, pair_of(0.490691155f));
    float h0, h1, a0, a1, e0, e1;
    unpair(fma2(nx, p, fma2(nx, pair_of(0.398942292f), pair_of(0.5f))), a0, a1);
    unpair(mul2(s, pair_of(-0.72134752f)), e0, e1);
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e0));
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e1));
    unpair(mul2(pair_of(e0, e1), q), h0, h1);
    if (fabsf(v0) <= 1.6f) h0 = a0;                    // (NaN takes the other branch and stays)
    if (fabsf(v1) <= 1.6f) h1 = a1;
    unpair(fma2(nx, pair_of(h0, h1), pair_of(fmaxf(v0, 0.f), fmaxf(v1, 0.f))), v0, v1);
}
__device__ __forceinline__ float gelu_erf(float v) {
    float other = 0.f;
    gelu_erf2(v, other);
    return v;
}

// Activations of the epilogue; P carries `act` and the limits of the GEMM's arguments.
template <class P>
__device__ __forceinline__ float apply_act(float v, const P& p) {
    switch (p.act) {
        case OVB_ACT_GELU_ERF: return gelu_erf(v);
        case OVB_ACT_RELU: return v > 0.f ? v : 0.f;
        case OVB_ACT_SILU: return v / (1.0f + __expf(-v));
        case OVB_ACT_GELU_TANH: {
            float u = 0.7978845608028654f * (v + 0.044715f * v * v * v);
            return 0.5f * v * (1.0f + tanhf(u));
        }
        case OVB_ACT_RELU2: return v > 0.f ? v * v : 0.f;
        case OVB_ACT_SOFTCAP: return soft_cap(v, p.act_limit);
        default: return v;
    }
}

// The same for N values. The choice is outside the loop: sixteen unrolled copies of the switch do not fit the instruction cache.
template <int N, class P>
__device__ __forceinline__ void apply_act_n(float (&v)[N], const P& p) {
    static_assert(N % 2 == 0, "pairs");
    switch (p.act) {
        case OVB_ACT_NONE: break;
        case OVB_ACT_GELU_ERF:
#pragma unroll
            for (int j = 0; j < N; j += 2) gelu_erf2(v[j], v[j + 1]);
            break;
        case OVB_ACT_SILU:
#pragma unroll
            for (int j = 0; j < N; ++j) v[j] = v[j] / (1.0f + __expf(-v[j]));
            break;
        case OVB_ACT_RELU:
#pragma unroll
            for (int j = 0; j < N; ++j) v[j] = v[j] > 0.f ? v[j] : 0.f;
            break;
        case OVB_ACT_RELU2:
#pragma unroll
            for (int j = 0; j < N; ++j) v[j] = v[j] > 0.f ? v[j] * v[j] : 0.f;
            break;
        default:                            // the rare ones: one copy of the code
#pragma unroll 1
            for (int j = 0; j < N; ++j) {
                float one = 0.f;
#pragma unroll
                for (int i = 0; i < N; ++i) one = i == j ? v[i] : one;
                one = apply_act(one, p);
#pragma unroll
                for (int i = 0; i < N; ++i) v[i] = i == j ? one : v[i];
            }
    }
}

// Clamped gate and up values with a sigmoid of adjustable slope (OVB_ACT_GLU_LIMITED).
template <class P>
__device__ __forceinline__ float glu_limited(const P& p, float g, float u) {
    g = fminf(g, p.act_limit);
    u = fminf(fmaxf(u, -p.act_limit), p.act_limit);
    return g / (1.0f + __expf(-p.act_slope * g)) * (u + p.act_shift);
}

// Integers to bf16 without shifts: the bits 0..7 of a bf16 are linear in value down to zero (sub-normals and the first binade have
// the same spacing), so an integer b < 256 in the low byte of a 16-bit lane reads as b * 2^-133, and a nibble in bits 4..7 as
// 16 q * 2^-133. One fused multiply-add by 2^127 (2^123) makes that (b - z) / 64, exact; the product with 64 * scale is then rounded
// once, like (b - z) * scale. u4: five integer instructions per eight weights instead of eight (shift and merge per pair), which
// bound the kernel (ALU pipe 67 % busy on average); u8: one per pair instead of conversions (XU pipe 76 % busy). Zero points are whole.
// 128256 x 4096 weights: u4 T = 1 109 -> 94 us, T = 64 125 -> 109 us; u8 T = 24 177 -> 119 us (cold caches).
struct RowScale {
    __nv_bfloat162 m, s;        // -z / 64 and 64 * scale, twice each
};
// `szp`: (scale, bias + zero point) of a row and group; bias 16 for u4, 0 for u8
__device__ __forceinline__ RowScale row_scale(__nv_bfloat162 szp, float bias) {
    const __nv_bfloat162 zz = __halves2bfloat162(__high2bfloat16(szp), __high2bfloat16(szp)), ss = __halves2bfloat162(__low2bfloat16(szp), __low2bfloat16(szp));
    return {__hmul2(__hsub2(__float2bfloat162_rn(bias), zz), __float2bfloat162_rn(0.015625f)), __hmul2(ss, __float2bfloat162_rn(64.f))};
}
__device__ __forceinline__ uint32_t lane_fma(uint32_t bits, uint32_t mul, const RowScale& r) {
    const __nv_bfloat162 v = __hmul2(__hfma2(*reinterpret_cast<__nv_bfloat162*>(&bits), *reinterpret_cast<__nv_bfloat162*>(&mul), r.m), r.s);
    return *reinterpret_cast<const uint32_t*>(&v);
}
constexpr uint32_t kTwo127 = 0x7F007F00u, kTwo123 = 0x7D007D00u;      // bf16 pairs
// Expand one u32 (8 packed u4 in the plugin nibble order) to 8 bf16: (q - zp) * scale.
__device__ __forceinline__ uint4 dequant_u4x8(uint32_t x, const RowScale& r) {
    const uint32_t y = x >> 8;
    return make_uint4(lane_fma(x & 0x000F000Fu, kTwo127, r), lane_fma(x & 0x00F000F0u, kTwo123, r), lane_fma(y & 0x000F000Fu, kTwo127, r),
                      lane_fma(y & 0x00F000F0u, kTwo123, r));
}
// Four bytes -> four bf16: (b - zp) * scale.
__device__ __forceinline__ void dequant_u8x4(uint32_t w, const RowScale& r, uint32_t& lo, uint32_t& hi) {
    lo = lane_fma(__byte_perm(w, 0u, 0x4140), kTwo127, r);
    hi = lane_fma(__byte_perm(w, 0u, 0x4342), kTwo127, r);
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

constexpr bool is_quant(int wmode) { return wmode == OVB_W_U4 || wmode == OVB_W_U8 || wmode == OVB_W_F8; }
constexpr int wq_bytes(int wmode) { return wmode == OVB_W_U4 ? TILE_N * 32 : ((wmode == OVB_W_U8 || wmode == OVB_W_F8) ? TILE_N * 64 : 0); }

// Four fp8 e4m3 values -> four bf16 (two words), each scaled: an e4m3 value at bits 4..10 (sign at 15) of a bf16 reads as
// value * 2^-120 (sub-normals included), and the per-block scale in `ss` already carries the 2^120. The weight is packed so that
// the first two values of a word lie in these bits of its two 16-bit lanes as they are; of the other two the sign is bit 11, the
// upper three exponent bits are bits 12..14 and the rest bits 0..3 (PackedWeight.from_f8_block). Five integer instructions for four
// values; the plain byte order takes nine, and those bound the kernel. A step
// of 32 tokens through two layers of a 70B model and its vocabulary projection: products 774 -> 618 us.
__device__ __forceinline__ void dequant_f8x4(uint32_t w, __nv_bfloat162 ss, uint32_t& lo, uint32_t& hi) {
    uint32_t t0 = w & 0x87F087F0u;
    uint32_t t1 = ((w << 4) & 0x80F080F0u) | ((w >> 4) & 0x07000700u);
    __nv_bfloat162 v0 = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&t0), ss);
    __nv_bfloat162 v1 = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&t1), ss);
    lo = *reinterpret_cast<uint32_t*>(&v0);
    hi = *reinterpret_cast<uint32_t*>(&v1);
}

// gemm_pair.cu: products of many tokens on pairs of CTAs. gemm_pair_takes() says whether it runs the problem.
bool gemm_pair_takes(const ovb_gemm_args* a);
int gemm_pair(const ovb_gemm_args* a, cudaStream_t stream);
// gemm_few.cu: products of up to 64 tokens with quantised weights.
bool gemm_few_takes(const ovb_gemm_args* a);
int gemm_few(const ovb_gemm_args* a, cudaStream_t stream);
// Clusters of this many CTAs that the current device holds, one CTA of gemm_few.cu's size per SM, asked of the driver once per device.
int cluster_capacity(int size);
// The RMS norm of a product's few rows, by the whole CTA: every thread holds HOLD pieces of eight columns of each of T rows of x (it reads the rows in
// whole, whatever part of K its CTA has) and calls put(token, piece of eight columns, normalised values). `part`: [warps][TMAX] floats of shared
// memory. The caller's barrier must follow. Loads come from L2: the rows were written by the kernel before.
template <int THREADS, int TMAX, int HOLD, class P, class F>
__device__ __forceinline__ void norm_rows(const P& p, float (*part)[TMAX], F&& put) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pieces = p.K >> 3;
    uint4 x[TMAX][HOLD], g[HOLD];
#pragma unroll
    for (int h = 0; h < HOLD; ++h) {
        const int k8 = threadIdx.x + h * THREADS;
        if (k8 < pieces) g[h] = __ldg(reinterpret_cast<const uint4*>(p.x_norm) + k8);
    }
#pragma unroll
    for (int t = 0; t < TMAX; ++t) {
        if (t >= p.T) break;
        int row = t;
        if (p.x_rows != nullptr) {
            row = p.x_rows[t];
            if (row < 0 || row >= p.x_count) row = 0;
        }
        const uint4* src = reinterpret_cast<const uint4*>(p.x + (size_t)row * p.ldx * 2);
#pragma unroll
        for (int h = 0; h < HOLD; ++h) {
            const int k8 = threadIdx.x + h * THREADS;
            if (k8 < pieces) x[t][h] = __ldcg(src + k8);
        }
    }
#pragma unroll
    for (int t = 0; t < TMAX; ++t) {
        if (t >= p.T) break;
        float ss = 0.f;
#pragma unroll
        for (int h = 0; h < HOLD; ++h)
            if (threadIdx.x + h * THREADS < pieces) {
                const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&x[t][h]);
#pragma unroll
                for (int j = 0; j < 8; ++j) ss += __bfloat162float(e[j]) * __bfloat162float(e[j]);
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) part[warp][t] = ss;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
#pragma unroll
    for (int t = 0; t < TMAX; ++t) {
        if (t >= p.T) break;
        float tot = lane < THREADS / 32 ? part[lane][t] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
        const float inv = rsqrtf(tot / float(p.K) + p.x_eps);
#pragma unroll
        for (int h = 0; h < HOLD; ++h) {
            const int k8 = threadIdx.x + h * THREADS;
            if (k8 >= pieces) continue;
            const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&x[t][h]);
            const __nv_bfloat16* ge = reinterpret_cast<const __nv_bfloat16*>(&g[h]);
            uint4 o;
            __nv_bfloat16* oe = reinterpret_cast<__nv_bfloat16*>(&o);
#pragma unroll
            for (int j = 0; j < 8; ++j) oe[j] = __float2bfloat16_rn(__bfloat162float(e[j]) * inv * __bfloat162float(ge[j]));
            put(t, k8, o);
        }
    }
}

// gemm_ring.cu: products of up to four tokens with u4 weights.
bool gemm_ring_takes(const ovb_gemm_args* a);
bool gemm_ring_norms(const ovb_gemm_args* a);
int gemm_ring(const ovb_gemm_args* a, cudaStream_t stream);
// gemm_stream.cu: products of few tokens, small ones.
bool gemm_stream_takes(const ovb_gemm_args* a);
bool gemm_stream_norms(const ovb_gemm_args* a);
int gemm_stream(const ovb_gemm_args* a, cudaStream_t stream);

}  // namespace ovb
