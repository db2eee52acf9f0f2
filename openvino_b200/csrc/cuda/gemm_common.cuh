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

// Activations of the epilogue; P carries `act` and the limits of the GEMM's arguments.
template <class P>
__device__ __forceinline__ float apply_act(float v, const P& p) {
    switch (p.act) {
        case OVB_ACT_GELU_ERF: return 0.5f * v * (1.0f + erff(v * 0.70710678118654752f));
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

// Clamped gate and up values with a sigmoid of adjustable slope (OVB_ACT_GLU_LIMITED).
template <class P>
__device__ __forceinline__ float glu_limited(const P& p, float g, float u) {
    g = fminf(g, p.act_limit);
    u = fminf(fmaxf(u, -p.act_limit), p.act_limit);
    return g / (1.0f + __expf(-p.act_slope * g)) * (u + p.act_shift);
}

// Expand one u32 (8 packed u4 in the plugin nibble order) to 8 bf16: (q - zp) * scale.
// A nibble placed in mantissa bits 3..6 of bf16 16.0 (0x4180) reads as 16 + q exactly.
__device__ __forceinline__ uint4 dequant_u4x8(uint32_t x, __nv_bfloat162 zz, __nv_bfloat162 ss) {
    uint32_t t[4];
    t[0] = ((x << 3) & 0x00780078u) | 0x41804180u;
    t[1] = ((x >> 1) & 0x00780078u) | 0x41804180u;
    t[2] = ((x >> 5) & 0x00780078u) | 0x41804180u;
    t[3] = ((x >> 9) & 0x00780078u) | 0x41804180u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&t[i]);
        v = __hmul2(__hsub2(v, zz), ss);
        t[i] = *reinterpret_cast<uint32_t*>(&v);
    }
    return make_uint4(t[0], t[1], t[2], t[3]);
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

// Four fp8 e4m3 bytes -> four bf16 (two words), each scaled: an e4m3 byte placed at bits 4..10 (sign at 15) of a bf16
// reads as value * 2^-120 (sub-normals included), and the per-block scale in `ss` already carries the 2^120.
__device__ __forceinline__ void dequant_f8x4(uint32_t w, __nv_bfloat162 ss, uint32_t& lo, uint32_t& hi) {
    const uint32_t y0 = __byte_perm(w, 0u, 0x4140), y1 = __byte_perm(w, 0u, 0x4342);
    uint32_t t0 = ((y0 << 8) & 0x80008000u) | ((y0 << 4) & 0x07F007F0u);
    uint32_t t1 = ((y1 << 8) & 0x80008000u) | ((y1 << 4) & 0x07F007F0u);
    __nv_bfloat162 v0 = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&t0), ss);
    __nv_bfloat162 v1 = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&t1), ss);
    lo = *reinterpret_cast<uint32_t*>(&v0);
    hi = *reinterpret_cast<uint32_t*>(&v1);
}

// gemm_pair.cu: products of many tokens on pairs of CTAs. gemm_pair_takes() says whether it runs the problem.
bool gemm_pair_takes(const ovb_gemm_args* a);
int gemm_pair(const ovb_gemm_args* a, cudaStream_t stream);

}  // namespace ovb
