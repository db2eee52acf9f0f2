// Products of up to four tokens with u4 weights: out[T, N] = epilogue(X[T, K] * dequant(W[N, K])^T), a single user's decode step.
//
// What bounds it: the read of the weights. gemm_stream.cu, which ran all of these before and keeps the small ones, reads them into registers: a few
// units per warp are on their way, and its warps meet after every 32 rows (128256 x 4096 with the norm before it 75.5 us, here 59.8; the products of
// a step of one token through four layers of an 8B model 258 -> 200). Here
//  * one lane streams stages of 128 rows x 256 columns (18 KB, one bulk copy) into a ring of 6 to 10 of them, requested before the kernel that
//    writes the tokens is done;
//  * sixteen warps share a stage: warp w of a half takes 16 rows and 128 columns. ldmatrix hands a lane the 32-bit word (8 nibbles) that its place in
//    the A fragment of mma.sync wants, without bank conflicts: the columns of K are permuted inside a piece of 32, for the tokens alike;
//  * weights enter the products as exact small integers and a group's scale is applied to its fp32 sum, as in gemm_stream.cu: nothing is rounded
//    before the sums;
//  * a warp keeps its rows for the whole of K: the halves meet once per 128 rows. One CTA per SM works off several tiles; where there are
//    fewer tiles than SMs, the CTAs of a cluster share K and push their sums to the first one (st.async).
#include <mutex>

#include "gemm_common.cuh"
#include "mma_sync.cuh"

namespace ovb {

constexpr int kRingThreads = 17 * 32;                             // 16 warps that multiply, one that fetches
constexpr int kRingStage = 4 * 4608;
constexpr int kRingTokens = 4;
constexpr int kRingMaxSlots = 10;
constexpr int kRingSmem = 216 * 1024;                             // the blocks of a norm fit beside a CTA
constexpr int kRingMaxX = 64 * 1024;
constexpr int kRingHold = 2;                                      // pieces of a token that a thread holds for a norm: up to 8192 columns

struct RingParams {
    const uint8_t* w;
    const uint8_t* x;
    void* out;
    const void* bias;
    const void* residual;
    int* status;
    int T, N, K;
    int ldx, ldo, ldr;
    int ring;
    int act, out_f32;
    float act_limit, act_slope, act_shift;
    const void* x_norm;
    const int* x_rows;
    float x_eps;
    int x_count;
};

__device__ __forceinline__ void ring_barrier() { asm volatile("bar.sync 1, 512;" ::: "memory"); }

__global__ void __launch_bounds__(kRingThreads, 1) gemm_ring_kernel(const RingParams p) {
    using E = __nv_bfloat16;
    extern __shared__ __align__(128) uint8_t ring_smem[];
    const int P = p.ring, T = p.T;
    uint32_t csize;
    const uint32_t crank = cluster_ctarank();
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
    uint8_t* ring = ring_smem;
    float* red = reinterpret_cast<float*>(ring + P * kRingStage);               // [2][half][token][row]
    float* recv = red + 4 * kRingTokens * 128;                                  // [rank][token][row] (first CTA of a cluster)
    uint64_t* full = reinterpret_cast<uint64_t*>(recv + 8 * kRingTokens * 128);
    uint64_t* empty = full + kRingMaxSlots;
    uint64_t* recv_full = empty + kRingMaxSlots;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(recv_full + 1);
    uint8_t* xs = reinterpret_cast<uint8_t*>(recv_full + 2);                    // [piece of 32 columns][token] of 64 bytes

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles = p.N / TILE_N, step = (int)(gridDim.x / csize), first = (int)(blockIdx.x / csize);
    const int ks = p.K / 256, s0 = (int)crank * ks / (int)csize, nks = ((int)crank + 1) * ks / (int)csize - s0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < P; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 16);
        }
        mbar_init(recv_full, 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    __syncthreads();
    cluster_arrive();                                             // the first CTA's barrier is ready for its peers

    if (warp == 16) {
        if (lane == 0) {
            int slot = 0;
            uint32_t par = 1;
            bool ok = true;
            for (int tile = first; ok && tile < tiles; tile += step) {
                const uint8_t* src = p.w + ((size_t)tile * (p.K / TILE_K) + 4 * s0) * 4608;
                for (int j = 0; j < nks; ++j) {
                    ok = mbar_wait(&empty[slot], par, abort_flag, p.status);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&full[slot], kRingStage);
                    bulk_load_1d(ring + slot * kRingStage, src, kRingStage, &full[slot]);
                    src += kRingStage;
                    if (++slot == P) { slot = 0; par ^= 1; }
                }
            }
            if (OVB_PDL_GEMM) {
                pdl_wait();
                pdl_trigger();
            }
        }
        __syncwarp();
        cluster_wait();
    } else {
        const int half = warp >> 3, g = lane >> 2, t = lane & 3, row0 = (warp & 7) * 16;
        pdl_wait();
        // the tokens of this CTA's part of K, in 16-byte pieces
        if (p.x_norm != nullptr) {
            __shared__ float squares[16][kRingTokens];
            norm_rows<512, kRingTokens, kRingHold>(p, squares, [&](int tok, int k8, uint4 v) {
                const int k = k8 - s0 * 32;
                if (k >= 0 && k < nks * 32) *reinterpret_cast<uint4*>(xs + ((size_t)(k >> 2) * T + tok) * 64 + (k & 3) * 16) = v;
            });
            ring_barrier();
        } else {
            const int per = nks * 32;                             // pieces of a token
            for (int i = threadIdx.x; i < per * T; i += 512) {
                const int tok = i / per, k8 = i - tok * per;
                cp_async16(xs + ((size_t)(k8 >> 2) * T + tok) * 64 + (k8 & 3) * 16, p.x + ((size_t)tok * p.ldx + (size_t)s0 * 256 + k8 * 8) * 2, true);
            }
            cp_async_commit();
            cp_async_wait<0>();
            ring_barrier();
        }
        cluster_wait();
        const bool gated = p.act == OVB_ACT_SWIGLU || p.act == OVB_ACT_GLU_LIMITED;
        const uint32_t lane_off = smem_u32(ring) + half * 9216 + (lane >> 4) * 2048 + (row0 + (lane & 15)) * 16;
        const uint32_t sz_off = smem_u32(ring) + half * 9216 + 4096 + (row0 + g) * 4;
        // (columns behind the last token repeat it: nothing reads their sums)
        const uint32_t xlane = smem_u32(xs) + half * 4 * T * 64 + min(g, T - 1) * 64 + t * 16, xpiece = T * 64;
        int slot = 0, turn = 0;
        uint32_t par = 0;
        bool ok = true;
        for (int tile = first; tile < tiles; tile += step) {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            for (int j = 0; ok && j < nks; ++j) {
                ok = mbar_wait(&full[slot], par, abort_flag, p.status);
                if (!ok) break;
                uint32_t q[2][4], sz[2];
#pragma unroll
                for (int c = 0; c < 2; ++c) ldsm_x4(lane_off + slot * kRingStage + c * 4608, q[c][0], q[c][1], q[c][2], q[c][3]);
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sz[0]) : "r"(sz_off + slot * kRingStage));
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sz[1]) : "r"(sz_off + slot * kRingStage + 32));
                uint32_t minus[2];                                // -z / 64 (the table holds 16 + z), twice each
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const __nv_bfloat162 zz = __high2bfloat162(*reinterpret_cast<const __nv_bfloat162*>(&sz[i]));
                    const __nv_bfloat162 m = __hfma2(zz, __float2bfloat162_rn(-0.015625f), __float2bfloat162_rn(0.25f));
                    minus[i] = *reinterpret_cast<const uint32_t*>(&m);
                }
                auto whole = [&](uint32_t bits, uint32_t mul, uint32_t m) {
                    const __nv_bfloat162 v = __hfma2(*reinterpret_cast<__nv_bfloat162*>(&bits), *reinterpret_cast<__nv_bfloat162*>(&mul), *reinterpret_cast<__nv_bfloat162*>(&m));
                    return *reinterpret_cast<const uint32_t*>(&v);
                };
                float part[4] = {};
                uint32_t xa = xlane + j * 8 * xpiece;
#pragma unroll
                for (int s = 0; s < 4; ++s) {                     // pieces of 32 columns
                    const uint4 xb = lds128(xa);
                    xa += xpiece;
                    const uint32_t lo = q[s >> 1][(s & 1) * 2], hi = q[s >> 1][(s & 1) * 2 + 1], ly = lo >> 8, hy = hi >> 8;
                    const uint32_t a0[4] = {whole(lo & 0x000F000Fu, kTwo127, minus[0]), whole(hi & 0x000F000Fu, kTwo127, minus[1]),
                                            whole(lo & 0x00F000F0u, kTwo123, minus[0]), whole(hi & 0x00F000F0u, kTwo123, minus[1])};
                    const uint32_t a1[4] = {whole(ly & 0x000F000Fu, kTwo127, minus[0]), whole(hy & 0x000F000Fu, kTwo127, minus[1]),
                                            whole(ly & 0x00F000F0u, kTwo123, minus[0]), whole(hy & 0x00F000F0u, kTwo123, minus[1])};
                    mma16816<false>(part, a0, xb.x, xb.y);
                    mma16816<false>(part, a1, xb.z, xb.w);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[slot]);
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[e] += __uint_as_float(sz[e >> 1] << 16) * part[e];
                if (++slot == P) { slot = 0; par ^= 1; }
            }
            // the halves of K meet; another tile's sums go to the other buffer meanwhile
            float* mine = red + (turn * 2 + half) * kRingTokens * 128;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int tok = 2 * t + (e & 1);
                if (tok < T) mine[tok * 128 + row0 + (e >> 1) * 8 + g] = 64.f * acc[e];
            }
            ring_barrier();
            const float* a = red + turn * 2 * kRingTokens * 128;
            const float* b = a + kRingTokens * 128;
            if (crank != 0) {                                     // (one tile per cluster)
                if ((int)threadIdx.x < T * 32) {
                    const int i = threadIdx.x * 4;
                    uint32_t v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[e] = __float_as_uint(a[i + e] + b[i + e]);
                    st_async_v4(dsmem_addr(smem_u32(recv + crank * kRingTokens * 128 + i), 0), v, dsmem_addr(smem_u32(recv_full), 0));
                }
            } else {
                if (csize > 1) {
                    if (threadIdx.x == 0) mbar_arrive_expect_tx(recv_full, (csize - 1) * (uint32_t)T * 512);
                    ok = mbar_wait(recv_full, 0, abort_flag, p.status) && ok;
                }
                auto sum = [&](int i) {
                    float v = a[i] + b[i];
                    for (uint32_t z = 1; z < csize; ++z) v += recv[z * kRingTokens * 128 + i];
                    return v;
                };
                const int sh = gated ? 6 : 7;
                for (int i = threadIdx.x; ok && i < T << sh; i += 512) {
                    const int tok = i >> sh, r = i & ((1 << sh) - 1);
                    if (gated) {
                        const float gv = sum(tok * 128 + r), uv = sum(tok * 128 + 64 + r);
                        reinterpret_cast<E*>(p.out)[(size_t)tok * p.ldo + tile * 64 + r] =
                            from_float<E>(p.act == OVB_ACT_SWIGLU ? gv / (1.0f + __expf(-gv)) * uv : glu_limited(p, gv, uv));
                    } else {
                        const int oc = tile * TILE_N + r;
                        float v = sum(i);
                        if (p.bias) v += to_float(reinterpret_cast<const E*>(p.bias)[oc]);
                        v = apply_act(v, p);
                        if (p.residual) v += to_float(reinterpret_cast<const E*>(p.residual)[(size_t)tok * p.ldr + oc]);
                        if (p.out_f32) reinterpret_cast<float*>(p.out)[(size_t)tok * p.ldo + oc] = v;
                        else reinterpret_cast<E*>(p.out)[(size_t)tok * p.ldo + oc] = from_float<E>(v);
                    }
                }
            }
            turn ^= 1;
        }
    }
    __syncthreads();
    if (csize > 1) {                                              // no CTA leaves while a peer may still store to it
        cluster_arrive();
        cluster_wait();
    }
    if (*abort_flag) {      // copies that are still in flight land before the shared memory is used again
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        __syncthreads();
    }
}

// --------------------------------------------------------------------------------------------- host
struct RingPlan {
    int splits, ctas, ring, smem;
};

// Splits of K: none where the tiles fill the SMs; otherwise one tile per cluster, the clusters as large as the device holds that many.
static bool ring_plan(int T, int N, int K, RingPlan* f) {
    const int tiles = N / TILE_N, ks = K / 256;
    int s = 1;
    for (int c = 2; c <= 8 && c <= ks && tiles < 148; ++c)
        if (tiles <= cluster_capacity(c)) s = c;
    f->splits = s;
    f->ctas = (tiles < 148 ? tiles : 148) * s;
    const int x = ceil_div(ks, s) * 512 * T, fixed = 12 * kRingTokens * 128 * 4 + (2 * kRingMaxSlots + 2) * 8;
    if (x > kRingMaxX) return false;
    f->ring = (kRingSmem - x - fixed) / kRingStage;
    if (f->ring > kRingMaxSlots) f->ring = kRingMaxSlots;
    f->smem = f->ring * kRingStage + x + fixed;
    return true;
}

// Below, a launch costs as much either way (2048 x 2048 5.7 us, gemm_stream.cu 5.2; 1024 x 4096 5.7 / 5.8; 4096 x 4096 6.9 / 7.6).
constexpr int64_t kRingMinWeights = 8ll << 20;

bool gemm_ring_takes(const ovb_gemm_args* a) {
    if (a->wmode != OVB_W_U4 || a->T > kRingTokens || a->comm != nullptr || a->group_offsets != nullptr || a->group_mode == 3 || a->block_t != 0 || a->splits > 1) return false;
    if (a->N % TILE_N != 0 || a->K % 256 != 0 || a->group_size % 128 != 0 || a->w_kb_stride != 0 || (int64_t)a->N * a->K < kRingMinWeights) return false;
    RingPlan f;
    return ring_plan(a->T, a->N, a->K, &f);
}

bool gemm_ring_norms(const ovb_gemm_args* a) { return a->K <= kRingHold * 512 * 8; }

int gemm_ring(const ovb_gemm_args* a, cudaStream_t stream) {
    const bool gated = a->act == OVB_ACT_SWIGLU || a->act == OVB_ACT_GLU_LIMITED;
    RingPlan f;
    if (!ring_plan(a->T, a->N, a->K, &f)) return ERR_UNSUPPORTED;
    RingParams p;
    memset(&p, 0, sizeof(p));
    p.w = static_cast<const uint8_t*>(a->w);
    p.x = static_cast<const uint8_t*>(a->x);
    p.out = a->out;
    p.bias = a->bias;
    p.residual = a->residual;
    p.status = status_word();
    p.T = a->T;
    p.N = a->N;
    p.K = a->K;
    p.ldx = a->ldx ? a->ldx : a->K;
    p.ldo = a->ldo ? a->ldo : (gated ? a->N / 2 : a->N);
    p.ldr = a->ldr ? a->ldr : a->N;
    p.ring = f.ring;
    p.act = a->act;
    p.out_f32 = a->out_f32;
    p.act_limit = a->act_limit;
    p.act_slope = a->act_slope;
    p.act_shift = a->act_shift;
    p.x_norm = a->x_norm;
    p.x_rows = a->x_rows;
    p.x_eps = a->x_eps;
    p.x_count = a->x_count;
    {
        static std::mutex mu;
        static uint64_t configured = 0;         // one bit per device
        int dev = 0;
        OVB_CHECK_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lk(mu);
        if (!(configured & (1ull << (dev & 63)))) {
            OVB_CHECK_CUDA(cudaFuncSetAttribute(gemm_ring_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRingSmem));
            OVB_CHECK_CUDA(cudaFuncSetAttribute(gemm_ring_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
            configured |= 1ull << (dev & 63);
        }
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(f.ctas);
    cfg.blockDim = dim3(kRingThreads);
    cfg.dynamicSmemBytes = f.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = f.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    OVB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, gemm_ring_kernel, static_cast<const RingParams>(p)));
    OVB_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace ovb
