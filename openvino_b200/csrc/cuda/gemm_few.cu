// Products of up to 64 tokens with quantised weights: out[T, N] = epilogue(X[T, K] * dequant(W[N, K])^T), a decode step's or a short prompt's.
//
// What has to bound it: the read of the weights. The kernel of gemm_sm100.cu, which keeps short sums (few_is_faster), takes up to three times as long
// as that read: the one warp that issues its MMAs competes with the expanding warps for issue slots, and a launch costs 8 to 10 us beyond its
// bytes, most of it in the reduction over the splits of K.
//  * One CTA per SM, persistent: warp 0 streams the weights into a ring (requested before the kernel that writes the tokens is done), warp 1 the
//    tokens, warps 6 and 7 issue the MMAs, warps 8 .. 11 are the epilogue, under the main loop of the next tile, and two or three groups of four
//    warps (one per quarter of the tensor memory's lanes) expand, each a stage of its own.
//  * A stage is 256 columns of K: one copy for the weights, one for the tokens. With 128 columns the copying lanes, between busy warps, were what
//    the kernel waited for (128256 x 4096 u4, 16 tokens: 82 us, now 69; u8 107, now 90: 5.9 TB/s).
//  * Two issuing warps, each with an accumulator of its own: between warps that expand, one of them was what the kernel waited for (128256 x 4096 u8,
//    24 tokens now: 5.8 TB/s, issue slots 58 % busy, tensor pipe 19 %).
//  * The S CTAs of a cluster share the columns of K. Partial sums are pushed: every CTA owns a share of the tile's outputs, the others store their
//    sums straight into its shared memory (st.async, counted on an mbarrier), it adds them in the order of the ranks (the same bits on every run)
//    and writes the outputs. One way through the cluster instead of a barrier, a read and a barrier.
//  * Expanded weights go to tensor memory, as in gemm_sm100.cu, with the same rounding.
// A decode step of 24 tokens (8B, four layers, u8): 684 -> 609 us, products 414 -> 345; of 32 tokens (70B, two layers, fp8): 868 -> 777 us.
#include <mutex>

#include "cluster_table.h"
#include "gemm_common.cuh"

namespace ovb {

constexpr int kFewGroups = 3;                                  // groups of four expanding warps, at most
constexpr int kFewIssuers = 2;                                 // warps that issue MMAs
constexpr int kFewStageK = 256;                                // columns of K of a stage: 128 for either issuer
constexpr int kFewThreads = (12 + 4 * kFewGroups) * 32;
constexpr int kFewBound = 896;                                 // (see kFewSmem)
constexpr int kFewMaxRing = 12, kFewMaxX = 8, kFewA = 3;        // slots of packed weights, of tokens, of expanded weights
constexpr int kFewBarBytes = 1024;
// 40 KB of registers (u4: 768 threads of 72; 8-bit weights start 640) and 11 KB of shared memory stay free: a block of a norm or a rotation (256
// threads of up to 40) fits beside a CTA, so that it starts, and requests its weights, while they still run. The kernel's launch bound names 896
// threads, more than any plan starts, for these 72 registers: bound to 768 it takes 80, and 16 KB would be left.
constexpr int kFewSmem = 216 * 1024;
constexpr int kFewTokens = 64;                                 // largest T

struct FewParams {
    const uint8_t* w;
    const uint32_t* sz;
    void* out;
    const void* bias;
    const void* residual;
    int* status;
    int T, N, K;
    int ldo, ldr;
    int kb_stride;             // u4: chunks between weight tiles
    int gpk;                   // columns per scale group / 128
    int nt;                    // token columns of the product: T rounded up to 16
    int ring, xslots, bufs, groups;
    int unit_cap;              // output units that a CTA owns, at most
    int act, out_f32;
    float act_limit, act_slope, act_shift;
};

// Bytes of a stage in the ring: u4 four packed chunks with their pairs; 8-bit twice 128 x 128 bytes (the pairs lie behind the ring)
constexpr int few_slot(int wmode) { return wmode == OVB_W_U4 ? 2 * 9216 : 2 * 16384; }
constexpr int few_pairs(int wmode) { return wmode == OVB_W_U4 ? 0 : 2 * 512; }

// The eight MMAs of a stage and their commits, called by a whole warp with uniform arguments: one lane issues them all. db: descriptor of the
// first k-block's tokens, `second`: distance to the second's.
__device__ __forceinline__ void few_mma_stage(uint32_t d, uint32_t ta, uint64_t db, uint64_t second, uint32_t idesc, uint32_t acc, uint32_t done, uint32_t xdone) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 b0, b1, b2, b3, b4, b5, b6;\n\t.reg .b32 a1, a2, a3, a4, a5, a6, a7;\n\t"
        "add.s64 b0, %2, 2;\n\tadd.s64 b1, %2, 4;\n\tadd.s64 b2, %2, 6;\n\tadd.s64 b3, %2, %3;\n\tadd.s64 b4, b3, 2;\n\tadd.s64 b5, b3, 4;\n\tadd.s64 b6, b3, 6;\n\t"
        "add.s32 a1, %1, 8;\n\tadd.s32 a2, %1, 16;\n\tadd.s32 a3, %1, 24;\n\tadd.s32 a4, %1, 32;\n\tadd.s32 a5, %1, 40;\n\tadd.s32 a6, %1, 48;\n\tadd.s32 a7, %1, 56;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %4, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b0, %4, 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b1, %4, 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b2, %4, 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a4], b3, %4, 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a5], b4, %4, 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a6], b5, %4, 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a7], b6, %4, 1;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t}"
        ::"r"(d), "r"(ta), "l"(db), "l"(second), "r"(idesc), "r"(acc), "r"(done), "r"(xdone)
        : "memory");
}

template <int WMODE>
__global__ void __launch_bounds__(kFewBound, 1)
gemm_few_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const FewParams p) {
    using E = __nv_bfloat16;
    constexpr int SLOT = few_slot(WMODE), PAIRS = few_pairs(WMODE);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int P = p.ring, XS = p.xslots, NT = p.nt;
    const int xbytes = NT * 512;                                  // four k-blocks of the token tile
    uint8_t* ring = smem;
    uint8_t* xbuf = ring + P * SLOT;
    uint8_t* recv = xbuf + XS * xbytes;                           // [source][unit][quarter][row] of four tokens
    uint32_t csize, crank = cluster_ctarank();
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
    uint8_t* pairs = recv + csize * p.unit_cap * 1024;
    uint64_t* p_full = reinterpret_cast<uint64_t*>(pairs + P * PAIRS);
    uint64_t* p_empty = p_full + kFewMaxRing;
    uint64_t* x_full = p_empty + kFewMaxRing;
    uint64_t* x_empty = x_full + kFewMaxX;
    uint64_t* a_full = x_empty + kFewMaxX;                        // [slot][issuer]
    uint64_t* a_empty = a_full + 2 * kFewA;
    uint64_t* acc_full = a_empty + 2 * kFewA;                     // [buffer][issuer]
    uint64_t* acc_empty = acc_full + 4;
    uint64_t* recv_full = acc_empty + 4;
    uint64_t* recv_free = recv_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(recv_free + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles = p.N / TILE_N, clusters = (int)(gridDim.x / csize), first = (int)(blockIdx.x / csize);
    const int ks = p.K / kFewStageK, s0 = (int)crank * ks / (int)csize, nks = ((int)crank + 1) * ks / (int)csize - s0;
    const int my_tiles = (tiles - first + clusters - 1) / clusters, total = my_tiles * nks;
    // Every cluster walks its part of K from a place of its own: CTAs that asked for the same tokens at the same time would queue at the few
    // slices of L2 that hold them.
    const int turn = first % nks;
    const int acc_cols = 2 * p.bufs * NT;                         // tensor memory: [buffer][issuer] accumulators, then the expanded stages

    if (threadIdx.x == 0) {
        for (int s = 0; s < P; ++s) {
            mbar_init(&p_full[s], 1);
            mbar_init(&p_empty[s], 4);
        }
        for (int s = 0; s < XS; ++s) {
            mbar_init(&x_full[s], 1);
            mbar_init(&x_empty[s], 2);
        }
        for (int s = 0; s < 2 * kFewA; ++s) {
            mbar_init(&a_full[s], 4);
            mbar_init(&a_empty[s], 1);
        }
        for (int b = 0; b < 4; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 4);
        }
        mbar_init(recv_full, 4);
        mbar_init(recv_free, 4 * csize);
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmX);
        if (WMODE != OVB_W_U4) tma_prefetch_desc(&tmW);
    }
    if (warp == 2) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    // the barriers of this CTA are ready for its peers; who talks to them waits first, the others at their end
    cluster_arrive();

    if (warp == 0) {
        // ------------------------------------------------------------ weights
        if (lane == 0) {
            int slot = 0;
            uint32_t par = 1;
            bool ok = true;
            for (int tile = first; ok && tile < tiles; tile += clusters) {
                const uint8_t* src = p.w + ((size_t)tile * p.kb_stride + 4 * s0) * 4608;
                int k = turn;
                for (int j = 0; j < nks; ++j) {
                    ok = mbar_wait(&p_empty[slot], par, abort_flag, p.status);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&p_full[slot], SLOT + PAIRS);
                    if (WMODE == OVB_W_U4) {
                        bulk_load_1d(ring + slot * SLOT, src + (size_t)k * SLOT, SLOT, &p_full[slot]);
                    } else {
                        tma_load_3d(ring + slot * SLOT, &tmW, &p_full[slot], 0, tile * TILE_N, 2 * (s0 + k));
                        for (int h = 0; h < 2; ++h)
                            bulk_load_1d(pairs + slot * PAIRS + h * 512, p.sz + (size_t)((2 * (s0 + k) + h) / p.gpk) * p.N + tile * TILE_N, 512, &p_full[slot]);
                    }
                    if (++k == nks) k = 0;
                    if (++slot == P) { slot = 0; par ^= 1; }
                }
            }
            if (OVB_PDL_GEMM) {
                pdl_wait();
                pdl_trigger();
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ tokens
        if (lane == 0) {
            pdl_wait();
            int slot = 0, k = turn;
            uint32_t par = 1;
            for (int i = 0; i < total; ++i) {
                if (!mbar_wait(&x_empty[slot], par, abort_flag, p.status)) break;
                mbar_arrive_expect_tx(&x_full[slot], xbytes);
                tma_load_3d(xbuf + slot * xbytes, &tmX, &x_full[slot], 0, 0, 4 * (s0 + k));
                if (++k == nks) k = 0;
                if (++slot == XS) { slot = 0; par ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp >= 8 - kFewIssuers && warp < 8) {
        // ------------------------------------------------------------ MMA issuers (warp-uniform, see gemm_sm100.cu)
        // Two warps, one for the first 128 columns of every stage and one for the others, each with an accumulator of its own: the waits,
        // eight MMAs and commits of a stage take one warp, between the expanding ones, longer than the read of its weights.
        const uint32_t idesc = umma_idesc_f16(TILE_N, NT, true);
        const int me = warp - (8 - kFewIssuers);
        const uint64_t desc0 = umma_desc_k_sw128(smem_u32(xbuf) + me * (xbytes >> 1), 1024);
        int a = 0, xs = 0, buf = 0, it = 0;
        uint32_t apar = 0, xpar = 0, accpar = 1;
        bool ok = true, a_ready = false, x_ready = false;
        for (int i = 0; ok && i < my_tiles; ++i) {
            ok = mbar_wait(&acc_empty[buf * 2 + me], accpar, abort_flag, p.status);
            const uint32_t d = tmem_base + uint32_t((buf * 2 + me) * NT);
            for (int j = 0; ok && j < nks; ++j) {
                if (!x_ready) ok = mbar_wait(&x_full[xs], xpar, abort_flag, p.status);
                if (!a_ready) ok = ok && mbar_wait(&a_full[a * 2 + me], apar, abort_flag, p.status);
                if (!ok) break;
                const uint32_t ta = tmem_base + uint32_t(acc_cols + (a * 2 + me) * 64), done = smem_u32(&a_empty[a * 2 + me]), xdone = smem_u32(&x_empty[xs]);
                const uint64_t db = desc0 + (uint64_t)((xs * xbytes) >> 4);
                if (++a == kFewA) { a = 0; apar ^= 1; }
                if (++xs == XS) { xs = 0; xpar ^= 1; }
                if (++it < total) {                               // answered while the MMAs are issued
                    a_ready = mbar_test(&a_full[a * 2 + me], apar);
                    x_ready = mbar_test(&x_full[xs], xpar);
                }
                tc_fence_after_sync();
                few_mma_stage(d, ta, db, (uint64_t)(xbytes >> 6), idesc, j > 0 ? 1u : 0u, done, xdone);
            }
            if (ok) umma_commit_elect(&acc_full[buf * 2 + me]);
            if (++buf == p.bufs) { buf = 0; accpar ^= 1; }
        }
        __syncwarp();
    } else if (warp >= 12) {
        // ------------------------------------------------------------ expansion: the groups take the stages in turn
        const int G = p.groups;
        const int g = (warp - 12) >> 2, q = warp & 3, row = q * 32 + lane;
        const uint32_t a_lane = tmem_base + (uint32_t(q * 32) << 16) + uint32_t(acc_cols);
        int slot = g % P, a = g % kFewA;
        uint32_t ppar = (g / P) & 1, apar = ((g / kFewA) & 1) ^ 1;
        constexpr int LD = WMODE == OVB_W_U4 ? 4 : 8;
        bool ok = true;
        for (int i = g; ok && i < total; i += G) {
            ok = mbar_wait(&p_full[slot], ppar, abort_flag, p.status);
#pragma unroll 1
            for (int h = 0; ok && h < 2; ++h) {
                const uint32_t base = smem_u32(ring + slot * SLOT) + h * (SLOT / 2);
                uint32_t szw;
                uint4 pk[LD];                                     // 128 values of a row
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(szw) : "r"(WMODE == OVB_W_U4 ? base + 4096 + row * 4 : smem_u32(pairs + slot * PAIRS) + h * 512 + row * 4));
#pragma unroll
                for (int j = 0; j < LD; ++j) pk[j] = lds128(WMODE == OVB_W_U4 ? base + (j >> 1) * 4608 + (j & 1) * 2048 + row * 16 : base + row * 128 + ((j ^ (row & 7)) << 4));
                ok = mbar_wait(&a_empty[a * 2 + h], apar, abort_flag, p.status);
                if (!ok) break;
                const uint32_t dst = a_lane + uint32_t((a * 2 + h) * 64);
                const __nv_bfloat162 szp = *reinterpret_cast<const __nv_bfloat162*>(&szw);
                const RowScale rs = row_scale(szp, WMODE == OVB_W_U4 ? 16.f : 0.f);
                const __nv_bfloat162 ss = __halves2bfloat162(__low2bfloat16(szp), __low2bfloat16(szp));
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint32_t r[16];
                    if (WMODE == OVB_W_U4) {
                        const uint32_t xs[4] = {pk[j].x, pk[j].y, pk[j].z, pk[j].w};
#pragma unroll
                        for (int n = 0; n < 4; ++n) {
                            const uint4 e = dequant_u4x8(xs[n], rs);
                            r[4 * n] = e.x; r[4 * n + 1] = e.y; r[4 * n + 2] = e.z; r[4 * n + 3] = e.w;
                        }
                    } else {
#pragma unroll
                        for (int b = 0; b < 2; ++b) {
                            const uint4 w = pk[(2 * j + b) % LD];
                            const uint32_t xs[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                            for (int n = 0; n < 4; ++n) {
                                if (WMODE == OVB_W_F8) dequant_f8x4(xs[n], ss, r[b * 8 + 2 * n], r[b * 8 + 2 * n + 1]);
                                else dequant_u8x4(xs[n], rs, r[b * 8 + 2 * n], r[b * 8 + 2 * n + 1]);
                            }
                        }
                    }
                    tmem_st_x16(dst + j * 16, r);
                }
                __syncwarp();
                if (lane == 0 && h == 1) mbar_arrive(&p_empty[slot]);
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[a * 2 + h]);
            }
            slot += G;
            while (slot >= P) { slot -= P; ppar ^= 1; }
            a += G;
            while (a >= kFewA) { a -= kFewA; apar ^= 1; }
        }
        __syncwarp();
    } else if (warp >= 8) {
        // ------------------------------------------------------------ epilogue
        // A unit is four tokens of 64 rows: quarter h and quarter h + 2 of the tile's rows (gate and up of the same channels in a gated MLP).
        const int q = warp & 3;
        const int units = NT >> 1, S = (int)csize, rank = (int)crank;
        const int inv = 65536 / units + 1;                        // u * S / units for u * S <= 8 * 32
        auto start_of = [&](int r) { return (r * units + S - 1) / S; };
        const int u0 = start_of(rank), mine = start_of(rank + 1) - u0;
        const uint32_t recv_a = smem_u32(recv), full_a = smem_u32(recv_full), free_a = smem_u32(recv_free);
        const bool gated = p.act == OVB_ACT_SWIGLU || p.act == OVB_ACT_GLU_LIMITED;
        int buf = 0;
        uint32_t accpar = 0;
        cluster_wait();                                           // the peers' barriers are initialised
        pdl_wait();                                               // from here on outputs are written and the residual is read
        for (int i = 0, tile = first; i < my_tiles; ++i, tile += clusters) {
            bool ok = mbar_wait(&acc_full[buf * 2], accpar, abort_flag, p.status) && mbar_wait(&acc_full[buf * 2 + 1], accpar, abort_flag, p.status);
            if (ok && i > 0) ok = mbar_wait(recv_free, (uint32_t)(i - 1) & 1u, abort_flag, p.status);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after_sync();
            const uint32_t src = tmem_base + (uint32_t(q * 32) << 16) + uint32_t(buf * 2 * NT);
            for (int c = 0; c < NT; c += 16) {
                uint32_t r[16];
                uint32_t more[16];
                tmem_ld_x16(src + c, r);
                tmem_ld_x16(src + NT + c, more);
                tmem_ld_wait();
#pragma unroll
                for (int k = 0; k < 16; ++k) r[k] = __float_as_uint(__uint_as_float(r[k]) + __uint_as_float(more[k]));
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int u = ((c >> 2) + k) * 2 + (q & 1), owner = (u * S * inv) >> 16, ou = u - start_of(owner);
                    const uint32_t at = (uint32_t)((rank * p.unit_cap + ou) * 1024 + (q >> 1) * 512 + lane * 16);
                    if (owner == rank) sts128(recv_a + at, make_uint4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]));
                    else st_async_v4(dsmem_addr(recv_a + at, (uint32_t)owner), r + 4 * k, dsmem_addr(full_a, (uint32_t)owner));
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&acc_empty[buf * 2]);
                mbar_arrive(&acc_empty[buf * 2 + 1]);
                if (q == 0) mbar_arrive_expect_tx(recv_full, (uint32_t)((S - 1) * mine * 1024));
                else mbar_arrive(recv_full);
            }
            if (++buf == p.bufs) { buf = 0; accpar ^= 1; }
            const int n0 = tile * TILE_N;
            E res[8];
            auto fetch = [&](int w) {
                const int u = u0 + w, tok = (u >> 1) * 4, r = (u & 1) * 32 + lane;
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const E* rp = reinterpret_cast<const E*>(p.residual) + (size_t)(tok + t) * p.ldr + n0 + r;
                    res[t] = tok + t < p.T ? rp[0] : from_float<E>(0.f);
                    res[4 + t] = tok + t < p.T ? rp[64] : from_float<E>(0.f);
                }
            };
            if (p.residual != nullptr && q < mine) fetch(q);
            ok = mbar_wait(recv_full, (uint32_t)i & 1u, abort_flag, p.status);
            if (!__all_sync(0xffffffffu, ok)) break;
            for (int w = q; w < mine; w += 4) {
                float lo[4] = {0.f, 0.f, 0.f, 0.f}, hi[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
                for (int z = 0; z < S; ++z) {
                    const float4* at = reinterpret_cast<const float4*>(recv + (z * p.unit_cap + w) * 1024) + lane;
                    const float4 a = at[0], b = at[32];
                    lo[0] += a.x; lo[1] += a.y; lo[2] += a.z; lo[3] += a.w;
                    hi[0] += b.x; hi[1] += b.y; hi[2] += b.z; hi[3] += b.w;
                }
                const int u = u0 + w, tok = (u >> 1) * 4, r = (u & 1) * 32 + lane;
                if (gated) {
                    E* o = reinterpret_cast<E*>(p.out) + (size_t)tok * p.ldo + tile * 64 + r;
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const float v = p.act == OVB_ACT_SWIGLU ? lo[t] / (1.0f + __expf(-lo[t])) * hi[t] : glu_limited(p, lo[t], hi[t]);
                        if (tok + t < p.T) o[(size_t)t * p.ldo] = from_float<E>(v);
                    }
                } else {
                    const float b0 = p.bias ? to_float(reinterpret_cast<const E*>(p.bias)[n0 + r]) : 0.f;
                    const float b1 = p.bias ? to_float(reinterpret_cast<const E*>(p.bias)[n0 + r + 64]) : 0.f;
                    float v[8];
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        v[t] = lo[t] + b0;
                        v[4 + t] = hi[t] + b1;
                    }
                    apply_act_n(v, p);
                    if (p.residual != nullptr) {
#pragma unroll
                        for (int t = 0; t < 8; ++t) v[t] += to_float(res[t]);
                        if (w + 4 < mine) fetch(w + 4);
                    }
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        if (tok + t >= p.T) continue;
                        const size_t at = (size_t)(tok + t) * p.ldo + n0 + r;
                        if (p.out_f32) {
                            reinterpret_cast<float*>(p.out)[at] = v[t];
                            reinterpret_cast<float*>(p.out)[at + 64] = v[4 + t];
                        } else {
                            reinterpret_cast<E*>(p.out)[at] = from_float<E>(v[t]);
                            reinterpret_cast<E*>(p.out)[at + 64] = from_float<E>(v[4 + t]);
                        }
                    }
                }
            }
            __syncwarp();
            // the shares of this tile have been read: the peers may send the next one's (after the last tile a peer may be gone)
            if (lane == 0 && i + 1 < my_tiles)
                for (uint32_t z = 0; z < csize; ++z) arrive_cluster(dsmem_addr(free_a, z));
        }
        __syncwarp();
    }
    if (warp < 8 || warp >= 12) cluster_wait();
    // ---------------------------------------------------------------- tear-down; no CTA leaves while a peer may still store to it
    tc_fence_before_sync();
    __syncthreads();
    if (csize > 1) {
        cluster_arrive();
        cluster_wait();
    }
    if (*abort_flag) {      // copies that are still in flight land before the shared memory is used again
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 2) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

// --------------------------------------------------------------------------------------------- host
struct FewPlan {
    int splits, clusters, ring, xslots, bufs, groups, unit_cap, smem;
};

// Shared and tensor memory of a plan. Where they fit, 110 KB (u4) or 135 KB of weights are on their way, and up to four stages of tokens
// (28672 x 4096 u4, 32 tokens: 28.4 us with four, 30.4 with two). Nibbles take more instructions per byte than 8-bit weights: three groups expand
// them (128256 x 4096, 16 tokens: 69 us, two groups 79 us), two the others (u8: 91 us, three 99 us).
static bool few_layout(int wmode, int nt, FewPlan* f) {
    const int xb = nt * 512, slot = few_slot(wmode) + few_pairs(wmode);
    f->unit_cap = ceil_div(nt / 2, f->splits);
    f->bufs = nt <= 32 ? 2 : 1;                                   // 2 * bufs * nt + kFewA * 128 columns of tensor memory
    const int left = kFewSmem - 1024 - kFewBarBytes - f->splits * f->unit_cap * 1024;
    // A slot belongs to one group (the ring is a multiple of the groups): its wait for the slot's next filling then starts after the last one
    // has landed. A wait for a phase must not start two phases early.
    f->groups = wmode == OVB_W_U4 ? 3 : 2;
    for (f->xslots = 4; f->xslots >= 2; --f->xslots) {
        f->ring = (left - f->xslots * xb) / slot;
        if (f->ring > kFewMaxRing) f->ring = kFewMaxRing;
        f->ring -= f->ring % f->groups;
        if (f->ring >= (wmode == OVB_W_U4 ? 6 : 4)) break;
    }
    if (f->xslots < 2) {                                          // 8-bit weights, 64 tokens: three stages of one group each
        f->xslots = 2;
        f->groups = 3;
        f->ring = 3;
    }
    f->smem = 1024 + kFewBarBytes + f->splits * f->unit_cap * 1024 + f->xslots * xb + f->ring * slot;
    return f->smem <= kFewSmem;
}

static int ask_cluster_capacity(int size) {
    auto kern = gemm_few_kernel<OVB_W_U4>;
    int n = 0;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(size * 64);
    cfg.blockDim = dim3(kFewThreads);
    cfg.dynamicSmemBytes = kFewSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = size;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kFewSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return n;
}

int cluster_capacity(int size) {
    static ClusterTable table;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        (void)cudaGetLastError();
        dev = -1;
    }
    return table.get(dev, size, [size] { return ask_cluster_capacity(size); });
}

// Splits of K. Time of a candidate (us): rounds of tiles, each as long as its stages take an SM or their bytes take HBM at 6.3 TB/s, whichever is
// longer, and an exchange of the sums per round, which the next round's products do not hide: 0.45 per peer and 0.03 per token.
static bool few_plan(int wmode, int T, int N, int K, int forced, FewPlan* best) {
    const int nt = (T + 15) / 16 * 16, ks = K / kFewStageK, tiles = N / TILE_N;
    const double stage_us = (wmode == OVB_W_U4 ? 0.47 : 0.51) + (nt <= 48 ? 0.001 * nt : 0.2);      // (measured, one CTA per tile)
    const double bytes_us = (few_slot(wmode) + few_pairs(wmode)) / 6.3e6;
    double best_t = 1e30;
    for (int s = 1; s <= 8 && s <= ks; ++s) {
        if (forced > 0 && s != forced) continue;
        FewPlan f;
        f.splits = s;
        if (!few_layout(wmode, nt, &f)) continue;
        f.clusters = cluster_capacity(s);
        const int per = ceil_div(ks, s), full = tiles / f.clusters, rest = tiles % f.clusters;
        auto round_us = [&](int clusters) {
            const double sm = per * stage_us, hbm = (double)clusters * s * per * bytes_us;
            return (sm > hbm ? sm : hbm) + (s > 1 ? 0.45 * (s - 1) + 0.03 * nt : 0.0);
        };
        const double t = full * round_us(f.clusters) + (rest > 0 ? round_us(rest) : 0.0);
        if (f.clusters > tiles) f.clusters = tiles;
        if (t < best_t - 1e-9) {
            best_t = t;
            *best = f;
        }
    }
    return best_t < 1e30;
}

// Where it is the faster one, against gemm_sm100.cu: the smallest K, by token columns (16, 32, 48, 64) and tiles of 128 rows (up to 8, 16, 32, 64, 148, 296,
// more). A tile costs the exchange of its sums and its epilogue, which grow with the tokens and which short sums do not hide, and 149 to 296 tiles
// are one wave of the other kernel's two CTAs per SM and two rounds here. Measured with cold weights behind a norm, which is included, and back to back; a
// product stays here where either way it is not the slower one, since behind a longer kernel that leaves SMs idle (a short prompt's attention) its weights are
// fetched meanwhile (37 tokens, 4096 x 4096 u4 after the attention: 5 us less than the other kernel; behind a norm 0.96 of it, back to back 1.05).
// us here / there, back to back: u4, 16 tokens 128256 x 4096 65.5 / 89, 4096 x 14336 14.9 / 18.2, 28672 x 1024 11.5 / 10.8; 37 tokens 28672 x 4096 26.6 /
// 28.2, 20480 x 1024 14.6 / 11.5; u8, 24 tokens 6144 x 4096 11.8 / 14.6, 1024 x 1024 7.4 / 5.4; 48 tokens 24576 x 2048 20.0 / 19.2; 64 tokens 8192 x 28672
// 58 / 74, 1024 x 1024 10.8 / 6.9, 28672 x 4096 40.5 / 36.6. With 64 token columns the MMAs bind a stage, so that half the bytes gain u4 weights little.
static bool few_is_faster(int wmode, int T, int tiles, int K) {
    constexpr int never = 1 << 30;
    static constexpr int u4[4][7] = {{256, 256, 256, 256, 1024, 1536, 256}, {2048, 2048, 3072, 2048, 2048, 3072, 1536}, {6144, 2048, 3072, 2048, 3072, 4096, 3072},
                                     {never, never, never, never, never, never, never}};
    static constexpr int bytes[4][7] = {{256, 256, 256, 256, 512, 1024, 256}, {2048, 2048, 3072, 1536, 2048, 2048, 1024}, {6144, 2048, 2048, 1024, 1536, 4096, 1536},
                                        {8192, 2048, 4096, 2048, 3072, 8192, 3072}};
    const int col = tiles <= 8 ? 0 : tiles <= 16 ? 1 : tiles <= 32 ? 2 : tiles <= 64 ? 3 : tiles <= 148 ? 4 : tiles <= 296 ? 5 : 6, row = (T - 1) / 16;
    // a few tiles more than clusters of two: one CTA per tile leaves half of the SMs idle (10240 x 6144 u8, 64 tokens 27.6 / 23.6, 10240 x 8192, 37 tokens 28.3 / 27.3)
    if (wmode != OVB_W_U4 && tiles > 74 && tiles <= 90 && K >= 6144 && K <= 8192) return false;
    return K >= (wmode == OVB_W_U4 ? u4 : bytes)[row][col];
}

bool gemm_few_takes(const ovb_gemm_args* a) {
    if (!is_quant(a->wmode) || a->T > kFewTokens || a->comm != nullptr || a->group_offsets != nullptr || a->group_mode == 3 || a->block_t != 0) return false;
    if (a->N % TILE_N != 0 || a->K % kFewStageK != 0 || a->group_size % 128 != 0 || a->w_kb_stride != 0) return false;
    if (a->splits > 8 || a->splits > a->K / kFewStageK) return false;
    if (a->splits == 0 && !few_is_faster(a->wmode, a->T, a->N / TILE_N, a->K)) return false;
    FewPlan f;
    return few_plan(a->wmode, a->T, a->N, a->K, a->splits, &f);
}

template <int WMODE>
static int run_few(const ovb_gemm_args* a, cudaStream_t stream) {
    const bool gated = a->act == OVB_ACT_SWIGLU || a->act == OVB_ACT_GLU_LIMITED;
    FewPlan f;
    if (!few_plan(WMODE, a->T, a->N, a->K, a->splits, &f)) return ERR_UNSUPPORTED;
    FewParams p;
    memset(&p, 0, sizeof(p));
    p.w = static_cast<const uint8_t*>(a->w);
    p.sz = static_cast<const uint32_t*>(a->scales);
    p.out = a->out;
    p.bias = a->bias;
    p.residual = a->residual;
    p.status = status_word();
    p.T = a->T;
    p.N = a->N;
    p.K = a->K;
    p.ldo = a->ldo ? a->ldo : (gated ? a->N / 2 : a->N);
    p.ldr = a->ldr ? a->ldr : a->N;
    p.kb_stride = a->K / TILE_K;
    p.gpk = a->group_size / 128;
    p.nt = (a->T + 15) / 16 * 16;
    p.ring = f.ring;
    p.xslots = f.xslots;
    p.bufs = f.bufs;
    p.groups = f.groups;
    p.unit_cap = f.unit_cap;
    p.act = a->act;
    p.out_f32 = a->out_f32;
    p.act_limit = a->act_limit;
    p.act_slope = a->act_slope;
    p.act_shift = a->act_shift;
    CUtensorMap tmW, tmX;
    const int ldx = a->ldx ? a->ldx : a->K;
    // [block of columns][row][64 tokens' values or 128 bytes]: a stage of either operand is one copy
    if (int rc = make_tmap_blocks(&tmX, a->x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a->T, a->K, (uint64_t)ldx * 2, p.nt, TILE_K, kFewStageK / TILE_K)) return rc;
    if (WMODE == OVB_W_U4) tmW = tmX;
    else if (int rc = make_tmap_blocks(&tmW, a->w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a->N, a->K, (uint64_t)a->K, TILE_N, 128, kFewStageK / 128)) return rc;
    auto kern = gemm_few_kernel<WMODE>;
    {
        static std::mutex mu;
        static uint64_t configured = 0;         // one bit per device
        int dev = 0;
        OVB_CHECK_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lk(mu);
        if (!(configured & (1ull << (dev & 63)))) {
            OVB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kFewSmem));
            OVB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
            configured |= 1ull << (dev & 63);
        }
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(f.clusters * f.splits);
    cfg.blockDim = dim3((12 + 4 * f.groups) * 32);
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
    OVB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, tmW, tmX, static_cast<const FewParams>(p)));
    OVB_CHECK_CUDA(cudaGetLastError());
    return 0;
}

int gemm_few(const ovb_gemm_args* a, cudaStream_t stream) {
    switch (a->wmode) {
        case OVB_W_U4: return run_few<OVB_W_U4>(a, stream);
        case OVB_W_U8: return run_few<OVB_W_U8>(a, stream);
        default: return run_few<OVB_W_F8>(a, stream);
    }
}

}  // namespace ovb
