// Products of many tokens: out[T, N] = epilogue(X[T, K] * W[N, K]^T) on pairs of CTAs (tcgen05, cta_group::2).
//
// What bounds it: the tensor pipe. A pair of SMs works on one tile of 256 weight rows x up to 256 tokens: every CTA loads its
// 128 weight rows and HALF of the token tile, so that a k-block costs 32 KB of shared memory per SM for 256 x 256 x 64 products (a
// single CTA with a 128 x 256 tile needs 48 KB for half of them). The kernel is persistent, and the accumulator exists twice in
// tensor memory (2 x 256 columns): the epilogue of a tile runs under the main loop of the next.
//  * warp 0: TMA producer; both CTAs report their bytes on the barrier of the even CTA, whose warp 1 issues the MMAs of the pair
//  * warps 4 .. 11: epilogue, straight from the accumulator to global memory (no staging of the tile)
//  * the token tile is any multiple of 32 up to 256, chosen on the host so that the last wave of tiles is nearly full; the tiles of one that
//    is not are cut (pick_pair_tile)
// Quantised weights are expanded into 16-bit tiles first, a piece of at most kScratchBytes at a time, where that takes less time than the
// fused expansion of gemm_sm100.cu, which is repeated for every token tile (expansion_pays).
// Measured on B200, one launch, T = 8192, 28672 x 4096 int8 weights with the fused gate: 2452 us in the single-CTA kernel, 1274 us here
// (expansion included, 1.51 PFLOP/s); T = 999, the same in bf16: 271 -> 159 us; top-2 of 8 experts, 4096 rows, 28672 x 4096: 969 -> 728 us.
// Counters (2048 tokens, bf16, 1.54 PFLOP/s): tensor pipe 85 % of the cycles, weights and tokens read once.
#include <mutex>

#include "gemm_common.cuh"

namespace ovb {

constexpr int kPairStages = 6;
constexpr int kPairThreads = 384;
constexpr int kPairStageBytes = 32768;              // 128 weight rows and up to 128 tokens, 64 columns of 16 bits
constexpr int kPairExchange = 16384;                // gate / up values on their way between the epilogue warps
constexpr int kPairSmem = kPairStages * kPairStageBytes + kPairExchange + 1024 + 1024;
constexpr int kPairBand = 8;                        // pairs of weight tiles per rasterisation band
constexpr int64_t kScratchBytes = 128ll << 20;

struct PairParams {
    void* out;
    const void* bias;
    const void* residual;
    int* status;
    const int* group_off;
    int T, N, K;
    int ldo, ldr;
    int bt;
    int full_tiles, cut;                            // (not grouped) tiles from full_tiles on are cut into `cut` parts along the tokens
    int kb_stride;                                  // chunks between consecutive weight tiles
    int num_groups, group_mode;
    int act, out_f32;
    float act_limit, act_slope, act_shift;
};

// Forms of the kernel: whole tiles; tiles of the last wave cut along the tokens; groups, whose rows are shared out evenly among as many tiles as
// they need, each as wide as that. (Groups of about 512 rows need two tiles of 256 or three of 192; tiles of 256 and a rest cost three of 256.) The
// token box that is loaded stays p.bt / 2 rows: boxes of 16 rows, as many as the tile has, took 1390 us where one wide box takes 817 (8 experts,
// 4096 rows, 28672 x 4096). us with equal tiles -> even
// ones: that product 780 -> 728, 4096 x 14336 443 -> 390 (341 with 512 rows in each group); 64 experts, 8192 rows, 3072 x 2048: 275 -> 185; 128
// experts, 32768 rows, 1536 x 2048: 454 -> 318; 8 experts, 16384 rows, 4096 x 14336: the same. 256 is the best limit: with 192 the first took 813.
constexpr int kPairWhole = 0, kPairCut = 1, kPairEven = 2;

struct PairTile {
    int n0;            // first weight row of the pair
    int t0, t_end;     // first token row, one past the last valid one
    int w_tile, w_kb;  // first weight tile of the pair and first k-block in the stack
    int bt;            // tokens of the tile
    bool valid;
};

__device__ __forceinline__ void pair_coords(int idx, int tiles_n, int tiles_t, int& n, int& t) {
    const int band_sz = kPairBand * tiles_t;
    const int band = idx / band_sz, r = idx - band * band_sz;
    const int in_band = min(kPairBand, tiles_n - band * kPairBand);
    t = r / in_band;
    n = band * kPairBand + (r - t * in_band);
}

template <int FORM>
__device__ __forceinline__ PairTile pair_tile(const PairParams& p, int idx) {
    const int tiles_n = (p.N + 255) / 256;
    PairTile r;
    int n, t;
    r.w_kb = 0;
    r.bt = p.bt;
    if (p.group_off == nullptr) {
        const int tiles_t = (p.T + p.bt - 1) / p.bt;
        int part = 0;
        if (FORM == kPairCut && idx >= p.full_tiles) {
            part = (idx - p.full_tiles) % p.cut;
            idx = p.full_tiles + (idx - p.full_tiles) / p.cut;
            r.bt = p.bt / p.cut;
        }
        r.valid = idx < tiles_n * tiles_t;
        pair_coords(r.valid ? idx : 0, tiles_n, tiles_t, n, t);
        r.t0 = t * p.bt + part * r.bt;
        r.t_end = p.T;
        r.w_tile = n * 2;
    } else {
        int g = 0, acc = 0, begin = 0, end = 0;
        for (; g < p.num_groups; ++g) {
            begin = __ldg(p.group_off + g);
            end = min(__ldg(p.group_off + g + 1), p.T);
            const int cnt = (max(0, end - begin) + p.bt - 1) / p.bt * tiles_n;
            if (idx < acc + cnt) break;
            acc += cnt;
        }
        r.valid = g < p.num_groups;
        if (!r.valid) return r;
        pair_coords(idx - acc, tiles_n, (end - begin + p.bt - 1) / p.bt, n, t);
        if (FORM == kPairEven) {
            const int rows = end - begin, n_t = (rows + p.bt - 1) / p.bt;
            r.bt = ((rows + n_t - 1) / n_t + 31) & ~31;         // at most p.bt; n_t tiles of this width hold all rows, n_t - 1 do not
        }
        r.t0 = begin + t * r.bt;
        r.t_end = end;
        r.w_tile = n * 2 + (p.group_mode == 1 ? g * (p.N / TILE_N) : 0);
        r.w_kb = p.group_mode == 2 ? g * (p.K / TILE_K) : 0;
    }
    r.n0 = n * 256;
    return r;
}

// Tensor load into this CTA's shared memory, bytes reported on the barrier at the same offset in the even CTA of the pair.
__device__ __forceinline__ void pair_load_2d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar & 0xFEFFFFFFu), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void pair_mma_elect(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrive on the barrier at this offset in both CTAs once the MMAs issued so far are done.
__device__ __forceinline__ void pair_commit_elect(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
        ::"r"(smem_u32(bar)), "h"((uint16_t)3)
        : "memory");
}
template <bool F16, int FORM>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const PairParams p, const __grid_constant__ CUtensorMap tmCut) {
    using E = typename Elem<F16>::type;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float* exchange = reinterpret_cast<float*>(smem + kPairStages * kPairStageBytes);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kPairStages * kPairStageBytes + kPairExchange);
    uint64_t* full = bars;                           // [stages] even CTA: both CTAs' tiles have landed
    uint64_t* empty = bars + kPairStages;            // [stages] both CTAs: the stage has been read
    uint64_t* acc_full = bars + 2 * kPairStages;     // [2] both CTAs: accumulator complete
    uint64_t* acc_empty = acc_full + 2;              // [2] even CTA: accumulator drained by the 16 epilogue warps of the pair
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* went_well = abort_flag + 1;        // [2]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kPairStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 16);
        }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmW);
        tma_prefetch_desc(&tmX);
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_arrive();
    cluster_wait();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const int pairs = (int)gridDim.x >> 1, first = (int)blockIdx.x >> 1;
    const int num_kb = p.K / TILE_K;
    // weights may have been expanded by the kernel before this one, and the group offsets come from an earlier one
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            const int tiles_n128 = p.N / TILE_N;
            int s = 0;
            uint32_t phase = 1;
            bool ok = true;
            for (int idx = first; ok; idx += pairs) {
                const PairTile t = pair_tile<FORM>(p, idx);
                if (!t.valid) break;
                // an odd last tile: the second CTA loads the first one's rows again and stores nothing
                const int own = (t.n0 / TILE_N + (int)rank) < tiles_n128 ? (int)rank : 0;
                int w_row = ((t.w_tile + own) * p.kb_stride + t.w_kb) * TILE_N;
                const int x_row = t.t0 + (int)rank * (t.bt / 2);
                const uint32_t tx = 2u * (TILE_N * 128 + ((FORM == kPairEven ? p.bt : t.bt) / 2) * 128);
                const CUtensorMap* tm = FORM != kPairCut || t.bt == p.bt ? &tmX : &tmCut;
                for (int kb = 0; kb < num_kb; ++kb) {
                    ok = mbar_wait(&empty[s], phase, abort_flag, p.status);
                    if (!ok) break;
                    const uint32_t st = smem_u32(smem) + s * kPairStageBytes, bar = smem_u32(&full[s]);
                    if (rank == 0) mbar_arrive_expect_tx(&full[s], tx);
                    pair_load_2d(st, &tmW, bar, 0, w_row);
                    pair_load_2d(st + TILE_N * 128, tm, bar, kb * TILE_K, x_row);
                    w_row += TILE_N;
                    if (++s == kPairStages) { s = 0; phase ^= 1; }
                }
            }
            if (OVB_PDL_GEMM) pdl_trigger();
        }
        __syncwarp();
    } else if (warp == 1) {
        if (rank == 0) {
            const uint64_t desc0 = umma_desc_k_sw128(smem_u32(smem), 1024);
            int s = 0, buf = 0;
            uint32_t phase = 0, acc_phase = 1;
            bool ok = true;
            for (int idx = first; ok; idx += pairs) {
                const PairTile t = pair_tile<FORM>(p, idx);
                if (!t.valid) break;
                const uint32_t idesc = umma_idesc_f16(256, t.bt, !F16);
                ok = mbar_wait(&acc_empty[buf], acc_phase, abort_flag, p.status);
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t d = tmem_base + uint32_t(buf * 256);
                for (int kb = 0; kb < num_kb; ++kb) {
                    ok = mbar_wait(&full[s], phase, abort_flag, p.status);
                    if (!ok) break;
                    tc_fence_after_sync();
                    const uint64_t da = desc0 + (uint64_t)((s * kPairStageBytes) >> 4), db = da + (uint64_t)((TILE_N * 128) >> 4);
#pragma unroll
                    for (int k = 0; k < TILE_K / 16; ++k) pair_mma_elect(d, da + 2 * k, db + 2 * k, idesc, (kb | k) ? 1u : 0u);
                    pair_commit_elect(&empty[s]);
                    if (++s == kPairStages) { s = 0; phase ^= 1; }
                }
                if (!ok) break;
                pair_commit_elect(&acc_full[buf]);
                if (++buf == 2) { buf = 0; acc_phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp >= 4) {
        const int q = warp & 3, half = (warp - 4) >> 2;
        const int odd = lane & 1;
        const bool gated = p.act == OVB_ACT_SWIGLU || p.act == OVB_ACT_GLU_LIMITED;
        const uint32_t drained0 = dsmem_addr(smem_u32(&acc_empty[0]), 0);
        int buf = 0;
        uint32_t acc_phase = 0;
        for (int idx = first;; idx += pairs) {
            const PairTile t = pair_tile<FORM>(p, idx);
            if (!t.valid) break;
            const int cols = t.bt / 2, cbeg = half * cols;       // this warp's token columns
            const int n0 = t.n0 + (int)rank * TILE_N;
            const bool store = n0 < p.N;
            const int oc = n0 + q * 32 + lane;
            const float bias_v = p.bias != nullptr && store ? to_float(reinterpret_cast<const E*>(p.bias)[oc]) : 0.f;
            // two tokens at a time: neighbouring lanes exchange a value, so that each holds two adjacent columns of one token
            const E* res = reinterpret_cast<const E*>(p.residual) + (size_t)(t.t0 + cbeg + odd) * p.ldr + (oc & ~1);
            const bool has_res = p.residual != nullptr && store;
            uint32_t rn[8];
            auto fetch = [&](int c) {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    rn[j] = (t.t0 + cbeg + c + 2 * j + odd < t.t_end) ? __ldcg(reinterpret_cast<const uint32_t*>(res + (size_t)(c + 2 * j) * p.ldr)) : 0u;
            };
            if (has_res) fetch(0);
            // one thread polls and says how it ended; the others wait at the barrier, so that all eight warps go on or leave together
            // (the warps of a gate / up pair meet at barriers of their own)
            if (threadIdx.x == 128) went_well[buf] = mbar_wait(&acc_full[buf], acc_phase, abort_flag, p.status) ? 1 : 0;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (!went_well[buf]) break;
            tc_fence_after_sync();
            const uint32_t src = tmem_base + (uint32_t(q * 32) << 16) + uint32_t(buf * 256 + cbeg);
            for (int c = 0; c < cols; c += 16) {
                uint32_t r[16];
                tmem_ld_x16(src + c, r);
                tmem_ld_wait();
                if (c + 16 >= cols) {                            // last read of the accumulator by this warp
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) arrive_cluster(drained0 + buf * 8);
                }
                const int tok = t.t0 + cbeg + c;
                if (gated) {
                    // Rows 0..63 of the tile are the gate, 64..127 the up values of the same channels: the warps of the two halves
                    // swap eight tokens each and finish the eight that they keep.
                    const bool up_warp = q >= 2;
                    float* box = exchange + ((half * 2 + (q & 1)) * 2) * 256;      // [2][8 tokens][32 channels] of this pair of warps
                    float* to = box + (up_warp ? 0 : 256);
                    const float* from = box + (up_warp ? 256 : 0);
#pragma unroll
                    for (int j = 0; j < 8; ++j) to[j * 32 + lane] = __uint_as_float(up_warp ? r[j] : r[8 + j]);
                    asm volatile("bar.sync %0, 64;" ::"r"(2 + half * 2 + (q & 1)) : "memory");
                    const int first_tok = tok + (up_warp ? 8 : 0);
                    float v[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float other = from[j * 32 + lane], mine = __uint_as_float(up_warp ? r[8 + j] : r[j]);
                        const float g = up_warp ? other : mine, u = up_warp ? mine : other;
                        v[j] = p.act == OVB_ACT_SWIGLU ? g / (1.0f + __expf(-g)) * u : glu_limited(p, g, u);
                    }
                    asm volatile("bar.sync %0, 64;" ::"r"(2 + half * 2 + (q & 1)) : "memory");
                    const int ch = (n0 >> 1) + (q & 1) * 32 + lane;
                    E* o = reinterpret_cast<E*>(p.out) + (size_t)(first_tok + odd) * p.ldo + (ch & ~1);
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const float got = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
                        E pair[2] = {from_float<E>(odd ? got : v[j]), from_float<E>(odd ? v[j + 1] : got)};
                        if (store && first_tok + j + odd < t.t_end) *reinterpret_cast<uint32_t*>(o + (size_t)j * p.ldo) = *reinterpret_cast<uint32_t*>(pair);
                    }
                } else if (p.out_f32) {
                    float* o = reinterpret_cast<float*>(p.out) + (size_t)tok * p.ldo + oc;
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]) + bias_v;
                    apply_act_n(v, p);
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (store && tok + j < t.t_end) o[(size_t)j * p.ldo] = v[j];
                } else {
                    uint32_t rc[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) rc[j] = rn[j];
                    if (has_res && c + 16 < cols) fetch(c + 16);
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]) + bias_v;
                    apply_act_n(v, p);
                    E* o = reinterpret_cast<E*>(p.out) + (size_t)(tok + odd) * p.ldo + (oc & ~1);
#pragma unroll
                    for (int j = 0; j < 16; j += 2) {
                        const float got = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
                        float a = odd ? got : v[j], b = odd ? v[j + 1] : got;
                        if (has_res) {
                            const E* re = reinterpret_cast<const E*>(&rc[j >> 1]);
                            a += to_float(re[0]);
                            b += to_float(re[1]);
                        }
                        E pair[2] = {from_float<E>(a), from_float<E>(b)};
                        if (store && tok + j + odd < t.t_end) *reinterpret_cast<uint32_t*>(o + (size_t)j * p.ldo) = *reinterpret_cast<uint32_t*>(pair);
                    }
                }
            }
            if (++buf == 2) { buf = 0; acc_phase ^= 1; }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        // copies that are still in flight land before the shared memory is reused
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        __syncthreads();
    }
    cluster_arrive();
    cluster_wait();
    if (warp == 2) {
        tc_fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    }
}

// Quantised rows [0, rows) of a weight -> 16-bit tiles (the layout of ovb_pack_w16), the same values that the fused expansion
// gives. What bounds it: memory, 2.5 (u4) or 3 bytes per weight. Eight neighbouring lanes write the eight 16-byte pieces of a row's
// k-block, a whole 128-byte line; a thread takes four rows, so four loads are in flight.
template <int WMODE>
__global__ void __launch_bounds__(256) expand_weights_kernel(const uint8_t* __restrict__ w, const uint32_t* __restrict__ sz, uint4* __restrict__ out,
                                                             int n_base, int N, int KB, int kb_stride, int kpg) {
    pdl_enter();
    const int chunk = blockIdx.x;                       // (weight tile, k-block)
    const int tile = chunk / KB, kb = chunk - tile * KB;
    const int u = threadIdx.x & 7, r0 = threadIdx.x >> 3;
    uint4* dst = out + (size_t)chunk * 1024;
    if (WMODE == OVB_W_U4) {
        const uint8_t* src = w + ((size_t)(n_base / TILE_N + tile) * kb_stride + kb) * (TILE_N * 36);
        uint32_t q[4], s[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = r0 + i * 32;
            q[i] = __ldg(reinterpret_cast<const uint32_t*>(src + (u >> 2) * (TILE_N * 16) + r * 16 + (u & 3) * 4));
            s[i] = __ldg(reinterpret_cast<const uint32_t*>(src + TILE_N * 32 + r * 4));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = r0 + i * 32;
            const __nv_bfloat162 szp = *reinterpret_cast<const __nv_bfloat162*>(&s[i]);
            dst[r * 8 + (u ^ (r & 7))] = dequant_u4x8(q[i], row_scale(szp, 16.f));
        }
    } else {
        const size_t K = (size_t)KB * TILE_K;
        uint2 q[4];
        uint32_t s[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int n = n_base + tile * TILE_N + r0 + i * 32;
            q[i] = __ldg(reinterpret_cast<const uint2*>(w + (size_t)n * K + kb * TILE_K + u * 8));
            s[i] = __ldg(sz + (size_t)(kb / kpg) * N + n);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = r0 + i * 32;
            const __nv_bfloat162 szp = *reinterpret_cast<const __nv_bfloat162*>(&s[i]);
            uint32_t o[4];
            if (WMODE == OVB_W_F8) {
                const __nv_bfloat162 ss2 = __halves2bfloat162(__low2bfloat16(szp), __low2bfloat16(szp));
                dequant_f8x4(q[i].x, ss2, o[0], o[1]);
                dequant_f8x4(q[i].y, ss2, o[2], o[3]);
            } else {
                const RowScale rs = row_scale(szp, 0.f);
                dequant_u8x4(q[i].x, rs, o[0], o[1]);
                dequant_u8x4(q[i].y, rs, o[2], o[3]);
            }
            dst[r * 8 + (u ^ (r & 7))] = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
}

// --------------------------------------------------------------------------------------------- host
// Pairs of CTAs that are resident at a time (GPCs with an odd number of free SMs hold fewer than SMs / 2).
template <bool F16>
static int resident_pairs(int* pairs) {
    static std::mutex mu;
    static int known[64] = {0};
    int dev = 0;
    OVB_CHECK_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    if (known[dev & 63] == 0) {
        auto kern = gemm_pair_kernel<F16, kPairWhole>;
        OVB_CHECK_CUDA(cudaFuncSetAttribute(gemm_pair_kernel<F16, kPairCut>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem));
        OVB_CHECK_CUDA(cudaFuncSetAttribute(gemm_pair_kernel<F16, kPairEven>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem));
        OVB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem));
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3(148);
        cfg.blockDim = dim3(kPairThreads);
        cfg.dynamicSmemBytes = kPairSmem;
        int n = 0;
        OVB_CHECK_CUDA(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
        known[dev & 63] = n < 1 ? 1 : n;
    }
    *pairs = known[dev & 63];
    return 0;
}

// The last wave, when it would leave most pairs idle: its tiles are cut along the tokens, into parts of a multiple of 32 and so few that each pair
// has at most one.
static int pick_cut(int bt, int rest, int pairs) {
    int best = 1;
    for (int f = 2; f <= 8; ++f)
        if (rest > 0 && rest * f <= pairs && bt % (32 * f) == 0) best = f;
    return best;
}

// Token tile: the smallest estimate of waves x (tile + 32); the constant stands for what a wave costs beside its MMAs (the pair that
// finishes last, the epilogue of the last tile). With 999 tokens a 256-token tile of the 4096 x 4096 product fills 64 of 74 pairs
// once, 6144 rows fill them 1.3 times and take 192-token tiles (two full waves) instead.
// A cut last wave has to be cheaper by 3 %. Its parts read their 256 weight rows once each and take 166 of these units with 32 tokens, 182 with 64, 214 with
// 128 (100 products of 192 to 3000 tokens, K 2048 to 14336). us without / with it, gate and up of 28672 x 4096: 512 tokens 98.8 / 89.6, 999: 166.7 /
// 160.3; 4096 x 14336, 4096 tokens: 331 / 315; 19200 x 2048, 512 tokens: 48.6 / 37.4. Where 72 parts stand for 12 tiles it costs as much as it gives or more
// (10240 x 8192, 768 tokens: 101 / 109, 8192 x 4096, 900: 66 / 75), and so it does where nearly every pair has a tile (4096 x 4096, 1024 tokens,
// one cut wave of 64 tiles: 31 / 34) and where the sum is short (4096 x 1024, 4096 tokens: 36.3 / 37.0).
constexpr int kCutMinK = 2048;
static int pick_pair_tile(int T, int N, int K, int pairs, int* cut) {
    const int tiles_n = ceil_div(N, 256);
    int best = 256, best_cut = 1;
    double best_t = 1e30;
    for (int bt = 256; bt >= 64; bt -= 32) {
        const double t = (double)ceil_div(tiles_n * ceil_div(T, bt), pairs) * (bt + 32);
        if (t < best_t * 0.999) { best_t = t; best = bt; }
    }
    if (cut == nullptr || K < kCutMinK || (int64_t)tiles_n * ceil_div(T, 64) > (1 << 24)) return best;
    best_t *= 0.97;
    for (int bt = 256; bt >= 64; bt -= 32) {
        const int tiles = tiles_n * ceil_div(T, bt), parts = tiles < pairs ? 1 : pick_cut(bt, tiles % pairs, pairs);
        const double t = (double)(tiles / pairs) * (bt + 32) + 0.5 * bt / parts + 150;
        if (parts > 1 && t < best_t) { best_t = t; best = bt; best_cut = parts; }
    }
    *cut = best_cut;
    return best;
}

// Rows of a quantised weight that are expanded at a time: as many as the scratch holds, fewer where that saves waves.
static int pick_piece(int T, int N, int K, int bt, int pairs, int64_t scratch_bytes) {
    const int64_t max_rows = scratch_bytes / ((int64_t)K * 2) / 256 * 256;
    if (max_rows >= N) return N;
    if (max_rows < 256) return 0;
    const int tiles_t = ceil_div(T, bt), total = ceil_div(N, 256), most = (int)(max_rows / 256);
    int best = most;
    long long best_w = 1ll << 60;
    for (int r = most; r >= (most + 1) / 2; --r) {
        const int whole = total / r, rest = total - whole * r;
        const long long w = (long long)whole * ceil_div(r * tiles_t, pairs) + (rest ? ceil_div(rest * tiles_t, pairs) : 0);
        if (w < best_w) { best_w = w; best = r; }
    }
    return best * 256;
}

// From how many tokens on: 16-bit weights above one 128-token tile of the single-CTA kernel; quantised weights from 1024 on, where
// expansion_pays says so (for bytes the two are already equal at about 400 tokens: 28672 x 4096, 384 tokens, 201 / 166 us; the callers
// provide scratch memory from 1024 on).
constexpr int kPairMinTokens = 129;
constexpr int kPairMinTokensQuant = 1024;

// Is the expansion with a product of 16-bit tiles after it faster than the fused one? Both are estimated in microseconds, constants fitted
// to 156 measured pairs (the products of an 8B and a 70B model in u4, u8 and fp8, 1024 to 8192 tokens, cold caches): the faster one is
// chosen in all but four, which lose 2 to 5 %. Fused / expanded, us: u4 28672 x 4096 1024 tokens 264 / 226, 8192 tokens 2006 / 1252; 4096 x
// 14336 1024 tokens 86 / 112; 57344 x 8192 1024 tokens 793 / 986; u8 4096 x 14336 1024 tokens 158 / 118. The expansion loses where it writes
// many bytes for few tokens, and where K is so long that a piece of the scratch memory does not fill the machine: 8192 x 28672 1024 tokens,
// u4 324 / 685, u8 575 / 691.
static bool expansion_pays(const ovb_gemm_args* a) {
    constexpr int kPairs = 74, kSMs = 148;
    const bool u4 = a->wmode == OVB_W_U4, gated = a->act == OVB_ACT_SWIGLU || a->act == OVB_ACT_GLU_LIMITED;
    // fused: waves of 128 x 256 tiles
    const double k_us = a->K * 1e-3, fused_wave = (u4 ? 3.5 : 0.0) + (gated ? 10.0 : 0.0) + k_us * (u4 ? 6.2 : a->wmode == OVB_W_U8 ? 10.6 : 11.0);
    const double fused = ceil_div(ceil_div(a->N, TILE_N) * ceil_div(a->T, 256), kSMs) * fused_wave;
    // expanded: launches and bytes of the expansion, waves of 256 x bt tiles of every piece
    const int bt = pick_pair_tile(a->T, a->N, a->K, kPairs, nullptr), piece = pick_piece(a->T, a->N, a->K, bt, kPairs, kScratchBytes);
    if (piece <= 0) return false;
    int pieces = 0, waves = 0;
    for (int n = 0; n < a->N; n += piece, ++pieces) waves += ceil_div(ceil_div(a->N - n < piece ? a->N - n : piece, 256) * ceil_div(a->T, bt), kPairs);
    const double expanded = 3.0 * pieces + (double)a->N * a->K * 2 / (1 << 20) * (u4 ? 0.30 : 0.36) + waves * k_us * 5.7 * (bt + 32) / 288;
    return expanded < fused;
}

static bool pair_shape(const ovb_gemm_args* a) {
    const bool quant = is_quant(a->wmode);
    const bool swiglu = a->act == OVB_ACT_SWIGLU || a->act == OVB_ACT_GLU_LIMITED;
    const int ldo = a->ldo ? a->ldo : (swiglu ? a->N / 2 : a->N), ldr = a->ldr ? a->ldr : a->N;
    if (a->comm != nullptr || a->group_mode == 3 || a->K % TILE_K != 0 || a->N % TILE_N != 0) return false;
    if (!quant && !a->w_tiled) return false;
    if (a->T < (quant ? kPairMinTokensQuant : kPairMinTokens)) return false;
    if (a->group_offsets != nullptr) {
        if (quant || a->block_t < 128 || a->bias != nullptr || a->residual != nullptr) return false;
    } else if (a->block_t != 0 || a->splits > 1) {
        return false;
    } else if (ceil_div(a->N, 256) * ceil_div(a->T, 64) < 37) {
        return false;           // less than half of the pairs would have a tile: the other kernel splits K over a cluster
    }
    if (quant && (a->w_kb_stride != 0 || a->group_size <= 0 || !expansion_pays(a))) return false;
    if (a->out_f32) {
        if (a->residual != nullptr || swiglu || (reinterpret_cast<uintptr_t>(a->out) & 3) != 0) return false;
    } else {
        if (ldo % 2 != 0 || (reinterpret_cast<uintptr_t>(a->out) & 3) != 0) return false;
        if (a->residual != nullptr && (ldr % 2 != 0 || (reinterpret_cast<uintptr_t>(a->residual) & 3) != 0)) return false;
    }
    return true;
}

bool gemm_pair_takes(const ovb_gemm_args* a) {
    if (!pair_shape(a)) return false;
    return !is_quant(a->wmode) || (a->scratch != nullptr && (reinterpret_cast<uintptr_t>(a->scratch) & 15) == 0 && a->scratch_bytes >= (int64_t)256 * a->K * 2);
}

template <bool F16>
static int run_pair(const ovb_gemm_args* a, cudaStream_t stream) {
    const bool quant = is_quant(a->wmode);
    const bool swiglu = a->act == OVB_ACT_SWIGLU || a->act == OVB_ACT_GLU_LIMITED;
    const bool grouped = a->group_offsets != nullptr;
    int pairs = 0;
    if (int rc = resident_pairs<F16>(&pairs)) return rc;
    PairParams p;
    memset(&p, 0, sizeof(p));
    p.status = status_word();
    p.group_off = a->group_offsets;
    p.T = a->T;
    p.K = a->K;
    p.ldo = a->ldo ? a->ldo : (swiglu ? a->N / 2 : a->N);
    p.ldr = a->ldr ? a->ldr : a->N;
    p.cut = 1;
    p.bt = grouped ? 256 : pick_pair_tile(a->T, a->N, a->K, pairs, quant ? nullptr : &p.cut);
    p.num_groups = a->num_groups;
    p.group_mode = a->group_mode;
    p.act = a->act;
    p.out_f32 = a->out_f32;
    p.act_limit = a->act_limit;
    p.act_slope = a->act_slope;
    p.act_shift = a->act_shift;
    const int KB = a->K / TILE_K;
    const CUtensorMapDataType dt16 = F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    CUtensorMap tmW, tmX, tmCut;
    const int ldx = a->ldx ? a->ldx : a->K;
    if (int rc = make_tmap_2d(&tmX, a->x, dt16, 2, a->T, a->K, (uint64_t)ldx * 2, p.bt / 2, TILE_K, true)) return rc;
    const int piece = quant ? pick_piece(a->T, a->N, a->K, p.bt, pairs, a->scratch_bytes) : a->N;
    if (piece <= 0) {
        set_error("ovb_gemm: the scratch memory does not hold one tile of expanded weights");
        return ERR_TOO_LARGE;
    }
    const int esz = a->out_f32 ? 4 : 2;
    for (int n = 0; n < a->N; n += piece) {
        const int rows = a->N - n < piece ? a->N - n : piece;
        const void* w = a->w;
        int64_t w_chunks;               // 16 KB chunks from `w` to the end of what the problem reads
        if (quant) {
            const dim3 grid(rows / TILE_N * KB);
            const int kpg = a->group_size / TILE_K;
            const uint8_t* wq = static_cast<const uint8_t*>(a->w);
            const uint32_t* sz = static_cast<const uint32_t*>(a->scales);
            uint4* dst = static_cast<uint4*>(a->scratch);
            if (a->wmode == OVB_W_U4) OVB_CHECK_CUDA(launch_pdl(expand_weights_kernel<OVB_W_U4>, grid, dim3(256), 0, stream, wq, sz, dst, n, a->N, KB, KB, kpg));
            else if (a->wmode == OVB_W_U8) OVB_CHECK_CUDA(launch_pdl(expand_weights_kernel<OVB_W_U8>, grid, dim3(256), 0, stream, wq, sz, dst, n, a->N, KB, KB, kpg));
            else OVB_CHECK_CUDA(launch_pdl(expand_weights_kernel<OVB_W_F8>, grid, dim3(256), 0, stream, wq, sz, dst, n, a->N, KB, KB, kpg));
            w = a->scratch;
            p.kb_stride = KB;
            w_chunks = (int64_t)(rows / TILE_N) * KB;
        } else {
            p.kb_stride = a->w_kb_stride > 0 ? a->w_kb_stride : KB * (grouped && a->group_mode == 2 ? a->num_groups : 1);
            const int tiles = rows / TILE_N * (grouped && a->group_mode == 1 ? a->num_groups : 1);
            w_chunks = (int64_t)(tiles - 1) * p.kb_stride + (int64_t)KB * (grouped && a->group_mode == 2 ? a->num_groups : 1);
        }
        // the chunks are already in the swizzled order of the MMA: plain boxes of 128 rows of 128 bytes
        if (int rc = make_tmap_2d(&tmW, w, dt16, 2, (uint64_t)w_chunks * TILE_N, TILE_K, 128, TILE_N, TILE_K, false)) return rc;
        p.N = rows;
        p.out = static_cast<uint8_t*>(a->out) + (size_t)(swiglu ? n / 2 : n) * esz;
        p.bias = a->bias ? static_cast<const uint8_t*>(a->bias) + (size_t)n * 2 : nullptr;
        p.residual = a->residual ? static_cast<const uint8_t*>(a->residual) + (size_t)n * 2 : nullptr;
        // every group may end with a partial row tile
        int64_t tiles = (int64_t)ceil_div(rows, 256) * (ceil_div(a->T, p.bt) + (grouped ? a->num_groups : 0));
        p.full_tiles = p.cut > 1 ? (int)(tiles / pairs * pairs) : 0;
        tmCut = tmX;
        if (p.cut > 1) tiles = p.full_tiles + (tiles - p.full_tiles) * p.cut;
        if (p.cut > 1)
            if (int rc = make_tmap_2d(&tmCut, a->x, dt16, 2, a->T, a->K, (uint64_t)ldx * 2, p.bt / p.cut / 2, TILE_K, true)) return rc;
        const int grid = 2 * (int)(tiles < pairs ? tiles : pairs);
        OVB_CHECK_CUDA(launch_pdl(grouped ? gemm_pair_kernel<F16, kPairEven> : p.cut > 1 ? gemm_pair_kernel<F16, kPairCut> : gemm_pair_kernel<F16, kPairWhole>, dim3(grid), dim3(kPairThreads), kPairSmem, stream, tmW, tmX, p, tmCut));
        OVB_CHECK_CUDA(cudaGetLastError());
    }
    return 0;
}

int gemm_pair(const ovb_gemm_args* a, cudaStream_t stream) { return a->wmode == OVB_W_F16 ? run_pair<true>(a, stream) : run_pair<false>(a, stream); }

}  // namespace ovb

extern "C" int64_t ovb_gemm_scratch_bytes(const ovb_gemm_args* a) {
    using namespace ovb;
    if (!is_quant(a->wmode) || !pair_shape(a)) return 0;
    const int64_t all = (int64_t)a->N * a->K * 2, least = (int64_t)256 * a->K * 2;
    return all < kScratchBytes ? (all < least ? least : all) : (kScratchBytes > least ? kScratchBytes : least);
}
