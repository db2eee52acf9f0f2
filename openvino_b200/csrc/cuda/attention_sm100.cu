// Flash attention on the 5th-generation tensor cores (tcgen05 + TMEM + TMA): ragged paged prefill / mixed batches and
// dense (encoder) attention. Same semantics and parameters as pa_prefill_kernel in attention.cu, which stays as the
// fallback for shapes this kernel does not serve.
//
// Roles of the reference kernels this fills: src/plugins/intel_gpu/src/graph/impls/ocl_v2/sdpa_micro.cl:141 (prefill
// SDPA), paged_attention_opt.cl:64 (paged prefill), src/plugins/intel_cpu/src/nodes/kernels/scaled_attn/executor_pa.cpp:1470.
//
// One CTA owns 128 stacked query rows of one (sequence, KV head): row r = g * TOK + t is query head g of the group and the
// t-th token of the tile (TOK = 128 / G tokens), so that K/V pages are fetched once for the G heads that share them.
//
//   warp 4 (one lane)  : TMA. Q tile once (G boxes per 64-column half), then per 128-key tile the K and V pages of the
//                        sequence's block table, 16 keys x 64 columns per box, 128-byte swizzle, two stages.
//   warp 5 (elected)   : tcgen05.mma.  S[j] = Q K_j^T (both operands in shared memory, accumulator S in tensor memory,
//                        double buffered), then O += P_j V_j with P_j read from tensor memory (.ts form) and V_j as an
//                        MN-major shared-memory operand (V rows are keys, i.e. the reduction dimension). QK of tile j + 1
//                        is issued before PV of tile j, so the tensor core works on it while the softmax of tile j runs.
//   warps 0-3          : softmax, one thread per query row (no shuffles): tcgen05.ld of the row of S, masks, running
//                        maximum and sum in the exp2 domain, P as 16-bit pairs back into tensor memory (tcgen05.st).
//                        The running maximum is only raised when the tile's maximum exceeds it by more than 8 (a factor
//                        of 256): the accumulator O, which lives in tensor memory, then has to be rescaled only a few
//                        times per row instead of once per tile. Epilogue: O / l -> 16-bit -> global.
//
// Tensor memory (512 columns): S0 0..127, S1 128..255, O 256..256+DV-1, P0 and P1 (64 columns each) behind it.
// Every wait is bounded (mbar_wait) and reports through the status word.
#include <float.h>
#include <math_constants.h>

#include <atomic>
#include <type_traits>

#include "attention.cuh"
#include "common.cuh"
#include "debug_bounds.cuh"
#include "sm100_ptx.cuh"

namespace ovb {

OVB_DEBUG_LIMITS_DEFINE

namespace {

constexpr int kBM = 128;   // stacked query rows per CTA
constexpr int kBK = 128;   // keys per tile
constexpr int kPage = 16;  // keys per TMA box (= the cache block size)

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// MN-major shared-memory operand with the 128-byte swizzle: 64 elements (128 bytes) of the MN dimension are contiguous, rows
// of the reduction dimension are 128 bytes apart, 8-row groups `sbo` bytes apart, 64-element MN blocks `lbo` bytes apart.
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
    d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}

template <bool F16>
__device__ __forceinline__ uint32_t pack16(float lo, float hi) {
    if (F16) {
        __half2 v = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&v);
    }
    return pack_bf16x2(lo, hi);
}

// Where keys and values come from: pages of the cache, dense tensors, or rows expanded from a latent cache (PaKParams::kv_rows).
enum : int { SRC_PAGED = 0, SRC_DENSE = 1, SRC_LATENT = 2 };

// Tokens per tile for a group of g query heads: whole 8-row groups, so that every head's rows start on a swizzle boundary.
__host__ __device__ constexpr int tile_tokens(int g) { return kBM / g / 8 * 8; }

// KH / RH / VH: 64-column (128-byte) parts of a key row, of its shared second part, and of a value row. A part that reaches past
// the end of a cache row is filled with zeros by the copy, so any size that is a multiple of 8 is served; what the query tile
// holds behind a head's columns meets those zeros. GT: query heads per KV head, 0 = at run time (p.group).
// BIAS (dense): a value per key is added to its scaled scores.
// TWO (dense heads of 64): S and P are kept once (256 columns of tensor memory), so that two CTAs share an SM and one's exponentials run beside the
// other's products; the scores are read twice, 32 at a time, instead of being held.
template <int KH, int RH, int VH, int GT, int SRC, bool F16, bool BIAS = false, bool TWO = false>
__global__ void __launch_bounds__(192, TWO ? 2 : 1)
pa_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                     const __grid_constant__ CUtensorMap tmR, PaKParams p, int* status) {
    static_assert(SRC == SRC_DENSE || (!BIAS && !TWO), "dense attention");
    constexpr bool PAGED = SRC != SRC_DENSE;                   // ragged batch with a descriptor
    constexpr int DK = (KH + RH) * 64, DV = VH * 64;
    const int G = GT > 0 ? GT : p.group;
    const int TOK = tile_tokens(G);            // tokens per tile
    constexpr int Q_BYTES = kBM * DK * 2, K_BYTES = kBK * DK * 2, V_BYTES = kBK * DV * 2;
    constexpr int SB = TWO ? 1 : 2;            // copies of S and P
    constexpr uint32_t TM_S = 0, TM_O = SB * 128, TM_P = SB * 128 + DV, TM_COLS = SB == 1 ? 256 : 512;   // tensor-memory columns
    constexpr uint32_t IDESC_QK = umma_idesc_f16(kBM, kBK, !F16);
    constexpr uint32_t IDESC_PV = umma_idesc_f16(kBM, DV, !F16) | (1u << 16);   // B operand MN-major

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + Q_BYTES;                // two stages
    uint8_t* sV = sK + 2 * K_BYTES;            // two stages
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + 2 * V_BYTES);
    uint64_t* q_full = bars;
    uint64_t* k_full = bars + 1;               // [2]
    uint64_t* v_full = bars + 3;               // [2]
    uint64_t* kv_empty = bars + 5;             // [2] PV of the tile in the stage has retired
    uint64_t* s_full = bars + 7;               // [2] QK of the tile has retired
    uint64_t* s_free = bars + 9;               // [2] the softmax threads are done with S
    uint64_t* p_full = bars + 11;              // [2] P written
    uint64_t* pv_done = bars + 13;             // [2] PV of the tile has retired (O may be touched, P may be overwritten)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* s_work = const_cast<int*>(abort_flag) + 1;   // [2]
    float* sBias = reinterpret_cast<float*>(bars + 32);   // BIAS: of all keys, times log2(e)

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.y;
    pdl_enter_attn();

    // ---- (sequence, q tile) of this CTA: tiles are numbered sequence by sequence; the grid is walked backwards so that the
    // tiles with the longest causal context start first
    if (threadIdx.x == 0) {
        const int bx = gridDim.x - 1 - blockIdx.x;
        int acc = 0, found = -1, tile = 0;
        for (int b = 0; b < p.B; ++b) {
            const int ql = PAGED ? p.subsequence_begins[b + 1] - p.subsequence_begins[b] : p.dense_S;
            const int nt = (ql + TOK - 1) / TOK;
            if (bx < acc + nt) { found = b; tile = bx - acc; break; }
            acc += nt;
        }
        s_work[0] = found;
        s_work[1] = tile;
        *abort_flag = 0;
        mbar_init(q_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&kv_empty[i], 1);
            mbar_init(&s_full[i], 1);
            mbar_init(&s_free[i], kBM);
            mbar_init(&p_full[i], kBM);
            mbar_init(&pv_done[i], 1);
        }
        mbar_fence_init();
    }
    // (The PV product reads whole pages only: its k-steps are 16 keys = one page, and steps past the last loaded page are
    // not issued, so stale shared memory never reaches the tensor core as V. Stale K rows only produce masked columns of S.)
    __syncthreads();
    const int b = s_work[0];
    if (b < 0) return;                          // (uniform) nothing allocated yet
    if (warp == 5) {
        tmem_alloc(tmem_slot, TM_COLS);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    const int qtile = s_work[1];
    const int tok_begin = PAGED ? p.subsequence_begins[b] : b * p.dense_S;
    const int q_len = PAGED ? p.subsequence_begins[b + 1] - tok_begin : p.dense_S;
    const int past = PAGED ? p.past_lens[b] : 0;
    const int blk_begin = PAGED ? p.block_indices_begins[b] : 0;
    const int tq0 = qtile * TOK;
    const int tq1 = min(q_len, tq0 + TOK);
    const int kv_total = PAGED ? past + q_len : p.dense_S;
    const int kv_end = p.causal ? min(kv_total, past + tq1) : kv_total;
    const int kv_start = PAGED ? first_visible_key(past + tq0, p.sliding_window, p.chunk) / kBK * kBK : 0;
    const int lo_last = PAGED ? first_visible_key(past + tq1 - 1, p.sliding_window, p.chunk) : 0;   // of the tile's last token
    const int ntiles = (kv_end - kv_start + kBK - 1) / kBK;

    if (warp == 4) {
        // ------------------------------------------------------------------ TMA producer
        // One lane posts the byte counts; then every lane issues the boxes of its own (page, half): a single thread that
        // issues the 64 small copies of a tile one after the other is slower than the tensor core consumes them.
        if (lane == 0) {
            mbar_arrive_expect_tx(q_full, G * TOK * DK * 2);
            for (int g = 0; g < G; ++g)
                for (int hf = 0; hf < KH + RH; ++hf)
                    tma_load_2d(sQ + hf * (kBM * 128) + g * (TOK * 128), &tmQ, q_full,
                                (h * G + g) * p.q_head + (hf < KH ? hf * 64 : p.q_shared + (hf - KH) * 64), tok_begin + tq0);
        }
        // row of key 0 of this sequence in contiguous key / value rows
        const int row_base = SRC == SRC_DENSE ? b * p.dense_S : SRC == SRC_LATENT ? p.kv_rows[b] - latent_first_key(past, p.sliding_window) : 0;
        for (int j = 0; j < ntiles; ++j) {
            const int st = j & 1;
            if (j >= 2 && !mbar_wait(&kv_empty[st], ((j >> 1) - 1) & 1, abort_flag, status)) break;
            const int j0 = kv_start + j * kBK;
            const int npages = (min(kv_end, j0 + kBK) - j0 + kPage - 1) / kPage;
            if (lane == 0) {
                mbar_arrive_expect_tx(&k_full[st], npages * kPage * DK * 2);
                mbar_arrive_expect_tx(&v_full[st], npages * kPage * DV * 2);
            }
            __syncwarp();
            for (int u = lane; u < npages * (KH + RH + VH); u += 32) {      // keys first
                const int part = u / npages, pg = u % npages;
                int row = row_base + j0 + pg * kPage, col_k = h * p.k_head, col_v = h * p.v_head;
                if (SRC == SRC_PAGED || (RH > 0 && part >= KH && part < KH + RH)) {
                    const int blk = OVB_DBG_BLOCK(p.block_indices[blk_begin + j0 / kPage + pg]);
                    row = SRC == SRC_PAGED ? (blk * p.Hkv + h) * kPage : blk * kPage;
                    col_k = col_v = 0;
                }
                uint8_t* dk = sK + st * K_BYTES + part * (kBK * 128) + pg * (kPage * 128);
                if (part < KH) tma_load_2d(dk, &tmK, &k_full[st], col_k + part * 64, row);
                else if (RH > 0 && part < KH + RH) tma_load_2d(dk, &tmR, &k_full[st], p.shared_col + (part - KH) * 64, row);
                else tma_load_2d(sV + st * V_BYTES + (part - KH - RH) * (kBK * 128) + pg * (kPage * 128), &tmV, &v_full[st], col_v + (part - KH - RH) * 64, row);
            }
        }
        __syncwarp();
    } else if (warp == 5) {
        // ------------------------------------------------------------------ MMA issuer (warp-uniform flow, one elected lane issues)
        bool ok = mbar_wait(q_full, 0, abort_flag, status);
        const uint64_t dq = umma_desc_k_sw128(smem_u32(sQ), 1024);
        for (int j = 0; j <= ntiles && ok; ++j) {
            if (j < ntiles) {
                const int st = j & 1, sb = j % SB;
                ok = ok && mbar_wait(&k_full[st], (j >> 1) & 1, abort_flag, status);
                if (j >= SB) ok = ok && mbar_wait(&s_free[sb], (j / SB - 1) & 1, abort_flag, status);
                if (!ok) break;
                tc_fence_after_sync();
                const uint64_t dk = umma_desc_k_sw128(smem_u32(sK + st * K_BYTES), 1024);
#pragma unroll
                for (int ks = 0; ks < DK / 16; ++ks) {
                    const uint64_t off = (uint64_t)(((ks >> 2) * (kBM * 128) + (ks & 3) * 32) >> 4);
                    umma_f16_ss_elect(tmem + TM_S + sb * kBK, dq + off, dk + off, IDESC_QK, ks > 0 ? 1u : 0u);
                }
                umma_commit_elect(&s_full[sb]);
            }
            if (j >= 1) {
                const int i = j - 1, st = i & 1, sb = i % SB;
                ok = ok && mbar_wait(&v_full[st], (i >> 1) & 1, abort_flag, status);
                ok = ok && mbar_wait(&p_full[sb], (i / SB) & 1, abort_flag, status);
                if (!ok) break;
                tc_fence_after_sync();
                const int keys = min(kBK, kv_end - (kv_start + i * kBK));
                const int ksteps = (keys + 15) / 16;
                const uint64_t dv = umma_desc_mn_sw128(smem_u32(sV + st * V_BYTES), kBK * 128, 1024);
                for (int kk = 0; kk < ksteps; ++kk)
                    umma_f16_ts_elect(tmem + TM_O, tmem + TM_P + sb * 64 + kk * 8, dv + (uint64_t)((kk * 16 * 128) >> 4), IDESC_PV,
                                      (i > 0 || kk > 0) ? 1u : 0u);
                umma_commit_elect(&kv_empty[st]);
                umma_commit_elect(&pv_done[sb]);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ softmax: one thread per stacked query row
        const int r = threadIdx.x;                       // 0..127 = tensor-memory lane
        const int g = r / TOK, tl = r % TOK;
        const int qpos = past + tq0 + tl;
        const bool row_valid = (tq0 + tl) < q_len && (GT > 0 || g < G);
        const int lo_row = PAGED ? first_visible_key(qpos, p.sliding_window, p.chunk) : 0;
        const uint32_t lane_base = tmem + (uint32_t(warp * 32) << 16);
        float m_used = -CUDART_INF_F, l_sum = 0.f;
        bool ok = true;
        const float scale = BIAS ? 1.f : p.scale_log2;        // (biased scores are scaled when the bias is added)
        if (BIAS) {
            using E = typename std::conditional<F16, __half, __nv_bfloat16>::type;
            const E* kb = reinterpret_cast<const E*>(p.key_bias) + (size_t)b * p.bias_stride;
            // A finite value stays finite: bf16's lowest, times log2(e), would be -inf, and a sequence all of whose keys have it gets the mean of its
            // values, as any equal scores do.
            for (int i = r; i < ntiles * kBK; i += kBM) {
                const float v = i < kv_total ? float(kb[i]) : 0.f, w = v * 1.4426950408889634f;
                sBias[i] = isinf(w) && !isinf(v) ? copysignf(FLT_MAX, v) : w;
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        for (int j = 0; j < ntiles && ok; ++j) {
            const int st = j % SB;
            ok = mbar_wait(&s_full[st], (j / SB) & 1, abort_flag, status);
            if (!ok) break;
            tc_fence_after_sync();
            const int j0 = kv_start + j * kBK;
            // does any row of the tile need a mask? (uniform over the CTA)
            const bool need_mask = (j0 + kBK > kv_end) || (p.causal && (j0 + kBK - 1 > past + tq0)) ||
                                   j0 < lo_last;
            int hi = kBK, lo = 0;                        // keys [lo, hi) of the tile are visible to this row
            if (need_mask) {
                hi = min(hi, kv_end - j0);
                if (p.causal) hi = min(hi, qpos - j0 + 1);
                lo = max(lo, lo_row - j0);
                if (!row_valid) hi = 0;
            }
            // 32 scores of the row, biased and masked (SB == 1)
            auto scores = [&](int c, uint32_t* w) {
                tmem_ld_x16(lane_base + TM_S + c, w);
                tmem_ld_x16(lane_base + TM_S + c + 16, w + 16);
                tmem_ld_wait();
                if (BIAS) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        const float4 kb = *reinterpret_cast<const float4*>(sBias + j0 + c + i);
                        w[i] = __float_as_uint(fmaf(__uint_as_float(w[i]), p.scale_log2, kb.x));
                        w[i + 1] = __float_as_uint(fmaf(__uint_as_float(w[i + 1]), p.scale_log2, kb.y));
                        w[i + 2] = __float_as_uint(fmaf(__uint_as_float(w[i + 2]), p.scale_log2, kb.z));
                        w[i + 3] = __float_as_uint(fmaf(__uint_as_float(w[i + 3]), p.scale_log2, kb.w));
                    }
                }
                if (need_mask) {
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (c + i < lo || c + i >= hi) w[i] = __float_as_uint(-CUDART_INF_F);
                }
            };
            uint32_t v[SB == 1 ? 32 : kBK];
            float mx[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
            if constexpr (SB == 1) {
#pragma unroll 1
                for (int c = 0; c < kBK; c += 32) {
                    scores(c, v);
#pragma unroll
                    for (int i = 0; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(v[i]));
                }
            } else {
                // The whole row of S goes to registers in one round trip to tensor memory (eight loads in flight, one wait);
                // S is then free for the QK product of tile j + 2 while this thread still works on the values.
#pragma unroll
                for (int c = 0; c < kBK; c += 16) tmem_ld_x16(lane_base + TM_S + st * kBK + c, v + c);
                tmem_ld_wait();
                tc_fence_before_sync();
                mbar_arrive(&s_free[st]);
                if (BIAS) {
#pragma unroll
                    for (int i = 0; i < kBK; i += 4) {
                        const float4 kb = *reinterpret_cast<const float4*>(sBias + j0 + i);
                        v[i] = __float_as_uint(fmaf(__uint_as_float(v[i]), p.scale_log2, kb.x));
                        v[i + 1] = __float_as_uint(fmaf(__uint_as_float(v[i + 1]), p.scale_log2, kb.y));
                        v[i + 2] = __float_as_uint(fmaf(__uint_as_float(v[i + 2]), p.scale_log2, kb.z));
                        v[i + 3] = __float_as_uint(fmaf(__uint_as_float(v[i + 3]), p.scale_log2, kb.w));
                    }
                }
                // maximum of the visible part of the row (four independent chains)
                if (need_mask) {
#pragma unroll
                    for (int i = 0; i < kBK; ++i) {
                        const bool vis = i >= lo && i < hi;
                        if (!vis) v[i] = __float_as_uint(-CUDART_INF_F);
                        mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(v[i]));
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < kBK; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(v[i]));
                }
            }
            float m_tile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale;   // scale > 0: max commutes with scaling
            // raise the running maximum only when the tile exceeds it by a factor of 2^8; the rescale of O is warp-collective
            const bool raise = m_tile > m_used + 8.f;
            if (__any_sync(0xffffffffu, raise)) {
                const float factor = !raise ? 1.f : (m_used == -CUDART_INF_F ? 0.f : fast_exp2(m_used - m_tile));
                if (j > 0) {
                    ok = mbar_wait(&pv_done[(j - 1) % SB], ((j - 1) / SB) & 1, abort_flag, status);
                    if (!ok) break;
                    tc_fence_after_sync();
#pragma unroll 1
                    for (int c = 0; c < DV; c += 32) {
                        uint32_t o[32];
                        tmem_ld_x16(lane_base + TM_O + c, o);
                        tmem_ld_x16(lane_base + TM_O + c + 16, o + 16);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
                        tmem_st_x16(lane_base + TM_O + c, o);
                        tmem_st_x16(lane_base + TM_O + c + 16, o + 16);
                    }
                    tmem_st_wait();
                }
                if (raise) {
                    l_sum *= factor;
                    m_used = m_tile;
                }
            }
            const float neg_m = (m_used == -CUDART_INF_F) ? 0.f : -m_used;
            float ls[4] = {0.f, 0.f, 0.f, 0.f};
            if constexpr (SB == 1) {
                // P of the tile before must have been consumed
                if (j >= 1) {
                    ok = mbar_wait(&pv_done[0], (j - 1) & 1, abort_flag, status);
                    if (!ok) break;
                }
#pragma unroll 1
                for (int c = 0; c < kBK; c += 32) {
                    scores(c, v);
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float e0 = fast_exp2(fmaf(__uint_as_float(v[i]), scale, neg_m));
                        const float e1 = fast_exp2(fmaf(__uint_as_float(v[i + 1]), scale, neg_m));
                        ls[(i >> 1) & 3] += e0 + e1;
                        v[i >> 1] = pack16<F16>(e0, e1);
                    }
                    tmem_st_x16(lane_base + TM_P + c / 2, v);
                }
                l_sum += (ls[0] + ls[1]) + (ls[2] + ls[3]);
                tc_fence_before_sync();
                mbar_arrive(&s_free[0]);
            } else {
                // exponentials (masked entries are -inf: exp2 gives 0), row sum, P as 16-bit pairs (packed in place)
#pragma unroll
                for (int i = 0; i < kBK; i += 2) {
                    const float e0 = fast_exp2(fmaf(__uint_as_float(v[i]), scale, neg_m));
                    const float e1 = fast_exp2(fmaf(__uint_as_float(v[i + 1]), scale, neg_m));
                    ls[(i >> 1) & 3] += e0 + e1;
                    v[i >> 1] = pack16<F16>(e0, e1);
                }
                l_sum += (ls[0] + ls[1]) + (ls[2] + ls[3]);
                // P of tile j - 2 (same buffer) must have been consumed
                if (j >= 2) {
                    ok = mbar_wait(&pv_done[st], ((j >> 1) - 1) & 1, abort_flag, status);
                    if (!ok) break;
                }
#pragma unroll
                for (int c = 0; c < kBK / 2; c += 16) tmem_st_x16(lane_base + TM_P + st * 64 + c, v + c);
            }
            tmem_st_wait();
            tc_fence_before_sync();
            mbar_arrive(&p_full[st]);
        }
        // ---- epilogue: O / l. The gate's row is requested before the last product is waited for.
        uint4 gw[DV / 8];
        const bool gated = p.gate != nullptr && !p.gate_scalar && row_valid;
        float head_gate = 1.f, sink = -CUDART_INF_F;
        if (row_valid) {
            if (p.gate != nullptr && p.gate_scalar) {
                const __nv_bfloat16 gv = reinterpret_cast<const __nv_bfloat16*>(p.gate)[(size_t)(tok_begin + tq0 + tl) * p.ld_gate + (size_t)(h * G + g) * p.gate_head];
                head_gate = __fdividef(1.f, 1.f + __expf(-__bfloat162float(gv)));
            }
            if (p.sink != nullptr) sink = p.sink[h * G + g] * 1.4426950408889634f;
        }
        if (gated) {
            const uint4* gate = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.gate) + (size_t)(tok_begin + tq0 + tl) * p.ld_gate +
                                                               (size_t)(h * G + g) * p.gate_head);
#pragma unroll
            for (int c = 0; c < DV / 8; ++c)
                if (c * 8 < p.dv_store) gw[c] = gate[c];
        }
        if (ok && ntiles > 0) ok = mbar_wait(&pv_done[(ntiles - 1) % SB], ((ntiles - 1) / SB) & 1, abort_flag, status);
        if (ok) {
            tc_fence_after_sync();
            if (sink != -CUDART_INF_F && m_used != -CUDART_INF_F) l_sum += exp2f(sink - m_used);
            const float inv = l_sum > 0.f ? head_gate / l_sum : 0.f;
            uint8_t* dst = reinterpret_cast<uint8_t*>(p.out) + ((size_t)(tok_begin + tq0 + tl) * p.ldo + (size_t)(h * G + g) * p.o_head) * 2;
#pragma unroll
            for (int c = 0; c < DV; c += 16) {
                if (c >= p.dv_store) break;
                uint32_t o[16];
                if (ntiles > 0) {
                    tmem_ld_x16(lane_base + TM_O + c, o);
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = 0u;
                }
                if (gated) {
                    const __nv_bfloat16* gv = reinterpret_cast<const __nv_bfloat16*>(gw + c / 8);
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__fdividef(__uint_as_float(o[i]), 1.f + __expf(-__bfloat162float(gv[i]))));
                }
                if (row_valid) {
                    uint4 w0, w1;
                    w0.x = pack16<F16>(__uint_as_float(o[0]) * inv, __uint_as_float(o[1]) * inv);
                    w0.y = pack16<F16>(__uint_as_float(o[2]) * inv, __uint_as_float(o[3]) * inv);
                    w0.z = pack16<F16>(__uint_as_float(o[4]) * inv, __uint_as_float(o[5]) * inv);
                    w0.w = pack16<F16>(__uint_as_float(o[6]) * inv, __uint_as_float(o[7]) * inv);
                    w1.x = pack16<F16>(__uint_as_float(o[8]) * inv, __uint_as_float(o[9]) * inv);
                    w1.y = pack16<F16>(__uint_as_float(o[10]) * inv, __uint_as_float(o[11]) * inv);
                    w1.z = pack16<F16>(__uint_as_float(o[12]) * inv, __uint_as_float(o[13]) * inv);
                    w1.w = pack16<F16>(__uint_as_float(o[14]) * inv, __uint_as_float(o[15]) * inv);
                    *reinterpret_cast<uint4*>(dst + c * 2) = w0;
                    *reinterpret_cast<uint4*>(dst + c * 2 + 16) = w1;
                }
            }
        }
    }

    // ---------------------------------------------------------------- tear-down
    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);   // copies still in flight land before the shared memory is reused
        __syncthreads();
    }
    if (warp == 5) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, TM_COLS);
    }
}

// Two query tiles per CTA (256 stacked rows) for long prompts: paged bf16 cache, head size 128, G query heads per KV head.
//
// What bounds the kernel above: with one tile per SM the softmax of a tile (128 exponentials of a thread, one warp per scheduler)
// and its two products follow one another, 3700 cycles per 128 x 128 tile where the tensor pipe needs 1024 and the exponentials
// 1024. Here warps 0-3 and 4-7 hold a tile each and take turns: while one tile's scores are being exponentiated, the tensor pipe
// works on the other's products, and both share the K and V tiles in shared memory (half the reads). Tensor memory is full with
// S and O of the two tiles (4 x 128 columns), so P overwrites the first half of its S, and the next QK product of a tile is issued
// after the PV product that reads P has retired. K and V stages are released on their own: K as soon as both QK products have
// read it, so that the next tile but one is on its way a whole turn earlier. A CTA whose second tile has no rows (a sequence's odd last
// tile, a decoding sequence) works on the first alone, one product after the other.
// One launch, cold caches, 32 query and 8 KV heads: 1 x 8191 tokens 873 us with one tile per CTA, 592 us here; 8 x 1024 198 and 139 us;
// 40 decoding sequences beside 2048 prompt tokens 149 and 132 us.
constexpr int kDuoThreads = 320;

template <int G>
__global__ void __launch_bounds__(kDuoThreads, 1)
pa_prefill_duo_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, PaKParams p,
                      int* status) {
    constexpr int D = 128, TOK = tile_tokens(G);
    constexpr int T_BYTES = kBM * D * 2;                        // a query, key or value tile
    constexpr uint32_t TM_S = 0, TM_O = 256;                    // + 128 for the second tile
    constexpr uint32_t IDESC_QK = umma_idesc_f16(kBM, kBK, true);
    constexpr uint32_t IDESC_PV = umma_idesc_f16(kBM, D, true) | (1u << 16);

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sQ = smem;                                         // two tiles
    uint8_t* sK = sQ + 2 * T_BYTES;                             // two stages
    uint8_t* sV = sK + 2 * T_BYTES;                             // two stages
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + 2 * T_BYTES);
    uint64_t* q_full = bars;
    uint64_t* k_full = bars + 1;               // [2 stages]
    uint64_t* v_full = bars + 3;               // [2 stages]
    uint64_t* k_empty = bars + 5;              // [2 stages] both QK products have read the stage
    uint64_t* v_empty = bars + 7;              // [2 stages] both PV products have read the stage
    uint64_t* s_full = bars + 9;               // [2 tiles] QK has retired (and with it the tile's PV product before it)
    uint64_t* p_full = bars + 11;              // [2 tiles] P written, S read
    uint64_t* pv_done = bars + 13;             // [2 tiles] PV has retired
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* s_work = const_cast<int*>(abort_flag) + 1;   // [2]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.y;
    pdl_enter_attn();
    if (threadIdx.x == 0) {
        const int bx = gridDim.x - 1 - blockIdx.x;
        int acc = 0, found = -1, tile = 0;
        for (int b = 0; b < p.B; ++b) {
            const int nt = (p.subsequence_begins[b + 1] - p.subsequence_begins[b] + 2 * TOK - 1) / (2 * TOK);
            if (bx < acc + nt) { found = b; tile = bx - acc; break; }
            acc += nt;
        }
        s_work[0] = found;
        s_work[1] = tile;
        *abort_flag = 0;
        mbar_init(q_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&k_empty[i], 1);
            mbar_init(&v_empty[i], 1);
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], kBM);
            mbar_init(&pv_done[i], 1);
        }
        mbar_fence_init();
    }
    __syncthreads();
    const int b = s_work[0];
    if (b < 0) return;                          // (uniform) nothing allocated yet
    if (warp == 9) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    const int tok_begin = p.subsequence_begins[b];
    const int q_len = p.subsequence_begins[b + 1] - tok_begin;
    const int past = p.past_lens[b];
    const int blk_begin = p.block_indices_begins[b];
    const int tq0 = s_work[1] * 2 * TOK;
    const int tq1 = min(q_len, tq0 + 2 * TOK);
    const int nq = tq0 + TOK < q_len ? 2 : 1;                   // query tiles with rows: one at the end of a sequence, or in a decoding one
    const int kv_end = p.causal ? past + tq1 : past + q_len;
    const int kv_start = first_visible_key(past + tq0, p.sliding_window, p.chunk) / kBK * kBK;
    const int ntiles = (kv_end - kv_start + kBK - 1) / kBK;

    if (warp == 8) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            mbar_arrive_expect_tx(q_full, nq * G * TOK * D * 2);
            for (int x = 0; x < nq; ++x)
                for (int g = 0; g < G; ++g)
                    for (int hf = 0; hf < 2; ++hf)
                        tma_load_2d(sQ + x * T_BYTES + hf * (kBM * 128) + g * (TOK * 128), &tmQ, q_full, (h * G + g) * p.q_head + hf * 64, tok_begin + tq0 + x * TOK);
        }
        bool ok = true;
        for (int j = 0; j < ntiles && ok; ++j) {
            const int st = j & 1;
            const int j0 = kv_start + j * kBK;
            const int npages = (min(kv_end, j0 + kBK) - j0 + kPage - 1) / kPage;
            for (int kv = 0; kv < 2 && ok; ++kv) {
                uint64_t* full = kv ? &v_full[st] : &k_full[st];
                if (j >= 2) ok = mbar_wait(kv ? &v_empty[st] : &k_empty[st], ((j >> 1) - 1) & 1, abort_flag, status);
                if (!ok) break;
                if (lane == 0) mbar_arrive_expect_tx(full, npages * kPage * D * 2);
                __syncwarp();
                if (lane < npages * 2) {                         // a lane per (half, page)
                    const int part = lane / npages, pg = lane % npages;
                    const int blk = OVB_DBG_BLOCK(p.block_indices[blk_begin + j0 / kPage + pg]);
                    tma_load_2d((kv ? sV : sK) + st * T_BYTES + part * (kBK * 128) + pg * (kPage * 128), kv ? &tmV : &tmK, full, part * 64, (blk * p.Hkv + h) * kPage);
                }
            }
        }
        __syncwarp();
    } else if (warp == 9) {
        // ------------------------------------------------------------------ MMA issuer (warp-uniform flow, one elected lane issues)
        bool ok = mbar_wait(q_full, 0, abort_flag, status);
        const uint64_t dq0 = umma_desc_k_sw128(smem_u32(sQ), 1024);
        auto qk = [&](int x, int st) {
            const uint64_t dq = dq0 + (uint64_t)((x * T_BYTES) >> 4), dk = umma_desc_k_sw128(smem_u32(sK + st * T_BYTES), 1024);
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
                const uint64_t off = (uint64_t)(((ks >> 2) * (kBM * 128) + (ks & 3) * 32) >> 4);
                umma_f16_ss_elect(tmem + TM_S + x * 128, dq + off, dk + off, IDESC_QK, ks > 0 ? 1u : 0u);
            }
            umma_commit_elect(&s_full[x]);
        };
        ok = ok && mbar_wait(&k_full[0], 0, abort_flag, status);
        if (ok) {
            tc_fence_after_sync();
            qk(0, 0);
            if (nq == 2) qk(1, 0);
            umma_commit_elect(&k_empty[0]);
        }
        for (int j = 0; j < ntiles && ok; ++j) {
            const int st = j & 1, nx = (j + 1) & 1;
            const uint32_t par = j & 1;
            const int ksteps = (min(kBK, kv_end - (kv_start + j * kBK)) + 15) / 16;
            const uint64_t dv = umma_desc_mn_sw128(smem_u32(sV + st * T_BYTES), kBK * 128, 1024);
            for (int x = 0; x < 2 && ok; ++x) {
                if (x >= nq) break;
                if (x == 0) ok = mbar_wait(&v_full[st], (j >> 1) & 1, abort_flag, status);
                ok = ok && mbar_wait(&p_full[x], par, abort_flag, status);
                if (!ok) break;
                tc_fence_after_sync();
                for (int kk = 0; kk < ksteps; ++kk)
                    umma_f16_ts_elect(tmem + TM_O + x * 128, tmem + TM_S + x * 128 + kk * 8, dv + (uint64_t)((kk * 16 * 128) >> 4), IDESC_PV, (j > 0 || kk > 0) ? 1u : 0u);
                umma_commit_elect(&pv_done[x]);
                if (x == 1 || nq == 1) umma_commit_elect(&v_empty[st]);
                if (j + 1 < ntiles) {
                    if (x == 0) ok = mbar_wait(&k_full[nx], ((j + 1) >> 1) & 1, abort_flag, status);
                    ok = ok && mbar_wait(&pv_done[x], par, abort_flag, status);     // P, which QK overwrites, has been read
                    if (!ok) break;
                    tc_fence_after_sync();
                    qk(x, nx);
                    if (x == 1 || nq == 1) umma_commit_elect(&k_empty[nx]);
                }
            }
        }
        __syncwarp();
    } else if ((warp >> 2) < nq) {
        // ------------------------------------------------------------------ softmax: one thread per stacked query row
        const int x = warp >> 2;                         // query tile of this thread
        // keys [lo_row, hi_row) from kv_start on are visible to this row, every row of the query tile sees those of [lo_last, lim). (With
        // three warps on a scheduler a thread has 168 registers: a whole row of 128 scores beside the rest of the loop's state spilled.)
        int hi_row, lo_row, lim, lo_last;
        {
            const int tl = x * TOK + (threadIdx.x & 127) % TOK, first_pos = past + tq0 + x * TOK;
            hi_row = tq0 + tl >= q_len ? 0 : p.causal ? min(kv_end, past + tq0 + tl + 1) : kv_end;
            lo_row = first_visible_key(past + tq0 + tl, p.sliding_window, p.chunk);
            lim = tq0 + (x + 1) * TOK > q_len ? 0 : p.causal ? min(kv_end, first_pos + 1) : kv_end;
            lo_last = first_visible_key(first_pos + TOK - 1, p.sliding_window, p.chunk);
            hi_row -= kv_start;
            lo_row -= kv_start;
            lim -= kv_start;
            lo_last -= kv_start;
        }
        const uint32_t tm_s = tmem + (uint32_t((warp & 3) * 32) << 16) + TM_S + x * 128;
        float m_used = -CUDART_INF_F, l_sum = 0.f;
        bool ok = true;
        for (int j = 0; j < ntiles && ok; ++j) {
            ok = mbar_wait(&s_full[x], j & 1, abort_flag, status);
            if (!ok) break;
            tc_fence_after_sync();
            const int j0 = j * kBK;
            const bool need_mask = j0 + kBK > lim || j0 < lo_last;       // (uniform over the four warps of the query tile)
            const int hi = hi_row - j0, lo = lo_row - j0;
            // the upper half of the row is read for its maximum and again for its exponentials: a whole row does not fit the registers
            uint32_t v[kBK / 2];
            float mx[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
            auto half_row = [&](int c0) {
#pragma unroll
                for (int c = 0; c < kBK / 2; c += 16) tmem_ld_x16(tm_s + c0 + c, v + c);
                tmem_ld_wait();
                if (need_mask) {
#pragma unroll
                    for (int i = 0; i < kBK / 2; ++i)
                        if (!(c0 + i >= lo && c0 + i < hi)) v[i] = __float_as_uint(-CUDART_INF_F);
                }
            };
            half_row(kBK / 2);
#pragma unroll
            for (int i = 0; i < kBK / 2; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(v[i]));
            half_row(0);
#pragma unroll
            for (int i = 0; i < kBK / 2; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(v[i]));
            const float m_tile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2;
            // raise the running maximum only when the tile exceeds it by a factor of 2^8; the rescale of O is warp-collective.
            // (S of this tile is there, so the PV product of the tile before has retired and O may be touched.)
            const bool raise = m_tile > m_used + 8.f;
            if (__any_sync(0xffffffffu, raise)) {
                const float factor = !raise ? 1.f : (m_used == -CUDART_INF_F ? 0.f : fast_exp2(m_used - m_tile));
                if (j > 0) {
#pragma unroll 1
                    for (int c = 0; c < D; c += 8) {             // (eight columns at a time: the row of S is in registers)
                        uint32_t o[8];
                        tmem_ld_x8(tm_s + (TM_O - TM_S) + c, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 8; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
                        tmem_st_x8(tm_s + (TM_O - TM_S) + c, o);
                    }
                    tmem_st_wait();
                }
                if (raise) {
                    l_sum *= factor;
                    m_used = m_tile;
                }
            }
            const float neg_m = (m_used == -CUDART_INF_F) ? 0.f : -m_used;
            float ls[4] = {0.f, 0.f, 0.f, 0.f};
            auto half_p = [&](int c0) {                  // P takes half the columns of S: those of the lower half first
#pragma unroll
                for (int c = 0; c < kBK / 4; c += 16) {
                    uint32_t pk[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float e0 = fast_exp2(fmaf(__uint_as_float(v[2 * (c + i)]), p.scale_log2, neg_m));
                        const float e1 = fast_exp2(fmaf(__uint_as_float(v[2 * (c + i) + 1]), p.scale_log2, neg_m));
                        ls[i & 3] += e0 + e1;
                        pk[i] = pack16<false>(e0, e1);
                    }
                    tmem_st_x16(tm_s + c0 + c, pk);
                }
            };
            half_p(0);
            half_row(kBK / 2);
            half_p(kBK / 4);
            l_sum += (ls[0] + ls[1]) + (ls[2] + ls[3]);
            tmem_st_wait();
            tc_fence_before_sync();
            mbar_arrive(&p_full[x]);
        }
        if (ok && ntiles > 0) ok = mbar_wait(&pv_done[x], (ntiles - 1) & 1, abort_flag, status);
        if (ok) {
            tc_fence_after_sync();
            const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
            uint32_t tid;                                // all of this is read again: nothing of it is kept through the loop
            asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
            const int b2 = *reinterpret_cast<volatile int*>(s_work), tq = *reinterpret_cast<volatile int*>(s_work + 1) * 2 * TOK;
            const int begin = __ldg(p.subsequence_begins + b2), len = __ldg(p.subsequence_begins + b2 + 1) - begin;
            const int r = tid & 127, g = r / TOK, tl = (int)(tid >> 7) * TOK + r % TOK;
            const bool row_valid = tq + tl < len;
            uint8_t* dst = reinterpret_cast<uint8_t*>(p.out) + ((size_t)(begin + tq + tl) * p.ldo + (size_t)((int)blockIdx.y * G + g) * p.o_head) * 2;
#pragma unroll
            for (int c = 0; c < D; c += 16) {
                uint32_t o[16];
                tmem_ld_x16(tm_s + (TM_O - TM_S) + c, o);
                tmem_ld_wait();
                if (row_valid) {
                    uint32_t w[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) w[i] = pack16<false>(__uint_as_float(o[2 * i]) * inv, __uint_as_float(o[2 * i + 1]) * inv);
                    *reinterpret_cast<uint4*>(dst + c * 2) = make_uint4(w[0], w[1], w[2], w[3]);
                    *reinterpret_cast<uint4*>(dst + c * 2 + 16) = make_uint4(w[4], w[5], w[6], w[7]);
                }
            }
        }
    }

    // ---------------------------------------------------------------- tear-down
    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);   // copies still in flight land before the shared memory is reused
        __syncthreads();
    }
    if (warp == 9) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, 512);
    }
}

template <int G>
int launch_duo(PaKParams p, int num_q_tiles, cudaStream_t stream) {
    p.q_head = p.o_head = p.dv_store = p.k_row = p.v_row = 128;
    p.ldo = p.Hq * 128;
    const int smem = 6 * kBM * 256 + 256 + 1024;
    auto kern = pa_prefill_duo_kernel<G>;
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    OVB_CHECK_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        OVB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured.fetch_or(bit, std::memory_order_release);
    }
    const CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const uint64_t rows = p.cache_rows > 0 ? (uint64_t)p.cache_rows : 1ull << 30;
    CUtensorMap tmQ, tmK, tmV;
    if (int rc = make_tmap_2d(&tmQ, p.q, dt, 2, (uint64_t)p.T, (uint64_t)p.ldq, (uint64_t)p.ldq * 2, tile_tokens(G), 64, true)) return rc;
    if (int rc = make_tmap_2d(&tmK, p.k_cache, dt, 2, rows, 128, 256, kPage, 64, true)) return rc;
    if (int rc = make_tmap_2d(&tmV, p.v_cache, dt, 2, rows, 128, 256, kPage, 64, true)) return rc;
    // a sequence of n single tiles has (n + 1) / 2 of these
    OVB_CHECK_CUDA(launch_pdl(kern, dim3((num_q_tiles + p.B + 1) / 2, p.Hkv), dim3(kDuoThreads), (size_t)smem, stream, tmQ, tmK, tmV, p, status_word()));
    return 0;
}

constexpr int kMaxBiasedKeys = 8192;

template <int KH, int RH, int VH, int G, int SRC, bool F16, bool BIAS = false, bool TWO = false>
int launch_tc_parts(const PaKParams& p, int num_q_tiles, cudaStream_t stream) {
    const int TOK = tile_tokens(G > 0 ? G : p.group);
    constexpr int plain = kBM * (KH + RH) * 128 + 2 * kBK * (KH + RH + VH) * 128 + 256 + 1024;
    const int smem = plain + (BIAS ? ceil_div(p.dense_S, kBK) * kBK * 4 : 0);
    auto kern = pa_prefill_tc_kernel<KH, RH, VH, G, SRC, F16, BIAS, TWO>;
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    OVB_CHECK_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        OVB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, plain + (BIAS ? kMaxBiasedKeys * 4 : 0)));
        configured.fetch_or(bit, std::memory_order_release);
    }
    const CUtensorMapDataType dt = F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    CUtensorMap tmQ, tmK, tmV, tmR;
    // Q rows are tokens; a box is the TOK tokens of a tile x 64 columns of one head (rows past T read as zeros)
    if (int rc = make_tmap_2d(&tmQ, p.q, dt, 2, (uint64_t)p.T, (uint64_t)p.ldq, (uint64_t)p.ldq * 2, TOK, 64, true)) return rc;
    if (SRC == SRC_PAGED) {
        // the cache seen as rows of one head: row = (block * Hkv + head) * 16 + slot
        const uint64_t rows = p.cache_rows > 0 ? (uint64_t)p.cache_rows : 1ull << 30;
        if (int rc = make_tmap_2d(&tmK, p.k_cache, dt, 2, rows, p.k_row, (uint64_t)p.k_row * 2, kPage, 64, true)) return rc;
        if (int rc = make_tmap_2d(&tmV, p.v_cache, dt, 2, rows, p.v_row, (uint64_t)p.v_row * 2, kPage, 64, true)) return rc;
    } else if (SRC == SRC_LATENT) {
        // pages of 16 rows that reach past a sequence's last key read the next sequence's rows (masked) or zeros behind the last
        const uint64_t rows = p.cache_rows > 0 ? (uint64_t)p.cache_rows : 1ull << 30;
        if (int rc = make_tmap_2d(&tmK, p.k_cache, dt, 2, (uint64_t)p.kv_total, (uint64_t)p.Hkv * p.k_head, (uint64_t)p.kv_ld * 2, kPage, 64, true)) return rc;
        if (int rc = make_tmap_2d(&tmV, p.v_cache, dt, 2, (uint64_t)p.kv_total, (uint64_t)p.Hkv * p.v_head, (uint64_t)p.kv_ld * 2, kPage, 64, true)) return rc;
        if (int rc = make_tmap_2d(&tmR, p.shared, dt, 2, rows, p.shared_row, (uint64_t)p.shared_row * 2, kPage, 64, true)) return rc;
    } else {
        const uint64_t rows = (uint64_t)p.B * p.dense_S;
        if (int rc = make_tmap_2d(&tmK, p.k_cache, dt, 2, rows, (uint64_t)p.ld_kv, (uint64_t)p.ld_kv * 2, kPage, 64, true)) return rc;
        if (int rc = make_tmap_2d(&tmV, p.v_cache, dt, 2, rows, (uint64_t)p.ld_kv, (uint64_t)p.ld_kv * 2, kPage, 64, true)) return rc;
    }
    if (SRC != SRC_LATENT) tmR = tmK;      // unused
    OVB_CHECK_CUDA(launch_pdl(kern, dim3(num_q_tiles, p.Hkv), dim3(192), (size_t)smem, stream, tmQ, tmK, tmV, tmR, p, status_word()));
    return 0;
}

// Heads of one size D packed without gaps.
void pack_heads(PaKParams* p, int D) {
    p->q_head = p->o_head = p->dv_store = p->k_row = p->v_row = p->k_head = p->v_head = D;
    p->ldo = p->Hq * D;
}

template <int D, int G>
int launch_tc(PaKParams p, int num_q_tiles, cudaStream_t stream) {
    pack_heads(&p, D);
    return launch_tc_parts<D / 64, 0, D / 64, G, SRC_PAGED, false>(p, num_q_tiles, stream);
}

// Two CTAs to an SM where there are more CTAs than SMs (heads of 64, fp16, us with one / with two: 16 x 384 tokens, 16 heads, with a mask 49 / 36); a
// CTA that has its SM to itself is faster with S and P twice (1 x 1024, 16 heads 14.6 / 18.0; 4 x 200, 12 heads 7.7 / 8.8; 1 x 40 5.4 / 6.0).
template <int D, bool F16>
int launch_dense(PaKParams p, int num_q_tiles, cudaStream_t stream) {
    pack_heads(&p, D);
    constexpr int P = D / 64;
    if constexpr (D == 64) {
        if (num_q_tiles * p.Hkv > 148)
            return p.key_bias != nullptr ? launch_tc_parts<P, 0, P, 1, SRC_DENSE, F16, true, true>(p, num_q_tiles, stream)
                                         : launch_tc_parts<P, 0, P, 1, SRC_DENSE, F16, false, true>(p, num_q_tiles, stream);
    }
    return p.key_bias != nullptr ? launch_tc_parts<P, 0, P, 1, SRC_DENSE, F16, true>(p, num_q_tiles, stream)
                                 : launch_tc_parts<P, 0, P, 1, SRC_DENSE, F16>(p, num_q_tiles, stream);
}

}  // namespace

// Two tiles to a CTA once single tiles would fill the machine twice (fewer are better spread over the SMs), and where the tokens make up
// as many full tiles as there are sequences. A sequence with one tile gains nothing from the second and takes about 15 % longer in that
// kernel, a pair of tiles 30 % less. One tile / two (us, cold, 32 and 8 heads, decoding sequences behind 1000 to 1300 tokens): 48 decoding +
// a portion of 16 tokens 89 / 103, 40 + 512 85 / 93, 40 + 1024 112 / 112, 47 + 2 x 1024 138 / 134, 40 + 2048 149 / 132; 64 x 20 108 / 120,
// 40 x 33 44 / 36.
bool two_query_tiles(int T, int B, int G, int Hkv) {
    const int tok = tile_tokens(G);
    return (int64_t)(T / tok + B) * Hkv >= 2 * 148 && T - B >= (int64_t)B * tok;
}

int launch_prefill_tc(const PaKParams& p, int D, int G, bool paged, bool f16, int num_q_tiles, cudaStream_t stream) {
    if (paged && p.block_size != kPage) return ERR_UNSUPPORTED;
    if (p.key_bias != nullptr && (paged || p.dense_S > kMaxBiasedKeys)) return ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(p.q) & 15) || (reinterpret_cast<uintptr_t>(p.k_cache) & 15) || (reinterpret_cast<uintptr_t>(p.v_cache) & 15) ||
        (reinterpret_cast<uintptr_t>(p.out) & 15) || p.ldq % 8 != 0 || (!paged && p.ld_kv % 8 != 0))
        return ERR_UNSUPPORTED;
    if (paged && !f16) {
        if (D == 128 && p.gate == nullptr && p.sink == nullptr && two_query_tiles(p.T, p.B, G, p.Hkv)) {
            switch (G) {
                case 1: return launch_duo<1>(p, num_q_tiles, stream);
                case 2: return launch_duo<2>(p, num_q_tiles, stream);
                case 4: return launch_duo<4>(p, num_q_tiles, stream);
                case 8: return launch_duo<8>(p, num_q_tiles, stream);
            }
        }
        if (D == 128) {
            switch (G) {
                case 1: return launch_tc<128, 1>(p, num_q_tiles, stream);
                case 2: return launch_tc<128, 2>(p, num_q_tiles, stream);
                case 4: return launch_tc<128, 4>(p, num_q_tiles, stream);
                case 8: return launch_tc<128, 8>(p, num_q_tiles, stream);
            }
        } else if (D == 64) {
            switch (G) {
                case 1: return launch_tc<64, 1>(p, num_q_tiles, stream);
                case 4: return launch_tc<64, 4>(p, num_q_tiles, stream);
            }
        }
    } else if (!paged && G == 1) {
        if (D == 64) return f16 ? launch_dense<64, true>(p, num_q_tiles, stream) : launch_dense<64, false>(p, num_q_tiles, stream);
        if (D == 128) return f16 ? launch_dense<128, true>(p, num_q_tiles, stream) : launch_dense<128, false>(p, num_q_tiles, stream);
    }
    return ERR_UNSUPPORTED;
}

int launch_window_tc(PaKParams p, int dk, int dshared, int dv, cudaStream_t stream) {
    const int kh = ceil_div(dk, 64), rh = ceil_div(dshared, 64), vh = ceil_div(dv, 64);
    if (p.block_size != kPage || p.group < 1 || p.group > 16 || kh + rh > 3 || rh > 1 || vh > 2) return ERR_UNSUPPORTED;
    auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    if (!aligned(p.q) || !aligned(p.k_cache) || !aligned(p.v_cache) || !aligned(p.out) || !aligned(p.shared)) return ERR_UNSUPPORTED;
    if (!p.gate_scalar && (!aligned(p.gate) || p.ld_gate % 8 || p.gate_head % 8)) return ERR_UNSUPPORTED;
    if (p.ldq % 8 || p.q_head % 8 || p.ldo % 8 || p.o_head % 8 || dv % 16 || p.k_row % 8 || p.v_row % 8) return ERR_UNSUPPORTED;
    p.dv_store = dv;
    const int tiles = p.T / tile_tokens(p.group) + p.B;      // upper bound of the tiles of all sequences
    if (rh > 0) {
        if (kh == 1) return vh == 1 ? launch_tc_parts<1, 1, 1, 1, SRC_LATENT, false>(p, tiles, stream) : launch_tc_parts<1, 1, 2, 1, SRC_LATENT, false>(p, tiles, stream);
        return vh == 1 ? launch_tc_parts<2, 1, 1, 1, SRC_LATENT, false>(p, tiles, stream) : launch_tc_parts<2, 1, 2, 1, SRC_LATENT, false>(p, tiles, stream);
    }
    switch (kh * 2 + vh) {
        case 3: return launch_tc_parts<1, 0, 1, 0, SRC_PAGED, false>(p, tiles, stream);
        case 4: return launch_tc_parts<1, 0, 2, 0, SRC_PAGED, false>(p, tiles, stream);
        case 5: return launch_tc_parts<2, 0, 1, 0, SRC_PAGED, false>(p, tiles, stream);
        case 6: return launch_tc_parts<2, 0, 2, 0, SRC_PAGED, false>(p, tiles, stream);
        case 7: return launch_tc_parts<3, 0, 1, 0, SRC_PAGED, false>(p, tiles, stream);
        case 8: return launch_tc_parts<3, 0, 2, 0, SRC_PAGED, false>(p, tiles, stream);
    }
    return ERR_UNSUPPORTED;
}

}  // namespace ovb

#ifdef OVB_DEBUG_BOUNDS
extern "C" int ovb_debug_set_limits_attention_tc(const ovb::DebugLimits* l) {
    OVB_CHECK_CUDA(cudaMemcpyToSymbol(ovb::g_dbg_limits, l, sizeof(*l)));
    return 0;
}
#endif
