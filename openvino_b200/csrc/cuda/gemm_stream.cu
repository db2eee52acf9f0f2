// Products of few tokens: out[T, N] = epilogue(X[T, K] * dequant(W[N, K])^T), bound by the read of the weights and by the launch.
//
// The path of gemm_sm100.cu takes every weight through shared memory, the expansion warps, tensor memory and a chain of barriers;
// with a handful of tokens that chain and the set-up of a launch (5 to 6 us for the smallest product), not HBM, set the pace. Here a
// lane reads the 16-byte pieces of its weight rows straight into registers, expands them there into the A fragments of mma.sync
// (16 x 8 x 16) and multiplies: no barrier inside a tile, no tensor map, no tensor memory. At these token counts the legacy tensor
// pipe has the rate that HBM asks for.
//  * A CTA owns 32 weight rows at a time (two m16 fragments; for a gated MLP 16 gate rows and the 16 up rows of the same channels),
//    its eight warps share K: warp w takes the units w, w + 8, ... of 128 (16-bit: 64) columns. The sums meet in shared memory.
//  * K columns are permuted inside a unit so that a lane's fragment elements are 16 consecutive bytes of a row, for the weights and
//    for the tokens alike; eight lanes read a whole 128-byte line.
//  * The group's scale is applied to the fp32 sums of a unit. The weights enter the products as exact small integers, so nothing is
//    rounded before the fp32 sums (the other kernel rounds every weight to bf16).
//  * Every warp stages the tokens of its own units (cp.async, fragment order: conflict-free 16-byte reads).
//  * The loop over (tile, unit) is flat: weight loads run ahead, also across tiles and before the wait for the kernel that writes
//    the tokens.
//  * Few tiles: a cluster of 2, 4 or 8 CTAs shares K, partial sums are read through distributed shared memory in rank order.
// What bounds it: the latency of its loads, with 16 warps on an SM and issue slots half used (128256 x 4096 u4 74 us, 4 TB/s). u4 weights of at
// least 8 M values go to gemm_ring.cu, which streams them through shared memory (60 us), and here stay the small ones, where the launch counts: a
// step of one token through a two-layer model of 256 channels takes 82 us without this kernel, 46 with it, 37 with the norms inside its products.
#include <mutex>

#include "gemm_common.cuh"
#include "mma_sync.cuh"

namespace ovb {

constexpr int kStreamThreads = 256;
constexpr int kStreamWarps = 8;
constexpr int kStreamNormTokens = 4;     // rows that a norm inside the product takes, of up to 2048 columns

struct StreamParams {
    const uint8_t* w;
    const uint8_t* x;
    const uint32_t* sz;
    void* out;
    const void* bias;
    const void* residual;
    int T, N, K;
    int ldx, ldo, ldr;
    int kb_stride;                      // chunks between weight tiles (tile-packed forms)
    int kpg;                            // units per scale group
    int units, units_per_split;
    int act, out_f32;
    float act_limit, act_slope, act_shift;
    const void* x_norm;
    const int* x_rows;
    float x_eps;
    int x_count;
};

constexpr int stream_unit(int wmode) { return wmode == OVB_W_BF16 ? 64 : 128; }      // columns of K in a unit

// Eight weights of a row -> four pairs: (q - z) / 64 exactly (see RowScale), fp8 values, or 16-bit weights as they are.
template <int WMODE>
__device__ __forceinline__ void stream_expand(const uint4* q, int s, uint32_t m, uint32_t p[4]) {
    auto whole = [&](uint32_t bits, uint32_t mul) {
        const __nv_bfloat162 v = __hfma2(*reinterpret_cast<__nv_bfloat162*>(&bits), *reinterpret_cast<__nv_bfloat162*>(&mul), *reinterpret_cast<__nv_bfloat162*>(&m));
        return *reinterpret_cast<const uint32_t*>(&v);
    };
    if (WMODE == OVB_W_U4) {
        const uint32_t w = s == 0 ? q[0].x : s == 1 ? q[0].y : s == 2 ? q[0].z : q[0].w, y = w >> 8;
        p[0] = whole(w & 0x000F000Fu, kTwo127);
        p[1] = whole(w & 0x00F000F0u, kTwo123);
        p[2] = whole(y & 0x000F000Fu, kTwo127);
        p[3] = whole(y & 0x00F000F0u, kTwo123);
    } else if (WMODE == OVB_W_BF16) {
        p[0] = q[s].x; p[1] = q[s].y; p[2] = q[s].z; p[3] = q[s].w;
    } else {
        const uint4 v = q[s >> 1];
        const uint32_t w0 = (s & 1) ? v.z : v.x, w1 = (s & 1) ? v.w : v.y;
        if (WMODE == OVB_W_F8) {
            const __nv_bfloat162 up = __halves2bfloat162(__ushort_as_bfloat16(0x7B80), __ushort_as_bfloat16(0x7B80));    // 2^120: the e4m3 value, exact
            dequant_f8x4(w0, up, p[0], p[1]);
            dequant_f8x4(w1, up, p[2], p[3]);
        } else {
            p[0] = whole(__byte_perm(w0, 0u, 0x4140), kTwo127);
            p[1] = whole(__byte_perm(w0, 0u, 0x4342), kTwo127);
            p[2] = whole(__byte_perm(w1, 0u, 0x4140), kTwo127);
            p[3] = whole(__byte_perm(w1, 0u, 0x4342), kTwo127);
        }
    }
}

template <int WMODE, bool F16>
__global__ void __launch_bounds__(kStreamThreads, 2) gemm_stream_kernel(const StreamParams p) {
    using E = typename Elem<F16>::type;
    constexpr bool QUANT = WMODE != OVB_W_BF16;
    constexpr int KU = stream_unit(WMODE), SP = KU / 32;          // SP: 8-column pieces that a lane holds of a row
    constexpr int LD = WMODE == OVB_W_U4 ? 1 : 2;                 // 16-byte loads of a lane per row and unit
    constexpr int DEPTH = WMODE == OVB_W_U4 ? 3 : 2;              // units in flight per warp
    constexpr int TP = 8, PITCH = 36;                             // tokens; floats between tokens of a warp's sums: no bank conflicts
    constexpr int RED = kStreamWarps * TP * PITCH;
    extern __shared__ __align__(16) uint8_t smem[];
    float* red = reinterpret_cast<float*>(smem);                  // [2][warp][token][row]: one tile is read while the next is written
    uint8_t* xs = reinterpret_cast<uint8_t*>(red + 2 * RED);      // [unit][piece][token][quad lane] of 16 bytes
    const int u_per = p.units_per_split;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    unsigned csize, crank;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
    const bool gated = p.act == OVB_ACT_SWIGLU || p.act == OVB_ACT_GLU_LIMITED;
    const int tiles = p.N / 32, first = (int)(blockIdx.x / csize), step = (int)(gridDim.x / csize);
    const int u0 = (int)crank * u_per, nu_all = max(0, min(p.units - u0, u_per));
    const int nu = (nu_all - warp + kStreamWarps - 1) / kStreamWarps;    // units of this warp: warp, warp + 8, ...
    const int my_tiles = first < tiles ? (tiles - first + step - 1) / step : 0;

    // weights of one unit: rows g, g + 8 of both fragments
    struct Unit {
        uint4 q[4][LD];
        uint32_t sz[4];
    };
    // The next unit to request: one address per lane, moved by constants; the second fragment lies `frag_rows` rows behind the first.
    const int frag_rows = gated ? 64 : 16;
    const uint8_t* src = nullptr;
    const uint32_t* src_sz = nullptr;
    int ld_tile = first, ld_u = 0, ld_left = my_tiles * max(nu, 0);
    auto seek = [&]() {                                                  // the first unit of tile ld_tile
        const int tile128 = ld_tile >> 2, r = (ld_tile & 3) * (gated ? 16 : 32) + g, u = u0 + warp;
        if (WMODE == OVB_W_U4) {
            const uint8_t* c = p.w + ((size_t)tile128 * p.kb_stride + 2 * u) * 4608;
            src = c + (t >> 1) * 4608 + (t & 1) * 2048 + r * 16;
            src_sz = reinterpret_cast<const uint32_t*>(c + 4096) + r;
        } else if (WMODE == OVB_W_BF16) {
            src = p.w + ((size_t)tile128 * p.kb_stride + u) * 16384 + r * 128;
        } else {
            src = p.w + (size_t)(tile128 * TILE_N + r) * p.K + (size_t)u * KU + t * (KU / 4);
            src_sz = p.sz + tile128 * TILE_N + r;
        }
    };
    auto request = [&](Unit& b) {
        if (ld_left <= 0) return;
        --ld_left;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int dr = (i < 2 ? 0 : frag_rows) + (i & 1) * 8;
            if (WMODE == OVB_W_U4) {
                b.q[i][0] = __ldg(reinterpret_cast<const uint4*>(src + dr * 16));
                b.sz[i] = __ldg(src_sz + dr);
            } else if (WMODE == OVB_W_BF16) {                            // 16-byte pieces 2t, 2t + 1 in the swizzled row (8 rows on: the same swizzle)
#pragma unroll
                for (int j = 0; j < LD; ++j) b.q[i][j] = __ldg(reinterpret_cast<const uint4*>(src + dr * 128 + ((2 * t + j) ^ g) * 16));
            } else {
#pragma unroll
                for (int j = 0; j < LD; ++j) b.q[i][j] = __ldg(reinterpret_cast<const uint4*>(src + (size_t)dr * p.K + j * 16));
                b.sz[i] = __ldg(src_sz + (size_t)((u0 + warp + ld_u * kStreamWarps) / p.kpg) * p.N + dr);
            }
        }
        if (++ld_u == nu) {
            ld_u = 0;
            ld_tile += step;
            if (ld_left > 0) seek();
        } else if (WMODE == OVB_W_U4) {
            src += kStreamWarps * 2 * 4608;
            src_sz += kStreamWarps * 2 * 4608 / 4;
        } else {
            src += kStreamWarps * (WMODE == OVB_W_BF16 ? 16384 : KU);
        }
    };
    Unit buf[DEPTH];
    if (ld_left > 0) seek();
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) request(buf[d]);            // weights are constants: before the wait

    pdl_wait();
    // the tokens of this warp's units: consecutive lanes copy consecutive 16-byte pieces of a token row
    constexpr int PPU = KU / 8;                                  // pieces of a unit
    if (!F16 && p.x_norm != nullptr) {
        __shared__ float squares[kStreamWarps][kStreamNormTokens];
        norm_rows<kStreamThreads, kStreamNormTokens, 1>(p, squares, [&](int n, int k8, uint4 v) {
            const int lu = k8 / PPU - u0, r = k8 % PPU;
            if (lu >= 0 && lu < nu_all) *reinterpret_cast<uint4*>(xs + ((size_t)((lu * SP + r % SP) * p.T + n) * 4 + r / SP) * 16) = v;
        });
        __syncthreads();
    } else
    for (int i = 0; i < nu; ++i) {
        const int lu = warp + i * kStreamWarps;
        for (int j = lane; j < p.T * PPU; j += 32) {
            const int n = j / PPU, r = j % PPU;
            cp_async16(xs + ((size_t)((lu * SP + r % SP) * p.T + n) * 4 + r / SP) * 16,
                       p.x + ((size_t)n * p.ldx + (size_t)(u0 + lu) * KU + r * 8) * 2, true);
        }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();

    float acc[2][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][e] = 0.f;

    // the sums of a finished tile: over the warps, over the cluster, then the epilogue
    int turn = 0;
    auto finish = [&](int tile) {
        float* mine = red + turn * RED + warp * TP * PITCH;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                mine[(2 * t + (e & 1)) * PITCH + m * 16 + (e >> 1) * 8 + g] = acc[m][e];
                acc[m][e] = 0.f;
            }
        if (csize > 1) {
            cluster_arrive();
            cluster_wait();
        } else {
            __syncthreads();
        }
        const float* all = red + turn * RED;
        const int sh = gated ? 4 : 5;                             // log2 of the outputs of a token
        const int total = p.T << sh;
        for (int e = (int)threadIdx.x + (int)crank * kStreamThreads; e < total; e += kStreamThreads * (int)csize) {
            const int tok = e >> sh, r = e & ((1 << sh) - 1);
            float v = 0.f, u = 0.f;
            if (csize == 1) {
#pragma unroll
                for (int k = 0; k < kStreamWarps; ++k) {
                    v += all[(k * TP + tok) * PITCH + r];
                    if (gated) u += all[(k * TP + tok) * PITCH + 16 + r];
                }
            } else {
#pragma unroll 2
                for (unsigned z = 0; z < csize; ++z) {
                    const uint32_t a = dsmem_addr(smem_u32(all + tok * PITCH + r), z);
#pragma unroll
                    for (int k = 0; k < kStreamWarps; ++k) {
                        float f;
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f) : "r"(a + k * TP * PITCH * 4) : "memory");
                        v += f;
                        if (gated) {
                            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f) : "r"(a + (k * TP * PITCH + 16) * 4) : "memory");
                            u += f;
                        }
                    }
                }
            }
            if (gated) {
                v = p.act == OVB_ACT_SWIGLU ? v / (1.0f + __expf(-v)) * u : glu_limited(p, v, u);
                reinterpret_cast<E*>(p.out)[(size_t)tok * p.ldo + (tile >> 2) * 64 + (tile & 3) * 16 + r] = from_float<E>(v);
            } else {
                const int oc = tile * 32 + r;
                if (p.bias) v += to_float(reinterpret_cast<const E*>(p.bias)[oc]);
                v = apply_act(v, p);
                if (p.residual) v += to_float(reinterpret_cast<const E*>(p.residual)[(size_t)tok * p.ldr + oc]);
                if (p.out_f32) reinterpret_cast<float*>(p.out)[(size_t)tok * p.ldo + oc] = v;
                else reinterpret_cast<E*>(p.out)[(size_t)tok * p.ldo + oc] = from_float<E>(v);
            }
        }
        turn ^= 1;
    };

    if (nu <= 0) {                                                // fewer units than warps: this one only takes part in the sums
        for (int j = 0; j < my_tiles; ++j) finish(first + j * step);
    } else {
        int tile = first, u = 0;
        const int total = my_tiles * nu;
        for (int it = 0; it < total; it += DEPTH) {
#pragma unroll
            for (int d = 0; d < DEPTH; ++d) {
                if (it + d < total) {
                    const int lu = warp + u * kStreamWarps;
                    float part[2][4];
                    uint32_t minus[4];                           // -z / 64 of the four rows, as pairs
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        minus[i] = 0u;
                        if (WMODE == OVB_W_U4 || WMODE == OVB_W_U8) {
                            const RowScale rs = row_scale(*reinterpret_cast<const __nv_bfloat162*>(&buf[d].sz[i]), WMODE == OVB_W_U4 ? 16.f : 0.f);
                            minus[i] = *reinterpret_cast<const uint32_t*>(&rs.m);
                        }
                    }
#pragma unroll
                    for (int m = 0; m < 2; ++m)
#pragma unroll
                        for (int e = 0; e < 4; ++e) part[m][e] = QUANT ? 0.f : acc[m][e];
#pragma unroll
                    for (int s = 0; s < SP; ++s) {
                        uint4 xb = make_uint4(0, 0, 0, 0);
                        if (g < p.T) xb = *reinterpret_cast<const uint4*>(xs + ((size_t)((lu * SP + s) * p.T + g) * 4 + t) * 16);
#pragma unroll
                        for (int m = 0; m < 2; ++m) {
                            uint32_t lo[4], hi[4];
                            stream_expand<WMODE>(buf[d].q[2 * m], s, minus[2 * m], lo);
                            stream_expand<WMODE>(buf[d].q[2 * m + 1], s, minus[2 * m + 1], hi);
                            const uint32_t a0[4] = {lo[0], hi[0], lo[1], hi[1]}, a1[4] = {lo[2], hi[2], lo[3], hi[3]};
                            mma16816<F16>(part[m], a0, xb.x, xb.y);
                            mma16816<F16>(part[m], a1, xb.z, xb.w);
                        }
                    }
#pragma unroll
                    for (int m = 0; m < 2; ++m)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            // the scale with the 64 of the expansion; fp8: the table's scales carry 2^120
                            const float sc = __uint_as_float(buf[d].sz[2 * m + (e >> 1)] << 16) * (WMODE == OVB_W_F8 ? 7.52316384526264e-37f : 64.f);
                            acc[m][e] = QUANT ? acc[m][e] + sc * part[m][e] : part[m][e];
                        }
                    request(buf[d]);
                    if (++u == nu) {
                        u = 0;
                        if (it + d + 1 == total && OVB_PDL_GEMM) pdl_trigger();
                        finish(tile);
                        tile += step;
                    }
                }
            }
        }
    }
    if (csize > 1) {        // a peer may still read this CTA's sums
        cluster_arrive();
        cluster_wait();
    }
}

// --------------------------------------------------------------------------------------------- host
constexpr int kStreamSmem = 112 * 1024;         // two CTAs on an SM

static int stream_smem(int wmode, int T, int units_per_split) { return 2 * kStreamWarps * 8 * 36 * 4 + units_per_split * stream_unit(wmode) * T * 2; }

// CTAs that share K. Time of a candidate: tiles that a cluster works off one after another, each as long as its bytes take at this
// CTA's part of 6 TB/s, or as long as its loads wait (0.8 us a round); a cluster barrier costs about 1 us. Clusters of four and eight take one
// tile each: their CTAs wait for the slowest at every tile (8192 x 28672 u4, four tokens, whose rows only fit shared memory by such
// clusters: 100 us, gemm_sm100.cu 59 us). 0: no split serves the problem well.
static int pick_stream_split(int wmode, int T, int N, int units, int* smem_bytes) {
    const double unit_us = 32.0 * stream_unit(wmode) * (wmode == OVB_W_U4 ? 0.5625 : wmode == OVB_W_BF16 ? 2.0 : 1.03) * 296 / 6.0e6;
    int best = 0;
    double best_t = 1e30;
    for (int s = 1; s <= 8; s *= 2) {
        if (s > 1 && units < 2 * s) break;
        const int per = ceil_div(units, s), smem = stream_smem(wmode, T, per);
        if (smem > kStreamSmem) continue;
        const int jobs = ceil_div(N / 32, 296 / s);
        if (s > 2 && jobs > 1) continue;
        const double bytes_us = per * unit_us, wait_us = 0.8 * ceil_div(per, kStreamWarps * 2);
        const double t = jobs * ((bytes_us > wait_us ? bytes_us : wait_us) + (s > 1 ? 1.0 : 0.3)) + per * T * 0.0006;
        if (t < best_t) { best_t = t; best = s; *smem_bytes = smem; }
    }
    return best;
}

// (u4 weights that gemm_ring.cu takes are asked for there first.)
// Where it is the faster one, cold weights, against gemm_sm100.cu (us): u4 128256 x 4096 T = 1 74 / 84, T = 8 82 / 84; 4096 x 14336 T = 1
// 14 / 20, T = 4 20 / 20, T = 8 22 / 20: up to four tokens. Bytes cost a lane twice the loads for the same weights: u8 128256 x 4096 T = 1
// 119 / 103, fp8 4096 x 14336 22 / 21, but 4096 x 4096 9 / 17, where the launch counts: up to 32 MB. 16-bit: likewise, up to 16 MB
// (14 MB 4 / 6; 33 MB 10 / 10; 50 MB 20 / 12), any eight tokens.
constexpr int kStreamMaxTokens16 = 8, kStreamMaxTokensQuant = 4;
constexpr int64_t kStreamMaxBytes16 = 16ll << 20, kStreamMaxBytes8 = 32ll << 20;

bool gemm_stream_takes(const ovb_gemm_args* a) {
    const bool swiglu = a->act == OVB_ACT_SWIGLU || a->act == OVB_ACT_GLU_LIMITED;
    if (a->T > (is_quant(a->wmode) ? kStreamMaxTokensQuant : kStreamMaxTokens16) || a->comm != nullptr || a->group_offsets != nullptr || a->group_mode == 3 || a->block_t != 0 || a->splits > 1) return false;
    if (a->N % (swiglu ? 128 : 32) != 0 || (reinterpret_cast<uintptr_t>(a->x) & 15) != 0 || (reinterpret_cast<uintptr_t>(a->w) & 15) != 0) return false;
    if (is_quant(a->wmode)) {
        if (a->K % 128 != 0 || a->group_size % 128 != 0 || a->w_kb_stride != 0) return false;
        if (a->wmode != OVB_W_U4 && (int64_t)a->N * a->K > kStreamMaxBytes8) return false;
    } else if (!a->w_tiled || a->K % 64 != 0 || (int64_t)a->N * a->K * 2 > kStreamMaxBytes16) {
        return false;
    }
    const int wm = a->wmode == OVB_W_F16 ? OVB_W_BF16 : a->wmode;
    int smem = 0;
    return pick_stream_split(wm, a->T, a->N, a->K / stream_unit(wm), &smem) > 0;
}

bool gemm_stream_norms(const ovb_gemm_args* a) { return a->wmode != OVB_W_F16 && a->T <= kStreamNormTokens && a->K <= kStreamThreads * 8; }

template <int WMODE, bool F16>
static int run_stream(const ovb_gemm_args* a, cudaStream_t stream) {
    const bool swiglu = a->act == OVB_ACT_SWIGLU || a->act == OVB_ACT_GLU_LIMITED;
    StreamParams p;
    memset(&p, 0, sizeof(p));
    p.w = static_cast<const uint8_t*>(a->w);
    p.x = static_cast<const uint8_t*>(a->x);
    p.sz = static_cast<const uint32_t*>(a->scales);
    p.out = a->out;
    p.bias = a->bias;
    p.residual = a->residual;
    p.T = a->T;
    p.N = a->N;
    p.K = a->K;
    p.ldx = a->ldx ? a->ldx : a->K;
    p.ldo = a->ldo ? a->ldo : (swiglu ? a->N / 2 : a->N);
    p.ldr = a->ldr ? a->ldr : a->N;
    p.kb_stride = a->w_kb_stride > 0 ? a->w_kb_stride : a->K / TILE_K;
    p.kpg = WMODE == OVB_W_BF16 ? 1 : a->group_size / stream_unit(WMODE);
    p.units = a->K / stream_unit(WMODE);
    p.act = a->act;
    p.out_f32 = a->out_f32;
    p.act_limit = a->act_limit;
    p.act_slope = a->act_slope;
    p.act_shift = a->act_shift;
    p.x_norm = a->x_norm;
    p.x_rows = a->x_rows;
    p.x_eps = a->x_eps;
    p.x_count = a->x_count;
    int smem = 0;
    const int splits = pick_stream_split(WMODE, a->T, a->N, p.units, &smem);
    p.units_per_split = ceil_div(p.units, splits);
    auto kern = gemm_stream_kernel<WMODE, F16>;
    {
        static std::mutex mu;
        static uint64_t configured = 0;         // one bit per device
        int dev = 0;
        OVB_CHECK_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lk(mu);
        if (!(configured & (1ull << (dev & 63)))) {
            OVB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem));
            OVB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
            configured |= 1ull << (dev & 63);
        }
    }
    const int resident = 296 / splits, tiles = a->N / 32;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((tiles < resident ? tiles : resident) * splits);
    cfg.blockDim = dim3(kStreamThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    OVB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<const StreamParams>(p)));
    OVB_CHECK_CUDA(cudaGetLastError());
    return 0;
}

int gemm_stream(const ovb_gemm_args* a, cudaStream_t stream) {
    switch (a->wmode) {
        case OVB_W_BF16: return run_stream<OVB_W_BF16, false>(a, stream);
        case OVB_W_F16: return run_stream<OVB_W_BF16, true>(a, stream);
        case OVB_W_U4: return run_stream<OVB_W_U4, false>(a, stream);
        case OVB_W_U8: return run_stream<OVB_W_U8, false>(a, stream);
        default: return run_stream<OVB_W_F8, false>(a, stream);
    }
}

}  // namespace ovb
