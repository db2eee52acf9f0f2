// Stochastic sampling: temperature, top-k, top-p (nucleus), multinomial draw. One CTA per row of logits.
//
// The kept set is {v : logit[v] >= t*}: t* is found by bisection on the logit value so that the set has at most top_k
// members and the smallest probability mass >= top_p (the same rule as sorting by probability and cutting, without
// sorting 128k entries). The draw walks the kept entries in index order with a block-wide prefix sum, so a
// (seed, step, row) triple always gives the same token. The role of openvino.genai's sampler
// (multinomial / top-k / top-p transforms over logits), which the reference keeps outside its runtime repository.
#include "common.cuh"
#include "sm100_ptx.cuh"
#include <cuda_bf16.h>
#include "store_types.cuh"

namespace ovb {

constexpr int kSampleThreads = 1024;

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Eight consecutive logits from element v on; elements at or past `end` read as -inf.
template <class E>
__device__ __forceinline__ void load8(const E* __restrict__ l, int v, int end, bool vec, float x[8]) {
    if (vec && v + 8 <= end) {
        if constexpr (sizeof(E) == 2) {
            const uint4 u = *reinterpret_cast<const uint4*>(l + v);
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                x[2 * j] = __uint_as_float(w[j] << 16);
                x[2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
            }
        } else {
            const float4 a = *reinterpret_cast<const float4*>(l + v), b = *reinterpret_cast<const float4*>(l + v + 4);
            x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
            x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = v + j < end ? ld_f32(l + v + j) : -INFINITY;
    }
}

// Count and mass over the 32 warps: every warp leaves its pair, and after one barrier each warp sums all pairs itself (same
// order in every warp). `most` is the largest count of a warp. The pairs alternate between two buffers (`turn`), so that one
// barrier per sum is enough.
struct Kept {
    int cnt, most;
    float mass;
};
__device__ __forceinline__ Kept sum_kept(int cnt, float mass, float (*part_mass)[32], int (*part_cnt)[32], int& turn) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    for (int o = 16; o > 0; o >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, o);
    if (lane == 0) { part_cnt[turn][warp] = cnt; part_mass[turn][warp] = mass; }
    __syncthreads();
    const int c = part_cnt[turn][lane];
    float m = part_mass[turn][lane];
    for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
    turn ^= 1;
    return {__reduce_add_sync(0xffffffffu, c), __reduce_max_sync(0xffffffffu, c), m};
}

// What bounds it: passes over the row, which lies in L2 (256 KB for 128k entries: about 2 us a pass for one SM). Every warp owns a
// contiguous piece of the row and reads it in whole 512-byte lines. The bisection goes over the whole row only until no warp keeps
// more than kListWarp entries; these then stay in registers for the remaining steps, which cost one barrier each.
// 24 rows of 128256 entries, top-k 50 and top-p 0.95: 646 us with scattered loads in all 30 passes, 71 us now.
constexpr int kListLane = 8, kListWarp = 32 * kListLane;

template <class E>
__global__ void __launch_bounds__(kSampleThreads) sample_kernel(const E* __restrict__ logits, int ld, int V, float inv_temp,
                                                                int top_k, float top_p, uint64_t seed, const int* __restrict__ step_ptr,
                                                                int* __restrict__ out_ids) {
    pdl_enter();
    __shared__ float part_mass[2][32];
    __shared__ int part_cnt[2][32];
    __shared__ float list[32][kListWarp];
    const int row = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const E* l = logits + (size_t)row * ld;
    const bool vec = (reinterpret_cast<uintptr_t>(l) & 15) == 0;
    const int per = ((V + 31) / 32 + 7) / 8 * 8;             // contiguous piece of a warp (index order matters for the draw)
    const int v0 = min(V, warp * per), v1 = min(V, v0 + per);
    int turn = 0;
    // calls f(x[8], first element) for the pieces of 256 elements of this warp, four loads in flight
    auto each = [&](auto&& f) {
        for (int base = v0; base < v1; base += 1024) {
            float x[4][8];
#pragma unroll
            for (int i = 0; i < 4; ++i) load8(l, base + i * 256 + lane * 8, v1, vec, x[i]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (base + i * 256 < v1) f(x[i], base + i * 256 + lane * 8);
        }
    };

    float mx = -INFINITY, mn = INFINITY;
    each([&](const float* x, int v) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            mx = fmaxf(mx, x[j]);
            if (v + j < v1) mn = fminf(mn, x[j]);
        }
    });
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    }
    if (lane == 0) { part_mass[0][warp] = mx; part_mass[1][warp] = mn; }
    __syncthreads();
    mx = part_mass[0][lane];
    mn = part_mass[1][lane];
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    }
    __syncthreads();

    const bool restrict_k = top_k > 0 && top_k < V, restrict_p = top_p < 1.f;
    float thr = -INFINITY;
    if (restrict_k || restrict_p) {
        // bisection on the threshold: keep(lo) is never smaller than the wanted set, keep(hi) may be
        // An entry more than 104 temperatures below the largest has no mass (e^-104 < 2^-149), so the range ends there: masked entries
        // (-inf, or the type's lowest value) would otherwise hold the bisection off the entries that count.
        float lo = fmaxf(mn, mx - 104.f / inv_temp), hi = mx, z = 0.f;
        int it = 0, most = V;            // most: largest number of entries >= lo in a warp's piece
        for (; it < 26 && most > kListWarp; ++it) {
            const float mid = 0.5f * (lo + hi);
            int cnt = 0;
            float mass = 0.f, all = 0.f;
            const bool first = it == 0;
            each([&](const float* x, int v) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const bool in = v + j < v1 && x[j] >= mid;
                    if (in || (first && v + j < v1)) {
                        const float e = __expf((x[j] - mx) * inv_temp);
                        all += e;
                        if (in) { ++cnt; mass += e; }
                    }
                }
            });
            if (first) z = sum_kept(0, all, part_mass, part_cnt, turn).mass;
            const Kept k = sum_kept(cnt, mass, part_mass, part_cnt, turn);
            // t* = max(t_k, t_p): the threshold may rise to mid while at least one active rule still holds there
            // (t_k = largest t with count(>= t) >= k, t_p = largest t with mass(>= t) >= p)
            const bool enough = (restrict_p && k.mass >= top_p * z) || (restrict_k && k.cnt >= top_k);
            if (enough) { lo = mid; most = k.most; } else hi = mid;
        }
        if (it < 26) {
            // the warp's entries >= lo, in index order, then eight to a lane
            int n = 0;
            each([&](const float* x, int v) {
                int c = 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) c += v + j < v1 && x[j] >= lo;
                if (__any_sync(0xffffffffu, c)) {
                    int at = c;
                    for (int o = 1; o < 32; o <<= 1) {
                        const int up = __shfl_up_sync(0xffffffffu, at, o);
                        if (lane >= o) at += up;
                    }
                    const int total = __shfl_sync(0xffffffffu, at, 31);
                    at += n - c;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (v + j < v1 && x[j] >= lo && at < kListWarp) list[warp][at++] = x[j];
                    n += total;
                }
            });
            __syncwarp();
            float lx[kListLane], le[kListLane];
#pragma unroll
            for (int j = 0; j < kListLane; ++j) {
                const bool in = lane + j * 32 < n;
                lx[j] = in ? list[warp][lane + j * 32] : -INFINITY;
                le[j] = in ? __expf((lx[j] - mx) * inv_temp) : 0.f;
            }
            if (it == 0) {          // a short row is its own list
                float all = 0.f;
#pragma unroll
                for (int j = 0; j < kListLane; ++j) all += le[j];
                z = sum_kept(0, all, part_mass, part_cnt, turn).mass;
            }
            for (; it < 26; ++it) {
                const float mid = 0.5f * (lo + hi);
                int cnt = 0;
                float mass = 0.f;
#pragma unroll
                for (int j = 0; j < kListLane; ++j)
                    if (lane + j * 32 < n && lx[j] >= mid) { ++cnt; mass += le[j]; }
                const Kept k = sum_kept(cnt, mass, part_mass, part_cnt, turn);
                const bool enough = (restrict_p && k.mass >= top_p * z) || (restrict_k && k.cnt >= top_k);
                if (enough) lo = mid; else hi = mid;
            }
        }
        thr = lo;
    }

    // the draw: prefix masses of the warps' pieces, then the warp that the target falls into walks its piece
    float local = 0.f;
    each([&](const float* x, int v) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (v + j < v1 && x[j] >= thr) local += __expf((x[j] - mx) * inv_temp);
    });
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if (lane == 0) part_mass[turn][warp] = local;
    __syncthreads();
    float upto = part_mass[turn][lane];
    for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += up;
    }
    const float total = __shfl_sync(0xffffffffu, upto, 31);
    const uint64_t r64 = mix64(seed ^ mix64(((uint64_t)(step_ptr ? *step_ptr : 0) << 20) ^ (uint64_t)row));
    const float u = (float)((r64 >> 40) + 0.5) * (1.0f / 16777216.0f);      // (0, 1], the last value rounds to 1
    const float target = u * total;
    // One warp draws, and every warp finds the same one: the first with kept mass whose prefix reaches the target. The prefixes are sums
    // in different orders, so they may fall by a unit in the last place from a warp to the next, and the total may lie above the last
    // kept warp's: a target in such a gap belongs to the last warp with kept mass.
    const bool has = part_mass[turn][lane] > 0.f;
    const uint32_t kept = __ballot_sync(0xffffffffu, has), reach = __ballot_sync(0xffffffffu, has && target <= upto);
    const int owner = reach ? __ffs(reach) - 1 : 31 - __clz(kept);          // -1: no mass at all
    const float below = __shfl_sync(0xffffffffu, upto, max(owner - 1, 0));
    const float before = owner > 0 ? below : 0.f;
    if (owner < 0) {                    // no distribution to draw from (NaN or infinite logits): the first of the largest entries
        int best = V;
        each([&](const float* x, int v) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (v + j < v1 && x[j] == mx) best = min(best, v + j);
        });
        best = __reduce_min_sync(0xffffffffu, best);
        if (lane == 0) part_cnt[turn][warp] = best;
        __syncthreads();
        best = __reduce_min_sync(0xffffffffu, part_cnt[turn][lane]);
        if (threadIdx.x == 0) out_ids[row] = best < V ? best : 0;
    } else if (warp == owner) {
        float acc = before;
        int pick = -1, last = -1;       // last: the last entry with mass, for a target that the rounding of the sums puts past it
        for (int base = v0; base < v1 && pick < 0; base += 256) {
            const int v = base + lane * 8;
            float x[8];
            load8(l, v, v1, vec, x);
            float own = 0.f;
            int own_last = -1;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float e = v + j < v1 && x[j] >= thr ? __expf((x[j] - mx) * inv_temp) : 0.f;
                if (e > 0.f) { own += e; own_last = v + j; }
            }
            float incl = own;
            for (int o = 1; o < 32; o <<= 1) {
                const float up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            const float left = __shfl_up_sync(0xffffffffu, incl, 1);
            const uint32_t hit = __ballot_sync(0xffffffffu, own_last >= 0 && acc + incl >= target);
            if (hit) {
                const int who = __ffs(hit) - 1;
                if (lane == who) {
                    float a = acc + (lane ? left : 0.f);
                    bool done = false;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float e = v + j < v1 && x[j] >= thr ? __expf((x[j] - mx) * inv_temp) : 0.f;
                        if (!done && e > 0.f) {
                            a += e;
                            pick = v + j;
                            done = a >= target;
                        }
                    }
                }
                pick = __shfl_sync(0xffffffffu, pick, who);
            } else {
                last = max(last, __reduce_max_sync(0xffffffffu, own_last));
                acc += __shfl_sync(0xffffffffu, incl, 31);
            }
        }
        if (lane == 0) out_ids[row] = pick >= 0 ? pick : last;
    }
}

__global__ void bump_kernel(int* p) {
    pdl_enter(); *p += 1; }

}  // namespace ovb

extern "C" {
namespace ovb {

// Uniform in the open interval (0, 1) from the top 23 bits of a hash: (k + 0.5) * 2^-23 with k < 2^23 needs 24 significant
// bits, so the fp32 sum is exact and the largest value is 1 - 2^-24 (with 24 bits of k the sum k + 0.5 would round to 2^24
// for k = 2^24 - 1, u would be exactly 1, and the Gumbel noise -log(-log(u)) would be +inf).
__host__ __device__ __forceinline__ float gumbel_uniform(uint64_t h) {
    return ((float)(h >> 41) + 0.5f) * (1.0f / 8388608.0f);
}

// Sampling over vocabulary shards without gathering the logits (Gumbel-max): argmax_i(logit_i / T + G_i) with
// G_i = -log(-log(u_i)) is a draw from softmax(logits / T) when the u_i are independent uniforms. u_i depends on the seed,
// the step word, the row and the GLOBAL token index only, so every tensor-parallel rank perturbs its own shard, reduces
// it to (best value, local index), and the usual arg-max exchange between the ranks picks the token.
__global__ void __launch_bounds__(kSampleThreads) gumbel_argmax_kernel(const __nv_bfloat16* __restrict__ logits, int ld, int V, int vocab_offset,
                                                                       float inv_temp, uint64_t seed, const int* __restrict__ step_ptr,
                                                                       int* __restrict__ out_ids, float* __restrict__ out_max) {
    pdl_enter();
    __shared__ float sv[kSampleThreads / 32];
    __shared__ int si[kSampleThreads / 32];
    const int row = blockIdx.x;
    const __nv_bfloat16* lr = logits + (size_t)row * ld;
    const uint64_t base = mix64(seed ^ mix64(((uint64_t)(step_ptr ? *step_ptr : 0) << 20) ^ (uint64_t)row));
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < V; i += kSampleThreads) {
        const uint64_t h = mix64(base ^ ((uint64_t)(uint32_t)(vocab_offset + i) * 0xD1B54A32D192ED03ull));
        const float u = gumbel_uniform(h);
        const float g = -__logf(-__logf(u));
        const float f = __bfloat162float(lr[i]) * inv_temp + g;
        if (f > best) { best = f; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { sv[warp] = best; si[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        best = lane < kSampleThreads / 32 ? sv[lane] : -INFINITY;
        bi = lane < kSampleThreads / 32 ? si[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (lane == 0) {
            out_ids[row] = bi == 0x7fffffff ? 0 : bi;
            if (out_max) out_max[row] = best;
        }
    }
}

}  // namespace ovb

using namespace ovb;

// out_ids[row] ~ softmax(logits[row] / temperature) restricted to the top_k most likely tokens and to the smallest
// set of probability mass >= top_p. top_k <= 0 and top_p >= 1 switch the restrictions off. `step` (device int, may be
// NULL) is mixed into the random stream, so replays of a captured graph draw fresh numbers when the word is bumped.
}  // extern "C"

template <class E>
static int sample_rows(const E* logits, int ld, int rows, int vocab, float temperature, int top_k, float top_p, uint64_t seed, const int* step, int* out_ids,
                       cudaStream_t stream) {
    OVB_REQUIRE(logits && out_ids && rows > 0 && vocab > 0 && temperature > 0.f, "ovb_sample: bad arguments (temperature must be > 0)");
    OVB_CHECK_CUDA(launch_pdl(sample_kernel<E>, dim3(rows), dim3(kSampleThreads), 0, stream, logits, ld, vocab, 1.0f / temperature, top_k,
                                                       top_p <= 0.f ? 1e-6f : top_p, seed, step, out_ids));
    OVB_CHECK_CUDA(cudaGetLastError());
    return 0;
}

extern "C" {

int ovb_sample(const void* logits, int ld, int rows, int vocab, float temperature, int top_k, float top_p, uint64_t seed,
               const int* step, int* out_ids, ovb_stream_t stream_) {
    return sample_rows((const __nv_bfloat16*)logits, ld, rows, vocab, temperature, top_k, top_p, seed, step, out_ids, static_cast<cudaStream_t>(stream_));
}

int ovb_sample_f32(const float* logits, int ld, int rows, int vocab, float temperature, int top_k, float top_p, uint64_t seed, const int* step, int* out_ids,
                   ovb_stream_t stream_) {
    return sample_rows(logits, ld, rows, vocab, temperature, top_k, top_p, seed, step, out_ids, static_cast<cudaStream_t>(stream_));
}

int ovb_sample_gumbel(const void* logits, int ld, int rows, int vocab, int vocab_offset, float temperature, uint64_t seed, const int* step,
                      int* out_ids, float* out_max, ovb_stream_t stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    OVB_REQUIRE(logits && out_ids && rows > 0 && vocab > 0 && temperature > 0.f, "ovb_sample_gumbel: bad arguments (temperature must be > 0)");
    OVB_CHECK_CUDA(launch_pdl(gumbel_argmax_kernel, dim3(rows), dim3(kSampleThreads), 0, stream, (const __nv_bfloat16*)logits, ld, vocab, vocab_offset, 1.0f / temperature, seed, step,
                                                              out_ids, out_max));
    OVB_CHECK_CUDA(cudaGetLastError());
    return 0;
}

// Host-side view of the hash -> uniform mapping of the Gumbel sampler (for tests of its range).
float ovb_gumbel_uniform(uint64_t h) { return gumbel_uniform(h); }

int ovb_bump(int* counter, ovb_stream_t stream_) {
    OVB_REQUIRE(counter != nullptr, "ovb_bump: null counter");
    OVB_CHECK_CUDA(launch_pdl(bump_kernel, dim3(1), dim3(1), 0, static_cast<cudaStream_t>(stream_), counter));
    OVB_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // extern "C"
