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

// The same for few rows of a large vocabulary: a cluster of eight CTAs per row, and the row stays in their registers (32 entries a thread, in index
// order: CTA, warp, piece of 256, lane). What bounds it then is the way between the CTAs, about 1.3 us for a step of the bisection: every CTA pushes its count and
// mass to all (st.async) and adds up the eight itself, in the same order. Once no CTA keeps more than kShareList entries, the kept ones go to all
// CTAs, each of which takes the remaining steps by itself.
// (A thread holds 16 words of its row and the steps of two forms in 64 registers, two CTAs to an SM: some 30 words are parked in local memory.)
constexpr int kShareThreads = 512, kShareCtas = 8, kShareList = 512;

struct ShareBox {                         // what the CTAs of a row send one another
    float4 got[2][kShareCtas];
    float list[kShareCtas * kShareList];
    uint64_t full[2], list_full;
};

__global__ void __launch_bounds__(kShareThreads, 2) sample_shared_kernel(const __nv_bfloat16* __restrict__ logits, int ld, int V, float inv_temp, int top_k, float top_p,
                                                                         uint64_t seed, const int* __restrict__ step_ptr, int* __restrict__ out_ids,
                                                                         int* __restrict__ status) {
    constexpr int WARPS = kShareThreads / 32;
    __shared__ __align__(16) ShareBox box;
    __shared__ float part_a[WARPS], part_b[WARPS], part_mass[2][32];
    __shared__ int part_cnt[2][32];
    __shared__ int counts[kShareCtas];                        // kept by the CTAs
    __shared__ volatile int abort_flag;
    const int rank = (int)cluster_ctarank(), row = blockIdx.x / kShareCtas, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&box.full[i], 1);
            mbar_arrive_expect_tx(&box.full[i], kShareCtas * 16);
        }
        mbar_init(&box.list_full, 1);
        mbar_fence_init();
        abort_flag = 0;
    }
    if (threadIdx.x < 64) part_mass[threadIdx.x >> 5][lane] = 0.f, part_cnt[threadIdx.x >> 5][lane] = 0;
    __syncthreads();
    cluster_arrive();
    cluster_wait();
    pdl_enter();
    const __nv_bfloat16* l = logits + (size_t)row * ld;
    const int per = ((V + kShareCtas - 1) / kShareCtas + 7) / 8 * 8, per_warp = ((per + WARPS - 1) / WARPS + 7) / 8 * 8;
    const int end = min(V, (rank + 1) * per), v0 = min(end, rank * per + warp * per_warp), v1 = min(end, v0 + per_warp);
    uint4 q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int v = v0 + i * 256 + lane * 8;
        if (v + 8 <= v1) {
            q[i] = *reinterpret_cast<const uint4*>(l + v);
        } else {
            uint16_t e[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) e[j] = v + j < v1 ? __bfloat16_as_ushort(l[v + j]) : (uint16_t)0xFF80u;
            q[i] = make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
        }
    }
    // f(value, index) for the thread's entries (an index at or past v1: none)
    auto each = [&](auto&& f) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t w[4] = {q[i].x, q[i].y, q[i].z, q[i].w};
#pragma unroll
            for (int j = 0; j < 8; ++j) f(__uint_as_float(j & 1 ? w[j >> 1] & 0xFFFF0000u : w[j >> 1] << 16), v0 + i * 256 + lane * 8 + j);
        }
    };
    bool ok = true;
    int turn = 0;
    uint32_t parity = 0;
    // every CTA's four values (valid in warp 0) to all CTAs
    auto exchange = [&](float a, float b, float c, float d) {
        if (warp == 0 && lane < kShareCtas) {
            const uint32_t v[4] = {__float_as_uint(a), __float_as_uint(b), __float_as_uint(c), __float_as_uint(d)};
            st_async_v4(dsmem_addr(smem_u32(&box.got[turn][rank]), lane), v, dsmem_addr(smem_u32(&box.full[turn]), lane));
        }
        ok = mbar_wait(&box.full[turn], parity, &abort_flag, status) && ok;
        // (a peer fills this turn's places again only after it has this CTA's next values, which are sent behind a barrier)
        if (threadIdx.x == 0) mbar_arrive_expect_tx(&box.full[turn], kShareCtas * 16);
        const float4* got = box.got[turn];
        turn ^= 1;
        if (turn == 0) parity ^= 1;
        return got;
    };
    auto warps_sum = [&](const float* parts) {               // the same order in every warp
        float v = lane < WARPS ? parts[lane] : 0.f;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
    auto warp_sum_f = [&](float v) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };

    float mx = -INFINITY, mn = INFINITY;
    each([&](float x, int v) {
        mx = fmaxf(mx, x);
        if (v < v1) mn = fminf(mn, x);
    });
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    }
    if (lane == 0) part_a[warp] = mx, part_b[warp] = mn;
    __syncthreads();
    if (warp == 0) {
        mx = lane < WARPS ? part_a[lane] : -INFINITY;
        mn = lane < WARPS ? part_b[lane] : INFINITY;
        for (int o = 16; o > 0; o >>= 1) {
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        }
    }
    {
        const float4* got = exchange(mx, mn, 0.f, 0.f);
        mx = -INFINITY;
        mn = INFINITY;
#pragma unroll
        for (int z = 0; z < kShareCtas; ++z) {
            mx = fmaxf(mx, got[z].x);
            mn = fminf(mn, got[z].y);
        }
    }

    const bool restrict_k = top_k > 0 && top_k < V, restrict_p = top_p < 1.f;
    float thr = -INFINITY;
    if (restrict_k || restrict_p) {
        // as in sample_kernel
        float lo = fmaxf(mn, mx - 104.f / inv_temp), hi = mx, z = 0.f;
        int it = 0, most = V;
        for (; it < 26 && most > kShareList; ++it) {
            const float mid = 0.5f * (lo + hi);
            int cnt = 0;
            float mass = 0.f, all = 0.f;
            each([&](float x, int v) {
                const bool in = v < v1 && x >= mid;
                if (in || (it == 0 && v < v1)) {
                    const float e = __expf((x - mx) * inv_temp);
                    all += e;
                    if (in) { ++cnt; mass += e; }
                }
            });
            cnt = __reduce_add_sync(0xffffffffu, cnt);
            mass = warp_sum_f(mass);
            if (it == 0) all = warp_sum_f(all);
            __syncthreads();                                  // (the parts of the step before have been read)
            if (lane == 0) {
                part_cnt[0][warp] = cnt;
                part_a[warp] = mass;
                part_b[warp] = all;
            }
            __syncthreads();
            const int c = __reduce_add_sync(0xffffffffu, lane < WARPS ? part_cnt[0][lane] : 0);
            const float4* got = exchange(__int_as_float(c), warps_sum(part_a), it == 0 ? warps_sum(part_b) : 0.f, 0.f);
            int total = 0, largest = 0;
            float m = 0.f, s = 0.f;
#pragma unroll
            for (int r = 0; r < kShareCtas; ++r) {
                const int n = __float_as_int(got[r].x);
                total += n;
                largest = max(largest, n);
                m += got[r].y;
                s += got[r].z;
            }
            if (it == 0) z = s;
            const bool enough = (restrict_p && m >= top_p * z) || (restrict_k && total >= top_k);
            if (enough) {
                lo = mid;
                most = largest;
                if (threadIdx.x < kShareCtas) counts[threadIdx.x] = __float_as_int(got[threadIdx.x].x);
            } else {
                hi = mid;
            }
        }
        if (it < 26) {
            // the kept entries of all CTAs, each CTA's in index order, padded to four
            int c = 0;
            each([&](float x, int v) { c += v < v1 && x >= lo; });
            // (a lane's entries lie in four pieces: their order inside the list does not matter, that it is always the same does)
            int at = c;
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, at, o);
                if (lane >= o) at += up;
            }
            __syncthreads();
            if (lane == 31) part_cnt[0][warp] = at;
            __syncthreads();
            int before = 0;
            for (int w = 0; w < warp; ++w) before += part_cnt[0][w];
            at += before - c;
            int begin = 0, mine = 0, bytes = 0;
#pragma unroll
            for (int r = 0; r < kShareCtas; ++r) {
                if (r < rank) begin += (counts[r] + 3) / 4 * 4;
                if (r == rank) mine = counts[r];
                bytes += (counts[r] + 3) / 4 * 16;
            }
            __shared__ __align__(16) float own[kShareList];
            each([&](float x, int v) {
                if (v < v1 && x >= lo && at < kShareList) own[at++] = x;
            });
            if (threadIdx.x < 4 && mine + threadIdx.x < (mine + 3) / 4 * 4) own[mine + threadIdx.x] = -INFINITY;
            if (threadIdx.x == 0) mbar_arrive_expect_tx(&box.list_full, bytes);
            __syncthreads();
            for (int i = threadIdx.x; i < (mine + 3) / 4 * kShareCtas; i += kShareThreads) {
                const int piece = i / kShareCtas, to = i % kShareCtas;
                const uint32_t* src = reinterpret_cast<const uint32_t*>(own + piece * 4);
                const uint32_t v[4] = {src[0], src[1], src[2], src[3]};
                st_async_v4(dsmem_addr(smem_u32(box.list + begin + piece * 4), to), v, dsmem_addr(smem_u32(&box.list_full), to));
            }
            ok = mbar_wait(&box.list_full, 0, &abort_flag, status) && ok;
            float lx[kShareCtas], le[kShareCtas];
#pragma unroll
            for (int j = 0; j < kShareCtas; ++j) {
                const int i = threadIdx.x + j * kShareThreads;
                lx[j] = i < bytes / 4 ? box.list[i] : -INFINITY;
                le[j] = lx[j] >= lo ? __expf((lx[j] - mx) * inv_temp) : 0.f;
            }
            int side = 1;
            for (; it < 26; ++it) {
                const float mid = 0.5f * (lo + hi);
                int cnt = 0;
                float mass = 0.f;
#pragma unroll
                for (int j = 0; j < kShareCtas; ++j)
                    if (lx[j] >= mid) { ++cnt; mass += le[j]; }
                const Kept k = sum_kept(cnt, mass, part_mass, part_cnt, side);
                const bool enough = (restrict_p && k.mass >= top_p * z) || (restrict_k && k.cnt >= top_k);
                if (enough) lo = mid; else hi = mid;
            }
        }
        thr = lo;
    }

    // the draw: prefix masses of the CTAs, of the owner's warps, then the warp that the target falls into walks its piece
    float local = 0.f;
    each([&](float x, int v) {
        if (v < v1 && x >= thr) local += __expf((x - mx) * inv_temp);
    });
    local = warp_sum_f(local);
    __syncthreads();
    if (lane == 0) part_a[warp] = local;
    __syncthreads();
    float upto = lane < WARPS ? part_a[lane] : 0.f;           // of the warps
    const bool has = upto > 0.f;
    for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += up;
    }
    const float4* got = exchange(__shfl_sync(0xffffffffu, upto, 31), 0.f, 0.f, 0.f);
    float sums[kShareCtas], total = 0.f;
#pragma unroll
    for (int r = 0; r < kShareCtas; ++r) sums[r] = total += got[r].x;
    const uint64_t r64 = mix64(seed ^ mix64(((uint64_t)(step_ptr ? *step_ptr : 0) << 20) ^ (uint64_t)row));
    const float u = (float)((r64 >> 40) + 0.5) * (1.0f / 16777216.0f);      // (0, 1], the last value rounds to 1
    const float target = u * total;
    int owner = -1, last = -1;                                // (see sample_kernel for targets between the prefixes)
#pragma unroll
    for (int r = 0; r < kShareCtas; ++r) {
        const bool mass = got[r].x > 0.f;
        if (mass) last = r;
        if (mass && owner < 0 && target <= sums[r]) owner = r;
    }
    if (owner < 0) owner = last;
    if (owner < 0) {                    // no distribution to draw from (NaN or infinite logits): the first of the largest entries
        int best = V;
        each([&](float x, int v) {
            if (v < v1 && x == mx) best = min(best, v);
        });
        best = __reduce_min_sync(0xffffffffu, best);
        __syncthreads();
        if (lane == 0) part_cnt[0][warp] = best;
        __syncthreads();
        best = __reduce_min_sync(0xffffffffu, lane < WARPS ? part_cnt[0][lane] : V);
        const float4* b = exchange(__int_as_float(best), 0.f, 0.f, 0.f);
        best = V;
        for (int r = 0; r < kShareCtas; ++r) best = min(best, __float_as_int(b[r].x));
        if (ok && rank == 0 && threadIdx.x == 0) out_ids[row] = best < V ? best : 0;
    } else if (rank == owner) {
        float base = 0.f;
#pragma unroll
        for (int r = 0; r < kShareCtas; ++r)
            if (r + 1 == rank) base = sums[r];
        const uint32_t kept = __ballot_sync(0xffffffffu, has), reach = __ballot_sync(0xffffffffu, has && target <= base + upto);
        const int who = reach ? __ffs(reach) - 1 : 31 - __clz(kept);
        const float below = __shfl_sync(0xffffffffu, upto, max(who - 1, 0));
        if (warp == who) {
            float acc = base + (who > 0 ? below : 0.f);
            int pick = -1, final_one = -1;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t w[4] = {q[i].x, q[i].y, q[i].z, q[i].w};
                const int v = v0 + i * 256 + lane * 8;
                float e[8], own = 0.f;
                int own_last = -1;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float x = __uint_as_float(j & 1 ? w[j >> 1] & 0xFFFF0000u : w[j >> 1] << 16);
                    e[j] = v + j < v1 && x >= thr ? __expf((x - mx) * inv_temp) : 0.f;
                    if (e[j] > 0.f) { own += e[j]; own_last = v + j; }
                }
                float incl = own;
                for (int o = 1; o < 32; o <<= 1) {
                    const float up = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += up;
                }
                const float left = __shfl_up_sync(0xffffffffu, incl, 1);
                const uint32_t hit = __ballot_sync(0xffffffffu, own_last >= 0 && acc + incl >= target);
                if (pick < 0 && hit) {
                    const int at = __ffs(hit) - 1;
                    float a = acc + (lane ? left : 0.f);
                    int found = own_last;
                    bool done = false;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (!done && e[j] > 0.f) {
                            a += e[j];
                            found = v + j;
                            done = a >= target;
                        }
                    pick = __shfl_sync(0xffffffffu, found, at);
                }
                final_one = max(final_one, __reduce_max_sync(0xffffffffu, own_last));
                acc += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (ok && lane == 0) out_ids[row] = pick >= 0 ? pick : final_one;
        }
    }
    cluster_arrive();       // no CTA leaves while a peer may still store to it
    cluster_wait();
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
    if constexpr (sizeof(E) == 2) {
        // A cluster holds up to 8 x 512 x 32 entries. It takes 26 us with up to 12 rows, 38 with up to 36 (their 296 CTAs are resident at a time), 71 with 48, 76 with
        // 64; a CTA per row takes the same for any of these numbers of rows: 33 us with 16384 entries, 39 with 32000, 51 with 65536, 85 with 128256 (top-k 50,
        // top-p 0.95, logits in L2). At the line: 6 rows of 16384 entries 26 / 33, 11 of 32000 26 / 39, 24 of 65536 37 / 52, 37 of 100352 62 / 76, 47 of 128256
        // 71 / 86; behind it 24 of 16384 36 / 34, 37 of 65536 59 / 52, 74 of 128256 94 / 87. Without top-k the kept set is large, its steps are all between the
        // CTAs, and the token of a flat distribution would depend on the order of its sums.
        if (top_k > 0 && top_k < vocab && vocab >= 16384 && (int64_t)rows * 2700 <= vocab && vocab <= kShareCtas * kShareThreads * 32 && ld % 8 == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0) {
            cudaLaunchConfig_t cfg;
            memset(&cfg, 0, sizeof(cfg));
            cfg.gridDim = dim3(rows * kShareCtas);
            cfg.blockDim = dim3(kShareThreads);
            cfg.stream = stream;
            cudaLaunchAttribute attr[2];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = kShareCtas;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[1].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = pdl_enabled() ? 2 : 1;
            OVB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, sample_shared_kernel, logits, ld, vocab, 1.0f / temperature, top_k, top_p <= 0.f ? 1e-6f : top_p, seed, step, out_ids,
                                              status_word()));
            return 0;
        }
    }
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
