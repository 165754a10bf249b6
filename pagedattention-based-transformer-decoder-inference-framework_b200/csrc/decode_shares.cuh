// decode_shares.cuh -- a list of equal work units cut into equal contiguous shares, for the kernels of decoded tokens
// (masked_decode.cu, latent_decode.cu).
//
// Token t of a launch has pre[t + 1] - pre[t] units in each of its `pairs` (kv heads, or runs of query heads); the list goes token by
// token, pair by pair.  Share w of pair p writes its sums to slot p + w: walking the list, every new share belongs to the
// next pair or the next worker, so no two meet.  The number of shares depends on the lengths of the sequences alone, never on
// the bound of the lengths that a launch was sized for: a launch made for longer sequences gives the same bits.
#pragma once
#include "seq_common.cuh"

namespace pa {
namespace shares {

constexpr int kMostTokens = 4096;

// pre[0 .. n] from the units of every token, by all threads of a CTA (two barriers)
template <typename F>
__device__ __forceinline__ void count_units(int* pre, int n, F units) {
    for (int t = threadIdx.x; t < n; t += blockDim.x) pre[t + 1] = units(t);
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int run = 0;
        for (int t0 = 0; t0 < n; t0 += 32) {
            int v = t0 + lane < n ? pre[t0 + lane + 1] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += u;
            }
            if (t0 + lane < n) pre[t0 + lane + 1] = run + v;
            run += __shfl_sync(0xffffffffu, v, 31);
        }
        if (lane == 0) pre[0] = 0;
    }
    __syncthreads();
}

// the token whose pairs hold unit f
__device__ __forceinline__ int find_token(const int* pre, int n, int64_t f, int pairs) {
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if ((int64_t)pre[mid] * pairs <= f) lo = mid;
        else hi = mid;
    }
    return lo;
}

// shares of a list of `total` units, at least `least` units each where there are that many; every share has a unit, so that no slot is
// read that was not written
__host__ __device__ __forceinline__ int64_t count(int64_t total, int workers, int least) {
    const int64_t n = (total + least - 1) / least;
    return n < workers ? n : workers;
}

static inline size_t pre_bytes(int tokens) { return ((size_t)(tokens + 1) * sizeof(int) + 15) / 16 * 16; }

}  // namespace shares
}  // namespace pa
