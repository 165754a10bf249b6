// moe_tc.cu -- the grouped matrix products of routed feed-forward experts on the 5th-generation tensor cores (tcgen05.mma
// kind::f16, bfloat16 operands, float accumulators in TMEM), for batches with more than a few rows per expert.  The pairs are
// sorted by expert (moe_sort_kernel); offsets[e] .. offsets[e + 1] are expert e's.
//
// Persistent: one CTA per SM walks tiles of 128 sorted pairs x 256 weight rows (MODE 0: 128 gate rows and the matching 128 up
// rows) of one expert, the row tiles of a strip of weight rows next to each other so that the strip stays in L2.
//   warp 0        TMA: weight boxes of 128 rows x 64 columns (and, MODE 1, the rows of the activations, which are sorted)
//   warp 1        TMEM allocation (two accumulators of 256 columns) and the elected thread that issues the products
//   warps 2-5     epilogue of tile j while the products of tile j + 1 run: accumulator -> activation or float rows, staged
//                 through shared memory so that a store instruction writes whole 128-byte row segments
//   warps 6-9     MODE 0 and 2: the token rows of the tile's pairs by 16-byte cp.async into the swizzled K-major A tile, two
//                 stages in flight per thread (a gather by TMA would need 32 four-row copies a stage from one thread)
// A routing weight on the expert's input is applied to the accumulated product, which is linear in it.
//
// What bounds it: what one SM takes in.  A stage (64 columns) is 4 x M128 N256 K16 = 512 cycles of tensor pipe, and its 48 KB would
// have to come at 96 B per cycle; about 50 are seen, and the pipe is busy 36 % of the time.  Measured, 16384 pairs of 8 experts,
// width 2048, ff 1024: gate / up 178 us = 770 TFLOP/s, down 67 us = 1030 TFLOP/s (mma.sync kernels of moe_ops.cu: 530 and 294 us).
//
// Every wait is bounded: on a protocol error the CTA raises a flag (pa_moe_tc_errors), lets its copies land, frees its TMEM and
// writes NaN into the rows of its tiles from there on.
#include "seq_common.cuh"
#include "tcgen05_utils.cuh"

namespace pa {
namespace mtc {

using namespace tc;

constexpr int BM = 128, BN = 256, BK = 64, ST = 4;
constexpr int A_BYTES = BM * 128, B_BYTES = BN * 128, STAGE = A_BYTES + B_BYTES;
constexpr int kMostExperts = 1024;

struct Args {
    const bf16_t* A;            // MODE 0, 2: token rows
    int64_t lda;
    int K, n_out, experts, top, act, n_strips;
    const int32_t* order;
    const float* a_scale;
    const int32_t* offsets;     // [experts + 1]
    bf16_t* out;                // MODE 0, 2: [pairs][n_out], sorted order
    float* out_f32;             // MODE 1: [pairs][n_out], (row, choice) order
    uint32_t polls;             // of a wait
};

__device__ int g_errors;

__device__ __forceinline__ float act_f32(float v, int act) {
    if (act == 1) return fmaxf(v, 0.f);
    if (act == 2) { const float r = fmaxf(v, 0.f); return r * r; }
    return silu_f32(v);
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__host__ __device__ constexpr int threads_for(int mode) { return mode == 1 ? 192 : 320; }
constexpr size_t smem_for(int experts) { return (size_t)ST * STAGE + 4 * 4096 + 256 + (size_t)(experts + 1) * 4 + 1024; }

// the walk over the tiles of all experts: every role of a CTA makes the same one
struct Walk {
    const int* start;           // [experts + 1] first tile of each expert
    const int32_t* off;
    int e, stride, t, strips, experts;
    int m0, rows, strip;
    __device__ __forceinline__ bool next() {
        t += stride;
        while (e < experts && t >= start[e + 1]) ++e;
        if (e >= experts) return false;
        const int i = t - start[e], mt = (start[e + 1] - start[e]) / strips, lo = __ldg(off + e);
        strip = i / mt;
        m0 = lo + (i - strip * mt) * BM;
        rows = min(BM, __ldg(off + e + 1) - m0);
        return true;
    }
};

template <int MODE>
__global__ void __launch_bounds__(threads_for(MODE), 1)
grouped_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const Args a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t stage_sm = base + ST * STAGE, bar0 = stage_sm + 4 * 4096;
    auto full = [&](int s) { return bar0 + s * 8; };
    auto empty = [&](int s) { return bar0 + (ST + s) * 8; };
    auto tfull = [&](int b) { return bar0 + (2 * ST + b) * 8; };
    auto tempty = [&](int b) { return bar0 + (2 * ST + 2 + b) * 8; };
    const uint32_t tmem_slot = bar0 + (2 * ST + 4) * 8, fail_sm = tmem_slot + 8;
    int* start = reinterpret_cast<int*>(smem_raw + (bar0 + 256 - smem_u32(smem_raw)));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(full(s), MODE == 1 ? 1 : 1 + 128);
            mbar_init(empty(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(tfull(b), 1);
            mbar_init(tempty(b), 128);
        }
        asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(fail_sm), "r"(0u) : "memory");
        mbar_fence_init();
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmW));
    }
    if (warp == 1) tmem_alloc(tmem_slot, 512);
    if (warp == 0) {            // tiles before every expert, by a scan over the experts
        int run = 0;
        for (int e0 = 0; e0 < a.experts; e0 += 32) {
            const int e = e0 + lane;
            int n = e < a.experts ? (__ldg(a.offsets + e + 1) - __ldg(a.offsets + e) + BM - 1) / BM * a.n_strips : 0;
            const int mine = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, n, o);
                if (lane >= o) n += v;
            }
            if (e < a.experts) start[e] = run + n - mine;
            run += __shfl_sync(0xffffffffu, n, 31);
        }
        if (lane == 0) start[a.experts] = run;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
    Walk w{start, a.offsets, 0, (int)gridDim.x, (int)blockIdx.x - (int)gridDim.x, a.n_strips, a.experts, 0, 0, 0};
    const int nk = (a.K + BK - 1) / BK, w_rows = MODE == 0 ? 2 * a.n_out : a.n_out;

    if (warp == 0) {
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 1;
            while (a.polls && w.next() && !tc_failed(fail_sm)) {       // 0: waits that are to run out, nothing is requested
                const int n0 = w.strip * (MODE == 0 ? BN / 2 : BN);
                const int r1 = w.e * w_rows + n0, r2 = r1 + (MODE == 0 ? a.n_out : BN / 2);
                for (int kt = 0; kt < nk; ++kt) {
                    if (!tc_wait(empty(s), ph, fail_sm, a.polls)) break;
                    const uint32_t st = base + s * STAGE;
                    mbar_arrive_expect_tx(full(s), MODE == 1 ? STAGE : B_BYTES);
                    tma_load_2d(st + A_BYTES, &tmW, kt * BK, r1, full(s));
                    tma_load_2d(st + A_BYTES + B_BYTES / 2, &tmW, kt * BK, r2, full(s));
                    if (MODE == 1) tma_load_2d(st, &tmA, kt * BK, w.m0, full(s));
                    if (++s == ST) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
            if (tc_failed(fail_sm)) __nanosleep(1000000);   // copies in flight land within microseconds
        }
    } else if (warp == 1) {
        constexpr uint32_t kIdesc = idesc_f16(BM, BN, 0, 0, 1);
        int s = 0, j = 0;
        uint32_t ph = 0;
        bool ok = true;         // false: a wait ran out, and no further product is issued
        for (; ok && w.next(); ++j) {
            const int b = j & 1;
            ok = __all_sync(0xffffffffu, tc_wait(tempty(b), ((uint32_t)(j >> 1) & 1u) ^ 1u, fail_sm, a.polls));
            tc_fence_after();
            for (int kt = 0; ok && kt < nk; ++kt) {
                ok = __all_sync(0xffffffffu, tc_wait(full(s), ph, fail_sm, a.polls));
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t st = base + s * STAGE;
#pragma unroll
                    for (int ks = 0; ks < BK / 16; ++ks)
                        umma_f16(tmem_base + b * BN, make_desc(st + ks * 32, 16, 1024), make_desc(st + A_BYTES + ks * 32, 16, 1024), kIdesc,
                                 kt > 0 || ks > 0 ? 1u : 0u);
                    umma_commit(empty(s));
                    if (kt == nk - 1) umma_commit(tfull(b));
                }
                __syncwarp();
                if (++s == ST) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp < 6) {
        const int qtr = warp & 3, row = qtr * 32 + lane;            // TMEM lane = row of the tile
        const uint32_t ebuf = stage_sm + qtr * 4096;
        constexpr int ECOLS = MODE == 1 ? 32 : 64;                  // output columns per round: 128 bytes of a row
        constexpr int ELEM = MODE == 1 ? 4 : 2, PER = 16 / ELEM;    // columns per 16-byte piece
        for (int j = 0; w.next(); ++j) {
            const int b = j & 1;
            const int n0 = w.strip * (MODE == 0 ? BN / 2 : BN);
            const int cols = min(MODE == 0 ? BN / 2 : BN, a.n_out - n0);
            int pair = -1;
            float sc = 1.f;
            if (row < w.rows && (MODE == 1 || a.a_scale)) {
                pair = __ldg(a.order + w.m0 + row);
                if (MODE != 1) sc = __ldg(a.a_scale + pair);
            }
            tc_wait(tfull(b), (uint32_t)(j >> 1) & 1u, fail_sm, a.polls);
            tc_fence_after();
            const bool lost = tc_failed(fail_sm);       // some wait of the CTA ran out: NaN from here on
            const uint32_t acc = tmem_base + ((uint32_t)(qtr * 32) << 16) + b * BN;
            for (int c0 = 0; c0 < cols; c0 += ECOLS) {
                if (MODE == 1) {
                    uint32_t v[32];
                    tmem_ld32(acc + c0, v);
                    tmem_wait_ld();
                    if (lost) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = 0x7fc00000u;
                    }
#pragma unroll
                    for (int p = 0; p < 8; ++p)
                        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(ebuf + lane * 128 + ((p ^ (lane & 7)) << 4)),
                                     "r"(v[4 * p]), "r"(v[4 * p + 1]), "r"(v[4 * p + 2]), "r"(v[4 * p + 3]) : "memory");
                } else {
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        uint32_t v[32], u[32];
                        tmem_ld32(acc + c0 + hf * 32, v);
                        if (MODE == 0) tmem_ld32(acc + BN / 2 + c0 + hf * 32, u);
                        tmem_wait_ld();
#pragma unroll
                        for (int p = 0; p < 4; ++p) {
                            float f[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                f[e] = act_f32(round_bf16(__uint_as_float(v[8 * p + e]) * sc), a.act);
                                if (MODE == 0) f[e] *= round_bf16(__uint_as_float(u[8 * p + e]) * sc);
                            }
                            uint4 o = bf16x8_pack(f);
                            if (lost) o = make_uint4(0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u);
                            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(ebuf + lane * 128 + (((hf * 4 + p) ^ (lane & 7)) << 4)),
                                         "r"(o.x), "r"(o.y), "r"(o.z), "r"(o.w) : "memory");
                        }
                    }
                }
                __syncwarp();
#pragma unroll
                for (int it = 0; it < 8; ++it) {
                    const int r = it * 4 + (lane >> 3), p = lane & 7, col = c0 + p * PER;
                    const uint4 v = lds_128(ebuf + r * 128 + ((p ^ (r & 7)) << 4));
                    const int64_t dst = MODE == 1 ? __shfl_sync(0xffffffffu, pair, r) : w.m0 + qtr * 32 + r;
                    if (qtr * 32 + r < w.rows && col < cols) {
                        if (MODE == 1) *reinterpret_cast<uint4*>(a.out_f32 + dst * a.n_out + n0 + col) = v;
                        else *reinterpret_cast<uint4*>(a.out + dst * a.n_out + n0 + col) = v;
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
            mbar_arrive_cnt(tempty(b));
        }
    } else {
        // MODE 0, 2: 8 lanes bring one row's 128 bytes of a stage; a thread has rows r0 + 16 i and one 16-byte piece of each
        const int t = threadIdx.x - 192, piece = t & 7, r0 = t >> 3;
        constexpr int LAG = 2;                      // stages whose copies are in flight while the next is issued
        int s = 0, sa = 0, issued = 0;
        uint32_t ph = 1;
        auto land = [&] {                           // the oldest stage in flight has landed: hand it over
            fence_proxy_async();                    // the products read it through the async proxy
            mbar_arrive_cnt(full(sa));
            if (++sa == ST) sa = 0;
        };
        while (w.next()) {
            const bf16_t* src[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = r0 + 16 * i;
                src[i] = r < w.rows ? a.A + (int64_t)(__ldg(a.order + w.m0 + r) / a.top) * a.lda + piece * 8 : nullptr;
            }
            for (int kt = 0; kt < nk; ++kt) {
                tc_wait(empty(s), ph, fail_sm, a.polls);
                const uint32_t st = base + s * STAGE;
                const bool in_k = kt * BK + piece * 8 < a.K;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = r0 + 16 * i;
                    const bool ok = src[i] && in_k;
                    cp_async_16(st + r * 128 + ((piece ^ (r & 7)) << 4), ok ? src[i] + kt * BK : a.A, ok);
                }
                cp_async_commit();
                if (issued++ >= LAG) {
                    cp_async_wait<LAG>();
                    land();
                }
                if (++s == ST) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
        if (issued > 1) {
            cp_async_wait<1>();
            land();
        }
        if (issued > 0) {
            cp_async_wait<0>();
            land();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        if (tc_failed(fail_sm)) {
            __nanosleep(1000000);
            if (lane == 0) atomicAdd(&g_errors, 1);
        }
        tmem_dealloc(tmem_base, 512);
    }
}

template <int MODE>
static int launch(const CUtensorMap& tmA, const CUtensorMap& tmW, const Args& a, int pairs, cudaStream_t st) {
    const size_t smem = smem_for(a.experts);
    cudaError_t e = cudaFuncSetAttribute(grouped_tc_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int64_t most = (int64_t)(pairs / BM + a.experts) * a.n_strips;
    const int sms = device_info().sm_count;
    grouped_tc_kernel<MODE><<<(unsigned)(most < sms ? most : sms), threads_for(MODE), smem, st>>>(tmA, tmW, a);
    PA_RETURN_LAUNCH_STATUS();
}

}  // namespace mtc

// mode 0: gate / up pairs, 1: down (rows scattered to (row, choice) order as float), 2: up.  PA_ERR_UNSUPPORTED: the caller's other
// kernels serve these operands.
int grouped_tc_launch(int mode, const void* A, int64_t lda, const void* W, int K, int n_out, int experts, const int32_t* order,
                      const float* a_scale, int top, const int32_t* offsets, int pairs, int act, void* out, cudaStream_t st, int polls) {
    using namespace mtc;
    const int64_t w_rows = (int64_t)experts * n_out * (mode == 0 ? 2 : 1);
    if (K % 8 || n_out % 8 || experts > kMostExperts || w_rows >= 0x7fffff00ll || (uintptr_t)out % 16) return PA_ERR_UNSUPPORTED;
    if ((uintptr_t)A % 16 || (uintptr_t)W % 16 || lda % 8) return PA_ERR_UNSUPPORTED;
    CUtensorMap tmA, tmW;
    if (!make_bf16_map(&tmW, W, w_rows, K, K, BN / 2)) return PA_ERR_UNSUPPORTED;
    tmA = tmW;
    if (mode == 1 && !make_bf16_map(&tmA, A, pairs, K, lda, BM)) return PA_ERR_UNSUPPORTED;
    const int strip = mode == 0 ? BN / 2 : BN;
    Args a{static_cast<const bf16_t*>(A), lda, K, n_out, experts, top, act, (n_out + strip - 1) / strip, order, a_scale, offsets,
           static_cast<bf16_t*>(out), static_cast<float*>(out), (uint32_t)polls};
    return mode == 0 ? launch<0>(tmA, tmW, a, pairs, st) : mode == 1 ? launch<1>(tmA, tmW, a, pairs, st) : launch<2>(tmA, tmW, a, pairs, st);
}

}  // namespace pa

using namespace pa;

PA_API int pa_moe_grouped_polls(int mode, const void* d_a, int64_t lda, const void* d_w, int K, int n_out, int experts, const int32_t* d_order,
                                const float* d_a_scale, int top, const int32_t* d_meta, int pairs, int act, void* d_out, int polls,
                                pa_stream_t stream) {
    PA_CHECK_ARG(mode >= 0 && mode <= 2 && d_a && d_w && d_order && d_meta && d_out && K > 0 && n_out > 0 && experts > 0 && top > 0 && pairs >= 0 &&
                 act >= 0 && act <= 2 && polls >= 0);
    if (pairs == 0) return PA_OK;
    return grouped_tc_launch(mode, d_a, lda, d_w, K, n_out, experts, d_order, d_a_scale, top, d_meta, pairs, act, d_out, as_stream(stream), polls);
}

PA_API int pa_moe_tc_errors(int* host_count) {
    PA_CHECK_ARG(host_count);
    return (int)cudaMemcpyFromSymbol(host_count, pa::mtc::g_errors, sizeof(int));
}
