// moe_tc.cu -- the grouped matrix products of routed feed-forward experts on the 5th-generation tensor cores (tcgen05.mma
// kind::f16, bfloat16 operands, float accumulators in TMEM), for batches with more than a few rows per expert.  The pairs are
// sorted by expert (moe_sort_kernel); offsets[e] .. offsets[e + 1] are expert e's.
//
// Persistent: one CTA per SM walks tiles of 128 sorted pairs x 256 weight rows (MODE 0: 128 gate rows and the matching 128 up
// rows) of one expert, the row tiles of a strip of weight rows next to each other so that the strip stays in L2.  Large batches go
// by pairs of CTAs (cta_group::2) where that pays (grouped_tc_pairs_pay): 256 sorted pairs x 256 weight rows, each CTA with its 128 rows and a half of the weight rows, so
// that a stage is 32 KB instead of 48.
//   warp 0        TMA: weight boxes of 128 rows x 64 columns, and the rows of A where they are sorted (MODE 1: the activations; pairs
//                 of CTAs: the token rows, copied into sorted order beforehand, which at 2048 columns takes 1.2 ns a row)
//   warp 1        TMEM allocation (two accumulators of 256 columns) and the elected thread that issues the products
//   next warps    epilogue of tile j while the products of tile j + 1 run: accumulator -> activation or float rows.  MODE 0 and 2 eight
//                 warps, as the activations of a tile take longer than its products with four; MODE 1 four
//   last 4 warps  one CTA, MODE 0 and 2: the token rows of the tile's pairs by 16-byte cp.async into the swizzled K-major A tile, two
//                 stages in flight per thread (four rows per TMA gather take about 100 cycles: 385 us where this takes 134)
// A routing weight on the expert's input is applied to the accumulated product, which is linear in it.
//
// What bounds it: the products' issue (a stage's 512 cycles of tensor pipe come every 740 in the pair) and, for down, the float
// rows (134 MB).  Measured, 16384 pairs of 8 experts, width 2048: ff 1024 gate / up 134 us (with four epilogue warps 164; by pairs of CTAs
// with the copy of the rows 131), down 65 us (one CTA 71); ff 2048 gate / up 220 us (one CTA 243), down 108 us (119).
//
// Every wait is bounded: on a protocol error the CTA raises a flag (pa_moe_tc_errors), lets its copies land, frees its TMEM and
// writes NaN into the rows of its tiles from there on.  A pair raises it in both CTAs: warps that gave up go through their tiles
// without waiting, so what they signal no longer says that an accumulator has been read, and no further product may be issued.
#include "cta_pair.cuh"
#include "seq_common.cuh"
#include "tcgen05_utils.cuh"

namespace pa {
namespace mtc {

using namespace tc;

constexpr int BM = 128, BN = 256, BK = 64;      // rows of a CTA's accumulator, its columns, and columns of a stage
constexpr int A_BYTES = BM * 128;
constexpr int kMostExperts = 1024;
constexpr int kPairFrom = 6144;                 // pairs (of row and expert) below which no launch goes by pairs of CTAs
__host__ __device__ constexpr int b_bytes(int ctas) { return BN / ctas * 128; }
__host__ __device__ constexpr int stages_for(int ctas) { return ctas == 2 ? 6 : 4; }

// ---- the pair (cta_pair.cuh)
// a box into this CTA's shared memory, its bytes counted by a barrier of the pair's first CTA
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                 "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// tc_wait for arrivals of the other CTA
__device__ __forceinline__ bool try_pair(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool wait_pair(uint32_t bar, uint32_t parity, uint32_t fail_sm, uint32_t polls) {
    for (uint32_t n = 0; !try_pair(bar, parity);) {
        if (++n > polls || ((n & 255u) == 0 && tc_failed(fail_sm))) {
            asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(fail_sm), "r"(1u) : "memory");
            return false;
        }
    }
    return true;
}

// a wait that ran out, in the other CTA of the pair too: ahead of whatever this thread signals next
__device__ __forceinline__ void tell_pair(uint32_t fail_there) {
    asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(fail_there), "r"(1u) : "memory");
}

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
    uint32_t epilogue_polls[2]; // of a wait of the epilogue warps, by their CTA's place in the pair
};

__device__ int g_errors;

__device__ __forceinline__ float act_f32(float v, int act) {
    if (act == 1) return fmaxf(v, 0.f);
    if (act == 2) { const float r = fmaxf(v, 0.f); return r * r; }
    return silu_f32(v);
}
// 32 bytes of an output row; !whole: the row ends after 16 of them (columns come in eights)
__device__ __forceinline__ void store_words(void* dst, const uint32_t* w, bool whole) {
    if (whole && ((uintptr_t)dst & 31) == 0) {
        asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]),
                     "r"(w[6]), "r"(w[7]) : "memory");
    } else {
        reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
        if (whole) reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__host__ __device__ constexpr int threads_for(int mode, int ctas) { return mode == 1 ? 192 : ctas == 2 ? 320 : 448; }
// epilogue warps.  MODE 0 and 2: two per 32 rows, a half of the columns each
__host__ __device__ constexpr int epilogue_warps(int mode) { return mode == 1 ? 4 : 8; }
constexpr size_t smem_for(int experts, int ctas, int mode) { return (size_t)stages_for(ctas) * (A_BYTES + b_bytes(ctas)) + (mode == 1 ? 4 * 4096 : 0) + 256 + (size_t)(experts + 1) * 4 + 1024; }

// the walk over the tiles of all experts: every role of a CTA makes the same one
template <int TILE_ROWS>
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
        m0 = lo + (i - strip * mt) * TILE_ROWS;
        rows = min(TILE_ROWS, __ldg(off + e + 1) - m0);
        return true;
    }
};

template <int MODE, int CTAS>
__global__ void __launch_bounds__(threads_for(MODE, CTAS), 1)
grouped_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const Args a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    constexpr int ST = stages_for(CTAS), B_BYTES = b_bytes(CTAS), STAGE = A_BYTES + B_BYTES, EPW = epilogue_warps(MODE);
    constexpr bool PAIR = CTAS == 2;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t stage_sm = base + ST * STAGE, bar0 = stage_sm + (MODE == 1 ? 4 * 4096 : 0);
    auto full = [&](int s) { return bar0 + s * 8; };
    auto empty = [&](int s) { return bar0 + (ST + s) * 8; };
    auto tfull = [&](int b) { return bar0 + (2 * ST + b) * 8; };
    auto tempty = [&](int b) { return bar0 + (2 * ST + 2 + b) * 8; };
    const uint32_t tmem_slot = bar0 + (2 * ST + 4) * 8, fail_sm = tmem_slot + 8;
    const int rank = PAIR ? (int)cluster_ctarank() : 0;     // in the pair; 0 issues the products of both
    int* start = reinterpret_cast<int*>(smem_raw + (bar0 + 256 - smem_u32(smem_raw)));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(full(s), PAIR ? 2 : MODE == 1 ? 1 : 1 + 128);     // the pair's first CTA counts for both
            mbar_init(empty(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(tfull(b), 1);
            mbar_init(tempty(b), PAIR ? 2 * EPW : EPW * 32);
        }
        asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(fail_sm), "r"(0u) : "memory");
        mbar_fence_init();
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmW));
    }
    if (warp == 1) {
        if (PAIR) tmem_alloc_pair(tmem_slot, 512);
        else tmem_alloc(tmem_slot, 512);
    }
    if (warp == 0) {            // tiles before every expert, by a scan over the experts
        int run = 0;
        for (int e0 = 0; e0 < a.experts; e0 += 32) {
            const int e = e0 + lane;
            int n = e < a.experts ? (__ldg(a.offsets + e + 1) - __ldg(a.offsets + e) + CTAS * BM - 1) / (CTAS * BM) * a.n_strips : 0;
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
    if (PAIR) cluster_sync();   // the other CTA's barriers and TMEM are there
    tc_fence_after();
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
    const int walkers = (int)gridDim.x / CTAS, me = (int)blockIdx.x / CTAS;
    Walk<CTAS * BM> w{start, a.offsets, 0, walkers, me - walkers, a.n_strips, a.experts, 0, 0, 0};
    const int nk = (a.K + BK - 1) / BK, w_rows = MODE == 0 ? 2 * a.n_out : a.n_out;

    if (warp == 0) {
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 1;
            while (a.polls && w.next() && !tc_failed(fail_sm)) {       // 0: waits that are to run out, nothing is requested
                const int n0 = w.strip * (MODE == 0 ? BN / 2 : BN);
                const int r1 = w.e * w_rows + n0, r2 = r1 + (MODE == 0 ? a.n_out : BN / 2);
                for (int kt = 0; kt < nk; ++kt) {
                    if (!tc_wait(empty(s), ph, fail_sm, a.polls)) {
                        if (PAIR) tell_pair(mapa_shared(fail_sm, rank ^ 1));
                        break;
                    }
                    const uint32_t st = base + s * STAGE;
                    constexpr int bytes = PAIR || MODE == 1 ? STAGE : B_BYTES;
                    if (PAIR) {             // this CTA's rows, and its half of the weight rows
                        const uint32_t bar = mapa_shared(full(s), 0);
                        if (rank == 0) mbar_arrive_expect_tx(full(s), bytes);
                        else mbar_remote_arrive_expect_tx(bar, bytes);
                        tma_load_2d_pair(st + A_BYTES, &tmW, kt * BK, rank == 0 ? r1 : r2, bar);
                        tma_load_2d_pair(st, &tmA, kt * BK, w.m0 + rank * BM, bar);
                    } else {
                        mbar_arrive_expect_tx(full(s), bytes);
                        tma_load_2d(st + A_BYTES, &tmW, kt * BK, r1, full(s));
                        tma_load_2d(st + A_BYTES + B_BYTES / 2, &tmW, kt * BK, r2, full(s));
                        if (MODE == 1) tma_load_2d(st, &tmA, kt * BK, w.m0, full(s));
                    }
                    if (++s == ST) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
            if (tc_failed(fail_sm)) __nanosleep(1000000);   // copies in flight land within microseconds
        }
    } else if (warp == 1) {
        constexpr uint32_t kIdesc = idesc_f16(CTAS * BM, BN, 0, 0, 1);
        int s = 0, j = 0;
        uint32_t ph = 0;
        auto wait = [&](uint32_t bar, uint32_t parity) {
            const bool ok = PAIR ? wait_pair(bar, parity, fail_sm, a.polls) : tc_wait(bar, parity, fail_sm, a.polls);
            if (PAIR && !ok) tell_pair(mapa_shared(fail_sm, rank ^ 1));
            return ok;
        };
        if (rank == 0 && elect_one()) {
            bool ok = true;             // false once a wait ran out, and no further product is issued
            for (; ok && w.next(); ++j) {
                const int b = j & 1;
                ok = wait(tempty(b), ((uint32_t)(j >> 1) & 1u) ^ 1u) && !(PAIR && tc_failed(fail_sm));
                for (int kt = 0; ok && kt < nk; ++kt) {
                    ok = wait(full(s), ph);
                    if (!ok) break;
                    const uint32_t st = base + s * STAGE, mine = empty(s);
                    if (++s == ST) {
                        s = 0;
                        ph ^= 1u;
                    }
                    tc_fence_after();
#pragma unroll
                    for (int ks = 0; ks < BK / 16; ++ks) {
                        const uint64_t da = make_desc(st + ks * 32, 16, 1024), db = make_desc(st + A_BYTES + ks * 32, 16, 1024);
                        if (PAIR) umma_f16_pair(tmem_base + b * BN, da, db, kIdesc, kt > 0 || ks > 0 ? 1u : 0u);
                        else umma_f16(tmem_base + b * BN, da, db, kIdesc, kt > 0 || ks > 0 ? 1u : 0u);
                    }
                    if (PAIR) {
                        umma_commit_pair(mine);
                        if (kt == nk - 1) umma_commit_pair(tfull(b));
                    } else {
                        umma_commit(mine);
                        if (kt == nk - 1) umma_commit(tfull(b));
                    }
                }
            }
        }
    } else if (warp < 2 + EPW) {
        const int qtr = warp & 3, row = qtr * 32 + lane;            // TMEM lane = row of the tile
        const int part = (warp - 2) / 4;                            // which of its columns
        constexpr int OUT = MODE == 0 ? BN / 2 : BN, MINE = OUT / (EPW / 4);
        for (int j = 0; w.next(); ++j) {
            const int b = j & 1, m0 = w.m0 + rank * BM, rows = w.rows - rank * BM;        // this CTA's
            const int n0 = w.strip * OUT, cols = min(OUT, a.n_out - n0);
            int dst = m0 + row;
            float sc = 1.f;
            if (row < rows && (MODE == 1 || a.a_scale)) {
                const int pair = __ldg(a.order + m0 + row);
                if (MODE == 1) dst = pair;
                else sc = __ldg(a.a_scale + pair);
            }
            if (!tc_wait(tfull(b), (uint32_t)(j >> 1) & 1u, fail_sm, a.epilogue_polls[rank]) && PAIR) tell_pair(mapa_shared(fail_sm, rank ^ 1));
            tc_fence_after();
            const bool lost = tc_failed(fail_sm);       // some wait of the CTA ran out: NaN from here on
            const uint32_t acc = tmem_base + ((uint32_t)(qtr * 32) << 16) + b * BN;
            for (int c0 = part * MINE; c0 < min(cols, (part + 1) * MINE); c0 += 32) {
                uint32_t v[32], u[32];
                tmem_ld32(acc + c0, v);
                if (MODE == 0) tmem_ld32(acc + BN / 2 + c0, u);
                tmem_wait_ld();
                if (MODE == 1) {
                    // through shared memory, so that a store instruction writes whole 128-byte row segments
                    const uint32_t ebuf = stage_sm + qtr * 4096;
                    if (lost) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = 0x7fc00000u;
                    }
#pragma unroll
                    for (int p = 0; p < 8; ++p)
                        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(ebuf + lane * 128 + ((p ^ (lane & 7)) << 4)),
                                     "r"(v[4 * p]), "r"(v[4 * p + 1]), "r"(v[4 * p + 2]), "r"(v[4 * p + 3]) : "memory");
                    __syncwarp();
#pragma unroll
                    for (int it = 0; it < 8; ++it) {
                        const int r = it * 4 + (lane >> 3), p = lane & 7, col = c0 + p * 4;
                        const uint4 x = lds_128(ebuf + r * 128 + ((p ^ (r & 7)) << 4));
                        const int to = __shfl_sync(0xffffffffu, dst, r);
                        if (qtr * 32 + r < rows && col < cols) *reinterpret_cast<uint4*>(a.out_f32 + (int64_t)to * a.n_out + n0 + col) = x;
                    }
                } else if (row < rows) {    // every thread its own row, whole 32-byte sectors where its address allows it
                    uint32_t o[16];
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float f[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            f[e] = act_f32(round_bf16(__uint_as_float(v[i + e]) * sc), a.act);
                            if (MODE == 0) f[e] *= round_bf16(__uint_as_float(u[i + e]) * sc);
                        }
                        o[i / 2] = lost ? 0x7fc07fc0u : pack_bf16x2(f[0], f[1]);
                    }
                    bf16_t* out = a.out + (int64_t)dst * a.n_out + n0 + c0;
#pragma unroll
                    for (int p = 0; p < 2; ++p)
                        if (cols - c0 - 16 * p > 0) store_words(out + 16 * p, o + 8 * p, cols - c0 - 16 * p >= 16);
                }
                __syncwarp();
            }
            tc_fence_before();
            if (PAIR) {
                __syncwarp();
                if (lane == 0) mbar_remote_arrive(mapa_shared(tempty(b), 0));
            } else {
                mbar_arrive_cnt(tempty(b));
            }
        }
    } else {
        // MODE 0, 2: 8 lanes bring one row's 128 bytes of a stage; a thread has rows r0 + 16 i and one 16-byte piece of each
        const int t = threadIdx.x - (2 + EPW) * 32, piece = t & 7, r0 = t >> 3;
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
    if (warp == 1 && tc_failed(fail_sm)) {      // in any of the CTA's roles: products and copies in flight end within microseconds
        __nanosleep(1000000);
        if (lane == 0) atomicAdd(&g_errors, 1);
        __syncwarp();
    }
    if (PAIR) cluster_sync();   // the other CTA may still read its accumulators or signal this one's barriers
    if (warp == 1) {
        tc_fence_after();
        if (PAIR) tmem_dealloc_pair(tmem_base, 512);
        else tmem_dealloc(tmem_base, 512);
    }
}

template <int MODE, int CTAS>
static int launch(const CUtensorMap& tmA, const CUtensorMap& tmW, const Args& a, int pairs, cudaStream_t st) {
    const size_t smem = smem_for(a.experts, CTAS, MODE);
    cudaError_t e = cudaFuncSetAttribute(grouped_tc_kernel<MODE, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int64_t most = (int64_t)(pairs / (CTAS * BM) + a.experts) * a.n_strips;
    const int walkers = device_info().sm_count / CTAS;
    const unsigned grid = (unsigned)(CTAS * (most < walkers ? most : walkers));
    if (CTAS == 1) {
        grouped_tc_kernel<MODE, CTAS><<<grid, threads_for(MODE, CTAS), smem, st>>>(tmA, tmW, a);
        PA_RETURN_LAUNCH_STATUS();
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads_for(MODE, CTAS));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CTAS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, grouped_tc_kernel<MODE, CTAS>, tmA, tmW, a);
}

// The token rows of the pairs in sorted order, 16 bytes a thread.  *count: how many pairs the sort gave a place; a pair whose id belongs
// to no expert (an identity output) has none, so order and out end there and may hold anything behind.
__global__ void __launch_bounds__(256) sorted_rows_kernel(const uint4* __restrict__ A, int64_t lda, const int32_t* __restrict__ order, int top,
                                                          const int32_t* __restrict__ count, int words, uint4* __restrict__ out) {
    const int64_t i0 = (int64_t)blockIdx.x * 256 + threadIdx.x, n = (int64_t)__ldg(count) * words, step = (int64_t)gridDim.x * 256;
    for (int64_t i = i0; i < n; i += 4 * step) {
        uint4 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int64_t j = i + k * step;
            if (j < n) v[k] = __ldg(A + (int64_t)(__ldg(order + j / words) / top) * lda + j % words);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int64_t j = i + k * step;
            if (j < n) out[j] = v[k];
        }
    }
}

}  // namespace mtc

// Whether a launch of this many pairs can go by pairs of CTAs: enough of them, and rows enough for tiles of 256.
bool grouped_tc_pairs_up(int pairs, int experts) { return pairs >= mtc::kPairFrom && (int64_t)pairs >= 256ll * experts; }

// Whether it should.  A tile of a pair takes 0.8 of the time of the two tiles of one CTA each, against which stand (us of one CTA a tile and
// of pairs, with the sorted rows where they are needed, 8 experts):
//  - a last tile of 256 that is half empty, for every expert: 1024 rows each are asked for (16 experts, down with ff 1024, width 2048:
//    8192 pairs 43.6 and 44.8, 16384 pairs 74.6 and 67.1);
//  - walkers with one round of tiles and little more: two are asked for (down, ff 1024, width 1024: 8192 pairs = 128 tiles 21.8 and 22.2,
//    12288 pairs 32.6 and 30.6);
//  - a tile's start and end, which few columns do not hide, and the activations: down asks for 1024 columns (8192 pairs, width 2048, ff 512:
//    27.9 and 30.2, ff 1024: 41.9 and 38.0), gate / up for 2048 (16384 pairs, ff 2048, width 1024: 146 and 169, width 2048: 243 and 220);
//  - for gate / up the copy of the rows, which the tiles of a row share: twelve strips (16384 pairs, width 2048, ff 512: 75 and 86, ff 1024: 134
//    and 131, ff 1536: 184 and 179; width 4096, ff 1024: 240 and 239, ff 2048: 456 and 420).
bool grouped_tc_pairs_pay(int mode, int pairs, int experts, int K, int n_out) {
    const int strip = mode == 0 ? mtc::BN / 2 : mtc::BN, strips = (n_out + strip - 1) / strip;
    return grouped_tc_pairs_up(pairs, experts) && (int64_t)pairs >= 1024ll * experts && (int64_t)(pairs / 256) * strips >= device_info().sm_count &&
           (mode == 1 ? K >= 1024 : K >= 2048 && strips >= 12);
}

// mode 0: gate / up pairs, 1: down (rows scattered to (row, choice) order as float), 2: up.  pair: by pairs of CTAs, which modes 0 and 2
// do where they are given scratch for the sorted rows.  PA_ERR_UNSUPPORTED: the caller's other kernels serve these operands.
int grouped_tc_launch(int mode, const void* A, int64_t lda, const void* W, int K, int n_out, int experts, const int32_t* order,
                      const float* a_scale, int top, const int32_t* offsets, int pairs, int act, void* out, cudaStream_t st, bool pair, void* rows, int polls,
                      int first_polls, int second_polls) {
    using namespace mtc;
    const int64_t w_rows = (int64_t)experts * n_out * (mode == 0 ? 2 : 1);
    if (K % 8 || n_out % 8 || experts > kMostExperts || w_rows >= 0x7fffff00ll || (uintptr_t)out % 16) return PA_ERR_UNSUPPORTED;
    if ((uintptr_t)A % 16 || (uintptr_t)W % 16 || lda % 8) return PA_ERR_UNSUPPORTED;
    CUtensorMap tmA, tmW;
    if (!make_bf16_map(&tmW, W, w_rows, K, K, BN / 2)) return PA_ERR_UNSUPPORTED;
    tmA = tmW;
    if (mode != 1 && (!rows || (uintptr_t)rows % 16)) pair = false;
    if (mode == 1 && !make_bf16_map(&tmA, A, pairs, K, lda, BM)) return PA_ERR_UNSUPPORTED;
    if (mode != 1 && pair) {
        if (!make_bf16_map(&tmA, rows, pairs, K, K, BM)) return PA_ERR_UNSUPPORTED;
        const int64_t blocks = ((int64_t)pairs * (K / 8) + 1023) / 1024, most = 8 * device_info().sm_count;
        sorted_rows_kernel<<<(unsigned)(blocks < most ? blocks : most), 256, 0, st>>>(static_cast<const uint4*>(A), lda / 8, order, top, offsets + experts, K / 8,
                                                                                      static_cast<uint4*>(rows));
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return (int)e;
    }
    const int strip = mode == 0 ? BN / 2 : BN;
    Args a{static_cast<const bf16_t*>(A), lda, K, n_out, experts, top, act, (n_out + strip - 1) / strip, order, a_scale, offsets,
           static_cast<bf16_t*>(out), static_cast<float*>(out), (uint32_t)polls, {(uint32_t)first_polls, (uint32_t)second_polls}};
    if (mode == 0) return pair ? launch<0, 2>(tmA, tmW, a, pairs, st) : launch<0, 1>(tmA, tmW, a, pairs, st);
    if (mode == 1) return pair ? launch<1, 2>(tmA, tmW, a, pairs, st) : launch<1, 1>(tmA, tmW, a, pairs, st);
    return pair ? launch<2, 2>(tmA, tmW, a, pairs, st) : launch<2, 1>(tmA, tmW, a, pairs, st);
}

}  // namespace pa

using namespace pa;

PA_API int pa_moe_grouped_waits(int mode, const void* d_a, int64_t lda, const void* d_w, int K, int n_out, int experts, const int32_t* d_order,
                                const float* d_a_scale, int top, const int32_t* d_meta, int pairs, int act, void* d_out, void* d_rows,
                                size_t rows_bytes, int polls, int first_polls, int second_polls, pa_stream_t stream) {
    PA_CHECK_ARG(mode >= 0 && mode <= 2 && d_a && d_w && d_order && d_meta && d_out && K > 0 && n_out > 0 && experts > 0 && top > 0 && pairs >= 0 &&
                 act >= 0 && act <= 2 && polls >= 0 && first_polls >= 0 && second_polls >= 0);
    if (pairs == 0) return PA_OK;
    if (d_rows && rows_bytes < (size_t)pairs * K * 2) return PA_ERR_WORKSPACE;
    return grouped_tc_launch(mode, d_a, lda, d_w, K, n_out, experts, d_order, d_a_scale, top, d_meta, pairs, act, d_out, as_stream(stream),
                             grouped_tc_pairs_up(pairs, experts), d_rows, polls, first_polls, second_polls);
}

PA_API int pa_moe_grouped_polls(int mode, const void* d_a, int64_t lda, const void* d_w, int K, int n_out, int experts, const int32_t* d_order,
                                const float* d_a_scale, int top, const int32_t* d_meta, int pairs, int act, void* d_out, int polls,
                                pa_stream_t stream) {
    return pa_moe_grouped_waits(mode, d_a, lda, d_w, K, n_out, experts, d_order, d_a_scale, top, d_meta, pairs, act, d_out, nullptr, 0, polls, polls,
                                polls, stream);
}

PA_API int pa_moe_tc_errors(int* host_count) {
    PA_CHECK_ARG(host_count);
    return (int)cudaMemcpyFromSymbol(host_count, pa::mtc::g_errors, sizeof(int));
}
