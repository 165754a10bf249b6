// attention_tc.cu -- softmax attention of prompt portions on the 5th-generation tensor cores (tcgen05.mma kind::f16, bfloat16
// operands, float accumulators in TMEM), for the ragged batches of the config-driven models.  Two forms of keys and values:
//
//   paged   one row per (token, kv head) in the page pools of masked_attention.cu, located through the page table; causal,
//           window (with kept first positions) and chunk masks, temperature, soft cap, distance biases, sinks, turned-back and
//           gated outputs, as described there
//   dense   keys and values of every head in plain buffers (latent attention in its expanded form, see
//           pa_latent_attention_expanded): a key is [kn columns of its head | rot columns all heads share]
//
// One CTA = NQ tiles of 128 query rows that share every staged key and value byte.  A row is a (query head, token) pair: the
// heads of one kv head are stacked (TB tokens x hg heads = 128 NQ rows), so with grouped heads a 64-token work item already
// fills the tensor core's 128 lanes twice and K/V are staged once for four heads; TB rows of one head are a multiple of 32, so a
// warp's rows have one head.  Persistent: a CTA walks its work items (Walk), and the barriers, the key ring and the score buffers run on
// through them, so that an item's keys, queries and first scores come under the end of the one before.  Keys are consumed in tiles of 64:
//   warps 0-3 (4-7)  softmax of query tile 0 (1), one thread per row = TMEM lane: tcgen05.ld of its 64 scores, modifiers and
//                    mask, online softmax in registers, P back to TMEM as bfloat16 over the scores it came from
//   next NQ warps    one elected thread each issues its tile's  S = Q K^T  (M128 N64, double buffered in TMEM, tile i + 1 under
//                    the softmax of tile i)  and  O += P V  (A operand from TMEM, V as the MN-major B operand)
//   last warp        producer: TMA boxes into a ring of 2 or 3 stages, SWIZZLE_128B (16-token boxes per page unit, or 64 rows)
// O keeps a per-row reference maximum that is raised only when a tile exceeds it by more than 2^8 (P stays below 2^8, and l and
// O share the reference, so O / l does not depend on it): rows are rescaled a few times instead of once per tile.
//
// What bounds it: the hand-offs between the pipes and the exponentials.  Per 64 keys and both query tiles the tensor pipe needs 1235 cycles
// (dim 128; 1620 at dim 192: an N = 64 product reads 6 KB of shared memory for 32 cycles of arithmetic) and the special-function
// unit 1024; a step takes 1940.  The two tiles' softmax warps run in step, 670 cycles of theirs are waits and TMEM accesses, and
// an issuing warp spends 780 on waits behind its own commits.  Measured, 4 x 2048 tokens causal: 16 query / 4 kv heads of 128
// paged 97 us = 710 TFLOP/s (a CTA per item, whose set-up and query load nothing overlapped, and the maximum before the
// exponentials: 111 us; mma.sync kernel 918 us); latent attention at 16 heads of 128 + 64 / 128, five ragged portions 107 us, and 38
// us for gathering the rows and building keys and values (absorbed form on mma.sync 1360 us).
// Slower: the two tiles' exponentials in turns (112 us: the issuing warps come too late), one issuing warp per kind of product
// instead of one per tile (108 to 110 us), tiles of 128 keys (150 us where this took 123), a quarter of the exponentials as a
// polynomial on the FMA pipe (105 and 101 us), the output 64 columns at a time (101 us).
//
// Every wait is bounded: on a protocol error the CTA raises a flag (pa_attention_tc_errors), waits for its copies, frees its
// TMEM and leaves NaN in its rows.
#include "masked_attention.cuh"
#include "softmax_tile.cuh"
#include "tcgen05_utils.cuh"

namespace pa {
namespace atc {

using namespace tc;

constexpr int QT = 128, KT = 64;

struct Args {
    MaskAttnParams p;
    int tb, hg, hchunks;     // tokens per head block, heads per CTA, head chunks per kv head
    int kn;                  // dense: key columns per head (multiple of 64); the shared block starts at k2_col of its buffer
    int k2_col;
    int upt;                 // paged: 16-token units per page
    int total_rows;          // rows of the pools: a box there is all zeros (out-of-bounds fill)
    int items;               // work items: tiles x units
};

__device__ int g_errors;

__host__ __device__ constexpr int q_bytes(int kb) { return kb * QT * 128; }
__host__ __device__ constexpr int stage_bytes(int kb, int vb) { return (kb + vb) * KT * 128; }
__host__ __device__ constexpr int stages_for(int kb, int nq) { return nq == 2 || kb == 3 ? 3 : 2; }
__host__ __device__ constexpr int threads_for(int nq) { return (5 * nq + 1) * 32; }
// Query buffers: two where they fit, so that the next item's queries come under the current one's products.  A CTA with a table of
// distance biases has no next item, and the table (up to 40 KB) takes the second one's place.
__host__ __device__ constexpr int q_bufs(int kb, int nq, bool table) { return nq == 2 && kb < 3 && !table ? 2 : 1; }
// barriers: kv_full, kv_empty [stage]; per query tile s_full, p_full, o_full [2], q_ready, q_free [2]
__host__ __device__ constexpr int nbar_for(int kb, int nq) { return 2 * stages_for(kb, nq) + 10 * nq; }
constexpr size_t smem_for(int kb, int vb, int nq, int qb) {
    return (size_t)nq * qb * q_bytes(kb) + stages_for(kb, nq) * stage_bytes(kb, vb) + nbar_for(kb, nq) * 8 + 8 + 4 + 4 * 4 + 1024;
}

// 32 bfloat16 numbers: two 32-byte sectors, each by one store where the row's address allows it
__device__ __forceinline__ void store_row32(bf16_t* dst, const uint32_t (&w)[16]) {
    if (((uintptr_t)dst & 31) == 0) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
            asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst + 16 * h), "r"(w[8 * h]), "r"(w[8 * h + 1]),
                         "r"(w[8 * h + 2]), "r"(w[8 * h + 3]), "r"(w[8 * h + 4]), "r"(w[8 * h + 5]), "r"(w[8 * h + 6]), "r"(w[8 * h + 7]) : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) reinterpret_cast<uint4*>(dst)[j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
    }
}

// One work item: the rows of a CTA's query tiles and the key tiles they see
template <int NQ>
struct Item {
    int row0, ntok, slot, pos0, g, h0, hend, kmax_c, n_tiles;
    int kmaxs[NQ], nts[NQ];
    MaSteps steps;
    bool whole;             // no box of query rows reaches past the item's
};
// entry x of an array that stays in registers
template <int NQ>
__device__ __forceinline__ int of_tile(const int (&v)[NQ], int x) { return NQ == 1 || x == 0 ? v[0] : v[NQ - 1]; }
struct RawItem { int row0, ntok, slot, pos0; };

// The walk over a CTA's items.  They are in order of falling length; every second round goes backwards through the CTAs, so that
// their sums are close.  The numbers of the next item are fetched an item ahead.
template <int NQ>
struct Walk {
    const Args& a;
    int round, idx;
    RawItem raw;
    __device__ __forceinline__ Walk(const Args& args) : a(args), round(0), idx(blockIdx.x) { fetch(); }
    __device__ __forceinline__ void fetch() {
        if (idx < 0) return;
        const int* t = a.p.tiles + 4 * (idx / (a.p.num_kv_heads * a.hchunks));
        raw = RawItem{__ldg(t), __ldg(t + 1), __ldg(t + 2), __ldg(t + 3)};
    }
    __device__ __forceinline__ bool next(Item<NQ>& it) {
        if (idx < 0) return false;
        const MaskAttnParams& p = a.p;
        const int un = idx % (p.num_kv_heads * a.hchunks), hpg = p.heads / p.num_kv_heads;
        it.row0 = raw.row0;
        it.ntok = min(raw.ntok, a.tb);
        it.slot = raw.slot;
        it.pos0 = raw.pos0;
        it.whole = it.ntok == a.tb;
        it.g = un / a.hchunks;
        it.h0 = it.g * hpg + un % a.hchunks * a.hg;
        it.hend = min(it.h0 + a.hg, (it.g + 1) * hpg);
        it.kmax_c = 0;
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int tok0 = x * QT % a.tb;
            const int last = min(it.ntok, tok0 + min(a.tb, QT)) - 1;
            it.kmaxs[x] = tok0 < it.ntok && it.h0 + x * QT / a.tb < it.hend ? it.pos0 + last + 1 : 0;
            it.kmax_c = max(it.kmax_c, it.kmaxs[x]);
        }
        it.steps = ma_steps(p, ma_first_key(p, it.pos0), it.kmax_c, KT);
        it.n_tiles = 0;
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            it.nts[x] = it.kmaxs[x] > 0 ? it.steps.head + (it.kmaxs[x] + KT - 1) / KT - it.steps.body0 : 0;
            it.n_tiles = max(it.n_tiles, it.nts[x]);
        }
        ++round;
        const int64_t at = (int64_t)round * gridDim.x + (round & 1 ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
        idx = at < a.items ? (int)at : -1;
        fetch();
        return true;
    }
};

// KB / VB: blocks of 64 columns of a key / a value; MOD: the score has more than a factor (soft cap or distance bias)
// QD: columns of a query (the last block may be part of one); QB: query buffers
template <int KB, int VB, int NQ, bool DENSE, bool MOD, int QD, int QB>
__global__ void __launch_bounds__(threads_for(NQ), NQ == 1 && KB < 3 ? 2 : 1)
attention_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmK2,
                    const __grid_constant__ CUtensorMap tmV, const Args a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    constexpr int ST = stages_for(KB, NQ), NBAR = nbar_for(KB, NQ), TMEM_COLS = NQ * 256, D = VB * 64;
    constexpr int Q_BYTES = q_bytes(KB), K_BYTES = KB * KT * 128, STAGE = stage_bytes(KB, VB);
    constexpr int W_MMA = 4 * NQ, W_PROD = 5 * NQ;
    constexpr float kLog2e = 1.4426950408889634f;
    const MaskAttnParams& p = a.p;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t kv_sm = base + NQ * QB * Q_BYTES, bar0 = kv_sm + ST * STAGE;
    auto q_sm = [&](int x, int buf) { return base + (x * QB + buf) * Q_BYTES; };
    auto kv_full = [&](int s) { return bar0 + s * 8; };
    auto kv_empty = [&](int s) { return bar0 + (ST + s) * 8; };
    // two barriers each, a tile's n-th key tile on barrier n & 1 (n counts on through the items): with S one tile ahead, waiter and
    // signaller are at most one phase apart
    auto s_full = [&](int x, int b) { return bar0 + (2 * ST + 10 * x + b) * 8; };
    auto p_full = [&](int x, int b) { return bar0 + (2 * ST + 10 * x + 2 + b) * 8; };
    auto o_full = [&](int x, int b) { return bar0 + (2 * ST + 10 * x + 4 + b) * 8; };
    auto q_ready = [&](int x, int b) { return bar0 + (2 * ST + 10 * x + 6 + b) * 8; };
    auto q_free = [&](int x, int b) { return bar0 + (2 * ST + 10 * x + 8 + b) * 8; };
    const uint32_t tmem_slot = bar0 + NBAR * 8, fail_sm = tmem_slot + 8, meta_sm = fail_sm + 4;
    float* bias_sm = reinterpret_cast<float*>(smem_raw + (meta_sm + 16 - smem_u32(smem_raw)));

    auto failed = [&] { return tc_failed(fail_sm); };
    auto wait = [&](uint32_t bar, uint32_t parity) { tc_wait(bar, parity, fail_sm); };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(kv_full(s), 1);
            mbar_init(kv_empty(s), NQ);
        }
        for (int x = 0; x < NQ; ++x)
            for (int b = 0; b < 2; ++b) {
                mbar_init(s_full(x, b), 1);
                mbar_init(p_full(x, b), QT);
                mbar_init(o_full(x, b), 1);
                mbar_init(q_ready(x, b), 1);
                mbar_init(q_free(x, b), 1);
            }
        asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(fail_sm), "r"(0u) : "memory");
        mbar_fence_init();
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmK));
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmV));
        if (DENSE) asm volatile("prefetch.tensormap [%0];" ::"l"(&tmK2));
    }
    if (warp == W_MMA) tmem_alloc(tmem_slot, TMEM_COLS);
    Walk<NQ> walk(a);
    Item<NQ> it;
    if (MOD && p.bias_kind == 2) {          // its CTAs have one item each
        Walk<NQ> mine(a);
        mine.next(it);
        const int nh = it.hend - it.h0;
        for (int i = threadIdx.x; i < nh * p.bias_len; i += blockDim.x)
            bias_sm[i] = p.bias[(int64_t)(i % p.bias_len) * p.heads + it.h0 + i / p.bias_len];
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));

    if (warp == W_PROD) {
        if (elect_one()) {
            int qn[NQ];                     // items so far in which a query tile has rows: its next buffer and phase
#pragma unroll
            for (int x = 0; x < NQ; ++x) qn[x] = 0;
            auto load_queries = [&](const Item<NQ>& q) {        // 64 rows of one head x 64 columns a box
#pragma unroll
                for (int x = 0; x < NQ; ++x) {
                    if (q.nts[x] == 0) continue;
                    const int buf = qn[x] % QB, nb = min(2, ((q.hend - q.h0) * a.tb - x * QT) / 64);     // blocks of 64 rows with a head
                    const uint32_t ph = (uint32_t)(qn[x]++ / QB & 1) ^ 1u;
                    if (!q.whole) continue;                     // the softmax threads bring these rows
                    wait(q_free(x, buf), ph);
                    if (failed()) return;
                    mbar_arrive_expect_tx(q_ready(x, buf), nb * KB * 8192);
                    for (int b = 0; b < nb; ++b) {
                        const int r = x * QT + b * 64, col = p.q_off + (q.h0 + r / a.tb) * QD;
#pragma unroll
                        for (int kb = 0; kb < KB; ++kb)
                            tma_load_2d(q_sm(x, buf) + kb * (QT * 128) + b * 8192, &tmQ, col + kb * 64, q.row0 + r % a.tb, q_ready(x, buf));
                    }
                }
            };
            int s = 0;
            uint32_t ph = 1;
            bool more = walk.next(it), ok = true;
            if (QB == 2) load_queries(it);
            while (more && ok) {
                const int32_t* trow = DENSE ? nullptr : p.table + ((int64_t)it.slot * p.num_kv_heads + it.g) * p.num_tiles;
                const bool slot_ok = DENSE || (unsigned)it.slot < (unsigned)p.num_slots;
                int pgn[4];
                auto load_pages = [&](int i) {
                    const int u0 = it.steps.step(i) * 4;
#pragma unroll
                    for (int uu = 0; uu < 4; ++uu) {
                        const int u = u0 + uu, t = u / a.upt;
                        int page = slot_ok && u * 16 < it.kmax_c && t < p.num_tiles ? __ldg(trow + t) : -1;
                        if ((unsigned)page >= (unsigned)p.total_pages) page = -1;
                        pgn[uu] = page >= 0 ? page * p.tile_size + (u - t * a.upt) * 16 : -1;
                    }
                };
                if (!DENSE) load_pages(0);
                Item<NQ> nxt;
                const bool has_next = walk.next(nxt);
                for (int i = 0; i < it.n_tiles; ++i) {
                    int r[4];
                    uint32_t mask = 0;
                    if (!DENSE) {
#pragma unroll
                        for (int uu = 0; uu < 4; ++uu) {
                            r[uu] = pgn[uu] >= 0 ? pgn[uu] : a.total_rows;     // unmapped: zeros, and its scores are masked
                            mask |= (pgn[uu] >= 0 ? 1u : 0u) << uu;
                        }
                        if (i + 1 < it.n_tiles) load_pages(i + 1);
                    }
                    wait(kv_empty(s), ph);
                    if (failed()) {
                        ok = false;
                        break;
                    }
                    const uint32_t st = kv_sm + s * STAGE;
                    if (!DENSE) asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(meta_sm + s * 4), "r"(mask) : "memory");
                    mbar_arrive_expect_tx(kv_full(s), STAGE);
                    if (DENSE) {
                        const int row = it.slot + it.steps.step(i) * KT;
#pragma unroll
                        for (int kb = 0; kb < KB - 1; ++kb) tma_load_2d(st + kb * 8192, &tmK, it.h0 * a.kn + kb * 64, row, kv_full(s));
                        tma_load_2d(st + (KB - 1) * 8192, &tmK2, a.k2_col, row, kv_full(s));
#pragma unroll
                        for (int vb = 0; vb < VB; ++vb) tma_load_2d(st + K_BYTES + vb * 8192, &tmV, it.h0 * D + vb * 64, row, kv_full(s));
                    } else {
#pragma unroll
                        for (int uu = 0; uu < 4; ++uu)
#pragma unroll
                            for (int kb = 0; kb < KB; ++kb) tma_load_2d(st + kb * 8192 + uu * 2048, &tmK, kb * 64, r[uu], kv_full(s));
#pragma unroll
                        for (int uu = 0; uu < 4; ++uu)
#pragma unroll
                            for (int vb = 0; vb < VB; ++vb) tma_load_2d(st + K_BYTES + vb * 8192 + uu * 2048, &tmV, vb * 64, r[uu], kv_full(s));
                    }
                    if (++s == ST) {
                        s = 0;
                        ph ^= 1u;
                    }
                    // the queries: with one buffer behind the item's first keys; with two, the next item's once this one has
                    // filled the ring (their buffer's last products are over by then)
                    if (QB == 1 && i == 0) load_queries(it);
                    if (QB == 2 && has_next && i == min(ST - 1, it.n_tiles - 1)) load_queries(nxt);
                }
                if (QB == 2 && has_next && ok && it.n_tiles == 0) load_queries(nxt);     // an item of no tokens has no keys to wait behind
                it = nxt;
                more = has_next;
            }
            if (failed()) {     // let the copies in flight land before the CTA's shared memory goes away
                for (int b = 0; b < ST; ++b) tc_let_land(kv_full(b), b < s ? ph ^ 1u : ph);
                __nanosleep(1000000);       // the queries: microseconds
            }
        }
    } else if (warp >= W_MMA) {
        constexpr uint32_t kIdescS = idesc_f16(QT, KT, 0, 0, 1), kIdescO = idesc_f16(QT, D, 0, 1, 1);
        const int x = warp - W_MMA;
        int s = 0, n = 0, qn = 0;           // stage; key tiles and items of this query tile so far
        uint32_t kv_ph = 0;
        while (walk.next(it)) {
            const int ntx = of_tile(it.nts, x), kmx = of_tile(it.kmaxs, x), qbuf = qn % QB;
            auto issue_S = [&](int i, int stage) {
                if (elect_one()) {
                    const uint32_t st = kv_sm + stage * STAGE, qx = q_sm(x, qbuf);
                    const int b = (n + i) & 1;
#pragma unroll
                    for (int ks = 0; ks < QD / 16; ++ks) {
                        const uint64_t da = make_desc(qx + (ks >> 2) * (QT * 128) + (ks & 3) * 32, 16, 1024);
                        const uint64_t db = make_desc(st + (ks >> 2) * (KT * 128) + (ks & 3) * 32, 16, 1024);
                        umma_f16(tmem_base + x * 2 * KT + b * KT, da, db, kIdescS, ks > 0 ? 1u : 0u);
                    }
                    umma_commit(s_full(x, b));
                    if (i == ntx - 1) umma_commit(q_free(x, qbuf));
                }
                __syncwarp();
            };
            if (it.n_tiles > 0) {
                wait(kv_full(s), kv_ph);
                if (ntx > 0) {
                    wait(q_ready(x, qbuf), (uint32_t)(qn / QB) & 1u);
                    tc_fence_after();
                    issue_S(0, s);
                }
            }
            for (int i = 0; i < it.n_tiles; ++i) {
                const int s_next = (s + 1 == ST) ? 0 : s + 1;
                if (i + 1 < it.n_tiles) {   // every issuer waits for every stage: its arrival on kv_empty belongs to THIS use of it
                    wait(kv_full(s_next), (s + 1 == ST) ? (kv_ph ^ 1u) : kv_ph);
                    tc_fence_after();
                    if (i + 1 < ntx) issue_S(i + 1, s_next);
                }
                if (i < ntx) {
                    const uint32_t st = kv_sm + s * STAGE;
                    const int b = (n + i) & 1, kp0 = it.steps.step(i) * KT, nvalid_c = min(KT, it.kmax_c - kp0);
                    if (nvalid_c & 15) {
                        // value rows past the last key may hold anything (0 x NaN = NaN): zeros (both issuers write the same)
                        const int r1 = (nvalid_c + 15) & ~15;
                        for (int idx = lane; idx < (r1 - nvalid_c) * (D / 8); idx += 32) {
                            const int r = nvalid_c + idx / (D / 8), c = idx % (D / 8);
                            const uint32_t addr = st + K_BYTES + (c >> 3) * 8192 + r * 128 + (((c & 7) ^ (r & 7)) << 4);
                            asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(addr), "r"(0u) : "memory");
                        }
                        fence_proxy_async();
                        __syncwarp();
                    }
                    // every row's thread has also read the last item's O by the time it hands over an item's first P
                    wait(p_full(x, b), (uint32_t)((n + i) >> 1) & 1u);
                    tc_fence_after();
                    if (elect_one()) {
                        const int ksteps = (min(KT, kmx - kp0) + 15) >> 4;  // keys past the tile's last token contribute nothing
                        for (int ks = 0; ks < ksteps; ++ks) {
                            const uint32_t ta = tmem_base + x * 2 * KT + b * KT + ks * 8;
                            const uint64_t db = make_desc(st + K_BYTES + ks * 2048, 8192, 1024);
                            umma_f16_ts(tmem_base + NQ * 2 * KT + x * D, ta, db, kIdescO, (i > 0 || ks > 0) ? 1u : 0u);
                        }
                        umma_commit(o_full(x, b));
                    }
                    __syncwarp();
                }
                if (elect_one()) umma_commit(kv_empty(s));
                __syncwarp();
                if (++s == ST) {
                    s = 0;
                    kv_ph ^= 1u;
                }
            }
            n += ntx;
            qn += ntx > 0;
        }
    } else {
        // ---- softmax: one thread per query row
        const int x = warp >> 2, qtr = warp & 3;
        const int wrow = x * QT + qtr * 32, tokw = wrow % a.tb, tok = tokw + lane;   // first row of this warp (its rows have one head)
        const uint32_t lane_base = (uint32_t)(qtr * 32) << 16;
        const uint32_t s_addr = tmem_base + lane_base + x * 2 * KT;
        const uint32_t o_addr = tmem_base + lane_base + NQ * 2 * KT + x * D;
        const int keep = p.mask_kind == 1 ? p.mask_keep : 0;
        const float inv_cap = MOD && p.softcap > 0.f ? 1.0f / p.softcap : 0.f;
        const float* brow = bias_sm + (int64_t)(wrow / a.tb) * p.bias_len;
        // P.V(t) is complete.  Unambiguous without consuming every phase: S(n) follows P.V(n - 2) on the pipe, so by the time a
        // thread works on tile n the barrier of P.V(n - 1) is in the phase asked for or just past it.
        auto pv_done = [&](int t) { wait(o_full(x, t & 1), (uint32_t)((t >> 1) & 1)); };
        int st_i = 0, n = 0, qn = 0;
        while (walk.next(it)) {
        const int nt = of_tile(it.nts, x), skipped = it.n_tiles - nt;
        if (nt == 0) {
            st_i = (st_i + skipped) % ST;
            continue;
        }
        const int head = min(it.h0 + wrow / a.tb, it.hend - 1);
        const int nw = it.h0 + wrow / a.tb < it.hend ? it.ntok : 0;     // a half of a tile may be past the last head: no rows
        const int qpos = tok < nw ? it.pos0 + tok : -1;
        if (!it.whole) {
            // the warp's query rows into the swizzled K-major A tile, whose last products this thread has seen complete
            const bf16_t* qsrc = static_cast<const bf16_t*>(p.q) + p.q_off + (int64_t)head * QD;
            const uint32_t qx = q_sm(x, qn % QB);
            constexpr int CH = QD / 8, PER = CH <= 32 ? 8 : 4;     // 16-byte pieces of a row; loads in flight per lane
#pragma unroll 1
            for (int i0 = 0; i0 < 32 * CH; i0 += 32 * PER) {
                uint4 v[PER];
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    const int idx = i0 + j * 32 + lane, r = idx / CH, c = idx % CH;
                    v[j] = make_uint4(0u, 0u, 0u, 0u);
                    if (r < 32 && tokw + r < nw) v[j] = __ldg(reinterpret_cast<const uint4*>(qsrc + (int64_t)(it.row0 + tokw + r) * p.q_stride) + c);
                }
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    const int idx = i0 + j * 32 + lane, r = idx / CH, c = idx % CH, rr = qtr * 32 + r;
                    if (r >= 32) continue;
                    const uint32_t addr = qx + (c >> 3) * (QT * 128) + rr * 128 + (((c & 7) ^ (rr & 7)) << 4);
                    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v[j].x), "r"(v[j].y), "r"(v[j].z), "r"(v[j].w) : "memory");
                }
            }
            fence_proxy_async();
            if (x == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
            else asm volatile("bar.sync 2, 128;" ::: "memory");
            if (qtr == 0 && lane == 0) mbar_arrive_cnt(q_ready(x, qn % QB));
        }
        const int rlo = qpos >= 0 ? ma_first_key(p, qpos) : 0;
        const float fs = p.scale * (p.head_scale ? p.head_scale[head] : 1.f);
        // MOD: scores become log2-domain numbers one by one; else they stay raw and the factor (made positive: a raw score
        // changes sign with it) enters the exponent's multiply-add
        const bool flip = !MOD && fs < 0.f;
        const float fe = MOD ? 1.f : fmaxf(fabsf(fs) * kLog2e, 1e-30f);
        const float slope = MOD && p.bias_kind == 1 ? p.bias[head] : 0.f;
        const float hb = p.head_bias ? p.head_bias[head] : 0.f;
        float m_ref = -INFINITY, l_run = 0.f;
#pragma unroll 1
        for (int i = 0; i < nt; ++i) {
            const int sb = (n + i) & 1, kp0 = it.steps.step(i) * KT;
            wait(s_full(x, sb), (uint32_t)((n + i) >> 1) & 1u);
            tc_fence_after();
            uint32_t mapped = 15u;      // the producer's note about this stage, older than the scores
            if (!DENSE) asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(mapped) : "r"(meta_sm + st_i * 4) : "memory");
            uint32_t sr[2][32];
            tmem_ld32(s_addr + sb * KT, sr[0]);
            tmem_ld32(s_addr + sb * KT + 32, sr[1]);
            tmem_wait_ld();
            const bool full = kp0 + KT - 1 <= qpos && (kp0 >= rlo || kp0 + KT <= keep) && mapped == 15u;
            if (MOD) {
#pragma unroll
                for (int k = 0; k < KT; ++k) {
                    float v = __uint_as_float(sr[k >> 5][k & 31]) * fs;
                    if (p.softcap > 0.f) v = p.softcap * ma_tanh(v * inv_cap);
                    const int dist = qpos - kp0 - k;
                    if (p.bias_kind == 1) v -= slope * (float)dist;
                    else if (p.bias_kind == 2) v += brow[max(0, min(dist, p.bias_len - 1))];
                    sr[k >> 5][k & 31] = __float_as_uint((v + hb) * kLog2e);
                }
            } else if (flip) {
#pragma unroll
                for (int k = 0; k < KT; ++k) sr[k >> 5][k & 31] ^= 0x80000000u;
            }
            if (!full) {
#pragma unroll
                for (int k = 0; k < KT; ++k) {
                    const int j = kp0 + k;
                    const bool vis = j <= qpos && (j >= rlo || j < keep) && ((mapped >> (k >> 4)) & 1u);
                    if (!vis) sr[k >> 5][k & 31] = 0xff800000u;
                }
            }
            // A row's reference rarely moves, so a tile that all rows of the warp see whole takes the exponentials with the one at
            // hand, without waiting for the maximum, and the scores' first half is on its way to TMEM under the second's exponentials
            auto pack = [](float lo, float hi) { return pack_bf16x2(lo, hi); };
            uint32_t w0[16], w1[16];
            uint64_t acc[2] = {0ull, 0ull};
            if (__all_sync(0xffffffffu, full && m_ref > -INFINITY)) {
                smx::exp_half(sr[0], fe, m_ref, w0, acc, pack);
                tmem_st16(s_addr + sb * KT, w0);
                const float mx = smx::row_max(sr) * fe;
                smx::exp_half(sr[1], fe, m_ref, w1, acc, pack);
                if (!__any_sync(0xffffffffu, mx > m_ref + 8.f)) {
                    tmem_st16(s_addr + sb * KT + 16, w1);
                    l_run += smx::sum_of(acc);
                    tmem_wait_st();
                    tc_fence_before();
                    mbar_arrive_cnt(p_full(x, sb));
                    if (++st_i == ST) st_i = 0;
                    continue;
                }
                acc[0] = acc[1] = 0ull;
                tmem_wait_st();
            }
            const float mx = smx::row_max(sr) * fe;
            const bool raise = mx > m_ref + 8.f || (m_ref == -INFINITY && mx > -INFINITY);
            const float m_new = raise ? mx : m_ref;
            const float corr = raise && m_ref != -INFINITY ? fast_exp2(m_ref - m_new) : 1.f;
            m_ref = m_new;
            smx::exp_half(sr[0], fe, m_ref, w0, acc, pack);
            smx::exp_half(sr[1], fe, m_ref, w1, acc, pack);
            const bool dead = m_ref == -INFINITY;       // nothing visible yet: the exponents above are NaN
            if (__any_sync(0xffffffffu, corr != 1.f)) {
                if (i > 0) pv_done(n + i - 1);
                tc_fence_after();
#pragma unroll
                for (int c4 = 0; c4 < D / 32; ++c4) {
                    uint32_t orr[32];
                    tmem_ld32(o_addr + c4 * 32, orr);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; ++j) orr[j] = __float_as_uint(__uint_as_float(orr[j]) * corr);
                    tmem_st32(o_addr + c4 * 32, orr);
                }
                l_run *= corr;
            }
            if (dead) {
#pragma unroll
                for (int k = 0; k < 16; ++k) w0[k] = w1[k] = 0u;
            } else {
                l_run += smx::sum_of(acc);
            }
            tmem_st16(s_addr + sb * KT, w0);
            tmem_st16(s_addr + sb * KT + 16, w1);
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive_cnt(p_full(x, sb));
            if (++st_i == ST) st_i = 0;
        }
        n += nt;
        ++qn;
        st_i = (st_i + skipped) % ST;
        pv_done(n - 1);
        tc_fence_after();
        float inv = 1.0f / l_run;
        if (p.sink) {                               // the reference maximum is in the log2 domain
            const float sk = p.sink[head] * kLog2e, mn = fmaxf(m_ref, sk);
            const float c = fast_exp2(m_ref - mn);
            inv = c / (l_run * c + fast_exp2(sk - mn));
        }
        if (failed()) inv = __int_as_float(0x7fc00000);
        // every thread writes its own row, whole 32-byte sectors at a time: the stores leave while the next item's scores come
        bf16_t* out = static_cast<bf16_t*>(p.out) + ((int64_t)(it.row0 + tok) * p.heads + head) * D;
        const bf16_t* gate = p.gate ? static_cast<const bf16_t*>(p.gate) + (int64_t)(it.row0 + tok) * p.gate_stride + p.gate_off + head * D : nullptr;
        const bool gate16 = ((uintptr_t)p.gate | (uintptr_t)(p.gate_stride * 2) | (uintptr_t)(p.gate_off * 2)) % 16 == 0;
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
            uint32_t o[32], w[16];
            tmem_ld32(o_addr + c0, o);
            tmem_wait_ld();
            if (qpos >= 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float f[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(o[j * 8 + e]) * inv;
                if (p.out_rot) {
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                        const int col = c0 + j * 8 + e;
                        const float u = f[e], v = f[e + 1];
                        f[e] = ma_unturn(p, it.row0 + tok, col, u, v);
                        f[e + 1] = ma_unturn(p, it.row0 + tok, col + 1, v, u);
                    }
                }
                if (gate) {
                    float g[8];
                    if (gate16) {
                        bf16x8_unpack(__ldg(reinterpret_cast<const uint4*>(gate + c0) + j), g);
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e) g[e] = __bfloat162float(gate[c0 + j * 8 + e]);
                    }
#pragma unroll
                    for (int e = 0; e < 8; ++e) f[e] *= sigmoid_f32(g[e]);
                }
                const uint4 v = bf16x8_pack(f);
                w[4 * j] = v.x; w[4 * j + 1] = v.y; w[4 * j + 2] = v.z; w[4 * j + 3] = v.w;
            }
            store_row32(out + c0, w);
            }
            __syncwarp();
        }
        }
        tc_fence_before();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == W_MMA) {
        tc_fence_after();
        if (failed()) {
            __nanosleep(1000000);       // products in flight write TMEM for microseconds at most
            if (lane == 0) atomicAdd(&g_errors, 1);
        }
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

template <int KB, int VB, int NQ, bool DENSE, bool MOD, int QD, int QB>
static int launch_bufs(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& k2, const CUtensorMap& v, const Args& a, int ntiles,
                       size_t extra, cudaStream_t st) {
    const size_t smem = smem_for(KB, VB, NQ, QB) + extra;
    if (smem > (size_t)device_info().max_smem_optin) return PA_ERR_UNSUPPORTED;
    const int64_t items = (int64_t)ntiles * a.p.num_kv_heads * a.hchunks;
    if (items > 0x7fffffff) return PA_ERR_INVALID_ARG;
    auto kern = attention_tc_kernel<KB, VB, NQ, DENSE, MOD, QD, QB>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    Args b = a;
    b.items = (int)items;
    // persistent, but where every item has a table of biases of its own in shared memory
    const int64_t most = (int64_t)device_info().sm_count * (NQ == 1 && KB < 3 ? 2 : 1);
    const int64_t ctas = a.p.bias_kind == 2 || items < most ? items : most;
    kern<<<(unsigned)ctas, threads_for(NQ), smem, st>>>(q, k, k2, v, b);
    PA_RETURN_LAUNCH_STATUS();
}

template <int KB, int VB, int NQ, bool DENSE, bool MOD, int QD = KB * 64>
static int launch(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& k2, const CUtensorMap& v, const Args& a, int ntiles, size_t extra,
                  cudaStream_t st) {
    if (MOD && a.p.bias_kind == 2) return launch_bufs<KB, VB, NQ, DENSE, MOD, QD, q_bufs(KB, NQ, MOD)>(q, k, k2, v, a, ntiles, extra, st);
    return launch_bufs<KB, VB, NQ, DENSE, MOD, QD, q_bufs(KB, NQ, false)>(q, k, k2, v, a, ntiles, extra, st);
}

// Rows of a CTA: tokens per head block and heads.  Four (two) heads of a kv head over 64 tokens where there are that many, so
// that the keys and values of a kv head are staged once for them; a head of its own takes its rows from its tokens.
static void plan(int hpg, int q_tiles, int& tb, int& hg) {
    if (hpg >= 3) {
        tb = 64;
        hg = 2 * q_tiles;
    } else if (hpg == 2) {
        tb = 64 * q_tiles;
        hg = 2;
    } else {
        tb = QT * q_tiles;
        hg = 1;
    }
}

}  // namespace atc

int masked_decode_errors(int* host_count);
int latent_decode_errors(int* host_count);

int masked_attention_tc_launch(const MaskAttnParams& p, int ntiles, int q_tiles, cudaStream_t st) {
    using namespace atc;
    const bool mod = p.softcap > 0.f || p.bias_kind != 0 || p.head_bias;
    if ((p.dim != 64 && p.dim != 128) || (p.vdim != 64 && p.vdim != 128) || p.sigm || p.key_scale || p.k_pool == p.v_pool)
        return PA_ERR_UNSUPPORTED;
    if (p.tile_size % 16 || p.q_stride % 8 || p.q_off % 8 || (uintptr_t)p.q % 16 || (uintptr_t)p.out % 16 ||
        (uintptr_t)p.k_pool % 16 || (uintptr_t)p.v_pool % 16)
        return PA_ERR_UNSUPPORTED;
    const int64_t rows = (int64_t)p.total_pages * p.tile_size;
    if (rows >= 0x7fffff00ll) return PA_ERR_UNSUPPORTED;
    Args a;
    a.p = p;
    plan(p.heads / p.num_kv_heads, q_tiles, a.tb, a.hg);
    a.hchunks = (p.heads / p.num_kv_heads + a.hg - 1) / a.hg;
    a.kn = a.k2_col = 0;
    a.upt = p.tile_size / 16;
    a.total_rows = (int)rows;
    const size_t extra = p.bias_kind == 2 ? (size_t)p.bias_len * a.hg * 4 : 0;
    if (extra > 40 * 1024) return PA_ERR_UNSUPPORTED;
    // the number of query rows is not known here: boxes are only taken of rows that a work item has
    CUtensorMap q, k, v;
    if (!make_bf16_map(&q, p.q, 0x7fffffff, p.q_off + (int64_t)p.heads * p.dim, p.q_stride, 64)) return PA_ERR_UNSUPPORTED;
    if (!make_bf16_map(&k, p.k_pool, rows, p.dim, p.dim, 16) || !make_bf16_map(&v, p.v_pool, rows, p.vdim, p.vdim, 16)) return PA_ERR_UNSUPPORTED;
#define PA_ATC(KB, VB)                                                                                            \
    if (p.dim == KB * 64 && p.vdim == VB * 64) {                                                                  \
        if (q_tiles == 2)                                                                                         \
            return mod ? launch<KB, VB, 2, false, true>(q, k, k, v, a, ntiles, extra, st) : launch<KB, VB, 2, false, false>(q, k, k, v, a, ntiles, extra, st); \
        return mod ? launch<KB, VB, 1, false, true>(q, k, k, v, a, ntiles, extra, st) : launch<KB, VB, 1, false, false>(q, k, k, v, a, ntiles, extra, st); \
    }
    PA_ATC(1, 1) PA_ATC(1, 2) PA_ATC(2, 1) PA_ATC(2, 2)
#undef PA_ATC
    return PA_ERR_UNSUPPORTED;
}

}  // namespace pa

using namespace pa;

PA_API int pa_masked_attention_tc_tile_tokens(int heads, int kv_heads, int dim, int vdim, int elem, int q_tiles) {
    if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || elem != 2 || (q_tiles != 1 && q_tiles != 2)) return 0;
    if ((dim != 64 && dim != 128) || (vdim != 64 && vdim != 128)) return 0;
    int tb, hg;
    atc::plan(heads / kv_heads, q_tiles, tb, hg);
    return tb;
}

PA_API int pa_masked_attention_tc_units(int heads, int kv_heads, int q_tiles) {
    if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || (q_tiles != 1 && q_tiles != 2)) return 0;
    int tb, hg;
    atc::plan(heads / kv_heads, q_tiles, tb, hg);
    return kv_heads * ((heads / kv_heads + hg - 1) / hg);
}

PA_API int pa_latent_attention_expanded(const void* d_q, int64_t q_stride, int q_off, const void* d_k, int64_t k_stride,
                                        const void* d_latent, int64_t latent_stride, int rot_off, const void* d_v,
                                        int64_t v_stride, int64_t kv_rows, const int32_t* d_q_tiles, int num_q_tiles, int heads,
                                        int dim, int rot_dim, int vdim, float scale, const float* d_sink, void* d_out, int q_tiles,
                                        pa_stream_t stream) {
    using namespace pa::atc;
    PA_CHECK_ARG(d_q && d_k && d_latent && d_v && d_q_tiles && d_out && num_q_tiles >= 0 && heads > 0 && kv_rows > 0 &&
                 (q_tiles == 1 || q_tiles == 2));
    if ((dim != 64 && dim != 128) || (vdim != 64 && vdim != 128) || rot_dim % 16 || rot_dim <= 0 || rot_dim > 64) return PA_ERR_UNSUPPORTED;
    if (q_stride % 8 || q_off % 8 || k_stride % 8 || latent_stride % 8 || v_stride % 8 || rot_off % 8) return PA_ERR_UNSUPPORTED;
    if (((uintptr_t)d_q | (uintptr_t)d_k | (uintptr_t)d_latent | (uintptr_t)d_v | (uintptr_t)d_out) % 16 || kv_rows >= 0x7fffff00ll)
        return PA_ERR_UNSUPPORTED;
    if (num_q_tiles == 0) return PA_OK;
    Args a;
    MaskAttnParams& p = a.p;
    p = MaskAttnParams{};
    p.q = d_q;
    p.q_stride = q_stride;
    p.q_off = q_off;
    p.num_kv_heads = p.heads = heads;
    p.tiles = d_q_tiles;
    p.dim = dim + rot_dim;
    p.vdim = vdim;
    p.scale = scale;
    p.out = d_out;
    p.sink = d_sink;
    plan(1, q_tiles, a.tb, a.hg);
    a.hchunks = 1;
    a.kn = dim;
    a.k2_col = rot_off;
    a.upt = 1;
    a.total_rows = (int)kv_rows;
    CUtensorMap q, k, k2, v;
    if (!make_bf16_map(&q, d_q, 0x7fffffff, q_off + (int64_t)heads * p.dim, q_stride, 64)) return PA_ERR_UNSUPPORTED;
    if (!make_bf16_map(&k, d_k, kv_rows, (uint64_t)heads * dim, k_stride, 64) || !make_bf16_map(&v, d_v, kv_rows, (uint64_t)heads * vdim, v_stride, 64) ||
        !make_bf16_map(&k2, d_latent, kv_rows, (uint64_t)rot_off + rot_dim, latent_stride, 64))
        return PA_ERR_UNSUPPORTED;
    cudaStream_t st = as_stream(stream);
#define PA_ATC(KB, VB, ROT)                                                                       \
    if (dim == (KB - 1) * 64 && vdim == VB * 64 && rot_dim == ROT)                                \
        return q_tiles == 2 ? launch<KB, VB, 2, true, false, (KB - 1) * 64 + ROT>(q, k, k2, v, a, num_q_tiles, 0, st)     \
                            : launch<KB, VB, 1, true, false, (KB - 1) * 64 + ROT>(q, k, k2, v, a, num_q_tiles, 0, st);
#define PA_ATC_ROT(ROT) PA_ATC(2, 1, ROT) PA_ATC(2, 2, ROT) PA_ATC(3, 1, ROT) PA_ATC(3, 2, ROT)
    PA_ATC_ROT(16) PA_ATC_ROT(32) PA_ATC_ROT(48) PA_ATC_ROT(64)
#undef PA_ATC_ROT
#undef PA_ATC
    return PA_ERR_UNSUPPORTED;
}

PA_API int pa_attention_tc_errors(int* host_count) {
    PA_CHECK_ARG(host_count);
    int n = 0, masked = 0, latent = 0;
    int rc = (int)cudaMemcpyFromSymbol(&n, pa::atc::g_errors, sizeof(int));
    if (rc == PA_OK) rc = masked_decode_errors(&masked);
    if (rc == PA_OK) rc = latent_decode_errors(&latent);
    *host_count = n + masked + latent;
    return rc;
}
