// masked_decode.cu -- masked_attention.cu's softmax attention for decoded tokens (one query token per sequence, bfloat16), with the
// keys of all sequences cut into equal shares.
//
// The work is a list of 16-key units: token by token, kv head by kv head, the units a query sees in order.  Every warp is a
// worker with an equal contiguous share of that list, whatever the lengths of the sequences: it streams its units through a
// ring of its own (TMA boxes of 16 keys x 64 columns, SWIZZLE_128B, page ids 32 units ahead), the query heads of the kv head
// are the rows of mma.sync m16n8k16 products (up to 16, the rest zero), and where its share leaves a (token, kv head) pair it
// writes the pair's running maximum, sum and weighted sum (decode_shares.cuh).  A second kernel, resident before the first ends
// (programmatic dependent launch), joins the shares of each pair and applies sink, turn and gate.
//
// The softmax weights enter the second product as bfloat16 for batches that give every SM a pair, as in masked_attention.cu's
// kernel with heads as rows; smaller batches, whose streaming kernel keeps them float, keep them float here too: three
// bfloat16 numbers add up to the 24 bits of a weight, for three products instead of one.
//
// What bounds it: HBM (busy 57 % of the time, with eight workers x 3 stages x 8 KB per SM in flight) and the chain of a unit in a warp,
// eight of which an SM has.  64 tokens, 16 query / 4 kv heads of 128, 2048 keys (268 MB): 56 us = 4.8 TB/s and 4 us for the
// join (heads as rows without a key split, masked_attention_mma_decode_kernel: 91 us); 8 tokens, 2 kv heads, 400 keys: 8.5 us
// (streaming kernel, one CTA per pair: 38 us).
#include "decode_shares.cuh"
#include "masked_attention.cuh"
#include "mma_utils.cuh"
#include "tcgen05_utils.cuh"

namespace pa {
namespace mdec {

// At least two units a share (GPU time with 2 / 3 / 4, kernel and join, each launched alone: 8 tokens of 128 to 640 keys, 2 kv heads 15.8 /
// 20.6 / 21.4 us, 4 x 300 keys, 4 kv heads 14.9 / 17.5 / 20.8 us, 20 x 300, 2 kv heads 15.8 / 19.3 / 19.9 us, 1 x 2000, 4 kv heads 20.3 /
// 19.8 / 21.4 us): a short chain per warp is worth more sums to join.
constexpr int kWarps = 8, kStages = 3, kUnit = 16, kRows = 16, kLeast = 2;

struct Args {
    MaskAttnParams p;
    int ntiles, hch, workers, rows;     // hch: chunks of 16 query heads per kv head; rows: query rows of a pair that are real
    int total_rows;
    uint32_t polls;                     // of a wait
    int* pre;                           // [ntiles + 1] units of one pair of every token, summed up
    float* part;                        // [slots][rows][2 + vdim]: maximum (log2), sum, weighted sums
};

__device__ int g_errors;

__device__ __forceinline__ int tile_units(const MaskAttnParams& p, int pos) {
    return ma_steps(p, ma_first_key(p, pos), pos + 1, kUnit).count;
}
// FLOAT_W: the weights of the second product are float (see above)
template <int DIM, int VDIM, bool FLOAT_W>
__global__ void __launch_bounds__(kWarps * 32, 1) masked_decode_kernel(const __grid_constant__ CUtensorMap tmK,
                                                                       const __grid_constant__ CUtensorMap tmV, const Args a) {
    constexpr int KB = DIM / 64, VB = VDIM / 64, STAGE = (KB + VB) * 2048, NT = VDIM / 8;
    constexpr float kLog2e = 1.4426950408889634f;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ int fail_word;
    const MaskAttnParams& p = a.p;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t ring = base + warp * kStages * STAGE, bar0 = base + kWarps * kStages * STAGE + warp * kStages * 8;
    int* pre = reinterpret_cast<int*>(smem_raw + (base - smem_u32(smem_raw)) + kWarps * kStages * (STAGE + 8));
    const uint32_t fail_sm = smem_u32(&fail_word);
    if (lane == 0) {
        for (int s = 0; s < kStages; ++s) mbar_init(bar0 + s * 8, 1);
        mbar_fence_init();
    }
    if (threadIdx.x == 0) fail_word = 0;
    shares::count_units(pre, a.ntiles, [&](int t) { return tile_units(p, __ldg(p.tiles + 4 * t + 3)); });
    if (blockIdx.x == 0)
        for (int t = threadIdx.x; t <= a.ntiles; t += blockDim.x) a.pre[t] = pre[t];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const int w = warp * gridDim.x + blockIdx.x;
    const int pairs = p.num_kv_heads * a.hch, hpg = p.heads / p.num_kv_heads;
    const int64_t total = (int64_t)pre[a.ntiles] * pairs;
    const int64_t ns = shares::count(total, a.workers, kLeast);
    const int64_t f_lo = w < ns ? total * w / ns : 0, f_hi = w < ns ? total * (w + 1) / ns : 0;
    if (f_lo >= f_hi) return;

    // ---- the copies: unit f's rows in the pools, 32 units at a time
    auto rows_of = [&](int64_t f) -> int {
        if (f >= f_hi) return -1;
        const int t = shares::find_token(pre, a.ntiles, f, pairs), per = pre[t + 1] - pre[t];
        const int rem = (int)(f - (int64_t)pre[t] * pairs), g = rem / per / a.hch, u = rem % per;
        const int4 tl = __ldg(reinterpret_cast<const int4*>(p.tiles) + t);
        const MaSteps st = ma_steps(p, ma_first_key(p, tl.w), tl.w + 1, kUnit);
        const int j = st.step(u) * kUnit, pt = j / p.tile_size;
        if ((unsigned)tl.z >= (unsigned)p.num_slots || pt >= p.num_tiles) return -1;
        const int page = __ldg(p.table + ((int64_t)tl.z * p.num_kv_heads + g) * p.num_tiles + pt);
        return (unsigned)page < (unsigned)p.total_pages ? page * p.tile_size + (j - pt * p.tile_size) : -1;
    };
    int rows_cur = rows_of(f_lo + lane), rows_nxt = rows_of(f_lo + 32 + lane);
    int64_t f_is = f_lo;                // next unit to request
    int is_stage = 0;
    uint32_t mapped = 0;                // bit s: the unit in stage s has a page
    auto issue = [&] {
        if (f_is >= f_hi) return;
        const int o = (int)(f_is - f_lo);
        if (o && (o & 31) == 0) {
            rows_cur = rows_nxt;
            rows_nxt = rows_of(f_is + 32 + lane);
        }
        const int row = __shfl_sync(0xffffffffu, rows_cur, o & 31);
        mapped = row >= 0 ? mapped | 1u << is_stage : mapped & ~(1u << is_stage);
        if (a.polls && elect_one()) {   // 0: a wait that is to run out
            const uint32_t st = ring + is_stage * STAGE, bar = bar0 + is_stage * 8;
            const int r = row >= 0 ? row : a.total_rows;        // no page: a box of zeros
            mbar_arrive_expect_tx(bar, STAGE);
#pragma unroll
            for (int b = 0; b < KB; ++b) tma_load_2d(st + b * 2048, &tmK, b * 64, r, bar);
#pragma unroll
            for (int b = 0; b < VB; ++b) tma_load_2d(st + (KB + b) * 2048, &tmV, b * 64, r, bar);
        }
        __syncwarp();
        ++f_is;
        if (++is_stage == kStages) is_stage = 0;
    };
#pragma unroll
    for (int s = 0; s < kStages; ++s) issue();

    // ---- the pair at hand
    int t = shares::find_token(pre, a.ntiles, f_lo, pairs);
    int per = pre[t + 1] - pre[t], pr, u;       // units of a pair of token t, pair within the token, unit within the pair
    {
        const int rem = (int)(f_lo - (int64_t)pre[t] * pairs);
        pr = rem / per;
        u = rem - pr * per;
    }
    uint32_t qf[DIM / 16][4];
    float o[NT][4], m[2], l[2], slope[2];
    int head[2], qpos, rlo;
    MaSteps steps;
    const int keep = p.mask_kind == 1 ? p.mask_keep : 0;
    auto open_pair = [&] {
        const int4 tl = __ldg(reinterpret_cast<const int4*>(p.tiles) + t);
        qpos = tl.w;
        rlo = ma_first_key(p, qpos);
        steps = ma_steps(p, rlo, qpos + 1, kUnit);
        const int g = pr / a.hch, h0 = g * hpg + pr % a.hch * kRows, hend = min(h0 + kRows, (g + 1) * hpg);
        const bf16_t* q = static_cast<const bf16_t*>(p.q) + (int64_t)tl.x * p.q_stride + p.q_off;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int h = h0 + (lane >> 2) + 8 * i;
            head[i] = h < hend ? h : -1;
            slope[i] = p.bias_kind == 1 && head[i] >= 0 ? p.bias[h] : 0.f;
            m[i] = -INFINITY;
            l[i] = 0.f;
#pragma unroll
            for (int ks = 0; ks < DIM / 16; ++ks)
#pragma unroll
                for (int hf = 0; hf < 2; ++hf)
                    qf[ks][2 * hf + i] = head[i] >= 0 ? __ldg(reinterpret_cast<const uint32_t*>(q + (int64_t)h * DIM + ks * 16 + hf * 8 + 2 * (lane & 3))) : 0u;
        }
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[n][c] = 0.f;
    };
    auto close_pair = [&] {
        const int64_t slot = (int64_t)t * pairs + pr + w;
        const int ld = 2 + VDIM;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = (lane >> 2) + 8 * i;
            float s = l[i] + __shfl_xor_sync(0xffffffffu, l[i], 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if (head[i] < 0) continue;
            float* dst = a.part + (slot * a.rows + r) * ld;
            if ((lane & 3) == 0) {
                dst[0] = m[i];
                dst[1] = s;
            }
#pragma unroll
            for (int n = 0; n < NT; ++n)
                *reinterpret_cast<float2*>(dst + 2 + n * 8 + 2 * (lane & 3)) = make_float2(o[n][2 * i], o[n][2 * i + 1]);
        }
    };
    open_pair();
    int stage = 0;
    uint32_t phase = 0;
    int64_t f = f_lo;
    for (; f < f_hi; ++f) {
        if (u == per) {
            close_pair();
            u = 0;
            if (++pr == pairs) {
                pr = 0;
                ++t;
                per = pre[t + 1] - pre[t];
            }
            open_pair();
        }
        const uint32_t ks_sm = ring + stage * STAGE, vs_sm = ks_sm + KB * 2048;
        if (!__all_sync(0xffffffffu, tc::tc_wait(bar0 + stage * 8, phase, fail_sm, a.polls))) break;
        const bool has = mapped >> stage & 1u;
        const int j0 = steps.step(u) * kUnit, valid = qpos + 1 - j0;
        if (valid < kUnit) {            // value rows past the query's own position may hold anything (0 x NaN = NaN)
            for (int i = lane; i < (kUnit - valid) * (VDIM / 8); i += 32) {
                const int r = valid + i / (VDIM / 8), c = i % (VDIM / 8);
                asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(vs_sm + (c >> 3) * 2048 + r * 128 + (((c & 7) ^ (r & 7)) << 4)),
                             "r"(0u) : "memory");
            }
            fence_proxy_async();
            __syncwarp();
        }
        float s[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int c = 0; c < 4; ++c) s[n][c] = 0.f;
        {
            const int r = (lane & 7) + ((lane >> 4) << 3);
#pragma unroll
            for (int ks = 0; ks < DIM / 16; ++ks) {
                const int c = (ks & 3) * 2 + ((lane >> 3) & 1);
                uint32_t b0, b1, b2, b3;
                ldsm_x4(ks_sm + (ks >> 2) * 2048 + r * 128 + ((c ^ (r & 7)) << 4), b0, b1, b2, b3);
                mma_bf16_16816(s[0], qf[ks], b0, b1);
                mma_bf16_16816(s[1], qf[ks], b2, b3);
            }
        }
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int i = c >> 1, j = j0 + n * 8 + 2 * (lane & 3) + (c & 1);
                const bool vis = has && head[i] >= 0 && j <= qpos && (j >= rlo || j < keep);
                s[n][c] = vis ? ma_score(p, s[n][c], qpos, j, head[i], slope[i]) * kLog2e : -INFINITY;
                mx[i] = fmaxf(mx[i], s[n][c]);
            }
        float ref[2], corr[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
            mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
            const float mn = fmaxf(m[i], mx[i]);
            ref[i] = mn == -INFINITY ? 0.f : mn;
            corr[i] = exp2f(m[i] - ref[i]);
            m[i] = mn;
        }
        if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                l[i] *= corr[i];
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    o[n][2 * i] *= corr[i];
                    o[n][2 * i + 1] *= corr[i];
                }
            }
        }
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                s[n][c] = exp2f(s[n][c] - ref[c >> 1]);
                l[c >> 1] += s[n][c];
            }
        const int vr = (lane & 7) + ((lane >> 3) & 1) * 8;
        auto load_values = [&](int np, uint32_t (&b)[4]) {
            ldsm_x4_trans(vs_sm + (np >> 2) * 2048 + vr * 128 + ((((np & 3) * 2 + (lane >> 4)) ^ (vr & 7)) << 4), b[0], b[1], b[2], b[3]);
        };
        if constexpr (!FLOAT_W) {
            const uint32_t pf[4] = {pack_bf16x2(s[0][0], s[0][1]), pack_bf16x2(s[0][2], s[0][3]), pack_bf16x2(s[1][0], s[1][1]),
                                    pack_bf16x2(s[1][2], s[1][3])};
#pragma unroll
            for (int np = 0; np < NT / 2; ++np) {
                uint32_t b[4];
                load_values(np, b);
                mma_bf16_16816(o[2 * np], pf, b[0], b[1]);
                mma_bf16_16816(o[2 * np + 1], pf, b[2], b[3]);
            }
        } else {
            uint32_t pf[3][4], vf[NT / 2][4];   // plane i of the weights: what the planes before it left
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float x = s[j >> 1][2 * (j & 1)], y = s[j >> 1][2 * (j & 1) + 1];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    pf[i][j] = pack_bf16x2(x, y);
                    x -= __uint_as_float(pf[i][j] << 16);
                    y -= __uint_as_float(pf[i][j] & 0xffff0000u);
                }
            }
#pragma unroll
            for (int np = 0; np < NT / 2; ++np) load_values(np, vf[np]);
            auto weigh = [&](const uint32_t (&w)[4]) {
#pragma unroll
                for (int np = 0; np < NT / 2; ++np) {
                    mma_bf16_16816(o[2 * np], w, vf[np][0], vf[np][1]);
                    mma_bf16_16816(o[2 * np + 1], w, vf[np][2], vf[np][3]);
                }
            };
            // a value that is not finite meets the first plane alone: a zero of the others would make NaN of an infinity
            const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
            __nv_bfloat162 probe = zero;        // 0 x value, summed up: NaN if any is not finite
#pragma unroll
            for (int np = 0; np < NT / 2; ++np)
#pragma unroll
                for (int j = 0; j < 4; ++j) probe = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&vf[np][j]), zero, probe);
            const bool apart = __any_sync(0xffffffffu, __hisnan(probe.x) || __hisnan(probe.y));
            if (apart) {
                weigh(pf[0]);
#pragma unroll
                for (int np = 0; np < NT / 2; ++np)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t v = vf[np][j];
                        vf[np][j] = ((v & 0x7f80u) == 0x7f80u ? 0u : v & 0xffffu) | ((v & 0x7f800000u) == 0x7f800000u ? 0u : v & 0xffff0000u);
                    }
            }
            weigh(pf[2]);                       // the small terms first
            weigh(pf[1]);
            if (!apart) weigh(pf[0]);
        }
        __syncwarp();                   // every lane has read the stage
        issue();                        // refills it
        ++u;
        if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
        }
    }
    if (f < f_hi) {                     // a wait ran out: the copies that were requested land, and the pairs from here on get NaN
        for (int64_t i = f; i < f_is; ++i) {
            const int at = stage + (int)(i - f);
            tc::tc_let_land(bar0 + at % kStages * 8, at < kStages ? phase : phase ^ 1u);
        }
        if (lane == 0) atomicAdd(&g_errors, 1);
        for (f += per - u; f < f_hi; f += per) {
            l[0] = l[1] = __int_as_float(0x7fc00000);
            close_pair();
            if (++pr == pairs) {
                pr = 0;
                ++t;
                per = pre[t + 1] - pre[t];
            }
            open_pair();
        }
        l[0] = l[1] = __int_as_float(0x7fc00000);
    }
    close_pair();
}

// One warp per (pair, query row); a lane has VDIM / 32 neighbouring columns.
template <int VDIM>
__global__ void __launch_bounds__(128) masked_decode_join_kernel(const Args a) {
    constexpr int NV = VDIM / 32;
    const MaskAttnParams& p = a.p;
    const int lane = threadIdx.x & 31;
    const int wid = blockIdx.x * 4 + (threadIdx.x >> 5);
    const int pairs = p.num_kv_heads * a.hch, hpg = p.heads / p.num_kv_heads;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (wid >= a.ntiles * pairs * a.rows) return;
    const int r = wid % a.rows, pair = wid / a.rows, t = pair / pairs, pr = pair % pairs;
    const int g = pr / a.hch, head = g * hpg + pr % a.hch * kRows + r;
    if (pr % a.hch * kRows + r >= hpg) return;
    const int64_t total = (int64_t)a.pre[a.ntiles] * pairs;
    const int per = a.pre[t + 1] - a.pre[t];
    const int64_t f0 = (int64_t)a.pre[t] * pairs + (int64_t)pr * per, f1 = f0 + per - 1;
    const int64_t ns = shares::count(total, a.workers, kLeast);
    const int w0 = (int)(((f0 + 1) * ns - 1) / total), w1 = (int)(((f1 + 1) * ns - 1) / total);
    const int ld = 2 + VDIM;
    const float* src = a.part + (((int64_t)pair + w0) * a.rows + r) * ld;
    const int64_t step = (int64_t)a.rows * ld;
    float mx = -INFINITY;
    for (int w = w0 + lane; w <= w1; w += 32) mx = fmaxf(mx, src[(w - w0) * step]);
    mx = warp_max(mx);
    const float ref = mx == -INFINITY ? 0.f : mx;
    float l = 0.f, acc[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) acc[i] = 0.f;
    // shares in order, four at a time so that their loads are in flight together
    for (int w = w0; w <= w1; w += 4) {
        float c[4], v[4][NV];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float* s = src + (min(w + k, w1) - w0) * step;
            c[k] = w + k <= w1 ? exp2f(s[0] - ref) : 0.f;
            l = fmaf(c[k], s[1], l);
#pragma unroll
            for (int i = 0; i < NV; i += 2) {
                const float2 x = *reinterpret_cast<const float2*>(s + 2 + lane * NV + i);
                v[k][i] = w + k <= w1 ? x.x : 0.f;      // 0 x infinity = NaN
                v[k][i + 1] = w + k <= w1 ? x.y : 0.f;
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int i = 0; i < NV; ++i) acc[i] = fmaf(c[k], v[k][i], acc[i]);
    }
    float inv = 1.0f / l;
    if (p.sink) {
        const float sk = p.sink[head] * 1.4426950408889634f, mn = fmaxf(mx, sk);
        const float c = exp2f(mx - mn);
        inv = c / (l * c + exp2f(sk - mn));
    }
    const int64_t row = p.tiles[4 * t];
    const int col = lane * NV;
#pragma unroll
    for (int i = 0; i < NV; i += 2) {
        float x = acc[i] * inv, y = acc[i + 1] * inv;
        if (p.out_rot) {
            const float x0 = x;
            x = ma_unturn(p, row, col + i, x0, y);
            y = ma_unturn(p, row, col + i + 1, y, x0);
        }
        if (p.gate) {
            x *= ma_gate<bf16_t>(p, row, head * VDIM + col + i);
            y *= ma_gate<bf16_t>(p, row, head * VDIM + col + i + 1);
        }
        *reinterpret_cast<uint32_t*>(static_cast<bf16_t*>(p.out) + row * p.heads * VDIM + (int64_t)head * VDIM + col + i) = pack_bf16x2(x, y);
    }
}

template <int DIM, int VDIM, bool FLOAT_W>
static int launch(const CUtensorMap& k, const CUtensorMap& v, const Args& a, cudaStream_t st) {
    const size_t smem = (size_t)kWarps * kStages * ((DIM + VDIM) / 64 * 2048 + 8) + (a.ntiles + 1) * 4 + 1024;
    cudaError_t e = cudaFuncSetAttribute(masked_decode_kernel<DIM, VDIM, FLOAT_W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int sms = device_info().sm_count;
    const int grid = a.workers < sms ? a.workers : sms;
    masked_decode_kernel<DIM, VDIM, FLOAT_W><<<grid, kWarps * 32, smem, st>>>(k, v, a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    const int64_t warps = (int64_t)a.ntiles * a.p.num_kv_heads * a.hch * a.rows;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((warps + 3) / 4));
    cfg.blockDim = dim3(128);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, masked_decode_join_kernel<VDIM>, a);
}

}  // namespace mdec
}  // namespace pa

using namespace pa;

PA_API int pa_masked_decode_workers(int num_tokens, int heads, int kv_heads, int64_t longest) {
    if (num_tokens <= 0 || kv_heads <= 0 || heads <= 0 || heads % kv_heads || longest <= 0) return 0;
    const int hch = (heads / kv_heads + mdec::kRows - 1) / mdec::kRows;
    const int64_t units = (int64_t)num_tokens * kv_heads * hch * ((longest + mdec::kUnit - 1) / mdec::kUnit), most = mdec::kWarps * device_info().sm_count;
    return (int)shares::count(units, (int)most, mdec::kLeast);
}

PA_API size_t pa_masked_decode_workspace_bytes(int num_tokens, int heads, int kv_heads, int vdim, int workers) {
    if (num_tokens <= 0 || kv_heads <= 0 || heads <= 0 || heads % kv_heads || vdim <= 0 || workers <= 0) return 0;
    const int hpg = heads / kv_heads, hch = (hpg + mdec::kRows - 1) / mdec::kRows, rows = hpg < mdec::kRows ? hpg : mdec::kRows;
    return shares::pre_bytes(num_tokens) + ((size_t)num_tokens * kv_heads * hch + workers) * rows * (2 + vdim) * sizeof(float);
}

namespace pa {
int masked_decode_errors(int* host_count) { return (int)cudaMemcpyFromSymbol(host_count, mdec::g_errors, sizeof(int)); }
}  // namespace pa

PA_API int pa_masked_decode_polls(const void* d_q, int64_t q_stride, int q_off, const void* d_k_pool, const void* d_v_pool,
                            const int32_t* d_table, int num_slots, int num_kv_heads, int num_tiles, int total_pages, int tile_size,
                            const int32_t* d_q_tiles, int num_q_tiles, int heads, int dim, int vdim, float scale, float softcap,
                            int mask_kind, int mask_size, int mask_keep, int bias_kind, const float* d_bias, int bias_len,
                            const float* d_head_scale, const float* d_sink, const float* d_out_rot, const float* d_head_bias,
                            const void* d_gate, int64_t gate_stride, int gate_off, void* d_out, int workers, void* d_workspace,
                            size_t workspace_bytes, int polls, pa_stream_t stream) {
    using namespace pa::mdec;
    PA_CHECK_ARG(polls >= 0);
    PA_CHECK_ARG(mask_keep >= 0 && (mask_keep == 0 || mask_kind == 1) && (!d_out_rot || vdim % 2 == 0));
    PA_CHECK_ARG(d_q && d_k_pool && d_v_pool && d_table && d_q_tiles && d_out && num_q_tiles >= 0);
    PA_CHECK_ARG(num_slots > 0 && num_kv_heads > 0 && num_tiles > 0 && total_pages > 0 && tile_size > 0);
    PA_CHECK_ARG(heads > 0 && heads % num_kv_heads == 0 && dim > 0 && vdim > 0 && softcap >= 0.f && workers > 0);
    PA_CHECK_ARG(mask_kind >= 0 && mask_kind <= 2 && (mask_kind == 0 || mask_size > 0));
    PA_CHECK_ARG(bias_kind >= 0 && bias_kind <= 2 && (bias_kind == 0 || d_bias) && (bias_kind != 2 || bias_len > 0));
    if (num_q_tiles == 0) return PA_OK;
    const int64_t rows = (int64_t)total_pages * tile_size;
    if ((dim != 64 && dim != 128) || (vdim != 64 && vdim != 128) || d_k_pool == d_v_pool || num_q_tiles > shares::kMostTokens || tile_size % 16 ||
        rows >= 0x7fffff00ll)
        return PA_ERR_UNSUPPORTED;
    if (((uintptr_t)d_k_pool | (uintptr_t)d_v_pool | (uintptr_t)d_q_tiles | (uintptr_t)d_workspace) % 16 || (uintptr_t)d_q % 4 ||
        (uintptr_t)d_out % 4 || q_stride % 2 || q_off % 2)
        return PA_ERR_UNSUPPORTED;
    if (!d_workspace || workspace_bytes < pa_masked_decode_workspace_bytes(num_q_tiles, heads, num_kv_heads, vdim, workers)) return PA_ERR_WORKSPACE;
    if (workers > kWarps * device_info().sm_count) return PA_ERR_INVALID_ARG;
    Args a;
    MaskAttnParams& p = a.p;
    p = MaskAttnParams{};
    p.q = d_q; p.q_stride = q_stride; p.q_off = q_off; p.k_pool = d_k_pool; p.v_pool = d_v_pool; p.table = d_table;
    p.num_slots = num_slots; p.num_kv_heads = num_kv_heads; p.num_tiles = num_tiles; p.total_pages = total_pages;
    p.tile_size = tile_size; p.tiles = d_q_tiles; p.heads = heads; p.dim = dim; p.vdim = vdim; p.scale = scale; p.softcap = softcap;
    p.mask_kind = mask_kind; p.mask_size = mask_size; p.mask_keep = mask_keep; p.bias_kind = bias_kind; p.bias = d_bias;
    p.bias_len = bias_len; p.out = d_out; p.head_scale = d_head_scale; p.sink = d_sink; p.out_rot = d_out_rot;
    p.head_bias = d_head_bias; p.gate = d_gate; p.gate_stride = gate_stride; p.gate_off = gate_off;
    const int hpg = heads / num_kv_heads;
    a.ntiles = num_q_tiles;
    a.hch = (hpg + kRows - 1) / kRows;
    a.rows = hpg < kRows ? hpg : kRows;
    a.workers = workers;
    a.total_rows = (int)rows;
    a.polls = (uint32_t)polls;
    a.pre = static_cast<int*>(d_workspace);
    a.part = reinterpret_cast<float*>(static_cast<char*>(d_workspace) + shares::pre_bytes(num_q_tiles));
    CUtensorMap k, v;
    if (!tc::make_bf16_map(&k, d_k_pool, rows, dim, dim, 16) || !tc::make_bf16_map(&v, d_v_pool, rows, vdim, vdim, 16)) return PA_ERR_UNSUPPORTED;
    cudaStream_t st = as_stream(stream);
    // bfloat16 weights where masked_attention.cu's kernel with heads as rows would serve the batch: a pair per SM, 16-byte query rows
    const bool rows16 = q_stride % 8 == 0 && q_off % 8 == 0 && (uintptr_t)d_q % 16 == 0;
    const bool float_w = !rows16 || (int64_t)num_q_tiles * num_kv_heads < device_info().sm_count;
#define PA_MDEC(D, V)                                                                                             \
    if (dim == D && vdim == V) return float_w ? launch<D, V, true>(k, v, a, st) : launch<D, V, false>(k, v, a, st)
    PA_MDEC(64, 64); PA_MDEC(64, 128); PA_MDEC(128, 64); PA_MDEC(128, 128);
#undef PA_MDEC
    return PA_ERR_UNSUPPORTED;
}

PA_API int pa_masked_decode(const void* d_q, int64_t q_stride, int q_off, const void* d_k_pool, const void* d_v_pool,
                            const int32_t* d_table, int num_slots, int num_kv_heads, int num_tiles, int total_pages, int tile_size,
                            const int32_t* d_q_tiles, int num_q_tiles, int heads, int dim, int vdim, float scale, float softcap,
                            int mask_kind, int mask_size, int mask_keep, int bias_kind, const float* d_bias, int bias_len,
                            const float* d_head_scale, const float* d_sink, const float* d_out_rot, const float* d_head_bias,
                            const void* d_gate, int64_t gate_stride, int gate_off, void* d_out, int workers, void* d_workspace,
                            size_t workspace_bytes, pa_stream_t stream) {
    return pa_masked_decode_polls(d_q, q_stride, q_off, d_k_pool, d_v_pool, d_table, num_slots, num_kv_heads, num_tiles, total_pages, tile_size,
                                  d_q_tiles, num_q_tiles, heads, dim, vdim, scale, softcap, mask_kind, mask_size, mask_keep, bias_kind, d_bias,
                                  bias_len, d_head_scale, d_sink, d_out_rot, d_head_bias, d_gate, gate_stride, gate_off, d_out, workers,
                                  d_workspace, workspace_bytes, (int)pa::tc::kPolls, stream);
}
