// latent_decode.cu -- attention through a low-rank latent (see latent_attention.cu) for decoded tokens, bfloat16, with the keys of
// all sequences cut into equal shares.
//
// The work is a list of 32-key units, token by token (and 16 query heads by 16 query heads).  Every CTA is a worker with an
// equal contiguous share of it: a producer warp brings whole pool rows in by TMA (boxes of 16 keys x 64 columns, SWIZZLE_128B)
// through a ring of 5 to 8 stages, and eight warps multiply.  The heads are the 16 rows of mma.sync m16n8k16 products.  A cached row
// serves both products: for the scores a warp takes 8 keys and half of the columns, the partial scores meet in shared memory
// behind the one barrier of a step, every warp keeps the softmax of all 32 keys, and for the weighted sums a warp owns an
// eighth of the latent columns -- nothing is computed twice but the 16 x 32 exponentials.  Shares that end inside a token are
// joined by a second kernel (decode_shares.cuh).
//
// What bounds it: the chain of a step (scores, exchange, exponentials, weighted sums), which all eight warps walk together; HBM
// is busy 40 % of the time with 180 KB in flight per SM.  64 tokens, 16 heads, rank 512 + 64, 2048 keys (151 MB): 49 us = 3.1 TB/s
// (latent_attention_mma_kernel with two key splits and its merge: 70 + 8 us); 8 tokens, 8 heads, rank 256 + 32, 400 keys: 8.7 us
// (13.6 us).
#include "decode_shares.cuh"
#include "mma_utils.cuh"
#include "seq_common.cuh"
#include "tcgen05_utils.cuh"

namespace pa {
namespace ldec {

// at least two units a share: opening and closing one costs about as much as that
constexpr int kUnit = 32, kRows = 16, kConsumers = 8, kThreads = (kConsumers + 1) * 32, kLeast = 2;
constexpr int kSLd = 40;                // row stride of the score exchange (floats): two rows apart do not share banks

__host__ __device__ constexpr int blocks_for(int kvr) { return kvr / 64 + 1; }      // 64-column blocks of a row; the last is the rotated part
__host__ __device__ constexpr int stage_bytes(int kvr) { return blocks_for(kvr) * kUnit * 128; }
__host__ __device__ constexpr int stages_for(int kvr) { return kvr >= 512 ? 5 : kvr >= 384 ? 6 : 8; }

struct Args {
    const bf16_t* q_lat;
    int64_t ql_rs, ql_hs;
    const bf16_t* q_rot;
    int64_t qr_rs, qr_hs;
    const int32_t* table;
    int num_slots, num_tiles, total_pages, tile_size;
    const int32_t* tiles;
    int ntiles, heads, hch, rows, rot_dim, workers, total_rows;
    uint32_t polls;             // of a wait
    float scale;
    const float* sink;
    bf16_t* out;
    int64_t o_rs, o_hs;
    int* pre;                   // [ntiles + 1] units of one pair of every token, summed up
    float* part;                // [slots][rows][2 + kv_rank]: maximum (log2), sum, weighted sums
};

__device__ int g_errors;

template <int KVR>
__global__ void __launch_bounds__(kThreads, 1) latent_decode_kernel(const __grid_constant__ CUtensorMap tmP, const Args a) {
    constexpr int VB = KVR / 64, STAGE = stage_bytes(KVR), ST = stages_for(KVR);
    constexpr int KP = KVR / 32 + 2;            // pairs of 16-column steps, the rotated part included (zeros past its end)
    constexpr int KPH = (KP + 1) / 2;           // of which a warp has at most this many
    constexpr int NT = KVR / 64;                // 8-column tiles of a warp's eighth of the latent
    constexpr float kLog2e = 1.4426950408889634f;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ int fail_word;
    __shared__ uint32_t meta[ST];
    __shared__ __align__(16) float Sx[2][2][kRows][kSLd];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, bar0 = base + ST * STAGE;
    auto full = [&](int s) { return bar0 + s * 8; };
    auto empty = [&](int s) { return bar0 + (ST + s) * 8; };
    int* pre = reinterpret_cast<int*>(smem_raw + (base - smem_u32(smem_raw)) + ST * STAGE + 2 * ST * 8);
    const uint32_t fail_sm = smem_u32(&fail_word);
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), kConsumers);
        }
        fail_word = 0;
        mbar_fence_init();
    }
    shares::count_units(pre, a.ntiles, [&](int t) { return (__ldg(a.tiles + 4 * t + 3) + kUnit) / kUnit; });
    if (blockIdx.x == 0)
        for (int t = threadIdx.x; t <= a.ntiles; t += blockDim.x) a.pre[t] = pre[t];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const int w = blockIdx.x, pairs = a.hch;
    const int64_t total = (int64_t)pre[a.ntiles] * pairs;
    const int64_t ns = shares::count(total, a.workers, kLeast);
    const int64_t f_lo = w < ns ? total * w / ns : 0, f_hi = w < ns ? total * (w + 1) / ns : 0;
    if (f_lo >= f_hi) return;

    if (warp == kConsumers) {
        // ---- producer: lane = (unit, half) of the next 16 units
        auto row_of = [&](int64_t f0) -> int {
            const int64_t f = f0 + (lane >> 1);
            if (f >= f_hi) return -1;
            const int t = shares::find_token(pre, a.ntiles, f, pairs), per = pre[t + 1] - pre[t];
            const int u = (int)(f - (int64_t)pre[t] * pairs) % per, j = u * kUnit + (lane & 1) * 16;
            const int4 tl = __ldg(reinterpret_cast<const int4*>(a.tiles) + t);
            const int pt = j / a.tile_size;
            if (j > tl.w || (unsigned)tl.z >= (unsigned)a.num_slots || pt >= a.num_tiles) return -1;
            const int page = __ldg(a.table + (int64_t)tl.z * a.num_tiles + pt);
            return (unsigned)page < (unsigned)a.total_pages ? page * a.tile_size + (j - pt * a.tile_size) : -1;
        };
        int cur = row_of(f_lo), nxt = row_of(f_lo + 16), s = 0;
        uint32_t ph = 1;
        for (int64_t f = f_lo; f < f_hi; ++f) {
            const int o = (int)(f - f_lo);
            if (o && (o & 15) == 0) {
                cur = nxt;
                nxt = row_of(f + 16);
            }
            const int r0 = __shfl_sync(0xffffffffu, cur, (o & 15) * 2), r1 = __shfl_sync(0xffffffffu, cur, (o & 15) * 2 + 1);
            if (!__all_sync(0xffffffffu, tc::tc_wait(empty(s), ph, fail_sm))) break;
            if (a.polls && elect_one()) {       // 0: a wait that is to run out
                meta[s] = (r0 >= 0 ? 1u : 0u) | (r1 >= 0 ? 2u : 0u);
                const uint32_t st = base + s * STAGE;
                mbar_arrive_expect_tx(full(s), STAGE);
#pragma unroll
                for (int b = 0; b <= VB; ++b) {
                    tma_load_2d(st + b * (kUnit * 128), &tmP, b * 64, r0 >= 0 ? r0 : a.total_rows, full(s));
                    tma_load_2d(st + b * (kUnit * 128) + 2048, &tmP, b * 64, r1 >= 0 ? r1 : a.total_rows, full(s));
                }
            }
            __syncwarp();
            if (++s == ST) {
                s = 0;
                ph ^= 1u;
            }
        }
        return;
    }

    // ---- consumers
    const int nkey = (warp & 3) * 8, kg = warp >> 2;            // scores: these 8 keys, this half of the columns
    const int p0 = kg ? KPH : 0, np_mine = kg ? KP - KPH : KPH;
    int t = shares::find_token(pre, a.ntiles, f_lo, pairs), per = pre[t + 1] - pre[t], pr, u;
    {
        const int rem = (int)(f_lo - (int64_t)pre[t] * pairs);
        pr = rem / per;
        u = rem - pr * per;
    }
    uint32_t qf[KPH][2][4];
    float o[NT][4], m[2], l[2];
    bool live[2];
    int qpos;
    auto open_pair = [&] {
        const int4 tl = __ldg(reinterpret_cast<const int4*>(a.tiles) + t);
        qpos = tl.w;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int h = pr * kRows + (lane >> 2) + 8 * i;
            live[i] = h < a.heads;
            m[i] = -INFINITY;
            l[i] = 0.f;
            const bf16_t* ql = a.q_lat + (int64_t)tl.x * a.ql_rs + (int64_t)h * a.ql_hs;
            const bf16_t* qr = a.q_rot + (int64_t)tl.x * a.qr_rs + (int64_t)h * a.qr_hs;
#pragma unroll
            for (int k = 0; k < KPH; ++k)
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        const int d = (p0 + k) * 32 + x * 16 + hf * 8 + 2 * (lane & 3);
                        uint32_t v = 0u;
                        if (live[i] && k < np_mine) {
                            if (d < KVR) v = __ldg(reinterpret_cast<const uint32_t*>(ql + d));
                            else if (d - KVR < a.rot_dim) v = __ldg(reinterpret_cast<const uint32_t*>(qr + d - KVR));
                        }
                        qf[k][x][2 * hf + i] = v;
                    }
        }
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[n][c] = 0.f;
    };
    auto close_pair = [&] {
        const int64_t slot = (int64_t)t * pairs + pr + w;
        const int ld = 2 + KVR;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = (lane >> 2) + 8 * i;
            float s = l[i] + __shfl_xor_sync(0xffffffffu, l[i], 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if (!live[i]) continue;
            float* dst = a.part + (slot * a.rows + r) * ld;
            if (warp == 0 && (lane & 3) == 0) {
                dst[0] = m[i];
                dst[1] = tc::tc_failed(fail_sm) ? __int_as_float(0x7fc00000) : s;       // a wait of some warp ran out before this pair's end
            }
#pragma unroll
            for (int n = 0; n < NT; ++n)
                *reinterpret_cast<float2*>(dst + 2 + warp * (KVR / 8) + n * 8 + 2 * (lane & 3)) = make_float2(o[n][2 * i], o[n][2 * i + 1]);
        }
    };
    open_pair();
    const float fs = a.scale * kLog2e;
    int stage = 0, buf = 0;
    uint32_t phase = 0;
    for (int64_t f = f_lo; f < f_hi; ++f) {
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
        const uint32_t st = base + stage * STAGE;
        tc::tc_wait(full(stage), phase, fail_sm, a.polls);     // if it runs out, on over whatever is there: close_pair leaves NaN
        const uint32_t mapped = meta[stage];
        const int j0 = u * kUnit, valid = qpos + 1 - j0;
        // scores of this warp's keys over its columns
        float s[2][4];
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int c = 0; c < 4; ++c) s[x][c] = 0.f;
        {
            const int r = nkey + (lane & 7);
#pragma unroll
            for (int k = 0; k < KPH; ++k) {
                if (k >= np_mine) break;
                const int chunk = (p0 + k) * 4 + (lane >> 3);
                uint32_t b0, b1, b2, b3;
                ldsm_x4(st + (chunk >> 3) * (kUnit * 128) + r * 128 + (((chunk & 7) ^ (r & 7)) << 4), b0, b1, b2, b3);
                mma_bf16_16816(s[0], qf[k][0], b0, b1);
                mma_bf16_16816(s[1], qf[k][1], b2, b3);
            }
        }
        *reinterpret_cast<float2*>(&Sx[buf][kg][lane >> 2][nkey + 2 * (lane & 3)]) = make_float2(s[0][0] + s[1][0], s[0][1] + s[1][1]);
        *reinterpret_cast<float2*>(&Sx[buf][kg][(lane >> 2) + 8][nkey + 2 * (lane & 3)]) = make_float2(s[0][2] + s[1][2], s[0][3] + s[1][3]);
        if (valid < kUnit) {            // rows past the query's own position may hold anything (0 x NaN = NaN)
            for (int i = threadIdx.x; i < (kUnit - valid) * (KVR / 8); i += kConsumers * 32) {
                const int r = valid + i / (KVR / 8), c = i % (KVR / 8);
                asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(st + (c >> 3) * (kUnit * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4)),
                             "r"(0u) : "memory");
            }
            fence_proxy_async();
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        // the softmax of all 32 keys; v[kk][..]: rows lane / 4 and + 8, keys 16 kk + 2 (lane % 4) + {0, 1, 8, 9}
        float v[2][2][4], mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int kk = 0; kk < 2; ++kk)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    const int r = (lane >> 2) + 8 * i, c = kk * 16 + hf * 8 + 2 * (lane & 3);
                    const float2 x = *reinterpret_cast<const float2*>(&Sx[buf][0][r][c]);
                    const float2 y = *reinterpret_cast<const float2*>(&Sx[buf][1][r][c]);
                    const bool page = mapped >> kk & 1u;
                    v[kk][i][2 * hf] = page && c < valid ? (x.x + y.x) * fs : -INFINITY;
                    v[kk][i][2 * hf + 1] = page && c + 1 < valid ? (x.y + y.y) * fs : -INFINITY;
                    mx[i] = fmaxf(mx[i], fmaxf(v[kk][i][2 * hf], v[kk][i][2 * hf + 1]));
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
        for (int kk = 0; kk < 2; ++kk) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    v[kk][i][c] = exp2f(v[kk][i][c] - ref[i]);
                    l[i] += v[kk][i][c];
                }
            const uint32_t pf[4] = {pack_bf16x2(v[kk][0][0], v[kk][0][1]), pack_bf16x2(v[kk][1][0], v[kk][1][1]),
                                    pack_bf16x2(v[kk][0][2], v[kk][0][3]), pack_bf16x2(v[kk][1][2], v[kk][1][3])};
            const int r = kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
            for (int np = 0; np < NT / 2; ++np) {
                const int chunk = warp * (KVR / 64) + np * 2 + (lane >> 4);
                uint32_t b0, b1, b2, b3;
                ldsm_x4_trans(st + (chunk >> 3) * (kUnit * 128) + r * 128 + (((chunk & 7) ^ (r & 7)) << 4), b0, b1, b2, b3);
                mma_bf16_16816(o[2 * np], pf, b0, b1);
                mma_bf16_16816(o[2 * np + 1], pf, b2, b3);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty(stage));
        buf ^= 1;
        ++u;
        if (++stage == ST) {
            stage = 0;
            phase ^= 1u;
        }
    }
    close_pair();
    if (threadIdx.x == 0 && tc::tc_failed(fail_sm)) {       // the copies that were requested land before the shared memory goes
        for (int b = 0; b < ST; ++b) tc::tc_let_land(full(b), b < stage ? phase : phase ^ 1u);
        atomicAdd(&g_errors, 1);
    }
}

// One warp per (pair, row); a lane has columns 2 lane + 64 i and the next.
template <int KVR>
__global__ void __launch_bounds__(128) latent_decode_join_kernel(const Args a) {
    constexpr int NV = KVR / 64;
    const int lane = threadIdx.x & 31;
    const int wid = blockIdx.x * 4 + (threadIdx.x >> 5);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (wid >= a.ntiles * a.hch * a.rows) return;
    const int r = wid % a.rows, pair = wid / a.rows, t = pair / a.hch, pr = pair % a.hch, head = pr * kRows + r;
    if (head >= a.heads) return;
    const int64_t total = (int64_t)a.pre[a.ntiles] * a.hch, ns = shares::count(total, a.workers, kLeast);
    const int per = a.pre[t + 1] - a.pre[t];
    const int64_t f0 = (int64_t)a.pre[t] * a.hch + (int64_t)pr * per, f1 = f0 + per - 1;
    const int w0 = (int)(((f0 + 1) * ns - 1) / total), w1 = (int)(((f1 + 1) * ns - 1) / total);
    const int ld = 2 + KVR;
    const float* src = a.part + (((int64_t)pair + w0) * a.rows + r) * ld;
    const int64_t step = (int64_t)a.rows * ld;
    float mx = -INFINITY;
    for (int w = w0 + lane; w <= w1; w += 32) mx = fmaxf(mx, src[(w - w0) * step]);
    mx = warp_max(mx);
    const float ref = mx == -INFINITY ? 0.f : mx;
    float l = 0.f;
    float2 acc[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) acc[i] = make_float2(0.f, 0.f);
    for (int w = w0; w <= w1; w += 2) {
        float c[2];
        float2 v[2][NV];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float* s = src + (min(w + k, w1) - w0) * step;
            c[k] = w + k <= w1 ? exp2f(s[0] - ref) : 0.f;
            l = fmaf(c[k], s[1], l);
#pragma unroll
            for (int i = 0; i < NV; ++i) v[k][i] = *reinterpret_cast<const float2*>(s + 2 + 2 * lane + 64 * i);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                acc[i].x = fmaf(c[k], v[k][i].x, acc[i].x);
                acc[i].y = fmaf(c[k], v[k][i].y, acc[i].y);
            }
    }
    float inv = 1.0f / l;
    if (a.sink) {
        const float sk = a.sink[head] * 1.4426950408889634f, mn = fmaxf(mx, sk);
        const float c = exp2f(mx - mn);
        inv = c / (l * c + exp2f(sk - mn));
    }
    bf16_t* dst = a.out + (int64_t)a.tiles[4 * t] * a.o_rs + (int64_t)head * a.o_hs;
#pragma unroll
    for (int i = 0; i < NV; ++i) *reinterpret_cast<uint32_t*>(dst + 2 * lane + 64 * i) = pack_bf16x2(acc[i].x * inv, acc[i].y * inv);
}

template <int KVR>
static int launch(const CUtensorMap& m, const Args& a, cudaStream_t st) {
    const size_t smem = (size_t)stages_for(KVR) * (stage_bytes(KVR) + 16) + (a.ntiles + 1) * 4 + 1024;
    cudaError_t e = cudaFuncSetAttribute(latent_decode_kernel<KVR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    latent_decode_kernel<KVR><<<a.workers, kThreads, smem, st>>>(m, a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    const int64_t warps = (int64_t)a.ntiles * a.hch * a.rows;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((warps + 3) / 4));
    cfg.blockDim = dim3(128);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, latent_decode_join_kernel<KVR>, a);
}

}  // namespace ldec
}  // namespace pa

using namespace pa;

PA_API int pa_latent_decode_workers(int num_tokens, int heads, int64_t longest) {
    if (num_tokens <= 0 || heads <= 0 || longest <= 0) return 0;
    const int64_t units = (int64_t)num_tokens * ((heads + ldec::kRows - 1) / ldec::kRows) * ((longest + ldec::kUnit - 1) / ldec::kUnit);
    return (int)shares::count(units, device_info().sm_count, ldec::kLeast);
}

PA_API size_t pa_latent_decode_workspace_bytes(int num_tokens, int heads, int kv_rank, int workers) {
    if (num_tokens <= 0 || heads <= 0 || kv_rank <= 0 || workers <= 0) return 0;
    const int hch = (heads + ldec::kRows - 1) / ldec::kRows, rows = heads < ldec::kRows ? heads : ldec::kRows;
    return shares::pre_bytes(num_tokens) + ((size_t)num_tokens * hch + workers) * rows * (2 + kv_rank) * sizeof(float);
}

namespace pa {
int latent_decode_errors(int* host_count) { return (int)cudaMemcpyFromSymbol(host_count, ldec::g_errors, sizeof(int)); }
}  // namespace pa

PA_API int pa_latent_decode_polls(const void* d_q_lat, int64_t ql_row_stride, int64_t ql_head_stride, const void* d_q_rot,
                            int64_t qr_row_stride, int64_t qr_head_stride, const void* d_pool, const int32_t* d_table, int num_slots,
                            int num_tiles, int total_pages, int tile_size, const int32_t* d_q_tiles, int num_q_tiles, int heads,
                            int kv_rank, int rot_dim, float scale, const float* d_sink, void* d_out, int64_t o_row_stride,
                            int64_t o_head_stride, int workers, void* d_workspace, size_t workspace_bytes, int polls, pa_stream_t stream) {
    using namespace pa::ldec;
    PA_CHECK_ARG(polls >= 0);
    PA_CHECK_ARG(d_q_lat && (d_q_rot || rot_dim == 0) && d_pool && d_table && d_q_tiles && d_out && num_q_tiles >= 0);
    PA_CHECK_ARG(num_slots > 0 && num_tiles > 0 && total_pages > 0 && tile_size > 0 && heads > 0 && kv_rank > 0 && rot_dim >= 0 && workers > 0);
    if (num_q_tiles == 0) return PA_OK;
    const int64_t rows = (int64_t)total_pages * tile_size;
    const int kd = kv_rank + rot_dim;
    if (kv_rank % 128 || kv_rank > 512 || rot_dim % 8 || rot_dim > 64 || tile_size % 16 || num_q_tiles > shares::kMostTokens || rows >= 0x7fffff00ll)
        return PA_ERR_UNSUPPORTED;
    if (((uintptr_t)d_pool | (uintptr_t)d_q_tiles | (uintptr_t)d_workspace) % 16 || ((uintptr_t)d_q_lat | (uintptr_t)d_q_rot | (uintptr_t)d_out) % 4 ||
        (ql_row_stride | ql_head_stride | qr_row_stride | qr_head_stride | o_row_stride | o_head_stride) % 2)
        return PA_ERR_UNSUPPORTED;
    if (!d_workspace || workspace_bytes < pa_latent_decode_workspace_bytes(num_q_tiles, heads, kv_rank, workers)) return PA_ERR_WORKSPACE;
    if (workers > device_info().sm_count) return PA_ERR_INVALID_ARG;
    Args a;
    a.q_lat = static_cast<const bf16_t*>(d_q_lat); a.ql_rs = ql_row_stride; a.ql_hs = ql_head_stride;
    a.q_rot = static_cast<const bf16_t*>(d_q_rot); a.qr_rs = qr_row_stride; a.qr_hs = qr_head_stride;
    a.table = d_table; a.num_slots = num_slots; a.num_tiles = num_tiles; a.total_pages = total_pages; a.tile_size = tile_size;
    a.tiles = d_q_tiles; a.ntiles = num_q_tiles; a.heads = heads; a.hch = (heads + kRows - 1) / kRows;
    a.rows = heads < kRows ? heads : kRows; a.rot_dim = rot_dim; a.workers = workers; a.total_rows = (int)rows; a.scale = scale;
    a.polls = (uint32_t)polls;
    a.sink = d_sink; a.out = static_cast<bf16_t*>(d_out); a.o_rs = o_row_stride; a.o_hs = o_head_stride;
    a.pre = static_cast<int*>(d_workspace);
    a.part = reinterpret_cast<float*>(static_cast<char*>(d_workspace) + shares::pre_bytes(num_q_tiles));
    CUtensorMap m;
    if (!tc::make_bf16_map(&m, d_pool, rows, kd, kd, 16)) return PA_ERR_UNSUPPORTED;
    cudaStream_t st = as_stream(stream);
    if (kv_rank == 128) return launch<128>(m, a, st);
    if (kv_rank == 256) return launch<256>(m, a, st);
    if (kv_rank == 384) return launch<384>(m, a, st);
    return launch<512>(m, a, st);
}

PA_API int pa_latent_decode(const void* d_q_lat, int64_t ql_row_stride, int64_t ql_head_stride, const void* d_q_rot,
                            int64_t qr_row_stride, int64_t qr_head_stride, const void* d_pool, const int32_t* d_table, int num_slots,
                            int num_tiles, int total_pages, int tile_size, const int32_t* d_q_tiles, int num_q_tiles, int heads,
                            int kv_rank, int rot_dim, float scale, const float* d_sink, void* d_out, int64_t o_row_stride,
                            int64_t o_head_stride, int workers, void* d_workspace, size_t workspace_bytes, pa_stream_t stream) {
    return pa_latent_decode_polls(d_q_lat, ql_row_stride, ql_head_stride, d_q_rot, qr_row_stride, qr_head_stride, d_pool, d_table, num_slots,
                                  num_tiles, total_pages, tile_size, d_q_tiles, num_q_tiles, heads, kv_rank, rot_dim, scale, d_sink, d_out,
                                  o_row_stride, o_head_stride, workers, d_workspace, workspace_bytes, (int)pa::tc::kPolls, stream);
}
