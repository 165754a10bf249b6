// recurrence_ops.cu -- matrix-state recurrences over a RAGGED batch (see seq_ops.cu for the batch description) and the
// small ops around them.
//
//   causal_conv_kernel        per-channel causal convolution over the tokens of a sequence (taps from the config, the
//                             last column of the weight is the current token's) + bias + silu; inputs before a portion's
//                             first token come from the sequence's state slot, which holds its last taps - 1 inputs
//   conv_state_kernel         state slot <- the last taps - 1 inputs of a portion (older ones slide out)
//   decay_scan_kernel         S_t = a_t S_{t-1} + k_t (s_t v_t)^T,  o_t = S_t^T q_t + skip * v_t   per head, S is dim x vdim,
//                             float, one slot per sequence.  The decay is a constant of the head (linear attention with
//                             decay), or a_t = exp(-exp(A_log) dt_t) with dt_t = softplus(raw_t + bias) and s_t = dt_t
//                             (selective state space); q / k may be shared by the heads of a group; q, k, v may pass silu;
//                             q and k may be rotated (halves) over their first dimensions and k scaled, in float, as they
//                             are staged
//   decay_chunk_* kernels     the same recurrence for long portions as a three-pass chunked scan (fold every chunk from a
//                             zero state, chain the chunks from the state slot, replay every chunk from its incoming state)
//   gated_norm_kernel         RMS norm in equal groups of a float row with a per-channel weight (optional) and a gate from
//                             another buffer: silu(gate) multiplied in BEFORE the norm, or sigmoid(gate) or silu(gate) AFTER
//
// States, decays and their logarithms, softplus, step sizes and the norms are float whatever the activation type.
#include "seq_common.cuh"

namespace pa {

// ---- causal convolution -----------------------------------------------------------------------------------------------
// chunks: [n][4] = first row, tokens, slot, offset of the first token within its portion.  A thread owns one channel of
// one chunk and slides a window of kMaxTaps inputs along it.
constexpr int kMaxTaps = 8;

template <typename T>
__global__ void __launch_bounds__(128) causal_conv_kernel(const T* __restrict__ in, int64_t in_stride, int in_off, int channels,
                                                          int taps, const float* __restrict__ w, const float* __restrict__ bias,
                                                          const float* __restrict__ state, const int32_t* __restrict__ chunks,
                                                          T* __restrict__ out, int64_t out_stride, int act) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= channels) return;
    const int* ch = chunks + 4 * blockIdx.y;
    const int row0 = ch[0], n = ch[1], slot = ch[2], off = ch[3];
    float wt[kMaxTaps], win[kMaxTaps];
#pragma unroll
    for (int i = 0; i < kMaxTaps; ++i) wt[i] = i < taps ? w[(int64_t)c * taps + (taps - 1 - i)] : 0.f;   // wt[i]: i tokens back
    const float b = bias ? bias[c] : 0.f;
    const float* st = state + (int64_t)slot * (taps - 1) * channels;
    // win[i] = input i + 1 tokens before the chunk's first token
#pragma unroll
    for (int i = 0; i < kMaxTaps - 1; ++i) {
        float v = 0.f;
        if (i < taps - 1) {
            const int t = off - 1 - i;                 // offset within the portion
            v = t >= 0 ? to_f32<T>(in[(int64_t)(row0 - 1 - i) * in_stride + in_off + c]) : st[(int64_t)(taps - 1 + t) * channels + c];
        }
        win[i + 1] = v;
    }
    for (int t = 0; t < n; ++t) {
        win[0] = to_f32<T>(in[(int64_t)(row0 + t) * in_stride + in_off + c]);
        float acc = b;
#pragma unroll
        for (int i = 0; i < kMaxTaps; ++i) acc = fmaf(wt[i], win[i], acc);
        out[(int64_t)(row0 + t) * out_stride + c] = from_f32<T>(act ? silu_f32(acc) : acc);
#pragma unroll
        for (int i = kMaxTaps - 1; i > 0; --i) win[i] = win[i - 1];
    }
}

template <typename T>
__global__ void __launch_bounds__(128) conv_state_kernel(const T* __restrict__ in, int64_t in_stride, int in_off, int channels,
                                                         int taps, const int32_t* __restrict__ seq_start,
                                                         const int32_t* __restrict__ seq_len, const int32_t* __restrict__ seq_slot,
                                                         float* __restrict__ state) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= channels) return;
    const int s = blockIdx.y, n = seq_len[s], r0 = seq_start[s];
    if (n <= 0) return;
    float* st = state + (int64_t)seq_slot[s] * (taps - 1) * channels;
    float nv[kMaxTaps];
#pragma unroll
    for (int i = 0; i < kMaxTaps - 1; ++i) {
        nv[i] = 0.f;
        if (i < taps - 1) {
            const int t = n - (taps - 1) + i;          // offset within the portion of the input that lands in place i
            nv[i] = t >= 0 ? to_f32<T>(in[(int64_t)(r0 + t) * in_stride + in_off + c]) : st[(int64_t)(taps - 1 + t) * channels + c];
        }
    }
#pragma unroll
    for (int i = 0; i < kMaxTaps - 1; ++i)
        if (i < taps - 1) st[(int64_t)i * channels + c] = nv[i];
}

// ---- the recurrence ---------------------------------------------------------------------------------------------------
struct DecayScanParams {
    const void* q; int64_t q_stride; int q_off;       // q of head h: q_off + (h / heads_per_group) * dim
    const void* k; int64_t k_stride; int k_off;
    const void* v; int64_t v_stride; int v_off;       // v of head h: v_off + h * vdim
    int heads, groups, dim, vdim;
    int act;                                          // 1: q, k and v pass silu as they are read
    const float* decay;                               // [heads] constant decays (dt == nullptr)
    const void* dt; int64_t dt_stride; int dt_off;    // raw step size of head h at dt_off + h
    const float* dt_bias; const float* a_log; const float* skip;   // [heads] each (dt != nullptr); skip may be null
    float* state;                                     // [slots][heads][dim][vdim]
    float* out; int64_t out_stride;                   // float rows [heads * vdim]
    // work items: [n][4] = first row, tokens, slot, kind-specific; mode 0: a portion from / to its state slot;
    // mode 1: fold a chunk from a zero state into part[item]; mode 2: replay a chunk from part[item] (no state written)
    const int32_t* items;
    int mode;
    int vec;                                          // every staged piece of q, k and v starts on a 16-byte boundary
    float* part;                                      // [items][heads][dim * vdim + 1]: state, then the chunk's total decay
    const float* rope; int rot_dims;                  // [rows][rot_dims / 2][cos, sin]: pairs (i, i + rot_dims / 2) of q and k
    float k_scale;                                    // multiplies k (constant decays)
};

constexpr int kDsTokens = 16;                         // tokens staged per step
constexpr int kDsMaxThreads = 128;

__device__ __forceinline__ float softplus_f32(float z) { return z > 20.f ? z : log1pf(expf(z)); }

template <typename T>
__device__ __forceinline__ void ds_load16(const T* __restrict__ p, float (&f)[16 / sizeof(T)]) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    if (sizeof(T) == 4) {
        f[0] = __uint_as_float(v.x); f[1] = __uint_as_float(v.y); f[2] = __uint_as_float(v.z); f[3] = __uint_as_float(v.w);
    } else {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[2 * i] = __uint_as_float(w[i] << 16);
            f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
}

// A thread keeps a DPT x CPT block of the state in registers: lane = (column group) * NSL + (row slice), so the NSL
// threads that share a column group cover NSL * DPT >= dim rows and their partial outputs meet in a shuffle reduction.
// q, k, v, the decays and the input scales of kDsTokens tokens are staged in shared memory per step (one 16-byte read of
// q and of k feeds 4 x CPT updates and as many output terms).  MODE 0: a portion from / to its state slot; 1: fold a
// chunk from a zero state into part[item] (no outputs); 2: replay a chunk from part[item] (no state written).
template <typename T, int DPT, int MODE, int CPT>
__global__ void __launch_bounds__(kDsMaxThreads) decay_scan_kernel(const DecayScanParams p, int NSL) {
    extern __shared__ __align__(16) float ds_smem[];
    const int dpad = NSL * DPT;
    const int ccols = blockDim.x / NSL * CPT;       // value columns of this CTA
    float* Qs = ds_smem;                               // [kDsTokens][dpad]
    float* Ks = Qs + kDsTokens * dpad;                 // [kDsTokens][dpad]
    float* Vs = Ks + kDsTokens * dpad;                 // [kDsTokens][ccols]
    float* As = Vs + kDsTokens * ccols;                // [kDsTokens] decay
    float* Ss = As + kDsTokens;                        // [kDsTokens] input scale
    const int slice = threadIdx.x % NSL, cgrp = threadIdx.x / NSL;
    const int h = blockIdx.y, cl = cgrp * CPT, c = blockIdx.z * ccols + cl;
    const int g = h / (p.heads / p.groups);
    const int* it = p.items + 4 * blockIdx.x;
    const int row0 = it[0], n = it[1], slot = it[2];
    const int d0 = slice * DPT;
    const int64_t sz = (int64_t)p.dim * p.vdim;

    float S[DPT][CPT];
    const float* src = MODE == 0 ? p.state + ((int64_t)slot * p.heads + h) * sz
                     : MODE == 2 ? p.part + ((int64_t)blockIdx.x * p.heads + h) * (sz + 1) : nullptr;
#pragma unroll
    for (int i = 0; i < DPT; ++i)
#pragma unroll
        for (int j = 0; j < CPT; ++j)
            S[i][j] = (MODE != 1 && d0 + i < p.dim && c + j < p.vdim) ? src[(int64_t)(d0 + i) * p.vdim + c + j] : 0.f;
    float total = 1.f;                                 // product of the decays (MODE 1)
    const float hd = p.dt ? 0.f : p.decay[h];
    const float a_rate = p.dt ? -expf(p.a_log[h]) : 0.f, dtb = p.dt ? p.dt_bias[h] : 0.f;
    const float skip = p.skip ? p.skip[h] : 0.f;
    const T* qb = static_cast<const T*>(p.q) + p.q_off + (int64_t)g * p.dim;
    const T* kb = static_cast<const T*>(p.k) + p.k_off + (int64_t)g * p.dim;
    const T* vb = static_cast<const T*>(p.v) + p.v_off + (int64_t)h * p.vdim + (int64_t)blockIdx.z * ccols;
    const int vcols = min(ccols, p.vdim - blockIdx.z * ccols);

    // rows whose pieces start on 16-byte boundaries are staged with 16-byte loads (`vec`, checked by the host); the columns
    // past dim / past this CTA's share of vdim are zeroed once and never written again
    constexpr int VN = 16 / sizeof(T);
    if (p.vec) {
        for (int idx = threadIdx.x; idx < kDsTokens * dpad; idx += blockDim.x) Qs[idx] = Ks[idx] = 0.f;
        for (int idx = threadIdx.x; idx < kDsTokens * ccols; idx += blockDim.x) Vs[idx] = 0.f;
    }
    for (int t0 = 0; t0 < n; t0 += kDsTokens) {
        const int nt = min(kDsTokens, n - t0);
        __syncthreads();
        if (p.vec) {
            const int kvecs = p.dim / VN, vvecs = vcols / VN;
            for (int idx = threadIdx.x; idx < nt * kvecs; idx += blockDim.x) {
                const int t = idx / kvecs, d = (idx % kvecs) * VN;
                float kf[VN], qf[VN];
                ds_load16<T>(kb + (int64_t)(row0 + t0 + t) * p.k_stride + d, kf);
                if (MODE != 1) ds_load16<T>(qb + (int64_t)(row0 + t0 + t) * p.q_stride + d, qf);
#pragma unroll
                for (int i = 0; i < VN; ++i) {
                    if (MODE == 1) qf[i] = 0.f;
                    if (p.act) { qf[i] = silu_f32(qf[i]); kf[i] = silu_f32(kf[i]); }
                }
#pragma unroll
                for (int i = 0; i < VN; i += 4) {
                    *reinterpret_cast<float4*>(Ks + t * dpad + d + i) = make_float4(kf[i], kf[i + 1], kf[i + 2], kf[i + 3]);
                    *reinterpret_cast<float4*>(Qs + t * dpad + d + i) = make_float4(qf[i], qf[i + 1], qf[i + 2], qf[i + 3]);
                }
            }
            for (int idx = threadIdx.x; idx < nt * vvecs; idx += blockDim.x) {
                const int t = idx / vvecs, cc = (idx % vvecs) * VN;
                float xf[VN];
                ds_load16<T>(vb + (int64_t)(row0 + t0 + t) * p.v_stride + cc, xf);
#pragma unroll
                for (int i = 0; i < VN; ++i)
                    if (p.act) xf[i] = silu_f32(xf[i]);
#pragma unroll
                for (int i = 0; i < VN; i += 4)
                    *reinterpret_cast<float4*>(Vs + t * ccols + cc + i) = make_float4(xf[i], xf[i + 1], xf[i + 2], xf[i + 3]);
            }
        } else {
        for (int idx = threadIdx.x; idx < nt * dpad; idx += blockDim.x) {
            const int t = idx / dpad, d = idx % dpad;
            float qv = 0.f, kv = 0.f;
            if (d < p.dim) {
                kv = to_f32<T>(kb[(int64_t)(row0 + t0 + t) * p.k_stride + d]);
                if (MODE != 1) qv = to_f32<T>(qb[(int64_t)(row0 + t0 + t) * p.q_stride + d]);
                if (p.act) { qv = silu_f32(qv); kv = silu_f32(kv); }
            }
            Qs[idx] = qv;
            Ks[idx] = kv;
        }
        for (int idx = threadIdx.x; idx < nt * ccols; idx += blockDim.x) {
            const int t = idx / ccols, cc = idx % ccols;
            float x = cc < vcols ? to_f32<T>(vb[(int64_t)(row0 + t0 + t) * p.v_stride + cc]) : 0.f;
            if (p.act) x = silu_f32(x);
            Vs[idx] = x;
        }
        }
        if (threadIdx.x < nt) {
            float a = hd, sc = p.k_scale;              // the key's factor rides on its value: only k v^T is kept
            if (p.dt) {
                const float raw = to_f32<T>(static_cast<const T*>(p.dt)[(int64_t)(row0 + t0 + threadIdx.x) * p.dt_stride + p.dt_off + h]);
                sc = softplus_f32(raw + dtb);
                a = expf(a_rate * sc);
            }
            As[threadIdx.x] = a;
            Ss[threadIdx.x] = sc;
        }
        __syncthreads();
        if (p.rope) {
            const int half = p.rot_dims >> 1;
            for (int idx = threadIdx.x; idx < nt * half; idx += blockDim.x) {
                const int t = idx / half, i = idx % half;
                const float2 cs = *reinterpret_cast<const float2*>(p.rope + ((int64_t)(row0 + t0 + t) * half + i) * 2);
                float* kr = Ks + t * dpad + i;
                const float ku = kr[0], kw = kr[half];
                kr[0] = ku * cs.x - kw * cs.y;
                kr[half] = kw * cs.x + ku * cs.y;
                if (MODE != 1) {
                    float* qr = Qs + t * dpad + i;
                    const float qu = qr[0], qw = qr[half];
                    qr[0] = qu * cs.x - qw * cs.y;
                    qr[half] = qw * cs.x + qu * cs.y;
                }
            }
            __syncthreads();
        }
        for (int t = 0; t < nt; ++t) {
            const float a = As[t], sc = Ss[t];
            float x[CPT];
            if (CPT == 4) {
                const float4 x4 = *reinterpret_cast<const float4*>(Vs + t * ccols + cl);
                x[0] = x4.x; x[1] = x4.y; x[CPT - 2] = x4.z; x[CPT - 1] = x4.w;
            } else {
                const float2 x2 = *reinterpret_cast<const float2*>(Vs + t * ccols + cl);
                x[0] = x2.x; x[1] = x2.y;
            }
            float xv[CPT], o[CPT];
#pragma unroll
            for (int j = 0; j < CPT; ++j) { xv[j] = x[j] * sc; o[j] = 0.f; }
            const float* kt = Ks + t * dpad + d0;
            const float* qt = Qs + t * dpad + d0;
#pragma unroll
            for (int i = 0; i < DPT; i += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(kt + i);
                const float kk[4] = {k4.x, k4.y, k4.z, k4.w};
                float qq[4] = {0.f, 0.f, 0.f, 0.f};
                if (MODE != 1) {
                    const float4 q4 = *reinterpret_cast<const float4*>(qt + i);
                    qq[0] = q4.x; qq[1] = q4.y; qq[2] = q4.z; qq[3] = q4.w;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int j = 0; j < CPT; ++j) {
                        S[i + u][j] = fmaf(a, S[i + u][j], kk[u] * xv[j]);
                        if (MODE != 1) o[j] = fmaf(S[i + u][j], qq[u], o[j]);
                    }
            }
            total *= a;
            if (MODE != 1) {
                for (int w = 1; w < NSL; w <<= 1)
#pragma unroll
                    for (int j = 0; j < CPT; ++j) o[j] += __shfl_xor_sync(0xffffffffu, o[j], w);
                if (slice == 0) {
                    float* dst = p.out + (int64_t)(row0 + t0 + t) * p.out_stride + (int64_t)h * p.vdim + c;
#pragma unroll
                    for (int j = 0; j < CPT; ++j)
                        if (c + j < p.vdim) dst[j] = fmaf(skip, x[j], o[j]);
                }
            }
        }
    }
    if (MODE == 2) return;
    float* dst = MODE == 0 ? p.state + ((int64_t)slot * p.heads + h) * sz : p.part + ((int64_t)blockIdx.x * p.heads + h) * (sz + 1);
#pragma unroll
    for (int i = 0; i < DPT; ++i)
#pragma unroll
        for (int j = 0; j < CPT; ++j)
            if (d0 + i < p.dim && c + j < p.vdim) dst[(int64_t)(d0 + i) * p.vdim + c + j] = S[i][j];
    if (MODE == 1 && threadIdx.x == 0 && blockIdx.z == 0) dst[sz] = total;
}

// ---- fold and replay of chunks of up to 64 tokens as matrix products (constant decays, bfloat16 rows) -----------------------
// With a constant decay d the tokens of a chunk need no walk:  fold   S = sum_t d^(n-1-t) k_t v_t^T
//                                                             replay o_t = sum_{s<=t} d^(t-s) (q_t . k_s) v_s + d^(t+1) S0^T q_t
// and both run on the tensor cores (mma.sync m16n8k16, float accumulators) WITHOUT giving up float operands: every float factor
// (rotated q and k, weighted k, the scores with their decays, the incoming state) is the sum of three bfloat16 numbers, 24 bits
// of it, and a product of two such factors keeps the six terms that reach 2^-24; the value rows are bfloat16 as they come.  One CTA
// of four warps per (chunk, head); a warp has 16 rows of the result.
// What bounds it: issue of ldmatrix and mma.sync.  4 x 2048 tokens, 16 heads of 64 x 128: fold 62 us, replay 154 us; the
// walk on the float pipe 141 and 231 us.  Error of the layer against float64 4.3e-3 either way (rounding of the result).
// A product adds zero times what a walk never meets (later tokens' values) and takes an infinity apart into planes.  So a chunk whose
// operands or incoming state hold a number that is not finite, or so large that a sum of products could overflow, is walked
// by the same CTA (dm_walk), as is a decay above one.  Looking for such numbers costs 2 us in the fold and 8 us in the replay.
constexpr int kDmTokens = 64, kDmDim = 64, kDmLd = kDmDim + 8, kDmThreads = 128;
constexpr float kDmMost = 68719476736.f;      // 2^36: 64 x 64 products of three such numbers stay below 2^120

__device__ __forceinline__ void dm_split(float x, bf16_t (&b)[3]) {
    b[0] = __float2bfloat16_rn(x);
    const float hi = __bfloat162float(b[0]);
    float r = isfinite(hi) ? x - hi : 0.f;
    b[1] = __float2bfloat16_rn(r);
    r -= __bfloat162float(b[1]);
    b[2] = __float2bfloat16_rn(r);
}
// the largest magnitudes seen, or NaN
__device__ __forceinline__ void dm_note(__nv_bfloat162& top, uint32_t pair) {
    top = __hmax2_nan(top, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&pair)));
}
__device__ __forceinline__ bool dm_big(__nv_bfloat162 top) { return !(__low2float(top) < kDmMost) || !(__high2float(top) < kDmMost); }
// two neighbouring columns split into three planes `plane` elements apart
__device__ __forceinline__ void dm_store2(bf16_t* dst, int plane, float x, float y, __nv_bfloat162& top) {
    bf16_t a[3], b[3];
    dm_split(x, a);
    dm_split(y, b);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        __nv_bfloat162 v;
        v.x = a[i];
        v.y = b[i];
        const uint32_t bits = *reinterpret_cast<const uint32_t*>(&v);
        if (i == 0) dm_note(top, bits);
        *reinterpret_cast<uint32_t*>(dst + i * plane) = bits;
    }
}
// rows of q or k of one head: rotated (halves), times f(token), zeros past the chunk's end
template <typename F>
__device__ __forceinline__ void dm_stage(const float* rope, int rot_dims, const bf16_t* src, int64_t stride, int row0, int n, bf16_t* dst,
                                         __nv_bfloat162& top, F f) {
    const int half = rope ? rot_dims >> 1 : 0;
    constexpr int U = 8;                                    // pieces of two columns whose loads are in flight together
#pragma unroll 1
    for (int i0 = 0; i0 < kDmTokens * kDmDim / 2; i0 += U * kDmThreads) {
        uint32_t xw[U], yw[U];
        float4 cs[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int idx = i0 + u * kDmThreads + threadIdx.x, t = idx / (kDmDim / 2), d = idx % (kDmDim / 2) * 2;
            const bool ok = t < n;
            const bf16_t* r = src + (int64_t)(row0 + (ok ? t : 0)) * stride;
            xw[u] = ok ? *reinterpret_cast<const uint32_t*>(r + d) : 0u;
            yw[u] = ok && d < half ? *reinterpret_cast<const uint32_t*>(r + d + half) : 0u;
            cs[u] = make_float4(1.f, 0.f, 1.f, 0.f);
            if (ok && d < half) cs[u] = *reinterpret_cast<const float4*>(rope + ((int64_t)(row0 + t) * half + d) * 2);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int idx = i0 + u * kDmThreads + threadIdx.x, t = idx / (kDmDim / 2), d = idx % (kDmDim / 2) * 2;
            if (d >= half && d < 2 * half) continue;        // the partners of the first half
            const float w = t < n ? f(t) : 0.f;
            const float x0 = __uint_as_float(xw[u] << 16), x1 = __uint_as_float(xw[u] & 0xffff0000u);
            const float y0 = __uint_as_float(yw[u] << 16), y1 = __uint_as_float(yw[u] & 0xffff0000u);
            if (d < half)
                dm_store2(dst + t * kDmLd + d + half, kDmTokens * kDmLd, (y0 * cs[u].x + x0 * cs[u].y) * w, (y1 * cs[u].z + x1 * cs[u].w) * w, top);
            dm_store2(dst + t * kDmLd + d, kDmTokens * kDmLd, (x0 * cs[u].x - y0 * cs[u].y) * w, (x1 * cs[u].z - y1 * cs[u].w) * w, top);
        }
    }
}
template <int VD>
__device__ __forceinline__ void dm_stage_values(const DecayScanParams& p, int h, int row0, int n, bf16_t* dst, __nv_bfloat162& top) {
    const bf16_t* vb = static_cast<const bf16_t*>(p.v) + p.v_off + (int64_t)h * VD;
#pragma unroll
    for (int i = 0; i < kDmTokens * VD / 8 / kDmThreads; ++i) {
        const int idx = i * kDmThreads + threadIdx.x, t = idx / (VD / 8), c = idx % (VD / 8) * 8;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (t < n) v = *reinterpret_cast<const uint4*>(vb + (int64_t)(row0 + t) * p.v_stride + c);
        *reinterpret_cast<uint4*>(dst + t * (VD + 8) + c) = v;
        dm_note(top, v.x);
        dm_note(top, v.y);
        dm_note(top, v.z);
        dm_note(top, v.w);
    }
}
// d^0 .. d^64
__device__ __forceinline__ void dm_powers(float d, float* pw) {
    for (int j = threadIdx.x; j <= kDmTokens; j += blockDim.x) {
        double r = 1.0, b = d;
        for (int e = j; e; e >>= 1, b *= b)
            if (e & 1) r *= b;
        pw[j] = (float)r;
    }
}
// o[n-tile] += A (16 x 16, fragment a) . B: 16 rows of a [.][ld] matrix from row k0, all VD columns
template <int VD>
__device__ __forceinline__ void dm_rows_product(float (&o)[VD / 8][4], const uint32_t (&a)[4], const bf16_t* B, int ld, int k0, int lane) {
#pragma unroll
    for (int np = 0; np < VD / 16; ++np) {
        uint32_t b0, b1, b2, b3;
        ldsm_x4_trans(smem_u32(B + (k0 + (lane & 7) + ((lane >> 3) & 1) * 8) * ld + np * 16 + (lane >> 4) * 8), b0, b1, b2, b3);
        mma_bf16_16816(o[2 * np], a, b0, b1);
        mma_bf16_16816(o[2 * np + 1], a, b2, b3);
    }
}

// The chunk token by token, a thread per column of the state.  Ks, Qs: [3][64][kDmLd] rotated and scaled rows in planes, of which `staged`
// (times `scale`) is brought in first, Vs: [64][VD + 8].  S0: the incoming state (null: zeros); Qs null: no outputs; end: where the state
// after the chunk goes (or null).  Out of line: the products around it keep their registers.
template <int VD>
__device__ __noinline__ void dm_walk(const float* rope, int rot_dims, const bf16_t* src, int64_t stride, int row0, int n, bf16_t* staged, float scale,
                                     const bf16_t* Ks, const bf16_t* Vs, const bf16_t* Qs, float a, const float* S0, float* out,
                                     int64_t out_stride, float* end) {
    __nv_bfloat162 top = __float2bfloat162_rn(0.f);
    dm_stage(rope, rot_dims, src, stride, row0, n, staged, top, [&](int) { return scale; });
    __syncthreads();
    const int c = threadIdx.x;
    if (c >= VD) return;
    auto whole = [](const bf16_t* x) {          // the three planes of a number, whose sum is exact
        return (__bfloat162float(x[2 * kDmTokens * kDmLd]) + __bfloat162float(x[kDmTokens * kDmLd])) + __bfloat162float(x[0]);
    };
    float S[kDmDim];
#pragma unroll
    for (int d = 0; d < kDmDim; ++d) S[d] = S0 ? S0[(int64_t)d * VD + c] : 0.f;
    for (int t = 0; t < n; ++t) {
        const float x = __bfloat162float(Vs[t * (VD + 8) + c]);
        float o = 0.f;
#pragma unroll
        for (int d = 0; d < kDmDim; ++d) {
            S[d] = fmaf(a, S[d], whole(Ks + t * kDmLd + d) * x);
            if (Qs) o = fmaf(S[d], whole(Qs + t * kDmLd + d), o);
        }
        if (Qs) out[t * out_stride + c] = o;
    }
    if (end) {
#pragma unroll
        for (int d = 0; d < kDmDim; ++d) end[(int64_t)d * VD + c] = S[d];
    }
}

template <int VD>
__global__ void __launch_bounds__(kDmThreads) decay_fold_mma_kernel(const DecayScanParams p) {
    extern __shared__ __align__(16) unsigned char dm_smem[];
    bf16_t* Ks = reinterpret_cast<bf16_t*>(dm_smem);                  // [3][64][kDmLd]
    bf16_t* Vs = Ks + 3 * kDmTokens * kDmLd;                          // [64][VD + 8]
    __shared__ float pw[kDmTokens + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = blockIdx.y, g = h / (p.heads / p.groups);
    const int* it = p.items + 4 * blockIdx.x;
    const int row0 = it[0], n = it[1];
    const float decay = p.decay[h];
    const bf16_t* kb = static_cast<const bf16_t*>(p.k) + p.k_off + (int64_t)g * kDmDim;
    const int64_t sz = (int64_t)kDmDim * VD;
    float* dst = p.part + ((int64_t)blockIdx.x * p.heads + h) * (sz + 1);
    __nv_bfloat162 top = __float2bfloat162_rn(fabsf(decay) <= 1.f ? 0.f : kDmMost);
    dm_powers(decay, pw);
    dm_stage_values<VD>(p, h, row0, n, Vs, top);
    __syncthreads();
    dm_stage(p.rope, p.rot_dims, kb, p.k_stride, row0, n, Ks, top, [&](int t) { return pw[n - 1 - t] * p.k_scale; });
    if (threadIdx.x == 0) dst[sz] = pw[n];
    if (__syncthreads_or(dm_big(top))) {
        dm_walk<VD>(p.rope, p.rot_dims, kb, p.k_stride, row0, n, Ks, p.k_scale, Ks, Vs, nullptr, decay, nullptr, nullptr, 0, dst);
        return;
    }
    float o[VD / 8][4];
#pragma unroll
    for (int i = 0; i < VD / 8; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) o[i][c] = 0.f;
#pragma unroll
    for (int x = 2; x >= 0; --x)                                      // the small terms first
#pragma unroll
        for (int ks = 0; ks < kDmTokens; ks += 16) {
            uint32_t a[4];                                            // rows = dimensions, read across the tokens' rows
            ldsm_x4_trans(smem_u32(Ks + (x * kDmTokens + ks + (lane & 7) + (lane >> 4) * 8) * kDmLd + warp * 16 + ((lane >> 3) & 1) * 8), a[0],
                          a[1], a[2], a[3]);
            dm_rows_product<VD>(o, a, Vs, VD + 8, ks, lane);
        }
#pragma unroll
    for (int i = 0; i < VD / 8; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) dst[(warp * 16 + (lane >> 2) + (c >> 1) * 8) * VD + i * 8 + 2 * (lane & 3) + (c & 1)] = o[i][c];
}

template <int VD>
__global__ void __launch_bounds__(kDmThreads, 2) decay_replay_mma_kernel(const DecayScanParams p) {
    extern __shared__ __align__(16) unsigned char dm_smem[];
    bf16_t* Ks = reinterpret_cast<bf16_t*>(dm_smem);                  // [3][64][kDmLd]
    bf16_t* Vs = Ks + 3 * kDmTokens * kDmLd;                          // [64][VD + 8]
    bf16_t* Ss = Vs + kDmTokens * (VD + 8);                           // [3][64][VD + 8]: first the queries, then the incoming state
    __shared__ float pw[kDmTokens + 1];
    __shared__ int big[kDmThreads / 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = blockIdx.y, g = h / (p.heads / p.groups);
    const int* it = p.items + 4 * blockIdx.x;
    const int row0 = it[0], n = it[1];
    const float decay = p.decay[h];
    const bf16_t* qb = static_cast<const bf16_t*>(p.q) + p.q_off + (int64_t)g * kDmDim;
    __nv_bfloat162 top = __float2bfloat162_rn(fabsf(decay) <= 1.f ? 0.f : kDmMost);
    dm_powers(decay, pw);
    dm_stage_values<VD>(p, h, row0, n, Vs, top);
    dm_stage(p.rope, p.rot_dims, static_cast<const bf16_t*>(p.k) + p.k_off + (int64_t)g * kDmDim, p.k_stride, row0, n, Ks, top, [&](int) { return p.k_scale; });
    dm_stage(p.rope, p.rot_dims, qb, p.q_stride, row0, n, Ss, top, [](int) { return 1.f; });
    __syncthreads();
    uint32_t qf[3][kDmDim / 16][4];
#pragma unroll
    for (int x = 0; x < 3; ++x)
#pragma unroll
        for (int ks = 0; ks < kDmDim / 16; ++ks)
            ldsm_x4(smem_u32(Ss + (x * kDmTokens + warp * 16 + (lane & 15)) * kDmLd + ks * 16 + (lane >> 4) * 8), qf[x][ks][0], qf[x][ks][1],
                    qf[x][ks][2], qf[x][ks][3]);
    __syncthreads();
    const int64_t sz = (int64_t)kDmDim * VD;
    const float* S0 = p.part + ((int64_t)blockIdx.x * p.heads + h) * (sz + 1);
#pragma unroll 1
    for (int i0 = 0; i0 < kDmDim * VD / 2; i0 += 16 * kDmThreads) {
        float x[16], y[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const int at = (i0 + u * kDmThreads + threadIdx.x) * 2;
            x[u] = S0[at];
            y[u] = S0[at + 1];
        }
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const int idx = i0 + u * kDmThreads + threadIdx.x, d = idx / (VD / 2), c = idx % (VD / 2) * 2;
            dm_store2(Ss + d * (VD + 8) + c, kDmDim * (VD + 8), x[u], y[u], top);
        }
    }
    const bool big_w = __any_sync(0xffffffffu, dm_big(top));
    if (lane == 0) big[warp] = big_w;
    // scores of this warp's tokens against the keys up to them
    float s[kDmTokens / 8][4];
#pragma unroll
    for (int i = 0; i < kDmTokens / 8; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) s[i][c] = 0.f;
#pragma unroll
    for (int np = 0; np < kDmTokens / 16; ++np) {
        if (np > warp) break;
#pragma unroll
        for (int ks = 0; ks < kDmDim / 16; ++ks)
#pragma unroll
            for (int y = 2; y >= 0; --y) {
                uint32_t b0, b1, b2, b3;
                ldsm_x4(smem_u32(Ks + (y * kDmTokens + np * 16 + (lane & 7) + ((lane >> 4) << 3)) * kDmLd + ks * 16 + ((lane >> 3) & 1) * 8), b0,
                        b1, b2, b3);
#pragma unroll
                for (int x = 2 - y; x >= 0; --x) {
                    mma_bf16_16816(s[2 * np], qf[x][ks], b0, b1);
                    mma_bf16_16816(s[2 * np + 1], qf[x][ks], b2, b3);
                }
            }
    }
    __syncthreads();                                                  // the state is staged
    float o[VD / 8][4];
#pragma unroll
    for (int i = 0; i < VD / 8; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) o[i][c] = 0.f;
#pragma unroll
    for (int y = 2; y >= 0; --y)
#pragma unroll
        for (int x = 2 - y; x >= 0; --x)
#pragma unroll
            for (int ks = 0; ks < kDmDim / 16; ++ks) dm_rows_product<VD>(o, qf[x][ks], Ss + y * kDmDim * (VD + 8), VD + 8, ks * 16, lane);
    const int t0 = warp * 16 + (lane >> 2);
    const float in0 = pw[t0 + 1], in1 = pw[t0 + 9];
#pragma unroll
    for (int i = 0; i < VD / 8; ++i) {
        o[i][0] *= in0;
        o[i][1] *= in0;
        o[i][2] *= in1;
        o[i][3] *= in1;
    }
#pragma unroll
    for (int kk = 0; kk < kDmTokens / 16; ++kk) {
        if (kk > warp) break;
        uint32_t a[3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {                                 // rows g, g + 8, then the second eight keys
            const int i = 2 * kk + (j >> 1), r = j & 1;
            bf16_t u[3], w[3];
            const int dist = t0 + 8 * r - (i * 8 + 2 * (lane & 3));
            dm_split(dist >= 0 ? s[i][2 * r] * pw[dist] : 0.f, u);
            dm_split(dist >= 1 ? s[i][2 * r + 1] * pw[dist - 1] : 0.f, w);
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                __nv_bfloat162 v;
                v.x = u[x];
                v.y = w[x];
                a[x][j] = *reinterpret_cast<const uint32_t*>(&v);
            }
        }
#pragma unroll
        for (int x = 2; x >= 0; --x) dm_rows_product<VD>(o, a[x], Vs, VD + 8, kk * 16, lane);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int t = t0 + 8 * r;
        if (t >= n) continue;
        float* dst = p.out + (int64_t)(row0 + t) * p.out_stride + (int64_t)h * VD + 2 * (lane & 3);
#pragma unroll
        for (int i = 0; i < VD / 8; ++i) *reinterpret_cast<float2*>(dst + i * 8) = make_float2(o[i][2 * r], o[i][2 * r + 1]);
    }
    __syncthreads();
    if (big[0] | big[1] | big[2] | big[3]) {
        dm_walk<VD>(p.rope, p.rot_dims, qb, p.q_stride, row0, n, Ss, 1.f, Ks, Vs, Ss, decay, S0,
                    p.out + (int64_t)row0 * p.out_stride + (int64_t)h * VD, p.out_stride, nullptr);
        return;
    }
}

// Whether the chunks run as matrix products: chunks of at most 64 tokens, bfloat16 rows, a constant decay, no activation, states of
// 64 x 64 or 64 x 128, and rows whose staged pieces are aligned.
static bool dm_ok(const DecayScanParams& p, int chunk_tokens, int elem) {
    return chunk_tokens > 0 && chunk_tokens <= kDmTokens && elem == 2 && !p.dt && !p.act && !p.skip && p.dim == kDmDim &&
           (p.vdim == 64 || p.vdim == 128) && p.rot_dims % 4 == 0 && (uintptr_t)p.rope % 16 == 0 && p.q_stride % 2 == 0 && p.q_off % 2 == 0 &&
           (uintptr_t)p.q % 4 == 0 && p.k_stride % 2 == 0 && p.k_off % 2 == 0 && (uintptr_t)p.k % 4 == 0 && p.v_stride % 8 == 0 &&
           p.v_off % 8 == 0 && (uintptr_t)p.v % 16 == 0 && p.out_stride % 2 == 0 && (uintptr_t)p.out % 8 == 0;
}
template <int VD, bool REPLAY>
static int dm_launch(const DecayScanParams& p, int num_items, cudaStream_t st) {
    const size_t smem = sizeof(bf16_t) * (3 * kDmTokens * kDmLd + kDmTokens * (VD + 8) + (REPLAY ? 3 * kDmDim * (VD + 8) : 0));
    auto kern = REPLAY ? decay_replay_mma_kernel<VD> : decay_fold_mma_kernel<VD>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    kern<<<dim3((unsigned)num_items, (unsigned)p.heads), kDmThreads, smem, st>>>(p);
    PA_RETURN_LAUNCH_STATUS();
}

// Chain pass of the chunked scan: per (portion, head, state element) walk the portion's chunks in order from the state
// slot; every chunk's folded state is replaced by its INCOMING state, and the slot gets the state after the last chunk.
__global__ void __launch_bounds__(256) decay_chunk_chain_kernel(float* __restrict__ part, int heads, int64_t sz,
                                                                const int32_t* __restrict__ seq_chunk0,
                                                                const int32_t* __restrict__ seq_nchunks,
                                                                const int32_t* __restrict__ seq_slot, float* __restrict__ state) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int h = blockIdx.y, s = blockIdx.z;
    if (e >= sz) return;
    const int n = seq_nchunks[s], k0 = seq_chunk0[s];
    if (n <= 0) return;
    float* sp = state + ((int64_t)seq_slot[s] * heads + h) * sz + e;
    float S = *sp;
    // the folded values of 8 chunks are read before any incoming state is written over them: the loads do not wait on
    // the chain
    constexpr int U = 8;
    for (int k = k0; k < k0 + n; k += U) {
        float A[U], B[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool ok = k + u < k0 + n;
            const float* pk = part + ((int64_t)(ok ? k + u : k) * heads + h) * (sz + 1);
            A[u] = ok ? pk[sz] : 1.f;
            B[u] = ok ? pk[e] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (k + u < k0 + n) part[((int64_t)(k + u) * heads + h) * (sz + 1) + e] = S;
            S = fmaf(A[u], S, B[u]);
        }
    }
    *sp = S;
}

// ---- gated group norm ---------------------------------------------------------------------------------------------------
// One warp per (row, group).  gate_mode 0: none; 1: y <- y * silu(gate) before the norm; 2: out <- norm(y) * sigmoid(gate);
// 3: out <- norm(y) * silu(gate).  weight may be null (ones).
template <typename T>
__global__ void __launch_bounds__(256) gated_norm_kernel(const float* __restrict__ y, int64_t rows, int inner, int groups,
                                                         const T* __restrict__ gate, int64_t gate_stride, int gate_off,
                                                         int gate_mode, const float* __restrict__ weight, float eps,
                                                         T* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= rows * groups) return;
    const int64_t r = w / groups;
    const int gsz = inner / groups, c0 = (int)(w % groups) * gsz;
    const float* yr = y + r * inner + c0;
    const T* gr = gate ? gate + r * gate_stride + gate_off + c0 : nullptr;
    float ss = 0.f;
    for (int j = lane; j < gsz; j += 32) {
        float v = yr[j];
        if (gate_mode == 1) v *= silu_f32(to_f32<T>(gr[j]));
        ss = fmaf(v, v, ss);
    }
    ss = warp_sum(ss);
    const float rn = 1.0f / sqrtf(ss / (float)gsz + eps);
    for (int j = lane; j < gsz; j += 32) {
        float v = yr[j];
        if (gate_mode == 1) v *= silu_f32(to_f32<T>(gr[j]));
        v *= rn;
        if (weight) v *= weight[c0 + j];
        if (gate_mode == 2) v *= sigmoid_f32(to_f32<T>(gr[j]));
        if (gate_mode == 3) v *= silu_f32(to_f32<T>(gr[j]));
        out[r * inner + c0 + j] = from_f32<T>(v);
    }
}

// the same for groups of whole words of four columns (at most 128 NV, aligned): a lane keeps its values in registers, so y and
// the gate are read once, 16 and 8 bytes at a time.  8192 rows of 16 groups of 128 (134 MB): 40 us, 68 us with single columns.
template <typename T, int NV>
__global__ void __launch_bounds__(256) gated_norm_vec_kernel(const float* __restrict__ y, int64_t rows, int inner, int groups,
                                                             const T* __restrict__ gate, int64_t gate_stride, int gate_off,
                                                             int gate_mode, const float* __restrict__ weight, float eps,
                                                             T* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= rows * groups) return;
    const int64_t r = w / groups;
    const int gsz = inner / groups, c0 = (int)(w - r * groups) * gsz;
    const float* yr = y + r * inner + c0;
    const T* gr = gate ? gate + r * gate_stride + gate_off + c0 : nullptr;
    float v[NV][4], gt[NV][4];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int j = 4 * lane + 128 * i;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < gsz) a = *reinterpret_cast<const float4*>(yr + j);
        v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w;
        if (gr && j < gsz) {
            if constexpr (sizeof(T) == 2) {
                const uint2 b = *reinterpret_cast<const uint2*>(gr + j);
                gt[i][0] = __uint_as_float(b.x << 16); gt[i][1] = __uint_as_float(b.x & 0xffff0000u);
                gt[i][2] = __uint_as_float(b.y << 16); gt[i][3] = __uint_as_float(b.y & 0xffff0000u);
            } else {
                const float4 b = *reinterpret_cast<const float4*>(gr + j);
                gt[i][0] = b.x; gt[i][1] = b.y; gt[i][2] = b.z; gt[i][3] = b.w;
            }
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) gt[i][c] = 0.f;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (gate_mode == 1) v[i][c] *= silu_f32(gt[i][c]);
            ss = fmaf(v[i][c], v[i][c], ss);
        }
    }
    ss = warp_sum(ss);
    const float rn = 1.0f / sqrtf(ss / (float)gsz + eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int j = 4 * lane + 128 * i;
        if (j >= gsz) continue;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            v[i][c] *= rn;
            if (weight) v[i][c] *= weight[c0 + j + c];
            if (gate_mode == 2) v[i][c] *= sigmoid_f32(gt[i][c]);
            if (gate_mode == 3) v[i][c] *= silu_f32(gt[i][c]);
        }
        T* o = out + r * inner + c0 + j;
        if constexpr (sizeof(T) == 2) *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16x2(v[i][0], v[i][1]), pack_bf16x2(v[i][2], v[i][3]));
        else *reinterpret_cast<float4*>(o) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
    }
}

// the same with one CTA per (row, group): groups of many values, or few rows
template <typename T>
__global__ void __launch_bounds__(256) gated_norm_block_kernel(const float* __restrict__ y, int inner, int groups,
                                                               const T* __restrict__ gate, int64_t gate_stride, int gate_off,
                                                               int gate_mode, const float* __restrict__ weight, float eps,
                                                               T* __restrict__ out) {
    __shared__ float sm[32];
    const int64_t r = blockIdx.x / groups;
    const int gsz = inner / groups, c0 = (int)(blockIdx.x % groups) * gsz;
    const float* yr = y + r * inner + c0;
    const T* gr = gate ? gate + r * gate_stride + gate_off + c0 : nullptr;
    float ss = 0.f;
    for (int j = threadIdx.x; j < gsz; j += blockDim.x) {
        float v = yr[j];
        if (gate_mode == 1) v *= silu_f32(to_f32<T>(gr[j]));
        ss = fmaf(v, v, ss);
    }
    ss = block_sum(ss, sm);
    const float rn = 1.0f / sqrtf(ss / (float)gsz + eps);
    for (int j = threadIdx.x; j < gsz; j += blockDim.x) {
        float v = yr[j];
        if (gate_mode == 1) v *= silu_f32(to_f32<T>(gr[j]));
        v *= rn;
        if (weight) v *= weight[c0 + j];
        if (gate_mode == 2) v *= sigmoid_f32(to_f32<T>(gr[j]));
        if (gate_mode == 3) v *= silu_f32(to_f32<T>(gr[j]));
        out[r * inner + c0 + j] = from_f32<T>(v);
    }
}

template <typename T, int DPT, int MODE, int CPT>
static int ds_launch(const DecayScanParams& p, int nitems, int NSL, cudaStream_t st) {
    // threads: enough column groups for vdim, whole warps, at most kDsMaxThreads
    int threads = (p.vdim + CPT - 1) / CPT * NSL;
    threads = (threads + 31) / 32 * 32;
    if (threads > kDsMaxThreads) threads = kDsMaxThreads;
    const int ccols = threads / NSL * CPT;
    DecayScanParams q = p;
    {   // 16-byte staging: pointers, row strides, column offsets, dim, vdim and a CTA's share of the columns all whole vectors
        const int VN = 16 / (int)sizeof(T);
        auto al = [&](const void* ptr, int64_t stride, int off) {
            return (uintptr_t)ptr % 16 == 0 && stride % VN == 0 && off % VN == 0;
        };
        q.vec = p.dim % VN == 0 && p.vdim % VN == 0 && ccols % VN == 0 && al(p.q, p.q_stride, p.q_off) &&
                al(p.k, p.k_stride, p.k_off) && al(p.v, p.v_stride, p.v_off);
    }
    const size_t smem = ((size_t)2 * kDsTokens * NSL * DPT + (size_t)kDsTokens * ccols + 2 * kDsTokens) * sizeof(float);
    if (smem > 200 * 1024) return PA_ERR_UNSUPPORTED;
    auto kern = decay_scan_kernel<T, DPT, MODE, CPT>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    dim3 grid((unsigned)nitems, (unsigned)p.heads, (unsigned)((p.vdim + ccols - 1) / ccols));
    kern<<<grid, threads, smem, st>>>(q, NSL);
    PA_RETURN_LAUNCH_STATUS();
}

// A thread's block of the state is DPT rows x CPT columns.  States of up to 64 rows: 16 x 4 (64 state registers, about
// twice the resident warps of 32 x 4; measured 1.3x faster at 64 rows).  Larger ones: 32 x 4.  Measured at 128 rows x 64
// columns: 16 x 4 (eight row slices, a three-round shuffle reduction) the same time, 32 x 2 (twice the warps, but twice
// the shared-memory operand reads per update) 1.6x slower -- the kernel is bound by those reads and the shuffles, so the
// block that feeds the most updates per read wins.
template <typename T, int MODE>
static int ds_dispatch(const DecayScanParams& p, int nitems, cudaStream_t st) {
    if (p.dim <= 8) return ds_launch<T, 8, MODE, 4>(p, nitems, 1, st);
    if (p.dim <= 64) return ds_launch<T, 16, MODE, 4>(p, nitems, p.dim <= 16 ? 1 : p.dim <= 32 ? 2 : 4, st);
    int NSL = 4;
    while (NSL * 32 < p.dim) NSL <<= 1;
    if (NSL > 32) return PA_ERR_UNSUPPORTED;
    return ds_launch<T, 32, MODE, 4>(p, nitems, NSL, st);
}

}  // namespace pa

using namespace pa;

PA_API int pa_causal_conv_silu(const void* d_in, int64_t in_stride, int in_off, int channels, int taps, const float* d_weight,
                               const float* d_bias, const float* d_state, const int32_t* d_chunks, int num_chunks,
                               void* d_out, int64_t out_stride, int elem, pa_stream_t stream) {
    return pa_causal_conv(d_in, in_stride, in_off, channels, taps, d_weight, d_bias, 1, d_state, d_chunks, num_chunks, d_out,
                          out_stride, elem, stream);
}

PA_API int pa_causal_conv(const void* d_in, int64_t in_stride, int in_off, int channels, int taps, const float* d_weight,
                          const float* d_bias, int act, const float* d_state, const int32_t* d_chunks, int num_chunks,
                          void* d_out, int64_t out_stride, int elem, pa_stream_t stream) {
    PA_CHECK_ARG(d_in && d_weight && (d_state || taps == 1) && d_chunks && d_out && channels > 0 && num_chunks >= 0);
    PA_CHECK_ARG(taps >= 1 && taps <= kMaxTaps && (act == 0 || act == 1));
    if (num_chunks == 0) return PA_OK;
    dim3 grid((unsigned)((channels + 127) / 128), (unsigned)num_chunks);
    PA_DISPATCH_ELEM(elem, causal_conv_kernel<T><<<grid, 128, 0, as_stream(stream)>>>(
                               static_cast<const T*>(d_in), in_stride, in_off, channels, taps, d_weight, d_bias, d_state,
                               d_chunks, static_cast<T*>(d_out), out_stride, act));
    PA_RETURN_LAUNCH_STATUS();
}

PA_API int pa_conv_state_update(const void* d_in, int64_t in_stride, int in_off, int channels, int taps,
                                const int32_t* d_seq_start, const int32_t* d_seq_len, const int32_t* d_seq_slot, int num_seqs,
                                float* d_state, int elem, pa_stream_t stream) {
    PA_CHECK_ARG(d_in && d_seq_start && d_seq_len && d_seq_slot && d_state && channels > 0 && num_seqs >= 0);
    PA_CHECK_ARG(taps >= 1 && taps <= kMaxTaps);
    if (num_seqs == 0 || taps == 1) return PA_OK;
    dim3 grid((unsigned)((channels + 127) / 128), (unsigned)num_seqs);
    PA_DISPATCH_ELEM(elem, conv_state_kernel<T><<<grid, 128, 0, as_stream(stream)>>>(
                               static_cast<const T*>(d_in), in_stride, in_off, channels, taps, d_seq_start, d_seq_len,
                               d_seq_slot, d_state));
    PA_RETURN_LAUNCH_STATUS();
}

PA_API size_t pa_decay_scan_workspace_bytes(int num_chunks, int heads, int dim, int vdim) {
    if (num_chunks <= 0 || heads <= 0 || dim <= 0 || vdim <= 0) return 0;
    return (size_t)num_chunks * heads * ((size_t)dim * vdim + 1) * sizeof(float);
}

PA_API int pa_decay_scan(const void* d_q, int64_t q_stride, int q_off, const void* d_k, int64_t k_stride, int k_off,
                         const void* d_v, int64_t v_stride, int v_off, int heads, int groups, int dim, int vdim, int act,
                         const float* d_decay, const void* d_dt, int64_t dt_stride, int dt_off, const float* d_dt_bias,
                         const float* d_a_log, const float* d_skip, float* d_state, float* d_out, int64_t out_stride,
                         const int32_t* d_items, int num_items, const int32_t* d_seq_chunk0, const int32_t* d_seq_nchunks,
                         const int32_t* d_seq_slot, int num_seqs, int chunked, void* d_workspace, size_t workspace_bytes,
                         int elem, pa_stream_t stream) {
    return pa_decay_scan_rotated(d_q, q_stride, q_off, d_k, k_stride, k_off, d_v, v_stride, v_off, heads, groups, dim, vdim, act,
                                 d_decay, d_dt, dt_stride, dt_off, d_dt_bias, d_a_log, d_skip, nullptr, 0, 1.0f, d_state, d_out,
                                 out_stride, d_items, num_items, d_seq_chunk0, d_seq_nchunks, d_seq_slot, num_seqs, chunked,
                                 d_workspace, workspace_bytes, elem, stream);
}

PA_API int pa_decay_scan_rotated(const void* d_q, int64_t q_stride, int q_off, const void* d_k, int64_t k_stride, int k_off,
                         const void* d_v, int64_t v_stride, int v_off, int heads, int groups, int dim, int vdim, int act,
                         const float* d_decay, const void* d_dt, int64_t dt_stride, int dt_off, const float* d_dt_bias,
                         const float* d_a_log, const float* d_skip, const float* d_rope, int rot_dims, float k_scale, float* d_state, float* d_out, int64_t out_stride,
                         const int32_t* d_items, int num_items, const int32_t* d_seq_chunk0, const int32_t* d_seq_nchunks,
                         const int32_t* d_seq_slot, int num_seqs, int chunked, void* d_workspace, size_t workspace_bytes,
                         int elem, pa_stream_t stream) {
    return pa_decay_scan_chunked(d_q, q_stride, q_off, d_k, k_stride, k_off, d_v, v_stride, v_off, heads, groups, dim, vdim, act, d_decay, d_dt,
                                 dt_stride, dt_off, d_dt_bias, d_a_log, d_skip, d_rope, rot_dims, k_scale, d_state, d_out, out_stride, d_items,
                                 num_items, d_seq_chunk0, d_seq_nchunks, d_seq_slot, num_seqs, chunked, d_workspace, workspace_bytes, elem, 0,
                                 stream);
}

PA_API int pa_decay_scan_chunked(const void* d_q, int64_t q_stride, int q_off, const void* d_k, int64_t k_stride, int k_off,
                         const void* d_v, int64_t v_stride, int v_off, int heads, int groups, int dim, int vdim, int act,
                         const float* d_decay, const void* d_dt, int64_t dt_stride, int dt_off, const float* d_dt_bias,
                         const float* d_a_log, const float* d_skip, const float* d_rope, int rot_dims, float k_scale, float* d_state, float* d_out, int64_t out_stride,
                         const int32_t* d_items, int num_items, const int32_t* d_seq_chunk0, const int32_t* d_seq_nchunks,
                         const int32_t* d_seq_slot, int num_seqs, int chunked, void* d_workspace, size_t workspace_bytes,
                         int elem, int chunk_tokens, pa_stream_t stream) {
    PA_CHECK_ARG(d_q && d_k && d_v && d_state && d_out && d_items && num_items >= 0);
    PA_CHECK_ARG(heads > 0 && groups > 0 && heads % groups == 0 && dim > 0 && vdim > 0);
    PA_CHECK_ARG(d_dt ? (d_dt_bias && d_a_log) : d_decay != nullptr);
    PA_CHECK_ARG(rot_dims >= 0 && rot_dims % 2 == 0 && rot_dims <= dim && (rot_dims == 0 || d_rope) && (!d_dt || k_scale == 1.0f));
    if (num_items == 0) return PA_OK;
    if (elem != 4 && elem != 2) return PA_ERR_UNSUPPORTED;
    DecayScanParams p;
    p.q = d_q; p.q_stride = q_stride; p.q_off = q_off; p.k = d_k; p.k_stride = k_stride; p.k_off = k_off;
    p.v = d_v; p.v_stride = v_stride; p.v_off = v_off; p.heads = heads; p.groups = groups; p.dim = dim; p.vdim = vdim;
    p.act = act; p.decay = d_decay; p.dt = d_dt; p.dt_stride = dt_stride; p.dt_off = dt_off; p.dt_bias = d_dt_bias;
    p.a_log = d_a_log; p.skip = d_skip; p.state = d_state; p.out = d_out; p.out_stride = out_stride; p.items = d_items;
    p.part = static_cast<float*>(d_workspace); p.rope = rot_dims ? d_rope : nullptr; p.rot_dims = rot_dims; p.k_scale = k_scale;
    cudaStream_t st = as_stream(stream);
#define PA_DS(MODE)                                                                                \
    do {                                                                                           \
        p.mode = MODE;                                                                             \
        const int rc = elem == 4 ? ds_dispatch<float, MODE>(p, num_items, st) : ds_dispatch<bf16_t, MODE>(p, num_items, st); \
        if (rc != PA_OK) return rc;                                                                \
    } while (0)
    if (!chunked) {
        PA_DS(0);
        return PA_OK;
    }
    PA_CHECK_ARG(d_seq_chunk0 && d_seq_nchunks && d_seq_slot && num_seqs > 0);
    if (!d_workspace || workspace_bytes < pa_decay_scan_workspace_bytes(num_items, heads, dim, vdim)) return PA_ERR_WORKSPACE;
    const bool products = dm_ok(p, chunk_tokens, elem);
    if (products) {
        const int rc = vdim == 64 ? dm_launch<64, false>(p, num_items, st) : dm_launch<128, false>(p, num_items, st);
        if (rc != PA_OK) return rc;
    } else {
        PA_DS(1);
    }
    const int64_t sz = (int64_t)dim * vdim;
    dim3 grid((unsigned)((sz + 255) / 256), (unsigned)heads, (unsigned)num_seqs);
    decay_chunk_chain_kernel<<<grid, 256, 0, st>>>(p.part, heads, sz, d_seq_chunk0, d_seq_nchunks, d_seq_slot, d_state);
    if (products) return vdim == 64 ? dm_launch<64, true>(p, num_items, st) : dm_launch<128, true>(p, num_items, st);
    PA_DS(2);
#undef PA_DS
    PA_RETURN_LAUNCH_STATUS();
}

PA_API int pa_gated_rms_norm(const float* d_y, int64_t rows, int inner, int groups, const void* d_gate, int64_t gate_stride,
                             int gate_off, int gate_mode, const float* d_weight, float eps, void* d_out, int elem,
                             pa_stream_t stream) {
    PA_CHECK_ARG(d_y && d_out && rows >= 0 && inner > 0 && groups > 0 && inner % groups == 0);
    PA_CHECK_ARG(gate_mode >= 0 && gate_mode <= 3 && (gate_mode == 0 || d_gate));
    if (rows == 0) return PA_OK;
    if (inner / groups >= 512 && rows * groups < (1 << 30)) {
        PA_DISPATCH_ELEM(elem, gated_norm_block_kernel<T><<<(unsigned)(rows * groups), 256, 0, as_stream(stream)>>>(
                                   d_y, inner, groups, static_cast<const T*>(d_gate), gate_stride, gate_off, gate_mode, d_weight,
                                   eps, static_cast<T*>(d_out)));
        PA_RETURN_LAUNCH_STATUS();
    }
    const int64_t threads = rows * groups * 32;
    const int gsz = inner / groups;
    const size_t word = (size_t)elem * 4;
    if (gsz % 4 == 0 && (elem == 2 || elem == 4) && (uintptr_t)d_y % 16 == 0 && (uintptr_t)d_out % word == 0 &&
        (!d_gate || ((uintptr_t)d_gate % word == 0 && gate_stride % 4 == 0 && gate_off % 4 == 0))) {
#define PA_GNORM(NV)                                                                                                     \
    PA_DISPATCH_ELEM(elem, (gated_norm_vec_kernel<T, NV><<<(unsigned)((threads + 255) / 256), 256, 0, as_stream(stream)>>>( \
                               d_y, rows, inner, groups, static_cast<const T*>(d_gate), gate_stride, gate_off, gate_mode, \
                               d_weight, eps, static_cast<T*>(d_out))))
        if (gsz <= 128) PA_GNORM(1);
        else if (gsz <= 256) PA_GNORM(2);
        else PA_GNORM(4);                       // below 512 here
#undef PA_GNORM
        PA_RETURN_LAUNCH_STATUS();
    }
    PA_DISPATCH_ELEM(elem, gated_norm_kernel<T><<<(unsigned)((threads + 255) / 256), 256, 0, as_stream(stream)>>>(
                               d_y, rows, inner, groups, static_cast<const T*>(d_gate), gate_stride, gate_off, gate_mode,
                               d_weight, eps, static_cast<T*>(d_out)));
    PA_RETURN_LAUNCH_STATUS();
}
