// masked_attention.cuh -- the operands of one masked-attention launch (masked_attention.cu, attention_tc.cu) and the small
// functions of its scores: what a key at position j gives a query at position i.
#pragma once
#include "seq_common.cuh"

namespace pa {

struct MaskAttnParams {
    const void* q;              // rows of the projection buffer; the query of head h starts at q_off + h * dim
    int64_t q_stride;
    int q_off;
    const void* k_pool;
    const void* v_pool;
    const int32_t* table;
    int num_slots, num_kv_heads, num_tiles, total_pages, tile_size;
    const int32_t* tiles;       // [ntiles][4]: first row, tokens, slot, position of the first token
    int heads, dim, vdim;
    float scale, softcap;
    int mask_kind, mask_size;
    int bias_kind, bias_len;
    const float* bias;          // kind 1: [heads]; kind 2: [bias_len][heads]
    void* out;                  // [rows][heads * vdim]
    const float* head_scale;    // [heads] or null
    const float* sink;          // [heads] or null
    int mask_keep;              // window masks: the first mask_keep positions stay visible
    const float* out_rot;       // [rows][vdim / 2][2] or null
    int sigm;                   // 1: weight = sigmoid(score), nothing divides the sum (no sink)
    const float* key_scale;     // [total_pages * tile_size] or null
    const float* head_bias;     // [heads] or null
    const void* gate;           // rows of the activation type; the gate of output column c of head h at gate_off + h * vdim + c
    int64_t gate_stride;
    int gate_off;
};

__device__ __forceinline__ int ma_first_key(const MaskAttnParams& p, int pos) {
    if (p.mask_kind == 1) return max(0, pos - p.mask_size + 1);
    if (p.mask_kind == 2) return pos / p.mask_size * p.mask_size;
    return 0;
}

__device__ __forceinline__ bool ma_visible(const MaskAttnParams& p, int i, int j) {
    if (j > i) return false;
    if (p.mask_kind == 1) return i - j < p.mask_size || j < p.mask_keep;
    if (p.mask_kind == 2) return i / p.mask_size == j / p.mask_size;
    return true;
}

// The key steps (runs of `keys` positions) the rows of a tile can see, in order: the steps of the kept first positions,
// then the steps from the first key of the tile's first token (ma_first_key) to its last token.  `first` = that first
// key, `total` = keys up to the tile's last token.
struct MaSteps {
    int head, body0, count;
    __device__ __forceinline__ int step(int n) const { return n < head ? n : body0 + n - head; }
};
__device__ __forceinline__ MaSteps ma_steps(const MaskAttnParams& p, int first, int total, int keys) {
    MaSteps s;
    s.body0 = first / keys;
    s.head = 0;
    if (p.mask_kind == 1 && p.mask_keep > 0) s.head = min(s.body0, (min(p.mask_keep, total) + keys - 1) / keys);
    s.count = s.head + (total + keys - 1) / keys - s.body0;
    return s;
}

// the softmax denominator with the sink of head h: returns the factor for the accumulated sums (and updates l)
__device__ __forceinline__ float ma_sink(const MaskAttnParams& p, int h, float m, float& l) {
    if (!p.sink) return 1.f;
    const float sk = p.sink[h];
    const float n = fmaxf(m, sk);
    const float c = m == -INFINITY ? 0.f : expf(m - n);
    l = l * c + expf(sk - n);
    return c;
}

// turns the pair (u, v) = columns (2m, 2m + 1) of batch row `row` back by the row's angle; even = this thread holds u
__device__ __forceinline__ float ma_unturn(const MaskAttnParams& p, int64_t row, int col, float mine, float other) {
    const float* t = p.out_rot + (row * (p.vdim >> 1) + (col >> 1)) * 2;
    return (col & 1) ? mine * t[0] - other * t[1] : mine * t[0] + other * t[1];
}

// the float score of (query position i, key position j, query head h) from the raw dot product
__device__ __forceinline__ float ma_score(const MaskAttnParams& p, float dot, int i, int j, int h, float slope) {
    float s = dot * p.scale;
    if (p.head_scale) s *= p.head_scale[h];
    if (p.softcap > 0.f) s = p.softcap * tanhf(s / p.softcap);
    if (p.bias_kind == 1) s -= slope * (float)(i - j);
    else if (p.bias_kind == 2) s += p.bias[(int64_t)min(i - j, p.bias_len - 1) * p.heads + h];
    if (p.head_bias) s += p.head_bias[h];
    return s;
}

// the factor of output column `col` (of all heads' columns) of batch row `row`
template <typename T>
__device__ __forceinline__ float ma_gate(const MaskAttnParams& p, int64_t row, int col) {
    return sigmoid_f32(to_f32<T>(static_cast<const T*>(p.gate)[row * p.gate_stride + p.gate_off + col]));
}

__device__ __forceinline__ float ma_tanh(float x) {        // 1 - 2 / (e^{2x} + 1), relative error ~1e-6
    const float e = __expf(2.0f * x);
    return 1.0f - __fdividef(2.0f, e + 1.0f);
}

// Prompt portions on tcgen05 (attention_tc.cu).  PA_ERR_UNSUPPORTED: a form, a shape or pointers that stay on mma.sync.
int masked_attention_tc_launch(const MaskAttnParams& p, int ntiles, int q_tiles, cudaStream_t st);

}  // namespace pa
