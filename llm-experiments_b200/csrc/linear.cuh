// Grouped, segmented linear layers (b2kv_linear): what the three kernels behind the entry point share.
#pragma once

#include "b2kv_common.cuh"

namespace b2kv {
namespace lin {

// a / b for b = 1 + exp(..), so from one on, infinity among it: the operator's quotient without its branch to a subroutine.  An
// approximate reciprocal, one step of Newton's for it, and the remainder a - q b, exact in a fused multiply-add, put right what is missing
// of the quotient (Markstein, IBM J. Res. Dev. 34, 1990).  Where the reciprocal would be a subnormal number b is scaled; where the
// remainder is no number (a or b infinite) or nothing is missing the first quotient stands.  For 1 + __expf(-a) and
// 1 + __expf(-1.702 a) it has the operator's bits for each of the 2^32 fp32 numbers a (tried).
__device__ __forceinline__ float quotient(float a, float b) {
    const float s = b > 0x1p100f ? 0x1p-64f : 1.0f;
    b *= s;
    float r = __fdividef(1.0f, b);
    r = fmaf(fmaxf(fmaf(-b, r, 1.0f), -1.0f), r, r);  // (the maximum: 0 for the reciprocal of infinity)
    const float q = a * r, left = fmaf(-q, b, a);
    return (left != 0.0f && fabsf(left) < INFINITY ? fmaf(left, r, q) : q) * s;
}

// x * sigmoid(1.702 x) of the clamped gate times the clamped up part plus one; silu(gate) * up.  An epilogue thread of a tiled product
// has 128 quotients one after the other per tile, whose latencies have to overlap (2975 rows, K = 2048, 10880
// gated columns beside 3648 plain ones: 192 us with the operator's division, 150 so; the experts' 17850 rows x 2816 gated columns: 308 and 230).
__device__ __forceinline__ float glu(int kind, float g, float u, float limit) {
    if (kind == B2KV_SEG_GLU_SILU) return quotient(g, 1.0f + __expf(-g)) * u;
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return quotient(g, 1.0f + __expf(-1.702f * g)) * (u + 1.0f);
}

// Kinds whose columns are (gate, up) pairs; kinds whose output is fp32.
__host__ __device__ constexpr bool is_pair(int kind) { return kind == B2KV_SEG_GLU_SILU || kind == B2KV_SEG_GLU_CLAMP; }
__host__ __device__ constexpr bool is_f32(int kind) { return kind == B2KV_SEG_F32 || kind >= B2KV_SEG_SOFTCAP; }

// sigmoid(z)^(1 / tau) through ln(sigmoid(z)) = min(z, 0) - ln(1 + u), u = exp(-|z|), which cancels on neither side.  Without
// branches or calls: ln(1 + u) = 2 atanh(s), s = u / (2 + u) <= 1/3, as a series whose first dropped term is below 2^-26 of it.
__device__ __forceinline__ float decay(float z, float inv_tau) {
    const float u = __expf(-fabsf(z)), s = __fdividef(u, 2.0f + u), s2 = s * s;
    float p = 1.0f / 15.0f;
    p = fmaf(p, s2, 1.0f / 13.0f);
    p = fmaf(p, s2, 1.0f / 11.0f);
    p = fmaf(p, s2, 1.0f / 9.0f);
    p = fmaf(p, s2, 1.0f / 7.0f);
    p = fmaf(p, s2, 1.0f / 5.0f);
    p = fmaf(p, s2, 1.0f / 3.0f);
    p = fmaf(p, s2, 1.0f);
    return __expf((fminf(z, 0.f) - 2.0f * s * p) * inv_tau);
}
__device__ __forceinline__ float decay_exact(float z, float tau) { return expf((fminf(z, 0.f) - log1pf(expf(-fabsf(z)))) / tau); }

// What happens to a single column before it is stored.
__device__ __forceinline__ float single(int kind, float v, float limit) {
    if (kind == B2KV_SEG_RELU2) {
        v = fmaxf(v, 0.f);
        return v * v;
    }
    if (kind == B2KV_SEG_DECAY) return decay(v, 1.0f / limit);
    return kind == B2KV_SEG_SOFTCAP ? limit * tanhf(v / limit) : v;
}

// Index of the segment that holds column c (segments are in column order).
__device__ __forceinline__ int segment_of(const b2kv_linear_args& a, int c) {
    int s = 0;
    while (s + 1 < a.n_seg && c >= a.seg[s].end) ++s;
    return s;
}

__device__ __forceinline__ int segment_first(const b2kv_linear_args& a, int s) { return s == 0 ? 0 : a.seg[s - 1].end; }

// Exact exponential for the fp32 path; the bf16 paths round the result to 8 bits anyway.
template <typename T>
__device__ __forceinline__ float glu_value(int kind, float g, float u, float limit) {
    if (sizeof(T) == 2) return glu(kind, g, u, limit);
    if (kind == B2KV_SEG_GLU_SILU) return g / (1.0f + expf(-g)) * u;
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.0f + expf(-1.702f * g)) * (u + 1.0f);
}

// The outputs of columns c and c + 1 (c even) of one row, from the sums of their products.
template <typename T>
__device__ __forceinline__ void finish_pair(const b2kv_linear_args& a, int g, int64_t out_row, int c, float v0, float v1) {
    const int s = segment_of(a, c);
    const b2kv_segment& sg = a.seg[s];
    const int local = c - segment_first(a, s);
    const int64_t base = out_row * sg.ld + static_cast<int64_t>(g) * (a.group_rows ? 0 : sg.group);
    const bool second = c + 1 < a.N;
    if (a.bias != nullptr) {
        v0 += a.bias[c];
        if (second) v1 += a.bias[c + 1];
    }
    if (is_pair(sg.kind)) {
        static_cast<T*>(sg.out)[base + local / 2] = Elt<T>::from_float(glu_value<T>(sg.kind, v0, v1, a.limit));
        return;
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        if (e == 1 && !second) break;
        float v = e ? v1 : v0;
        v = sizeof(T) == 4 && sg.kind == B2KV_SEG_DECAY ? decay_exact(v, a.limit) : single(sg.kind, v, a.limit);
        if (is_f32(sg.kind)) {
            if (a.residual != nullptr && sg.kind == B2KV_SEG_F32) v += a.residual[out_row * a.ld_residual + local + e];
            static_cast<float*>(sg.out)[base + local + e] = v;
        } else {
            static_cast<T*>(sg.out)[base + local + e] = Elt<T>::from_float(v);
        }
    }
}

}  // namespace lin

// fp32 on the CUDA cores; B2KV_ERR_UNSUPPORTED where rows are not made of 16-byte pieces.
int linear_f32(const b2kv_linear_args& a, void* stream);  // linear_f32.cu
// fp32 on the tensor cores, operands in three bf16 parts; same contract.
int linear_f32_tc(const b2kv_linear_args& a, int32_t* dev_status, void* stream);  // linear_f32_tc.cu

// bf16 kernels on the tensor cores; B2KV_ERR_UNSUPPORTED when the shape is not one they take.
int linear_rows_tc(const b2kv_linear_args& a, int32_t* dev_status, void* stream);   // linear_rows.cu
int linear_tiled_tc(const b2kv_linear_args& a, int32_t* dev_status, void* stream);  // gemm.cu

}  // namespace b2kv
