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

// Where the outputs of columns c and c + 1 (c even) go and what happens to the sums of their products, looked up once for all rows: the
// look-up is a chain of dependent loads, and the choice of what happens is more instructions than the rest (fp32, 16 input features, 693 rows x
// 1024 columns: 16.5 us with both per row, 4.3 so).
template <typename T>
struct Pair {
    void* out;            // column c of row 0
    const float* residual;
    int64_t ld, ld_residual;
    int kind;
    bool second, with_bias;  // second: there is a column c + 1
    float bias0, bias1, limit;

    __device__ __forceinline__ Pair(const b2kv_linear_args& a, int g, int c) {
        const int s = segment_of(a, c);
        const b2kv_segment& sg = a.seg[s];
        const int local = c - segment_first(a, s);
        const int64_t at = static_cast<int64_t>(g) * (a.group_rows ? 0 : sg.group) + (is_pair(sg.kind) ? local / 2 : local);
        kind = sg.kind, ld = sg.ld, ld_residual = a.ld_residual, limit = a.limit;
        second = c + 1 < a.N;
        out = is_f32(kind) ? static_cast<void*>(static_cast<float*>(sg.out) + at) : static_cast<void*>(static_cast<T*>(sg.out) + at);
        residual = a.residual != nullptr && kind == B2KV_SEG_F32 ? a.residual + local : nullptr;
        with_bias = a.bias != nullptr;
        bias0 = with_bias ? a.bias[c] : 0.f;
        bias1 = with_bias && second ? a.bias[c + 1] : 0.f;
    }
    // What is added to a row's outputs behind everything else.
    __device__ __forceinline__ float2 added(int64_t row) const {
        if (residual == nullptr) return make_float2(0.f, 0.f);
        const float* const r = residual + row * ld_residual;
        return make_float2(r[0], second ? r[1] : 0.f);
    }
    template <int kKind>
    __device__ __forceinline__ void store(int64_t row, float v0, float v1, float2 add) const {
        if (with_bias) v0 += bias0, v1 += bias1;
        if (is_pair(kKind)) {
            static_cast<T*>(out)[row * ld] = Elt<T>::from_float(glu_value<T>(kKind, v0, v1, limit));
            return;
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            if (e == 1 && !second) break;
            float v = e ? v1 : v0;
            v = sizeof(T) == 4 && kKind == B2KV_SEG_DECAY ? decay_exact(v, limit) : single(kKind, v, limit);
            if (is_f32(kKind)) {
                if (residual != nullptr) v += e ? add.y : add.x;
                static_cast<float*>(out)[row * ld + e] = v;
            } else {
                static_cast<T*>(out)[row * ld + e] = Elt<T>::from_float(v);
            }
        }
    }
};

template <int kKind>
struct Kind {
    static constexpr int value = kKind;
};
// fn(Kind<kind>): what happens to a column is chosen outside of the loop over rows.
template <typename F>
__device__ __forceinline__ void with_kind(int kind, F&& fn) {
    switch (kind) {
        case B2KV_SEG_F32: return fn(Kind<B2KV_SEG_F32>{});
        case B2KV_SEG_GLU_SILU: return fn(Kind<B2KV_SEG_GLU_SILU>{});
        case B2KV_SEG_GLU_CLAMP: return fn(Kind<B2KV_SEG_GLU_CLAMP>{});
        case B2KV_SEG_RELU2: return fn(Kind<B2KV_SEG_RELU2>{});
        case B2KV_SEG_SOFTCAP: return fn(Kind<B2KV_SEG_SOFTCAP>{});
        case B2KV_SEG_DECAY: return fn(Kind<B2KV_SEG_DECAY>{});
        default: return fn(Kind<B2KV_SEG_STORE>{});
    }
}

// Rows r0, r0 + step, .. below end of columns c and c + 1, `sums(r)` the two sums of row r, out_row0 the row that r = 0 goes to: four rows
// at a time, with what is added to them on its way together.
template <typename T, typename Sums>
__device__ __forceinline__ void finish_rows(const b2kv_linear_args& a, int g, int c, int64_t out_row0, int r0, int end, int step, Sums&& sums) {
    const Pair<T> pair(a, g, c);
    with_kind(pair.kind, [&](auto kind) {
        for (int r = r0; r < end; r += 4 * step) {
            float2 v[4], add[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (r + u * step < end) add[u] = pair.added(out_row0 + r + u * step), v[u] = sums(r + u * step);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (r + u * step < end) pair.template store<decltype(kind)::value>(out_row0 + r + u * step, v[u].x, v[u].y, add[u]);
        }
    });
}

// The outputs of columns c and c + 1 (c even) of one row, from the sums of their products.
template <typename T>
__device__ __forceinline__ void finish_pair(const b2kv_linear_args& a, int g, int64_t out_row, int c, float v0, float v1) {
    const Pair<T> pair(a, g, c);
    with_kind(pair.kind, [&](auto kind) { pair.template store<decltype(kind)::value>(out_row, v0, v1, pair.added(out_row)); });
}

}  // namespace lin

// fp32 on the CUDA cores; B2KV_ERR_UNSUPPORTED where rows are not made of 16-byte pieces.
int linear_f32(const b2kv_linear_args& a, void* stream);  // linear_f32.cu
// fp32 on the tensor cores, operands in three bf16 parts; same contract.  The parts are made ahead where there is scratch for them.
int linear_f32_tc(const b2kv_linear_args& a, void* workspace, size_t workspace_bytes, int32_t* dev_status, void* stream);  // linear_f32_tc.cu
size_t linear_f32_tc_workspace(const b2kv_linear_args& a);

// bf16 kernels on the tensor cores; B2KV_ERR_UNSUPPORTED when the shape is not one they take.
int linear_rows_tc(const b2kv_linear_args& a, int32_t* dev_status, void* stream);   // linear_rows.cu
int linear_tiled_tc(const b2kv_linear_args& a, const b2kv_linear_options& o, int32_t* dev_status, void* stream);  // gemm.cu

}  // namespace b2kv
