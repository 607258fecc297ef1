// Grouped-query attention, the parts on CUDA cores: norms and temperature of the queries with the cache append, and attention
// of single query rows for every shape and both storage types.
// These kernels may be scheduled ahead of the end of the kernel that writes their inputs, so no pointer to such data is
// const __restrict__: the compiler would take it for data that nothing writes and could load it before the wait.
#include "gqa.cuh"

#include <math.h>

#include <algorithm>

namespace b2kv {
namespace {

constexpr int kAppendThreads = 256;

__device__ __forceinline__ void narrow_store(float* p, const float (&f)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
}
__device__ __forceinline__ void narrow_store(__nv_bfloat16* p, const float (&f)[8]) {
    __nv_bfloat162 h[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
    *reinterpret_cast<uint4*>(p) = *reinterpret_cast<uint4*>(h);
}

// This thread's share of a row of n elements: 16-byte pieces when kVec (n a whole number of them), the first kKeep of which
// stay in registers.
template <typename T, bool kVec, int kKeep>
struct Row {
    static constexpr int kC = Elt<T>::kPerChunk;
    uint4 keep[kKeep];
    __device__ __forceinline__ uint4 piece(const T* src, int j) const {
        return reinterpret_cast<const uint4*>(src)[threadIdx.x + j * kAppendThreads];
    }
    __device__ __forceinline__ void load(const T* src, int n) {
        if (!kVec) return;
#pragma unroll
        for (int j = 0; j < kKeep; ++j)
            if (static_cast<int>(threadIdx.x) + j * kAppendThreads < n / kC) keep[j] = piece(src, j);
    }
    // fn(piece, index of its first element)
    template <typename F>
    __device__ __forceinline__ void each(const T* src, int n, F&& fn) const {
#pragma unroll
        for (int j = 0; j < kKeep; ++j)
            if (static_cast<int>(threadIdx.x) + j * kAppendThreads < n / kC) fn(keep[j], (threadIdx.x + j * kAppendThreads) * kC);
        for (int j = kKeep; static_cast<int>(threadIdx.x) + j * kAppendThreads < n / kC; ++j)
            fn(piece(src, j), (threadIdx.x + j * kAppendThreads) * kC);
    }
    __device__ __forceinline__ float squares(const T* src, int n) const {
        float sum = 0.f;
        if (kVec) {
            each(src, n, [&](const uint4& p, int) {
                float f[kC];
                Elt<T>::widen(p, f);
#pragma unroll
                for (int e = 0; e < kC; ++e) sum = fmaf(f[e], f[e], sum);
            });
        } else {
            for (int i = threadIdx.x; i < n; i += kAppendThreads) sum = fmaf(Elt<T>::to_float(src[i]), Elt<T>::to_float(src[i]), sum);
        }
        return sum;
    }
    // dst = src * factor * w (w NULL: src * factor); dst may be src.
    __device__ __forceinline__ void scaled(T* dst, const T* src, const float* w, float factor, int n) const {
        if (kVec) {
            each(src, n, [&](const uint4& p, int at) {
                float f[kC];
                Elt<T>::widen(p, f);
                if (w != nullptr) {
#pragma unroll
                    for (int e = 0; e < kC; e += 4) {
                        const float4 wv = *reinterpret_cast<const float4*>(w + at + e);
                        f[e] *= factor * wv.x, f[e + 1] *= factor * wv.y, f[e + 2] *= factor * wv.z, f[e + 3] *= factor * wv.w;
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < kC; ++e) f[e] *= factor;
                }
                narrow_store(dst + at, f);
            });
        } else {
            for (int i = threadIdx.x; i < n; i += kAppendThreads)
                dst[i] = Elt<T>::from_float(Elt<T>::to_float(src[i]) * (w != nullptr ? factor * w[i] : factor));
        }
    }
};

struct AppendArgs {
    const float *q_norm, *k_norm;
    const int32_t *row_slot, *row_pos;
    int32_t* dev_status;
    int64_t ld_y;
    int H, G, dim, vdim, n_slots, T_max, temp_every;
    float eps, temp_coef;
};

template <typename T, bool kVec>
__global__ void __launch_bounds__(kAppendThreads) gqa_append_kernel(T* y, T* k_cache, T* v_cache, const AppendArgs a) {
    __shared__ float part[2][kAppendThreads / 32];
    grid_launch_dependents();
    if (threadIdx.x == 0) grid_dependency_wait();
    __syncthreads();
    int slot, pos;
    if (!row_place(a.row_slot, a.row_pos, blockIdx.x, a.n_slots, a.T_max, slot, pos)) {
        if (threadIdx.x == 0) report_status(a.dev_status, B2KV_DEV_BAD_POSITION);
        return;
    }
    const int nq = a.H * a.dim, nk = a.G * a.dim, nv = a.G * a.vdim;
    T* q = y + static_cast<int64_t>(blockIdx.x) * a.ld_y;
    const T *k = q + nq, *v = k + nk;
    const bool own = k_cache != nullptr;
    // the first pieces of q, k and v stay in registers between the two passes, all loads on their way together
    Row<T, kVec, 2> rq;
    Row<T, kVec, 1> rk, rv;
    rq.load(q, nq);
    if (own) rk.load(k, nk), rv.load(v, nv);
    float sq = a.q_norm != nullptr ? rq.squares(q, nq) : 0.f;
    float sk = own && a.k_norm != nullptr ? rk.squares(k, nk) : 0.f;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        sq += __shfl_xor_sync(0xffffffffu, sq, off);
        sk += __shfl_xor_sync(0xffffffffu, sk, off);
    }
    if ((threadIdx.x & 31) == 0) part[0][threadIdx.x >> 5] = sq, part[1][threadIdx.x >> 5] = sk;
    __syncthreads();
    sq = sk = 0.f;
#pragma unroll
    for (int i = 0; i < kAppendThreads / 32; ++i) sq += part[0][i], sk += part[1][i];
    float fq = a.q_norm != nullptr ? 1.0f / sqrtf(sq / static_cast<float>(nq) + a.eps) : 1.f;
    if (a.temp_every > 0) fq *= 1.0f + a.temp_coef * logf(static_cast<float>((pos + 1) / a.temp_every) + 1.0f);
    if (a.q_norm != nullptr || a.temp_every > 0) rq.scaled(q, q, a.q_norm, fq, nq);
    if (!own) return;
    const int64_t place = static_cast<int64_t>(slot) * a.T_max + pos;
    const float fk = a.k_norm != nullptr ? 1.0f / sqrtf(sk / static_cast<float>(nk) + a.eps) : 1.f;
    rk.scaled(k_cache + place * nk, k, a.k_norm, fk, nk);
    rv.scaled(v_cache + place * nv, v, nullptr, 1.f, nv);
}

// One CTA per (head, query row); its warps take the visible tokens in turn, each with an online softmax of its own, and are merged at the end.
// A lane holds kPer elements of the query and of the output.  Two forms: four warps and token after token, and, where few rows are a chain of loads,
// sums over the warp and exponentials, eight warps and kTogether tokens at a time, which are on their way together and share the rest
// (three rows of 250 to 310 tokens, 12 heads of 64, fp32: 25 us and 12; the rule at launch_simt).
template <typename T, int kPer, int kWarps, int kTogether>
__global__ void __launch_bounds__(kWarps * 32) gqa_decode_kernel(const GqaDecodeArgs a) {
    extern __shared__ float sm_acc[];  // [kWarps][vdim]
    __shared__ float sm_m[kWarps], sm_l[kWarps];
    const int h = blockIdx.x, i = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int slot, pos;
    if (!row_place(a.row_slot, a.row_pos, i, a.n_slots, a.T_max, slot, pos)) {
        if (threadIdx.x == 0) report_status(a.dev_status, B2KV_DEV_BAD_POSITION);
        return;
    }
    const int g = h / (a.H / a.G);
    const T* qr = static_cast<const T*>(a.q) + i * a.ld_q + h * a.dim;
    const T* keys = static_cast<const T*>(a.k_cache) + (static_cast<int64_t>(slot) * a.T_max * a.G + g) * a.dim;
    const T* values = static_cast<const T*>(a.v_cache) + (static_cast<int64_t>(slot) * a.T_max * a.G + g) * a.vdim;
    const float slope = a.slopes != nullptr ? a.slopes[h] : 0.f;
    float q[kPer], acc[kPer];
#pragma unroll
    for (int c = 0; c < kPer; ++c) {
        const int d = c * 32 + lane;
        q[c] = d < a.dim ? Elt<T>::to_float(qr[d]) : 0.f;
        acc[c] = 0.f;
    }
    float m = -INFINITY, l = 0.f;
    if constexpr (kTogether == 1) {
        for (int t = warp; t <= pos; t += kWarps) {
            const T* key = keys + static_cast<int64_t>(t) * a.G * a.dim;
            const T* value = values + static_cast<int64_t>(t) * a.G * a.vdim;
            float v[kPer], s = 0.f;
#pragma unroll
            for (int c = 0; c < kPer; ++c) {
                const int d = c * 32 + lane;
                v[c] = d < a.vdim ? Elt<T>::to_float(value[d]) : 0.f;
                s = fmaf(q[c], d < a.dim ? Elt<T>::to_float(key[d]) : 0.f, s);
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
            s = s * a.scale - slope * static_cast<float>(pos - t);
            const float mn = fmaxf(m, s), f = expf(m - mn), p = expf(s - mn);
            l = l * f + p;
            m = mn;
#pragma unroll
            for (int c = 0; c < kPer; ++c) acc[c] = fmaf(acc[c], f, p * v[c]);
        }
    }
    for (int t0 = warp * kTogether; kTogether > 1 && t0 <= pos; t0 += kWarps * kTogether) {
        float v[kTogether][kPer], s[kTogether];
#pragma unroll
        for (int u = 0; u < kTogether; ++u) {
            const T* key = keys + static_cast<int64_t>(t0 + u) * a.G * a.dim;
            const T* value = values + static_cast<int64_t>(t0 + u) * a.G * a.vdim;
            const bool in = t0 + u <= pos;
            s[u] = 0.f;
#pragma unroll
            for (int c = 0; c < kPer; ++c) {
                const int d = c * 32 + lane;
                v[u][c] = in && d < a.vdim ? Elt<T>::to_float(value[d]) : 0.f;
                s[u] = fmaf(q[c], in && d < a.dim ? Elt<T>::to_float(key[d]) : 0.f, s[u]);
            }
        }
        float mn = m;
#pragma unroll
        for (int u = 0; u < kTogether; ++u) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) s[u] += __shfl_xor_sync(0xffffffffu, s[u], off);
            s[u] = s[u] * a.scale - slope * static_cast<float>(pos - t0 - u);
            if (t0 + u <= pos) mn = fmaxf(mn, s[u]);
        }
        const float f = expf(m - mn);
        l *= f;
        m = mn;
#pragma unroll
        for (int c = 0; c < kPer; ++c) acc[c] *= f;
#pragma unroll
        for (int u = 0; u < kTogether; ++u) {
            if (t0 + u > pos) break;
            const float p = expf(s[u] - mn);
            l += p;
#pragma unroll
            for (int c = 0; c < kPer; ++c) acc[c] = fmaf(p, v[u][c], acc[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < kPer; ++c)
        if (c * 32 + lane < a.vdim) sm_acc[warp * a.vdim + c * 32 + lane] = acc[c];
    if (lane == 0) sm_m[warp] = m, sm_l[warp] = l;
    __syncthreads();
    float mx = sm_m[0];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) mx = fmaxf(mx, sm_m[w]);
    float f[kWarps], sum = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        f[w] = expf(sm_m[w] - mx);
        sum += f[w] * sm_l[w];
    }
    T* out = static_cast<T*>(a.out) + i * a.ld_out + h * a.vdim;
    for (int d = threadIdx.x; d < a.vdim; d += kWarps * 32) {
        float o = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) o = fmaf(f[w], sm_acc[w * a.vdim + d], o);
        out[d] = Elt<T>::from_float(o / sum);
    }
}

// Runs of rows of one sequence in fp32 (prompt portions, which fp32 has no tensor-core form for): 16 rows of one head per CTA and 64
// tokens at a time, keys and values read into shared memory once for all of the rows.  A thread has 4 rows x 4 tokens of the scores
// and 4 rows x 4 columns (per 64) of the output, 64 multiply-adds for every eight 16-byte reads of shared memory; the 16 lanes of a
// row group keep the rows' softmax among themselves.  gqa_decode_kernel reads every key and value again for every row and reduces
// over the warp for every token: 174 us for 693 rows of three prompts (12 heads of 64, 4 of them for keys), against 90
// (100 with 32 rows: half as many warps to hide one another's waits).
// Rows of other sequences in the same 16 are taken in turn; a weight of zero is never multiplied with what a row must not see.
__device__ __forceinline__ void copy16_or_zero(void* dst, const void* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
constexpr int kRunRows = 16, kRunTokens = 64, kRunThreads = 64;

// kD: dim and vdim, rounded up; kLate: the last rows first.
template <int kD, bool kLate>
__global__ void __launch_bounds__(kRunThreads) gqa_run_f32_kernel(const __grid_constant__ GqaDecodeArgs a) {
    constexpr int kLd = kD + 4, kLdP = kRunTokens + 4, kCols = kD / 64;
    constexpr bool kAhead = kD > 64;
    extern __shared__ float4 sm_run[];
    float* const s_q = reinterpret_cast<float*>(sm_run);  // [rows][kLd]
    float* const s_k = s_q + kRunRows * kLd;              // [tokens][kLd]
    float* const s_v = s_k + kRunTokens * kLd;            // [tokens][kLd]
    float* const s_p = s_v + kRunTokens * kLd;            // [rows][kLdP]
    __shared__ int s_slot[kRunRows], s_pos[kRunRows];
    const int h = blockIdx.x, i0 = static_cast<int>(kLate ? gridDim.y - 1 - blockIdx.y : blockIdx.y) * kRunRows, n_rows = min(kRunRows, a.rows - i0);
    const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16, g = h / (a.H / a.G);
    grid_launch_dependents();
    grid_dependency_wait();
    if (tid < kRunRows) {
        int slot = -1, pos = -1;
        if (tid < n_rows && !row_place(a.row_slot, a.row_pos, i0 + tid, a.n_slots, a.T_max, slot, pos)) {
            report_status(a.dev_status, B2KV_DEV_BAD_POSITION);
            slot = pos = -1;
        }
        s_slot[tid] = slot, s_pos[tid] = pos;
    }
    const float* const q = static_cast<const float*>(a.q) + i0 * a.ld_q + h * a.dim;
    for (int i = tid; i < kRunRows * (kD / 4); i += kRunThreads) {
        const int r = i / (kD / 4), c = i % (kD / 4) * 4;
        *reinterpret_cast<float4*>(s_q + r * kLd + c) =
            r < n_rows && c < a.dim ? *reinterpret_cast<const float4*>(q + r * a.ld_q + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    const float slope = a.slopes != nullptr ? a.slopes[h] : 0.f;
    float m[4], l[4];
    float4 acc[4][kCols];
    int pos[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY, l[i] = 0.f, pos[i] = s_pos[ty * 4 + i];
#pragma unroll
        for (int c = 0; c < kCols; ++c) acc[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int first = 0; first < n_rows;) {
        // the run: rows [first, end) of one sequence, which see tokens up to last, all of them those up to all
        const int here = s_slot[first];
        int end = first, last = -1, all = 0x7fffffff;
        for (; end < n_rows && s_slot[end] == here; ++end) last = max(last, s_pos[end]), all = min(all, s_pos[end]);
        const bool alone = first == 0 && end == kRunRows;
        bool mine[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) mine[i] = ty * 4 + i >= first && ty * 4 + i < end;
        first = end;
        if (here < 0) continue;
        const int64_t base = static_cast<int64_t>(here) * a.T_max * a.G + g;
        const float* const keys = static_cast<const float*>(a.k_cache) + base * a.dim;
        const float* const values = static_cast<const float*>(a.v_cache) + base * a.vdim;
        // Rows of 128: keys and values come with copies of their own, the next tile's keys under this one's softmax and output, the next values
        // under the next scores (two prompts of 300 and 400 tokens, 8 heads: 62 us, 84 with the copies where they are waited for).  Of rows of 64 an SM
        // holds twice as many CTAs, which hide each other's loads (48 us so, 51 with copies ahead).
        auto request = [&](float* to, const float* from, int width, int t0) {
            if (t0 <= last) {
#pragma unroll 4
                for (int i = tid; i < kRunTokens * (kD / 4); i += kRunThreads) {
                    const int t = i / (kD / 4), c = i % (kD / 4) * 4;
                    const bool in = t0 + t <= last && c < width;
                    copy16_or_zero(to + t * kLd + c, in ? from + static_cast<int64_t>(t0 + t) * a.G * width + c : from, in);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        if (kAhead) {
            request(s_k, keys, a.dim, 0);
            request(s_v, values, a.vdim, 0);
        }
        for (int t0 = 0; t0 <= last; t0 += kRunTokens) {
            if (kAhead) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                __syncthreads();
#pragma unroll 4
                for (int i = tid; i < kRunTokens * (kD / 4); i += kRunThreads) {
                    const int t = i / (kD / 4), c = i % (kD / 4) * 4;
                    const bool in = t0 + t <= last;
                    *reinterpret_cast<float4*>(s_k + t * kLd + c) =
                        in && c < a.dim ? *reinterpret_cast<const float4*>(keys + static_cast<int64_t>(t0 + t) * a.G * a.dim + c)
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
                    *reinterpret_cast<float4*>(s_v + t * kLd + c) =
                        in && c < a.vdim ? *reinterpret_cast<const float4*>(values + static_cast<int64_t>(t0 + t) * a.G * a.vdim + c)
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
            __syncthreads();  // the keys are here
            float s[4][4] = {};
#pragma unroll 4
            for (int c = 0; c < a.dim; c += 4) {
                float4 qv[4], kv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    qv[i] = *reinterpret_cast<const float4*>(s_q + (ty * 4 + i) * kLd + c);
                    kv[i] = *reinterpret_cast<const float4*>(s_k + (tx + 16 * i) * kLd + c);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        s[i][j] = fmaf(qv[i].w, kv[j].w, fmaf(qv[i].z, kv[j].z, fmaf(qv[i].y, kv[j].y, fmaf(qv[i].x, kv[j].x, s[i][j]))));
            }
            if (kAhead) {
                __syncthreads();  // everybody has read them
                request(s_k, keys, a.dim, t0 + kRunTokens);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float mn = m[i];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int t = t0 + tx + 16 * j;
                    s[i][j] = mine[i] && t <= pos[i] ? s[i][j] * a.scale - slope * static_cast<float>(pos[i] - t) : -INFINITY;
                    mn = fmaxf(mn, s[i][j]);
                }
#pragma unroll
                for (int off = 8; off > 0; off >>= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, off));
                const float f = mn == m[i] ? 1.f : expf(m[i] - mn);
                m[i] = mn;
                l[i] *= f;
#pragma unroll
                for (int c = 0; c < kCols; ++c) acc[i][c].x *= f, acc[i][c].y *= f, acc[i][c].z *= f, acc[i][c].w *= f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int t = tx + 16 * j;
                    const float p = mine[i] && t0 + t <= pos[i] ? expf(s[i][j] - mn) : 0.f;
                    l[i] += p;
                    s_p[(ty * 4 + i) * kLdP + t] = p;
                }
            }
            if (kAhead) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                __syncthreads();  // the values are here
            } else {
                __syncwarp();  // a row's weights are written and read by the same 16 lanes
            }
            if (alone && t0 + kRunTokens - 1 <= all) {
                for (int t = 0; t < kRunTokens; t += 4) {
                    float4 p[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const float4*>(s_p + (ty * 4 + i) * kLdP + t);
#pragma unroll
                    for (int c = 0; c < kCols; ++c) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float4 v = *reinterpret_cast<const float4*>(s_v + (t + e) * kLd + c * 64 + tx * 4);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const float w = e == 0 ? p[i].x : (e == 1 ? p[i].y : (e == 2 ? p[i].z : p[i].w));
                                acc[i][c].x = fmaf(w, v.x, acc[i][c].x), acc[i][c].y = fmaf(w, v.y, acc[i][c].y);
                                acc[i][c].z = fmaf(w, v.z, acc[i][c].z), acc[i][c].w = fmaf(w, v.w, acc[i][c].w);
                            }
                        }
                    }
                }
            } else {
                // Tokens that not all rows see.  A weight of zero is no answer to a value that is not finite, so what a row must not
                // see counts as zero itself.
#pragma unroll 2
                for (int t = 0; t < kRunTokens; t += 4) {
                    if (t0 + t > last) break;
                    float4 p[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const float4*>(s_p + (ty * 4 + i) * kLdP + t);
#pragma unroll
                    for (int c = 0; c < kCols; ++c) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float4 v = *reinterpret_cast<const float4*>(s_v + (t + e) * kLd + c * 64 + tx * 4);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const bool sees = mine[i] && t0 + t + e <= pos[i];
                                const float w = e == 0 ? p[i].x : (e == 1 ? p[i].y : (e == 2 ? p[i].z : p[i].w));
                                acc[i][c].x = fmaf(w, sees ? v.x : 0.f, acc[i][c].x), acc[i][c].y = fmaf(w, sees ? v.y : 0.f, acc[i][c].y);
                                acc[i][c].z = fmaf(w, sees ? v.z : 0.f, acc[i][c].z), acc[i][c].w = fmaf(w, sees ? v.w : 0.f, acc[i][c].w);
                            }
                        }
                    }
                }
            }
            if (kAhead) {
                __syncthreads();  // everybody has read them
                request(s_v, values, a.vdim, t0 + kRunTokens);
            }
        }
    }
    float* const out = static_cast<float*>(a.out) + i0 * a.ld_out + h * a.vdim;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], off);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (s_slot[ty * 4 + i] < 0) continue;
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
            const float v[4] = {acc[i][c].x, acc[i][c].y, acc[i][c].z, acc[i][c].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int d = c * 64 + tx * 4 + e;
                if (d < a.vdim) out[static_cast<int64_t>(ty * 4 + i) * a.ld_out + d] = v[e] / l[i];
            }
        }
    }
}

template <int kD, bool kLate>
int launch_runs(const GqaDecodeArgs& a, void* stream) {
    constexpr size_t smem = ((kRunRows + 2 * kRunTokens) * (kD + 4) + kRunRows * (kRunTokens + 4)) * sizeof(float);
    static int resident[64] = {0};  // CTAs that the device holds
    int dev = 0;
    B2KV_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return B2KV_ERR_UNSUPPORTED;
    if (resident[dev] == 0) {
        B2KV_CUDA_TRY(cudaFuncSetAttribute(gqa_run_f32_kernel<kD, kLate>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        int n = 0;
        B2KV_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, gqa_run_f32_kernel<kD, kLate>, kRunThreads, smem));
        resident[dev] = n * device_sm_count();
    }
    OverlapLaunch launch(dim3(a.H, (a.rows + kRunRows - 1) / kRunRows), kRunThreads, smem, stream);
    // A prompt's late rows see the most tokens and must not be what is left at the end (352 CTAs of which 296 fit, rows of 128: 77 us, 62 with the
    // late rows first).  Of rows of 64, two and a half times as many fit, and the order that mixes late and early rows is better (57 us, 61 with
    // the late rows first, of 792 CTAs of which 740 fit; 48 and 54 of 528).
    if constexpr (kD > 64 && !kLate) {
        if (static_cast<long long>(launch.cfg.gridDim.x) * launch.cfg.gridDim.y > resident[dev]) return launch_runs<kD, true>(a, stream);
    }
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, gqa_run_f32_kernel<kD, kLate>, a));
    return B2KV_OK;
}

// For rows that the caller says come in runs, and enough of them (a CTA takes the sequences of its 16 rows one after the other, so that single rows of
// many sequences would be in line: 16 of them take as long as the one that sees most, times 16).
int launch_runs_f32(const GqaDecodeArgs& a, void* stream) {
    // Enough CTAs that the SMs are busy with 64 threads each: below, a CTA's chain of token tiles takes longer than rows one by one over as many SMs;
    // us row by row and as runs, in the order of CTAs.  Heads of 64 (and 32): 1 prompt of 160 over 8 heads (80) 15.4, 18.6; behind 500 tokens 68, 57;
    // 1 of 100 over 12 heads (84) 11.7, 13.9; 1 of 200 over 8 (104) 19.0, 23.8; behind 500 92, 65; 1 of 160 over 12 (120) 20.7, 18.8.  Heads of
    // 128, half as many CTAs per SM: 3 of 100 over 8 (152) 21, 29; behind 500 149, 180; 1 of 300 over 8 (152) 50, 53; behind 500 177, 132; 3 of 300 over
    // 4 (228) 69, 59.  Prompts mostly begin at their first token, and rows of several sequences in one CTA cost it twice, so the line is where runs
    // win without a past.
    const long long ctas = static_cast<long long>(a.H) * ((a.rows + kRunRows - 1) / kRunRows), sms = device_sm_count();
    const bool few = a.rows < 64 || (std::max(a.dim, a.vdim) <= 64 ? 4 * ctas < 3 * sms : 2 * ctas < 3 * sms);
    if ((few && tune_get("gqa_runs") == 0) || (a.rows + kRunRows - 1) / kRunRows > 65535) return B2KV_ERR_UNSUPPORTED;
    const int widest = std::max(a.dim, a.vdim);
    if (widest > 128 || a.dim % 4 || a.vdim % 4 || a.ld_q % 4 || !aligned16(a.q) || !aligned16(a.k_cache) || !aligned16(a.v_cache))
        return B2KV_ERR_UNSUPPORTED;
    return widest <= 64 ? launch_runs<64, false>(a, stream) : launch_runs<128, false>(a, stream);
}

template <typename T, int kPer>
int launch_simt_per(const GqaDecodeArgs& a, bool together, cudaStream_t stream) {
    constexpr int kTogether = kPer <= 4 ? 4 : 2;
    const int warps = together ? 8 : 4;
    const auto kernel = together ? gqa_decode_kernel<T, kPer, 8, kTogether> : gqa_decode_kernel<T, kPer, 4, 1>;
    kernel<<<dim3(a.H, a.rows), warps * 32, static_cast<size_t>(warps) * a.vdim * sizeof(float), stream>>>(a);
    B2KV_CUDA_TRY(cudaGetLastError());
    return B2KV_OK;
}

template <typename T>
int launch_simt(const GqaDecodeArgs& a, void* stream) {
    const int widest = a.dim > a.vdim ? a.dim : a.vdim;
    if (widest > 512 || a.rows > 65535) return B2KV_ERR_UNSUPPORTED;
    // Tokens together where a row's time is a chain that other CTAs do not hide, and there are tokens enough for all warps; us token after token and
    // together, fp32, 12 heads of 64: 3 rows of up to 16 tokens 3.3, 3.2; 100 8.6, 5.2; 2000 131, 57; 40 rows of 16 3.7, 4.2; 100 10.0, 8.1; 150 rows (1800
    // CTAs) of 100 17.1, 18.8; 400 55.0, 54.2; 2000 380, 301; 400 rows of 100 34.4, 41.7; 400 116, 126; 2000 808, 679.  In bf16 (sizes that the
    // tensor cores do not take) tokens share less: 12 heads of 60, 3 rows of 100 8.7, 8.4; 2000 133, 121; 150 rows of 400 57, 69.
    const long long ctas = static_cast<long long>(a.rows) * a.H, sms = device_sm_count();
    const bool together = sizeof(T) == 4 ? a.span > 32 && (ctas <= 5 * sms || (a.span >= 256 && ctas <= 9 * sms) || a.span >= 1024)
                                         : a.span >= 256 && ctas <= 4 * sms;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return widest <= 64 ? launch_simt_per<T, 2>(a, together, s) : widest <= 128 ? launch_simt_per<T, 4>(a, together, s) : launch_simt_per<T, 16>(a, together, s);
}

template <typename T>
int launch_append(T* y, T* k, T* v, const AppendArgs& a, int rows, void* stream) {
    constexpr int per = 16 / static_cast<int>(sizeof(T));
    const bool vec = aligned16(y) && aligned16(a.q_norm) && aligned16(a.k_norm) && aligned16(k) && aligned16(v) && a.ld_y % per == 0 && (a.H * a.dim) % per == 0 &&
                     (a.G * a.dim) % per == 0 && (a.G * a.vdim) % per == 0;
    OverlapLaunch launch(rows, kAppendThreads, 0, stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, vec ? gqa_append_kernel<T, true> : gqa_append_kernel<T, false>, y, k, v, a));
    return B2KV_OK;
}

}  // namespace
}  // namespace b2kv

using namespace b2kv;

extern "C" int b2kv_gqa_append(void* y, int64_t ld_y, int H, int G, int dim, int vdim, const float* q_norm, const float* k_norm,
                               float eps, float temp_coef, int temp_every, void* k_cache, void* v_cache,
                               const int32_t* row_slot, const int32_t* row_pos, int n_slots, int T_max, int rows, int dtype,
                               int32_t* dev_status, void* stream) {
    if (elt_bytes(dtype) == 0) return B2KV_ERR_UNSUPPORTED;
    if (!y || !row_pos || H <= 0 || G <= 0 || H % G != 0 || dim <= 0 || vdim <= 0 || rows <= 0 || n_slots <= 0 || T_max <= 0)
        return B2KV_ERR_BAD_ARG;
    if ((k_cache == nullptr) != (v_cache == nullptr)) return B2KV_ERR_BAD_ARG;
    const int64_t cols = static_cast<int64_t>(H) * dim + (k_cache ? static_cast<int64_t>(G) * (dim + vdim) : 0);
    if (ld_y < cols) return B2KV_ERR_BAD_ARG;
    const AppendArgs a{q_norm, k_norm, row_slot, row_pos, dev_status, ld_y, H, G, dim, vdim, n_slots, T_max, temp_every, eps, temp_coef};
    if (dtype == B2KV_DTYPE_F32)
        return launch_append(static_cast<float*>(y), static_cast<float*>(k_cache), static_cast<float*>(v_cache), a, rows, stream);
    return launch_append(static_cast<__nv_bfloat16*>(y), static_cast<__nv_bfloat16*>(k_cache), static_cast<__nv_bfloat16*>(v_cache),
                         a, rows, stream);
}

extern "C" size_t b2kv_gqa_decode_workspace_bytes(int rows, int H, int G, int vdim, int span, int dtype) {
    if (dtype != B2KV_DTYPE_BF16 || rows <= 0 || H <= 0 || G <= 0 || H % G != 0 || vdim <= 0 || span <= 0) return 0;
    return gqa_decode_tc_workspace(rows, H, G, vdim, span);
}

// singles: rows in front of those that come in runs (all rows: none do).
static int gqa_decode(const GqaDecodeArgs& a, int dtype, int path, int singles, void* workspace, size_t workspace_bytes, void* stream) {
    if (elt_bytes(dtype) == 0) return B2KV_ERR_UNSUPPORTED;
    if (!a.q || !a.k_cache || !a.v_cache || !a.out || !a.row_pos) return B2KV_ERR_BAD_ARG;
    if (a.n_slots <= 0 || a.T_max <= 0 || a.rows <= 0 || a.H <= 0 || a.G <= 0 || a.H % a.G != 0 || a.dim <= 0 || a.vdim <= 0 || a.span <= 0 ||
        path < 0 || path > 2 || singles < 0 || a.ld_q < static_cast<int64_t>(a.H) * a.dim || a.ld_out < static_cast<int64_t>(a.H) * a.vdim)
        return B2KV_ERR_BAD_ARG;
    if (path == 2 && dtype != B2KV_DTYPE_BF16) return B2KV_ERR_UNSUPPORTED;
    if (dtype == B2KV_DTYPE_BF16 && path != 1) {
        const int rc = gqa_decode_tc(a, workspace, workspace_bytes, stream);
        if (rc != B2KV_ERR_UNSUPPORTED || path == 2) return rc;
    }
    if (dtype == B2KV_DTYPE_F32 && path == 0 && singles < a.rows && a.row_slot != nullptr) {
        GqaDecodeArgs front = a, runs = a;
        front.rows = singles, runs.rows = a.rows - singles;
        runs.q = static_cast<const float*>(a.q) + singles * a.ld_q, runs.out = static_cast<float*>(a.out) + singles * a.ld_out;
        runs.row_slot = a.row_slot + singles, runs.row_pos = a.row_pos + singles;
        const int rc = launch_runs_f32(runs, stream);
        if (rc != B2KV_ERR_UNSUPPORTED) return rc != B2KV_OK || singles == 0 ? rc : launch_simt<float>(front, stream);
    }
    return dtype == B2KV_DTYPE_F32 ? launch_simt<float>(a, stream) : launch_simt<__nv_bfloat16>(a, stream);
}

extern "C" int b2kv_gqa_decode(const void* q, int64_t ld_q, const void* k_cache, const void* v_cache, void* out, int64_t ld_out,
                               const float* slopes, const int32_t* row_slot, const int32_t* row_pos, int n_slots, int T_max,
                               int rows, int H, int G, int dim, int vdim, int span, float scale, int dtype, int path,
                               void* workspace, size_t workspace_bytes, int32_t* dev_status, void* stream) {
    return gqa_decode({q, k_cache, v_cache, out, slopes, row_slot, row_pos, dev_status, ld_q, ld_out, n_slots, T_max, rows, H, G, dim, vdim,
                       span, scale}, dtype, path, rows, workspace, workspace_bytes, stream);
}

extern "C" int b2kv_gqa_decode_runs(const void* q, int64_t ld_q, const void* k_cache, const void* v_cache, void* out, int64_t ld_out,
                                    const float* slopes, const int32_t* row_slot, const int32_t* row_pos, int n_slots, int T_max,
                                    int rows, int H, int G, int dim, int vdim, int span, float scale, int dtype, int path, int singles,
                                    void* workspace, size_t workspace_bytes, int32_t* dev_status, void* stream) {
    return gqa_decode({q, k_cache, v_cache, out, slopes, row_slot, row_pos, dev_status, ld_q, ld_out, n_slots, T_max, rows, H, G, dim, vdim,
                       span, scale}, dtype, path, singles, workspace, workspace_bytes, stream);
}
