// Row operations around a 32-bit residual stream: the token rows that start it, RMS norms that read it, and layer norms that
// read it or add a sublayer's normed output to it.
// These kernels may be scheduled ahead of the end of the kernel that writes their inputs, so no pointer to such data is
// const __restrict__: the compiler would take it for data that nothing writes and could load it before the wait.
#include "b2kv_common.cuh"

namespace b2kv {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    uint2 u;
    u.x = *reinterpret_cast<const uint32_t*>(&lo);
    u.y = *reinterpret_cast<const uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(p) = u;
}

__device__ __forceinline__ float4 load4(const float* p, int i) { return reinterpret_cast<const float4*>(p)[i]; }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p, int i) {
    const uint2 u = reinterpret_cast<const uint2*>(p)[i];
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}

template <typename T>
__global__ void __launch_bounds__(kThreads) embed_rows_kernel(const T* table, const int32_t* ids,
                                                              float* out, T* copy, float scale, int dim, int vocab,
                                                              int32_t* dev_status, bool vec) {
    grid_launch_dependents();
    if (threadIdx.x == 0) grid_dependency_wait();
    __syncthreads();
    int id = ids[blockIdx.x];
    if (id < 0 || id >= vocab) {
        if (threadIdx.x == 0) report_status(dev_status, B2KV_DEV_BAD_TOKEN);
        id = id < 0 ? 0 : vocab - 1;
    }
    const T* src = table + static_cast<int64_t>(id) * dim;
    float* dst = out + static_cast<int64_t>(blockIdx.x) * dim;
    T* cp = copy == nullptr ? nullptr : copy + static_cast<int64_t>(blockIdx.x) * dim;
    // (four elements: a warp then writes whole lines of fp32, which are most of the bytes; 3548 rows of 2048 bf16 7.8 us, 9.7 element by
    // element, 12.9 with eight; 64 rows of 4096 2.3 and 4.3)
    if (vec) {
        for (int i = threadIdx.x; i < dim / 4; i += kThreads) {
            const float4 v = load4(src, i);
            const float4 o = make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale);
            store4(dst + 4 * i, o);
            if (cp != nullptr) store4(cp + 4 * i, o);
        }
        return;
    }
    for (int i = threadIdx.x; i < dim; i += kThreads) {
        const float v = Elt<T>::to_float(src[i]) * scale;
        dst[i] = v;
        if (cp != nullptr) cp[i] = Elt<T>::from_float(v);
    }
}

// Norms of rows.  A row of up to 1024 * kKeep elements stays in registers between the passes, and where there are more rows than CTAs
// fit the device, a CTA takes row after row and has the next one on its way under the sums of this one: with a CTA per row every row
// waits for a launch and for its loads (3548 rows of 2048: layer norm onto the residual 11.9 us, 14.5 with a CTA per row; 101 MB, 8.5 TB/s
// out of L2 and HBM.  64 rows of 4096, where weights come with the row: RMS norm 2.0 and 2.6).

// Sum over the CTA, the same in every thread.  `part` may be used again after the next __syncthreads.
__device__ __forceinline__ float block_sum(float v, float* part) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0.f;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) v += part[i];
    return v;
}

// Rows of up to 4096 elements are taken one after the other (wider ones leave no registers for the next).
constexpr bool row_after_row(int keep) { return keep <= 4; }

// CTAs for `rows` rows of such a kernel: as many as fit the device together.  `fit`: per device, 0 before the first call.
template <typename K>
int row_ctas(K kernel, int rows, int (&fit)[64]) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return rows;
    if (fit[dev] == 0) {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kThreads, 0) != cudaSuccess || n <= 0) {
            (void)cudaGetLastError();
            return rows;
        }
        fit[dev] = n * device_sm_count();
    }
    return rows < fit[dev] ? rows : fit[dev];
}

template <typename T, int kKeep>
__global__ void __launch_bounds__(kThreads) rmsnorm_kernel(const float* x, int64_t ld_x,
                                                           const int32_t* row_index, const float* w,
                                                           float w_offset, T* out, int64_t ld_out, int rows, int size,
                                                           float eps, bool vec) {
    __shared__ float part[2][kThreads / 32];
    grid_launch_dependents();
    if (threadIdx.x == 0) grid_dependency_wait();
    __syncthreads();
    auto row_of = [&](int r) { return x + static_cast<int64_t>(row_index ? row_index[r] : r) * ld_x; };
    if (!vec) {
        for (int r = blockIdx.x, odd = 0; r < rows; r += gridDim.x, odd ^= 1) {
            const float* xr = row_of(r);
            T* yr = out + static_cast<int64_t>(r) * ld_out;
            float sum = 0.f;
            for (int i = threadIdx.x; i < size; i += kThreads) sum = fmaf(xr[i], xr[i], sum);
            const float scale = 1.0f / sqrtf(block_sum(sum, part[odd]) / static_cast<float>(size) + eps);
            for (int i = threadIdx.x; i < size; i += kThreads) yr[i] = Elt<T>::from_float(xr[i] * scale * (w[i] + w_offset));
        }
        return;
    }
    const int chunks = size / 4;
    float4 next[kKeep], wv[kKeep];
    auto load = [&](int r) {
        const float* xr = row_of(r);
#pragma unroll
        for (int c = 0; c < kKeep; ++c) {
            const int i = threadIdx.x + c * kThreads;
            if (i < chunks) next[c] = reinterpret_cast<const float4*>(xr)[i];
        }
    };
    load(blockIdx.x);
#pragma unroll
    for (int c = 0; c < kKeep; ++c) {
        const int i = threadIdx.x + c * kThreads;
        if (i < chunks) wv[c] = reinterpret_cast<const float4*>(w)[i];
    }
    for (int r = blockIdx.x, odd = 0; r < rows; r += row_after_row(kKeep) ? gridDim.x : rows, odd ^= 1) {
        float4 keep[kKeep];
        float sum = 0.f;
#pragma unroll
        for (int c = 0; c < kKeep; ++c) {
            keep[c] = next[c];
            if (static_cast<int>(threadIdx.x) + c * kThreads < chunks)
                sum += (keep[c].x * keep[c].x + keep[c].y * keep[c].y) + (keep[c].z * keep[c].z + keep[c].w * keep[c].w);
        }
        if (row_after_row(kKeep) && r + static_cast<int>(gridDim.x) < rows) load(r + gridDim.x);
        const float scale = 1.0f / sqrtf(block_sum(sum, part[odd]) / static_cast<float>(size) + eps);
        T* yr = out + static_cast<int64_t>(r) * ld_out;
#pragma unroll
        for (int c = 0; c < kKeep; ++c) {
            const int i = threadIdx.x + c * kThreads;
            if (i < chunks) {
                float4 v = keep[c];
                v.x *= scale * (wv[c].x + w_offset), v.y *= scale * (wv[c].y + w_offset);
                v.z *= scale * (wv[c].z + w_offset), v.w *= scale * (wv[c].w + w_offset);
                store4(yr + 4 * i, v);
            }
        }
    }
}

template <typename T, int kKeep>
int launch_rmsnorm_keep(const float* x, int64_t ld_x, const int32_t* row_index, const float* w, float w_offset, T* out, int64_t ld_out,
                        int rows, int size, float eps, bool vec, void* stream) {
    static int fit[64] = {0};
    auto kernel = rmsnorm_kernel<T, kKeep>;
    OverlapLaunch launch(row_after_row(kKeep) ? row_ctas(kernel, rows, fit) : rows, kThreads, 0, stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, kernel, x, ld_x, row_index, w, w_offset, out, ld_out, rows, size, eps, vec));
    return B2KV_OK;
}

template <typename T>
int launch_rmsnorm(const float* x, int64_t ld_x, const int32_t* row_index, const float* w, float w_offset, T* out, int64_t ld_out,
                   int rows, int size, float eps, bool vec, void* stream) {
    // few registers per thread for rows of usual width
    auto launch = size <= 1024 ? launch_rmsnorm_keep<T, 1> : size <= 2048 ? launch_rmsnorm_keep<T, 2> : size <= 4096 ? launch_rmsnorm_keep<T, 4>
                  : size <= 8192 ? launch_rmsnorm_keep<T, 8> : launch_rmsnorm_keep<T, 16>;
    return launch(x, ld_x, row_index, w, w_offset, out, ld_out, rows, size, eps, vec, stream);
}

// A load that stays where it is: the compiler would have the residual's pieces wait until their sums are known.
__device__ __forceinline__ float4 load_now(const float* p, int i) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p + 4 * i));
    return v;
}

// kOne: a CTA per row, all of which are on the device at once; everything that is read is on its way together, with rows of up to 2048
// elements the weights as well (500 rows of 4096: 5.1 us, 6.2 row after row, for which fewer CTAs fit; 8 of 2048: 2.1 and 2.4).
template <typename T, int kKeep, bool kOne>
__global__ void __launch_bounds__(kThreads) layernorm_rows_kernel(const float* y, int64_t ld_y, const int32_t* row_index,
                                                                  const float* w, const float* b, float* x, int64_t ld_x,
                                                                  T* out, int64_t ld_out, int rows, int size, float eps, bool vec) {
    __shared__ float part[2][kThreads / 32];
    grid_launch_dependents();
    if (threadIdx.x == 0) grid_dependency_wait();
    __syncthreads();
    auto row_of = [&](int r) { return y + static_cast<int64_t>(row_index ? row_index[r] : r) * ld_y; };
    const float inv = 1.0f / static_cast<float>(size);
    if (!vec) {
        for (int r = blockIdx.x; r < rows; r += gridDim.x) {
            const float* yr = row_of(r);
            float* xr = x == nullptr ? nullptr : x + static_cast<int64_t>(r) * ld_x;
            T* outr = out == nullptr ? nullptr : out + static_cast<int64_t>(r) * ld_out;
            float sum = 0.f, sq = 0.f;
            for (int i = threadIdx.x; i < size; i += kThreads) sum += yr[i];
            const float mean = block_sum(sum, part[0]) * inv;
            for (int i = threadIdx.x; i < size; i += kThreads) sq = fmaf(yr[i] - mean, yr[i] - mean, sq);
            const float scale = 1.0f / sqrtf(block_sum(sq, part[1]) * inv + eps);
            for (int i = threadIdx.x; i < size; i += kThreads) {
                float v = fmaf((yr[i] - mean) * scale, w[i], b[i]);
                if (xr != nullptr) xr[i] = v = xr[i] + v;
                if (outr != nullptr) outr[i] = Elt<T>::from_float(v);
            }
        }
        return;
    }
    const int chunks = size / 4;
    float4 next[kKeep], next_res[kKeep];
    auto load = [&](int r) {
        const float* yr = row_of(r);
        const float* xr = x == nullptr ? nullptr : x + static_cast<int64_t>(r) * ld_x;
#pragma unroll
        for (int c = 0; c < kKeep; ++c) {
            const int i = threadIdx.x + c * kThreads;
            if (i < chunks) {
                next[c] = kOne ? load_now(yr, i) : reinterpret_cast<const float4*>(yr)[i];
                if (xr != nullptr) next_res[c] = kOne ? load_now(xr, i) : reinterpret_cast<const float4*>(xr)[i];
            }
        }
    };
    load(blockIdx.x);
    constexpr bool kWeightsAhead = kOne && kKeep <= 2;
    float4 w_ahead[kKeep], b_ahead[kKeep];
#pragma unroll
    for (int c = 0; c < kKeep && kWeightsAhead; ++c) {
        const int i = threadIdx.x + c * kThreads;
        if (i < chunks) w_ahead[c] = load_now(w, i), b_ahead[c] = load_now(b, i);
    }
    for (int r = blockIdx.x; r < rows; r += row_after_row(kKeep) ? gridDim.x : rows) {
        float* xr = x == nullptr ? nullptr : x + static_cast<int64_t>(r) * ld_x;
        T* outr = out == nullptr ? nullptr : out + static_cast<int64_t>(r) * ld_out;
        float4 keep[kKeep], res[kKeep];
        float sum = 0.f, sq = 0.f;
#pragma unroll
        for (int c = 0; c < kKeep; ++c) {
            keep[c] = next[c], res[c] = next_res[c];
            if (static_cast<int>(threadIdx.x) + c * kThreads < chunks) sum += (keep[c].x + keep[c].y) + (keep[c].z + keep[c].w);
        }
        if (!kOne && row_after_row(kKeep) && r + static_cast<int>(gridDim.x) < rows) load(r + gridDim.x);
        const float mean = block_sum(sum, part[0]) * inv;
#pragma unroll
        for (int c = 0; c < kKeep; ++c) {
            if (static_cast<int>(threadIdx.x) + c * kThreads < chunks) {
                keep[c].x -= mean, keep[c].y -= mean, keep[c].z -= mean, keep[c].w -= mean;
                sq += (keep[c].x * keep[c].x + keep[c].y * keep[c].y) + (keep[c].z * keep[c].z + keep[c].w * keep[c].w);
            }
        }
        const float scale = 1.0f / sqrtf(block_sum(sq, part[1]) * inv + eps);
#pragma unroll
        for (int c = 0; c < kKeep; ++c) {
            const int i = threadIdx.x + c * kThreads;
            if (i < chunks) {
                const float4 wv = kWeightsAhead ? w_ahead[c] : reinterpret_cast<const float4*>(w)[i];
                const float4 bv = kWeightsAhead ? b_ahead[c] : reinterpret_cast<const float4*>(b)[i];
                float4 v = keep[c];
                v.x = fmaf(v.x * scale, wv.x, bv.x), v.y = fmaf(v.y * scale, wv.y, bv.y);
                v.z = fmaf(v.z * scale, wv.z, bv.z), v.w = fmaf(v.w * scale, wv.w, bv.w);
                if (xr != nullptr) {
                    v.x += res[c].x, v.y += res[c].y, v.z += res[c].z, v.w += res[c].w;
                    store4(xr + 4 * i, v);
                }
                if (outr != nullptr) store4(outr + 4 * i, v);
            }
        }
        if (kOne) break;
    }
}

template <typename T, int kKeep>
int launch_layernorm_keep(const float* y, int64_t ld_y, const int32_t* row_index, const float* w, const float* b, float* x,
                          int64_t ld_x, T* out, int64_t ld_out, int rows, int size, float eps, bool vec, void* stream) {
    static int fit[64] = {0}, fit_one[64] = {0};
    auto kernel = layernorm_rows_kernel<T, kKeep, false>;
    int ctas = rows;
    if constexpr (row_after_row(kKeep)) {
        ctas = row_ctas(kernel, rows, fit);
        if (row_ctas(layernorm_rows_kernel<T, kKeep, true>, rows, fit_one) == rows) kernel = layernorm_rows_kernel<T, kKeep, true>, ctas = rows;
    }
    OverlapLaunch launch(ctas, kThreads, 0, stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, kernel, y, ld_y, row_index, w, b, x, ld_x, out, ld_out, rows, size, eps, vec));
    return B2KV_OK;
}

template <typename T>
int launch_layernorm_rows(const float* y, int64_t ld_y, const int32_t* row_index, const float* w, const float* b, float* x,
                          int64_t ld_x, T* out, int64_t ld_out, int rows, int size, float eps, bool vec, void* stream) {
    auto launch = size <= 1024 ? launch_layernorm_keep<T, 1> : size <= 2048 ? launch_layernorm_keep<T, 2> : size <= 4096 ? launch_layernorm_keep<T, 4>
                  : size <= 8192 ? launch_layernorm_keep<T, 8> : launch_layernorm_keep<T, 16>;
    return launch(y, ld_y, row_index, w, b, x, ld_x, out, ld_out, rows, size, eps, vec, stream);
}

}  // namespace
}  // namespace b2kv

using namespace b2kv;

extern "C" int b2kv_embed_rows(const void* table, const int32_t* ids, float* out, void* copy, float scale, int rows, int dim,
                               int vocab, int dtype, int32_t* dev_status, void* stream) {
    if (elt_bytes(dtype) == 0) return B2KV_ERR_UNSUPPORTED;
    if (!table || !ids || !out || rows <= 0 || dim <= 0 || vocab <= 0) return B2KV_ERR_BAD_ARG;
    const bool vec = dim % 4 == 0 && aligned16(table) && aligned16(out) && aligned16(copy);
    OverlapLaunch launch(rows, kThreads, 0, stream);
    if (dtype == B2KV_DTYPE_F32)
        B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, embed_rows_kernel<float>, static_cast<const float*>(table), ids, out,
                                         static_cast<float*>(copy), scale, dim, vocab, dev_status, vec));
    else
        B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, embed_rows_kernel<__nv_bfloat16>, static_cast<const __nv_bfloat16*>(table),
                                         ids, out, static_cast<__nv_bfloat16*>(copy), scale, dim, vocab, dev_status, vec));
    return B2KV_OK;
}

extern "C" int b2kv_layernorm_rows(const float* y, int64_t ld_y, const int32_t* row_index, const float* w, const float* b, float* x,
                                   int64_t ld_x, void* out, int64_t ld_out, int rows, int size, float eps, int dtype,
                                   void* stream) {
    if (elt_bytes(dtype) == 0) return B2KV_ERR_UNSUPPORTED;
    if (!y || !w || !b || (!x && !out) || rows <= 0 || size <= 0 || ld_y < size || (x && ld_x < size) || (out && ld_out < size))
        return B2KV_ERR_BAD_ARG;
    const bool vec = size % 4 == 0 && ld_y % 4 == 0 && size <= 16384 && aligned16(y) && aligned16(w) && aligned16(b) &&
                     (!x || (ld_x % 4 == 0 && aligned16(x))) && (!out || (ld_out % 4 == 0 && aligned16(out)));
    if (dtype == B2KV_DTYPE_F32)
        return launch_layernorm_rows(y, ld_y, row_index, w, b, x, ld_x, static_cast<float*>(out), ld_out, rows, size, eps, vec, stream);
    return launch_layernorm_rows(y, ld_y, row_index, w, b, x, ld_x, static_cast<__nv_bfloat16*>(out), ld_out, rows, size, eps, vec, stream);
}

extern "C" int b2kv_rmsnorm(const float* x, int64_t ld_x, const int32_t* row_index, const float* w, float w_offset, void* out,
                            int64_t ld_out, int rows, int size, float eps, int dtype, void* stream) {
    if (elt_bytes(dtype) == 0) return B2KV_ERR_UNSUPPORTED;
    if (!x || !w || !out || rows <= 0 || size <= 0 || ld_x < size || ld_out < size) return B2KV_ERR_BAD_ARG;
    const bool vec = size % 4 == 0 && ld_x % 4 == 0 && ld_out % 4 == 0 && size <= 16384 && aligned16(x) && aligned16(w) && aligned16(out);
    if (dtype == B2KV_DTYPE_F32) return launch_rmsnorm(x, ld_x, row_index, w, w_offset, static_cast<float*>(out), ld_out, rows, size, eps, vec, stream);
    return launch_rmsnorm(x, ld_x, row_index, w, w_offset, static_cast<__nv_bfloat16*>(out), ld_out, rows, size, eps, vec, stream);
}
