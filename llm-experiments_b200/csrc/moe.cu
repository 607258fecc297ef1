// Mixture of experts around the grouped products of b2kv_linear: expert choice, the sort of the chosen rows by expert, and
// the weighted sum of the experts' outputs onto the 32-bit residual stream.
// These kernels may be scheduled ahead of the end of the kernel that writes their inputs, so no pointer to such data is
// const __restrict__: the compiler would take it for data that nothing writes and could load it before the wait.
#include <math.h>

#include <algorithm>

#include "b2kv_common.cuh"

namespace b2kv {
namespace {

constexpr int kMaxExperts = 1024, kMaxTop = 64;
constexpr int kRouteWarps = 4, kRouteWarpsMany = 32;

// Largest value over a warp and, among equals, the lowest index.
__device__ __forceinline__ void warp_best(float& v, int& i) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, off);
        const int oi = __shfl_xor_sync(0xffffffffu, i, off);
        if (ov > v || (ov == v && oi < i)) v = ov, i = oi;
    }
}

__global__ void zero_counts_kernel(int32_t* counts, int n) {
    grid_launch_dependents();
    if (threadIdx.x == 0) grid_dependency_wait();
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) counts[i] = 0;
}

// A warp per row.  A score that is taken, or whose group is not kept, is replaced by -1 (scores are positive).  Many rows: what bounds it is the
// counting, two choices per nanosecond wherever they fall, so a CTA of 32 rows counts its own and adds them up expert by expert (3548
// rows, 6 of 64 experts: 9.7 us, 16.2 with every choice counted in memory; 8000 rows 10.1 and 32.8).
template <int kWarps>
__global__ void __launch_bounds__(kWarps * 32)
route_kernel(const float* logits, int64_t ld, int rows, int experts, int groups, int keep, int top,
             int32_t* idx, float* score, int32_t* counts) {
    extern __shared__ float sm_route[];
    grid_launch_dependents();
    if (threadIdx.x == 0) grid_dependency_wait();
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x * kWarps + warp;
    constexpr bool kOwnCounts = kWarps > kRouteWarps;
    int* const own = reinterpret_cast<int*>(sm_route + kWarps * 2 * experts);  // [experts]
    if (kOwnCounts) {
        for (int e = threadIdx.x; e < experts; e += kWarps * 32) own[e] = 0;
        __syncthreads();
    }
    if (!kOwnCounts && row >= rows) return;
    float* s = sm_route + warp * 2 * experts;  // scores
    float* best = s + experts;                 // largest score of every group (-1: taken)
    const float* z = logits + min(row, rows - 1) * ld;  // (a warp without a row stays for the barrier)
    float mx = -INFINITY;
    for (int e = lane; e < experts; e += 32) mx = fmaxf(mx, s[e] = z[e]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    float sum = 0.f;
    for (int e = lane; e < experts; e += 32) sum += s[e] = expf(s[e] - mx);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    for (int e = lane; e < experts; e += 32) s[e] = s[e] / sum;
    __syncwarp();
    if (keep < groups) {
        const int per = experts / groups;
        for (int g = lane; g < groups; g += 32) {
            float b = s[g * per];
            for (int e = 1; e < per; ++e) b = fmaxf(b, s[g * per + e]);
            best[g] = b;
        }
        __syncwarp();
        // what is not among the best is dropped: take the `keep` best away, the rest loses its experts
        for (int k = 0; k < keep; ++k) {
            float v = -2.f;
            int i = 0x7fffffff;
            for (int g = lane; g < groups; g += 32)
                if (best[g] > v) v = best[g], i = g;
            warp_best(v, i);
            if (i >= groups) i = k;  // scores that are not numbers: any group, but one that exists
            if (lane == 0) best[i] = -1.f;
            __syncwarp();
        }
        for (int e = lane; e < experts; e += 32)
            if (best[e / per] >= 0.f) s[e] = -1.f;
        __syncwarp();
    }
    for (int k = 0; k < top && row < rows; ++k) {
        float v = -2.f;
        int i = 0x7fffffff;
        for (int e = lane; e < experts; e += 32)
            if (s[e] > v) v = s[e], i = e;
        warp_best(v, i);
        if (i >= experts) i = k, v = 0.f;
        if (lane == 0) {
            idx[static_cast<int64_t>(row) * top + k] = i;
            score[static_cast<int64_t>(row) * top + k] = v;
            atomicAdd(kOwnCounts ? &own[i] : &counts[i], 1);
            s[i] = -1.f;
        }
        __syncwarp();
    }
    if (kOwnCounts) {
        __syncthreads();
        for (int e = threadIdx.x; e < experts; e += kWarps * 32)
            if (own[e] != 0) atomicAdd(&counts[e], own[e]);
    }
}

// A CTA per row, or per `per` of its choices: their places among the sorted rows, and the copies of the row there (128-bit when aligned).  The row is
// read once and its first pieces stay in registers; what bounds it is the copies' bytes (a CTA per choice, with the whole chain of
// loads before its first copy, took 38 us for 2975 rows of 4 KB and six choices, this one 25).
constexpr int kPlanThreads = 128;

template <bool kTable>  // the experts' first rows fit shared memory
__global__ void __launch_bounds__(kPlanThreads)
moe_plan_kernel(const int32_t* idx, int32_t* counts, int experts, int top, int32_t* offsets,
                int32_t* slot, const uint8_t* h, int64_t pitch_h, uint8_t* sorted,
                int64_t pitch_sorted, int row_bytes, bool vec, int per) {
    extern __shared__ int sm_plan[];  // [experts + 1]: row behind the last one of the experts before; then the places of the row's choices
    const int row = blockIdx.x, lane = threadIdx.x & 31, k_first = blockIdx.y * per, k_end = min(top, k_first + per);
    const bool writes = row == 0 && k_first == 0;  // the offsets
    int* const first = kTable ? sm_plan : offsets;  // (without a table one CTA writes them where they belong)
    int* const place = kTable ? sm_plan + experts + 1 : slot + static_cast<int64_t>(row) * top;
    constexpr int kKeep = 4;
    grid_launch_dependents();
    if (threadIdx.x == 0) grid_dependency_wait();
    __syncthreads();
    const uint8_t* src = h + static_cast<int64_t>(row) * pitch_h;
    uint4 keep[kKeep];
#pragma unroll
    for (int u = 0; u < kKeep; ++u) {
        const int i = threadIdx.x + u * kPlanThreads;
        if (vec && i < row_bytes / 16) keep[u] = reinterpret_cast<const uint4*>(src)[i];
    }
    if (threadIdx.x < 32) {
        int base = 0;
        for (int e0 = 0; e0 < experts && (kTable || writes); e0 += 32) {
            const int n = e0 + lane < experts ? counts[e0 + lane] : 0;
            int end = n;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, end, off);
                if (lane >= off) end += up;
            }
            if (e0 + lane < experts) first[e0 + lane] = base + end - n;
            base += __shfl_sync(0xffffffffu, end, 31);
        }
        if (lane == 0 && (kTable || writes)) first[experts] = base;
        __syncwarp();
        for (int k = k_first; k < k_end && !kTable; ++k) {
            const int e = idx[static_cast<int64_t>(row) * top + k];
            int before = 0;
            for (int i = lane; i < e; i += 32) before += counts[i];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) before += __shfl_xor_sync(0xffffffffu, before, off);
            if (lane == 0) place[k] = before + atomicAdd(&counts[experts + e], 1);
        }
        for (int k = k_first + lane; k < k_end && kTable; k += 32) {
            const int e = idx[static_cast<int64_t>(row) * top + k];
            place[k] = first[e] + atomicAdd(&counts[experts + e], 1);
            slot[static_cast<int64_t>(row) * top + k] = place[k];
        }
    }
    __syncthreads();
    if (writes && kTable)
        for (int i = threadIdx.x; i <= experts; i += kPlanThreads) offsets[i] = first[i];
    if (!vec) {
        for (int k = k_first; k < k_end; ++k)
            for (int i = threadIdx.x; i < row_bytes / 2; i += kPlanThreads)
                reinterpret_cast<uint16_t*>(sorted + place[k] * pitch_sorted)[i] = reinterpret_cast<const uint16_t*>(src)[i];
        return;
    }
    for (int k = k_first; k < k_end; ++k) {
        uint4* const dst = reinterpret_cast<uint4*>(sorted + place[k] * pitch_sorted);
#pragma unroll
        for (int u = 0; u < kKeep; ++u) {
            const int i = threadIdx.x + u * kPlanThreads;
            if (i < row_bytes / 16) dst[i] = keep[u];
        }
        for (int i = threadIdx.x + kKeep * kPlanThreads; i < row_bytes / 16; i += kPlanThreads) dst[i] = reinterpret_cast<const uint4*>(src)[i];
    }
}

template <typename T, int kAhead>  // kAhead: choices whose pieces are on their way together, with the row's own (1: as few registers as it goes)
__global__ void __launch_bounds__(256) moe_combine_kernel(float* x, int64_t ld_x, const T* y,
                                                          int64_t ld_y, const int32_t* slot,
                                                          const float* score, int top, int dim, bool vec) {
    __shared__ int32_t sl[kMaxTop];
    __shared__ float sc[kMaxTop];
    grid_launch_dependents();
    if (threadIdx.x == 0) grid_dependency_wait();
    __syncthreads();
    const int64_t row = blockIdx.x;
    if (threadIdx.x < top) {
        sl[threadIdx.x] = slot[row * top + threadIdx.x];
        sc[threadIdx.x] = score[row * top + threadIdx.x];
    }
    __syncthreads();
    float* xr = x + row * ld_x;
    if (vec) {
        constexpr int kC = Elt<T>::kPerChunk;
        for (int i = threadIdx.x; i < dim / kC; i += blockDim.x) {
            float acc[kC] = {};
            if constexpr (kAhead == 1) {
                for (int k = 0; k < top; ++k) {
                    float v[kC];
                    Elt<T>::widen(reinterpret_cast<const uint4*>(y + sl[k] * ld_y)[i], v);
#pragma unroll
                    for (int j = 0; j < kC; ++j) acc[j] = fmaf(sc[k], v[j], acc[j]);
                }
#pragma unroll
                for (int j = 0; j < kC / 4; ++j) {
                    float4* const p = reinterpret_cast<float4*>(xr + i * kC) + j;
                    const float4 o = *p;
                    *p = make_float4(o.x + acc[4 * j], o.y + acc[4 * j + 1], o.z + acc[4 * j + 2], o.w + acc[4 * j + 3]);
                }
                continue;
            }
            float4 o[kC / 4];
#pragma unroll
            for (int j = 0; j < kC / 4; ++j) o[j] = reinterpret_cast<const float4*>(xr + i * kC)[j];
            for (int k0 = 0; k0 < top; k0 += kAhead) {
                uint4 piece[kAhead];
#pragma unroll
                for (int k = 0; k < kAhead; ++k)
                    if (k0 + k < top) piece[k] = reinterpret_cast<const uint4*>(y + sl[k0 + k] * ld_y)[i];
#pragma unroll
                for (int k = 0; k < kAhead; ++k) {
                    if (k0 + k >= top) break;
                    float v[kC];
                    Elt<T>::widen(piece[k], v);
#pragma unroll
                    for (int j = 0; j < kC; ++j) acc[j] = fmaf(sc[k0 + k], v[j], acc[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < kC / 4; ++j) {
                o[j].x += acc[4 * j], o[j].y += acc[4 * j + 1], o[j].z += acc[4 * j + 2], o[j].w += acc[4 * j + 3];
                reinterpret_cast<float4*>(xr + i * kC)[j] = o[j];
            }
        }
        return;
    }
    for (int i = threadIdx.x; i < dim; i += blockDim.x) {
        float acc = 0.f;
        for (int k = 0; k < top; ++k) acc = fmaf(sc[k], Elt<T>::to_float(y[sl[k] * ld_y + i]), acc);
        xr[i] += acc;
    }
}

}  // namespace
}  // namespace b2kv

using namespace b2kv;

extern "C" int b2kv_route(const float* logits, int64_t ld, int rows, int experts, int groups, int keep, int top, int32_t* idx,
                          float* score, int32_t* counts, void* stream) {
    if (!logits || !idx || !score || !counts || rows <= 0 || experts <= 0 || ld < experts || groups <= 0 || keep <= 0 ||
        keep > groups || experts % groups != 0 || top <= 0 || top > keep * (experts / groups))
        return B2KV_ERR_BAD_ARG;
    if (experts > kMaxExperts || top > kMaxTop) return B2KV_ERR_UNSUPPORTED;
    OverlapLaunch zero(1, 256, 0, stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&zero.cfg, zero_counts_kernel, counts, 2 * experts));
    const size_t many_bytes = (static_cast<size_t>(kRouteWarpsMany) * 2 + 1) * experts * sizeof(float);
    // CTAs of 32 rows where many of their choices meet and there are choices enough for counting to be what takes the time; us with four rows and
    // with 32.  2048 rows: 4 of 32 experts 9.5, 8.4; 6 of 64 12.4, 11.9; 8 of 64 15.0, 12.8.  3001: 2 of 16 8.4, 8.6; 4 of 32 11.5, 10.8; 6 of 64
    // 15.9, 13.8.  8000: 2 of 16 15.7, 10.0; 6 of 64 36, 15.  With fewer that meet, 3001 rows: 4 of 64 12.1, 12.0; 6 of 96 12.9, 14.8; 6 of
    // 160 13.2, 16.0 (from some 4500 rows on it would pay there too: 4 of 64 16.1, 12.6; 8000 rows, 6 of 160 25, 18).  1500 rows, 6 of 64: 10.1 and 9.3, but
    // the kernel behind begins later, 18.8 and 20.4 together.
    const bool many = rows >= 2048 && static_cast<long long>(rows) * top >= 8192 && kRouteWarpsMany * top >= 3 * experts && many_bytes <= 48 * 1024;
    const int warps = many ? kRouteWarpsMany : kRouteWarps;
    OverlapLaunch launch((rows + warps - 1) / warps, warps * 32, many ? many_bytes : static_cast<size_t>(kRouteWarps) * 2 * experts * sizeof(float), stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, many ? route_kernel<kRouteWarpsMany> : route_kernel<kRouteWarps>, logits, ld, rows, experts, groups, keep,
                                     top, idx, score, counts));
    return B2KV_OK;
}

extern "C" int b2kv_moe_plan(const int32_t* idx, int32_t* counts, int rows, int experts, int top, int32_t* offsets,
                             int32_t* slot, const void* h, int64_t ld_h, void* sorted, int64_t ld_sorted, int dim, int dtype,
                             void* stream) {
    const int es = elt_bytes(dtype);
    if (es == 0) return B2KV_ERR_UNSUPPORTED;
    if (!idx || !counts || !offsets || !slot || !h || !sorted || rows <= 0 || experts <= 0 || top <= 0 || dim <= 0 || ld_h < dim ||
        ld_sorted < dim)
        return B2KV_ERR_BAD_ARG;
    if (static_cast<long long>(rows) * top > 0x7fffffffLL) return B2KV_ERR_UNSUPPORTED;
    const bool vec = (dim * es) % 16 == 0 && (ld_h * es) % 16 == 0 && (ld_sorted * es) % 16 == 0 && aligned16(h) && aligned16(sorted);
    const size_t bytes = (static_cast<size_t>(experts) + 1 + top) * sizeof(int);
    const bool table = bytes <= 48 * 1024;
    // Few rows: several CTAs for the choices of one, up to three per SM and of at least 32 KB of copies (by 16 bits they count eight times): one
    // after the other in one CTA they take longer than the row read again (8 rows of 32 KB, 64 choices: 84 us with a CTA per row, 34 so; with 300 rows of
    // 2 KB two CTAs per row take longer than one, 54 us and 45).
    const long long copied = static_cast<long long>(dim) * es * (vec ? 1 : 8) * top;
    const long long wanted = std::max<long long>(1, std::min<long long>(3LL * device_sm_count() / rows, copied / (32 * 1024)));
    const int most = static_cast<int>(std::min<long long>(wanted, top)), per = (top + most - 1) / most;
    const long long parts = (top + per - 1) / per;
    if (parts > 65535) return B2KV_ERR_UNSUPPORTED;
    OverlapLaunch launch(dim3(rows, static_cast<unsigned>(parts)), kPlanThreads, table ? bytes : 0, stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, table ? moe_plan_kernel<true> : moe_plan_kernel<false>, idx, counts, experts, top, offsets, slot,
                                     static_cast<const uint8_t*>(h), ld_h * es, static_cast<uint8_t*>(sorted), ld_sorted * es,
                                     dim * es, vec, per));
    return B2KV_OK;
}

extern "C" int b2kv_moe_combine(float* x, int64_t ld_x, const void* y, int64_t ld_y, const int32_t* slot, const float* score,
                                int rows, int top, int dim, int dtype, void* stream) {
    const int es = elt_bytes(dtype);
    if (es == 0) return B2KV_ERR_UNSUPPORTED;
    if (!x || !y || !slot || !score || rows <= 0 || top <= 0 || dim <= 0 || ld_x < dim || ld_y < dim) return B2KV_ERR_BAD_ARG;
    if (top > kMaxTop) return B2KV_ERR_UNSUPPORTED;
    const bool vec = (dim * es) % 16 == 0 && (ld_y * es) % 16 == 0 && ld_x % 4 == 0 && dim % 4 == 0 && aligned16(x) && aligned16(y);
    // Pieces on their way together pay unless registers then keep rows off the SM: two choices, rows by 16 bits, and many rows narrower
    // than a CTA (3000 rows, two choices: 4096 columns 24.0 us with six, 19.4 one by one; six choices: 41.1 and 42.8, 1024 columns 8.8 and 8.2;
    // 64 rows of 4096: 3.5 and 4.3).
    const bool ahead = vec && top > 2 && (top > 6 || dim * es / 16 >= 256 || rows <= 1024);
    OverlapLaunch launch(rows, 256, 0, stream);
    if (dtype == B2KV_DTYPE_F32)
        B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, ahead ? moe_combine_kernel<float, 6> : moe_combine_kernel<float, 1>, x, ld_x,
                                         static_cast<const float*>(y), ld_y, slot, score, top, dim, vec));
    else
        B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, ahead ? moe_combine_kernel<__nv_bfloat16, 6> : moe_combine_kernel<__nv_bfloat16, 1>, x, ld_x,
                                         static_cast<const __nv_bfloat16*>(y), ld_y, slot, score, top, dim, vec));
    return B2KV_OK;
}
