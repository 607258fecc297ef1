// b2kv_linear in fp32 on the CUDA cores, two kernels: what linear_f32_tc_kernel does not take, as rows grouped by expert, few rows and few
// input features.  Sums are fp32 multiply-adds, so what bounds them is that pipe (72 TFLOP/s over the chip at 1.9 GHz) for many rows and
// the weights' bytes for few.
//
// linear_f32_tile_kernel: 64 x 128 outputs per CTA of 128 threads, 8 x 8 per thread: 64 multiply-adds for every four 16-byte reads
// of shared memory, so the pipe and not the reads is what is busy.  Steps of 16 input features through two buffers; the next
// step's global reads are in flight (in registers) under the products of this one.  2000 rows of 16 experts, 768 x 1536: 292 us with
// linear_simt_kernel (one read of shared memory per two multiply-adds, nothing ahead of its use), 150 here.
//
// linear_f32_rows_kernel: up to 16 rows (a decode step, the wanted logits).  A thread keeps four neighbouring columns of every row;
// the warps of a CTA and the CTAs of a cluster share the input features, so w is read once, 512 bytes per warp at a time; the clusters'
// partial sums meet in distributed shared memory, in the order of the ranges (results do not depend on timing).  6 rows, 768 x 4096: 128 us
// with linear_simt_kernel, 14 here.
//
// linear_f32_thin_kernel: up to 32 input features and more than 16 rows (a low-rank bottleneck).  What they cost is the outputs and what happens to
// them, of which a tile of 64 x 128 has 64 per thread on a few SMs: a thread keeps two columns of w and goes through a few rows.  The sums
// are in the order of the tiles, to the bit.  1056 rows, 16 -> 384 decays: 6.8 us, 12.7 in tiles; 4000 rows,
// 32 -> 4096 as they are: 36.1 and 39.7.
#include <algorithm>

#include "linear.cuh"

namespace b2kv {
namespace linf32 {

constexpr int kBM = 64, kBN = 128, kStep = 16, kThreads = 128;
constexpr int kLdX = kBM + 4, kLdT = kBN + 4;

// Rows of a CTA's group, and where its operands start.
struct Operands {
    const float *x, *w;
    int first, n_rows;
};
__device__ __forceinline__ Operands operands(const b2kv_linear_args& a, int g) {
    Operands o{static_cast<const float*>(a.x), static_cast<const float*>(a.w) + static_cast<int64_t>(g) * a.group_w, 0, a.rows};
    if (a.group_rows != nullptr) {
        o.first = a.group_rows[g];
        o.n_rows = a.group_rows[g + 1] - o.first;
        o.x += static_cast<int64_t>(o.first) * a.ld_x;
    } else {
        o.x += static_cast<int64_t>(g) * a.group_x;
    }
    return o;
}

__global__ void __launch_bounds__(kThreads, 3) linear_f32_tile_kernel(const __grid_constant__ b2kv_linear_args a) {
    struct Ring {
        float x[2][kStep][kLdX], w[2][kStep][kBN];
    };
    __shared__ union {
        Ring ring;
        float tile[kBM][kLdT];
    } sm;
    grid_launch_dependents();
    grid_dependency_wait();
    const int g = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const Operands op = operands(a, g);
    const int row0 = blockIdx.y * kBM, col0 = blockIdx.x * kBN;
    if (row0 >= op.n_rows) return;

    // x: a warp reads one 16-byte piece of 32 rows (the same pieces of the other rows next); w: whole rows of 128 columns
    float4 xr[2], wr[4];
    auto read = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = row0 + lane + 32 * i, k = k0 + warp * 4;
            xr[i] = r < op.n_rows && k < a.K ? *reinterpret_cast<const float4*>(op.x + static_cast<int64_t>(r) * a.ld_x + k)
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + warp + 4 * i, c = col0 + lane * 4;
            wr[i] = k < a.K && c < a.N ? __ldg(reinterpret_cast<const float4*>(op.w + static_cast<int64_t>(k) * a.ld_w + c))
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto write = [&](int buf) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float* const dst = &sm.ring.x[buf][warp * 4][lane + 32 * i];
            dst[0] = xr[i].x, dst[kLdX] = xr[i].y, dst[2 * kLdX] = xr[i].z, dst[3 * kLdX] = xr[i].w;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(&sm.ring.w[buf][warp + 4 * i][lane * 4]) = wr[i];
    };
    // a warp has 32 rows x 64 columns, a thread rows r, r + 16 .. + 3 and columns c, c + 32 .. + 3 of them
    const int tr = (warp & 1) * 32 + (lane >> 3) * 4, tc = (warp >> 1) * 64 + (lane & 7) * 4;
    float acc[8][8] = {};
    read(0);
    write(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < a.K; k0 += kStep, buf ^= 1) {
        const bool more = k0 + kStep < a.K;
        if (more) read(k0 + kStep);
#pragma unroll
        for (int k = 0; k < kStep; ++k) {
            const float4 x0 = *reinterpret_cast<const float4*>(&sm.ring.x[buf][k][tr]);
            const float4 x1 = *reinterpret_cast<const float4*>(&sm.ring.x[buf][k][tr + 16]);
            const float4 w0 = *reinterpret_cast<const float4*>(&sm.ring.w[buf][k][tc]);
            const float4 w1 = *reinterpret_cast<const float4*>(&sm.ring.w[buf][k][tc + 32]);
            const float xv[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
            const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
        }
        if (more) write(buf ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; j += 4)
            *reinterpret_cast<float4*>(&sm.tile[tr + (i & 3) + (i >> 2) * 16][tc + j * 8]) =
                make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
    __syncthreads();
    const int c = (tid & 63) * 2;
    if (col0 + c >= a.N) return;
    lin::finish_rows<float>(a, g, col0 + c, op.first + row0, tid >> 6, min(kBM, op.n_rows - row0), 2,
                            [&](int r) { return *reinterpret_cast<const float2*>(&sm.tile[r][c]); });
}

constexpr int kRowsThreads = 256, kRowsCols = 128, kChunkK = 128;

template <int kR>
__global__ void __launch_bounds__(kRowsThreads) linear_f32_rows_kernel(const __grid_constant__ b2kv_linear_args a, int splits) {
    constexpr int kWarps = kRowsThreads / 32;
    __shared__ float4 xs[kChunkK][kR / 4];
    __shared__ float4 part[kWarps / 2][kR][kRowsCols / 4];
    grid_launch_dependents();
    grid_dependency_wait();
    const int g = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const Operands op = operands(a, g);
    const int split = splits > 1 ? static_cast<int>(cluster_rank()) : 0;
    const int c0 = static_cast<int>(blockIdx.x) / splits * kRowsCols, c = c0 + lane * 4;
    if (op.n_rows <= 0) return;
    const int chunks = (a.K + kChunkK - 1) / kChunkK;
    const int k_first = static_cast<int>(static_cast<long long>(chunks) * split / splits) * kChunkK;
    const int k_end = min(static_cast<int>(static_cast<long long>(chunks) * (split + 1) / splits) * kChunkK, a.K);
    float4 acc[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    constexpr int kMine = kChunkK / kWarps;  // input features of a chunk per warp: neighbours, so that w is read in long runs
    for (int k0 = k_first; k0 < k_end; k0 += kChunkK) {
        float4 wv[kMine];
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
            const int k = k0 + warp * kMine + i;
            wv[i] = k < k_end && c < a.N ? __ldg(reinterpret_cast<const float4*>(op.w + static_cast<int64_t>(k) * a.ld_w + c))
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
        for (int i = tid; i < kChunkK * kR; i += kRowsThreads) {
            const int r = i / kChunkK, k = i % kChunkK;
            reinterpret_cast<float*>(xs[k])[r] = r < op.n_rows && k0 + k < k_end ? op.x[static_cast<int64_t>(r) * a.ld_x + k0 + k] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
#pragma unroll
            for (int q = 0; q < kR / 4; ++q) {
                const float4 xq = xs[warp * kMine + i][q];
                const float xv[4] = {xq.x, xq.y, xq.z, xq.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float4& s = acc[q * 4 + e];
                    s.x = fmaf(xv[e], wv[i].x, s.x), s.y = fmaf(xv[e], wv[i].y, s.y);
                    s.z = fmaf(xv[e], wv[i].z, s.z), s.w = fmaf(xv[e], wv[i].w, s.w);
                }
            }
        }
    }
    // the warps' sums, halves of them at a time, then the ranges' (in order)
#pragma unroll
    for (int half = kWarps / 2; half > 0; half >>= 1) {
        __syncthreads();
        if (warp >= half && warp < 2 * half) {
#pragma unroll
            for (int r = 0; r < kR; ++r) part[warp - half][r][lane] = acc[r];
        }
        __syncthreads();
        if (warp < half) {
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                const float4 p = part[warp][r][lane];
                acc[r].x += p.x, acc[r].y += p.y, acc[r].z += p.z, acc[r].w += p.w;
            }
        }
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int r = 0; r < kR; ++r) part[0][r][lane] = acc[r];
    }
    if (splits > 1) cluster_sync();
    else __syncthreads();
    const int cp = (tid & 63) * 2;
    if (c0 + cp < a.N)
        lin::finish_rows<float>(a, g, c0 + cp, op.first, (tid >> 6) * splits + split, min(kR, op.n_rows), kRowsThreads / 64 * splits, [&](int r) {
            float2 v = make_float2(0.f, 0.f);
            for (int s = 0; s < splits; ++s) {
                const float2 p = peer_load2(peer_address(&part[0][r][0], s) + cp * 4);
                v.x += p.x, v.y += p.y;
            }
            return v;
        });
    __syncwarp();
    if (splits > 1) cluster_sync();
}

constexpr int kThinThreads = 128, kThinK = 32, kThinRows = 32;

template <int kK>
__global__ void __launch_bounds__(kThinThreads) linear_f32_thin_kernel(const __grid_constant__ b2kv_linear_args a, int row_tile) {
    __shared__ float xs[kThinRows][kK];
    grid_launch_dependents();
    grid_dependency_wait();
    const int row0 = static_cast<int>(blockIdx.y) * row_tile, n = min(row_tile, a.rows - row0);
    const int c = (static_cast<int>(blockIdx.x) * kThinThreads + threadIdx.x) * 2;
    const float* const x = static_cast<const float*>(a.x) + static_cast<int64_t>(row0) * a.ld_x;
    for (int i = threadIdx.x; i < n * kK; i += kThinThreads) {
        const int r = i / kK, k = i % kK;
        xs[r][k] = k < a.K ? x[static_cast<int64_t>(r) * a.ld_x + k] : 0.f;
    }
    float2 w[kK];  // (N is a multiple of 4)
#pragma unroll
    for (int k = 0; k < kK; ++k)
        w[k] = c < a.N && k < a.K ? *reinterpret_cast<const float2*>(static_cast<const float*>(a.w) + static_cast<int64_t>(k) * a.ld_w + c)
                                  : make_float2(0.f, 0.f);
    __syncthreads();
    if (c >= a.N) return;
    lin::finish_rows<float>(a, 0, c, row0, 0, n, 1, [&](int r) {
        float2 v = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < kK; ++k) v = __ffma2_rn(make_float2(xs[r][k], xs[r][k]), w[k], v);
        return v;
    });
}

}  // namespace linf32

int linear_f32(const b2kv_linear_args& a, void* stream) {
    using namespace linf32;
    if (a.dtype != B2KV_DTYPE_F32) return B2KV_ERR_UNSUPPORTED;
    // 16-byte pieces of rows of x and w; outputs and the residual have no rule
    if (!aligned16(a.x) || !aligned16(a.w) || a.K % 4 || a.N % 4 || a.ld_x % 4 || a.ld_w % 4 || a.group_x % 4 || a.group_w % 4)
        return B2KV_ERR_UNSUPPORTED;
    const int max_rows = a.group_rows ? a.max_group_rows : a.rows, sms = device_sm_count();
    const long long tiles_n = (a.N + kBN - 1) / kBN;
    if (max_rows <= 16) {
        // (the sums over the warps take longer than the products of a row: 3.4 us at K = 4, 2.9 with linear_simt_kernel; four rows 3.9 and 6.4)
        if (a.K < 16 && max_rows == 1) return B2KV_ERR_UNSUPPORTED;
        // ranges of at least one chunk, two CTAs per SM at most
        const long long tiles = tiles_n * a.groups;
        int splits = 1;
        const int forced = tune_get("matmul_splits");
        while (splits < 8 && (forced > 0 ? splits * 2 <= forced : tiles * splits * 2 <= 2 * sms && splits * 2 * kChunkK <= a.K)) splits *= 2;
        if (tiles_n * splits > 0x7fffffffLL || a.groups > 65535) return B2KV_ERR_UNSUPPORTED;
        OverlapLaunch launch(dim3(static_cast<unsigned>(tiles_n * splits), 1, a.groups), kRowsThreads, 0, stream, splits);
        B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg,
                                         max_rows <= 4 ? linear_f32_rows_kernel<4>
                                                       : (max_rows <= 8 ? linear_f32_rows_kernel<8> : linear_f32_rows_kernel<16>),
                                         a, splits));
        return B2KV_OK;
    }
    // (many rows of columns that leave a quarter and more of the threads idle: the tiles are better at the same sums, 8000 rows of 384 columns, K = 32,
    // 9.4 us and 11.9 by threads, 32000 of 96 14.4 and 15.8; fewer rows, 6000 of 96, 6.3 and 5.3)
    const long long thin_cols = (a.N / 2 + kThinThreads - 1) / kThinThreads;
    const bool idle = 4LL * a.N <= 3 * thin_cols * 2 * kThinThreads && a.rows * thin_cols >= (a.N <= 2 * kThinThreads ? 32000 : 16000);
    if (a.K <= kThinK && a.groups == 1 && a.group_rows == nullptr && !idle) {
        // rows per CTA: as few (eight) as leave all CTAs on the device at once (6000 rows, 16 -> 64: 750 CTAs of 8 rows, of which 740 fit, 4.7 us, 3.5
        // with 9; 4000 rows, 16 -> 768: 750 of 16 7.4, 6.5 with 17)
        const long long cols = thin_cols;
        const auto kernel = a.K <= 16 ? linear_f32_thin_kernel<16> : linear_f32_thin_kernel<32>;
        static int per_sm[2][64] = {};
        int dev = 0;
        B2KV_CUDA_TRY(cudaGetDevice(&dev));
        if (dev < 0 || dev >= 64) return B2KV_ERR_UNSUPPORTED;
        int& resident = per_sm[a.K <= 16][dev];
        if (resident == 0) B2KV_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, kThinThreads, 0));
        const long long fit = std::max(resident, 1) * static_cast<long long>(sms);
        const int row_tile = static_cast<int>(std::min<long long>(std::max<long long>((a.rows * cols + fit - 1) / fit, 8), kThinRows));
        const dim3 grid(static_cast<unsigned>(cols), static_cast<unsigned>((a.rows + row_tile - 1) / row_tile));
        if (grid.y <= 65535u) {
            OverlapLaunch launch(grid, kThinThreads, 0, stream);
            B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, kernel, a, row_tile));
            return B2KV_OK;
        }
    }
    const long long tiles_m = (max_rows + kBM - 1) / kBM;
    if (tiles_m > 65535 || a.groups > 65535 || tiles_n > 0x7fffffffLL) return B2KV_ERR_UNSUPPORTED;
    OverlapLaunch launch(dim3(static_cast<unsigned>(tiles_n), static_cast<unsigned>(tiles_m), a.groups), kThreads, 0, stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, linear_f32_tile_kernel, a));
    return B2KV_OK;
}

}  // namespace b2kv
