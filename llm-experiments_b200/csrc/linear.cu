// b2kv_linear: argument checks, the choice of the kernel, and two CUDA-core kernels: one for shapes and alignments that no other kernel
// takes (64 x 64 output tiles, 16 input features per step, 4 x 4 outputs per thread, fp32 accumulation) and one for few input features.
#include "linear.cuh"

namespace b2kv {
namespace lin {

constexpr int kTile = 64, kStep = 16, kThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kThreads) linear_simt_kernel(const b2kv_linear_args a) {
    __shared__ float xs[kStep][kTile + 4];
    __shared__ float ws[kStep][kTile + 4];
    const int g = blockIdx.z;
    int first = 0, n_rows = a.rows;
    const T* x = static_cast<const T*>(a.x);
    if (a.group_rows != nullptr) {
        first = a.group_rows[g];
        n_rows = a.group_rows[g + 1] - first;
        x += static_cast<int64_t>(first) * a.ld_x;
    } else {
        x += static_cast<int64_t>(g) * a.group_x;
    }
    const int row0 = blockIdx.y * kTile, col0 = blockIdx.x * kTile;
    if (row0 >= n_rows) return;
    const T* w = static_cast<const T*>(a.w) + static_cast<int64_t>(g) * a.group_w;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < a.K; k0 += kStep) {
        for (int i = threadIdx.x; i < kTile * kStep; i += kThreads) {
            const int r = i / kStep, k = i % kStep;
            xs[k][r] = (row0 + r < n_rows && k0 + k < a.K)
                           ? Elt<T>::to_float(x[static_cast<int64_t>(row0 + r) * a.ld_x + k0 + k]) : 0.f;
            const int wk = i / kTile, c = i % kTile;
            ws[wk][c] = (k0 + wk < a.K && col0 + c < a.N)
                            ? Elt<T>::to_float(w[static_cast<int64_t>(k0 + wk) * a.ld_w + col0 + c]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kStep; ++k) {
            float xv[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) xv[i] = xs[k][ty * 4 + i], wv[i] = ws[k][tx * 4 + i];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = row0 + ty * 4 + i;
        if (r >= n_rows) break;
        const int64_t out_row = first + r;
#pragma unroll
        for (int j = 0; j < 4; j += 2) {  // pairs of columns: boundaries of segments are even
            const int c = col0 + tx * 4 + j;
            if (c >= a.N) break;
            finish_pair<T>(a, g, out_row, c, acc[i][j], acc[i][j + 1]);
        }
    }
}

static int launch_simt(const b2kv_linear_args& a, void* stream) {
    const int max_rows = a.group_rows ? a.max_group_rows : a.rows;
    const dim3 grid((a.N + kTile - 1) / kTile, (max_rows + kTile - 1) / kTile, a.groups);
    if (grid.y > 65535u || grid.z > 65535u) return B2KV_ERR_UNSUPPORTED;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (a.dtype == B2KV_DTYPE_F32)
        linear_simt_kernel<float><<<grid, kThreads, 0, s>>>(a);
    else
        linear_simt_kernel<__nv_bfloat16><<<grid, kThreads, 0, s>>>(a);
    B2KV_CUDA_TRY(cudaGetLastError());
    return B2KV_OK;
}

// Products with few input features (a low-rank bottleneck): what they cost is the outputs, so there is nothing for the tensor
// cores to win.  A thread keeps two columns of w in registers and goes through a tile of rows, whose few elements lie in shared
// memory; neighbouring threads store neighbouring columns.  Four rows are under way together, a row's sums and what becomes of them being a chain,
// and what becomes of a column is chosen outside the loop (64 rows, 16 -> 1024 decays 3.6 -> 2.6 us; 16000 rows, 16 -> 2048 72 -> 62; 4000 rows,
// 32 -> 4096 in bf16 42 -> 29).
constexpr int kThinK = 32, kThinThreads = 128, kThinRows = 64;
constexpr int kThinAhead = 4;  // rows at a time

template <int kK>
__global__ void __launch_bounds__(kThinThreads) linear_thin_kernel(const __grid_constant__ b2kv_linear_args a, int row_tile) {
    __shared__ float4 xs[kThinRows][kK / 4];
    const int c = (blockIdx.x * kThinThreads + threadIdx.x) * 2;
    const bool live = c < a.N;
    const __nv_bfloat16* const w = static_cast<const __nv_bfloat16*>(a.w);
    float2 wr[kK], bias = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < kK; ++k) {
        wr[k] = make_float2(0.f, 0.f);
        if (live && k < a.K) wr[k] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(w + k * a.ld_w + c));
    }
    if (live && a.bias != nullptr) bias = make_float2(a.bias[c], a.bias[c + 1]);
    grid_launch_dependents();
    if (threadIdx.x == 0) grid_dependency_wait();
    __syncthreads();
    const int row0 = blockIdx.y * row_tile, n = min(row_tile, a.rows - row0);
    const __nv_bfloat16* const x = static_cast<const __nv_bfloat16*>(a.x) + row0 * a.ld_x;
    for (int i = threadIdx.x; i < n * kK; i += kThinThreads) {
        const int r = i / kK, k = i % kK;
        reinterpret_cast<float*>(xs[r])[k] = k < a.K ? __bfloat162float(x[r * a.ld_x + k]) : 0.f;
    }
    __syncthreads();
    if (!live) return;
    const b2kv_segment& sg = a.seg[0];
    const float* const residual = sg.kind == B2KV_SEG_F32 && a.residual != nullptr ? a.residual + static_cast<int64_t>(row0) * a.ld_residual + c : nullptr;
    with_kind(sg.kind, [&](auto of) {
        constexpr int kKind = decltype(of)::value;
        for (int r0 = 0; r0 < n; r0 += kThinAhead) {
            float2 v[kThinAhead];
#pragma unroll
            for (int u = 0; u < kThinAhead; ++u) v[u] = bias;
#pragma unroll
            for (int k = 0; k < kK; k += 4) {
#pragma unroll
                for (int u = 0; u < kThinAhead; ++u) {
                    const float4 xv = xs[r0 + u][k / 4];  // (behind the last row: whatever lies there)
                    v[u] = __ffma2_rn(make_float2(xv.x, xv.x), wr[k], v[u]);
                    v[u] = __ffma2_rn(make_float2(xv.y, xv.y), wr[k + 1], v[u]);
                    v[u] = __ffma2_rn(make_float2(xv.z, xv.z), wr[k + 2], v[u]);
                    v[u] = __ffma2_rn(make_float2(xv.w, xv.w), wr[k + 3], v[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < kThinAhead; ++u) v[u] = make_float2(single(kKind, v[u].x, a.limit), single(kKind, v[u].y, a.limit));
#pragma unroll
            for (int u = 0; u < kThinAhead; ++u) {
                if (r0 + u >= n) break;
                const int64_t row = row0 + r0 + u;
                if (is_f32(kKind)) {
                    if (residual != nullptr) {
                        const float2 add = *reinterpret_cast<const float2*>(residual + static_cast<int64_t>(r0 + u) * a.ld_residual);
                        v[u].x += add.x, v[u].y += add.y;
                    }
                    *reinterpret_cast<float2*>(static_cast<float*>(sg.out) + row * sg.ld + c) = v[u];
                } else {
                    *reinterpret_cast<__nv_bfloat162*>(static_cast<__nv_bfloat16*>(sg.out) + row * sg.ld + c) = __floats2bfloat162_rn(v[u].x, v[u].y);
                }
            }
        }
    });
}

static int launch_thin(const b2kv_linear_args& a, void* stream) {
    const b2kv_segment& sg = a.seg[0];
    if (a.dtype != B2KV_DTYPE_BF16 || a.K > kThinK || a.N % 2 || a.groups > 1 || a.group_rows || a.n_seg > 1 || is_pair(sg.kind))
        return B2KV_ERR_UNSUPPORTED;
    if (!aligned16(a.w) || !aligned16(sg.out) || a.ld_w % 2 || sg.ld % 2 || (a.residual && (!aligned16(a.residual) || a.ld_residual % 2)))
        return B2KV_ERR_UNSUPPORTED;
    // few rows: enough CTAs to be quick; many: the columns of w are loaded once per tile of rows, unless that leaves less than six CTAs
    // per SM (3548 rows x 1024 columns, then a row after the other: 29 us in tiles of 64, 18 in tiles of 16)
    int row_tile = a.rows > 1024 ? kThinRows : 8;
    const long long cols = (a.N / 2 + kThinThreads - 1) / kThinThreads;
    while (row_tile > 8 && cols * ((a.rows + row_tile - 1) / row_tile) < 6LL * device_sm_count()) row_tile /= 2;
    const auto kernel = a.K <= 16 ? linear_thin_kernel<16> : linear_thin_kernel<32>;
    static int per_sm[2][64] = {};
    int dev = 0;
    B2KV_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return B2KV_ERR_UNSUPPORTED;
    int& resident = per_sm[a.K <= 16][dev];
    if (resident == 0) B2KV_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, kThinThreads, 0));
    // a few CTAs more than fit the device would run behind all others (1056 rows, 16 -> 2048: 1056 of 8 rows, of which 1036 fit, 5.9 us, 5.3 with 9)
    const long long fit = static_cast<long long>(resident) * device_sm_count(), ctas = cols * ((a.rows + row_tile - 1) / row_tile);
    if (fit >= cols && ctas > fit && 4 * ctas <= 5 * fit)
        row_tile = static_cast<int>(std::min<long long>(kThinRows, std::max<long long>(row_tile, (a.rows + fit / cols - 1) / (fit / cols))));
    const dim3 grid(static_cast<unsigned>(cols), (a.rows + row_tile - 1) / row_tile);
    if (grid.y > 65535u) return B2KV_ERR_UNSUPPORTED;
    OverlapLaunch launch(grid, kThinThreads, 0, stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, kernel, a, row_tile));
    return B2KV_OK;
}

// A per-head product of many rows: the weight-streaming kernel on 128 rows at a time (the heads' matrices are small and
// stay in L2).
static int rows_in_slices(const b2kv_linear_args& all, int32_t* dev_status, void* stream) {
    const int es = elt_bytes(all.dtype);
    for (int r0 = 0; r0 < all.rows; r0 += 128) {
        b2kv_linear_args a = all;
        a.rows = all.rows - r0 < 128 ? all.rows - r0 : 128;
        a.x = static_cast<const char*>(all.x) + r0 * all.ld_x * es;
        if (all.residual) a.residual = all.residual + r0 * all.ld_residual;
        for (int s = 0; s < a.n_seg; ++s)
            a.seg[s].out = static_cast<char*>(all.seg[s].out) + r0 * all.seg[s].ld * (is_f32(all.seg[s].kind) ? 4 : es);
        const int rc = linear_rows_tc(a, dev_status, stream);
        if (rc != B2KV_OK) return rc;
    }
    return B2KV_OK;
}

}  // namespace lin
}  // namespace b2kv

using namespace b2kv;

extern "C" int b2kv_linear(const b2kv_linear_args* args, int32_t* dev_status, void* stream) {
    return b2kv_linear_opt(args, nullptr, dev_status, stream);
}

// More than 16 rows of fp32: the tensor cores, unless there are too few input features to be worth the parts.
static bool f32_on_tensor_cores(const b2kv_linear_args& a) { return a.path == 0 && a.dtype == B2KV_DTYPE_F32 && a.rows > 16 && a.K >= 128; }

extern "C" int b2kv_linear_opt(const b2kv_linear_args* args, const b2kv_linear_options* options, int32_t* dev_status, void* stream) {
    return b2kv_linear_ws(args, options, nullptr, 0, dev_status, stream);
}

extern "C" size_t b2kv_linear_workspace_bytes(const b2kv_linear_args* args) {
    return args != nullptr && args->rows > 0 && args->N > 0 && f32_on_tensor_cores(*args) ? linear_f32_tc_workspace(*args) : 0;
}

extern "C" int b2kv_linear_ws(const b2kv_linear_args* args, const b2kv_linear_options* options, void* workspace,
                              size_t workspace_bytes, int32_t* dev_status, void* stream) {
    if (args == nullptr) return B2KV_ERR_BAD_ARG;
    const b2kv_linear_args& a = *args;
    const b2kv_linear_options o = options != nullptr ? *options : b2kv_linear_options{};
    if (o.flags & ~B2KV_LINEAR_AHEAD) return B2KV_ERR_BAD_ARG;
    if (elt_bytes(a.dtype) == 0) return B2KV_ERR_UNSUPPORTED;
    if (!a.x || !a.w || a.rows <= 0 || a.K <= 0 || a.N <= 0 || a.groups <= 0 || a.path < 0 || a.path > 4) return B2KV_ERR_BAD_ARG;
    if (a.n_seg < 1 || a.n_seg > B2KV_MAX_SEGMENTS || a.seg[a.n_seg - 1].end != a.N) return B2KV_ERR_BAD_ARG;
    if (a.bias && a.groups > 1) return B2KV_ERR_BAD_ARG;
    if (a.group_rows && (a.max_group_rows <= 0 || a.max_group_rows > a.rows)) return B2KV_ERR_BAD_ARG;
    if (o.group_x_rows && (!a.group_rows || o.x_rows <= 0)) return B2KV_ERR_BAD_ARG;
    int first = 0;
    for (int s = 0; s < a.n_seg; ++s) {
        const b2kv_segment& sg = a.seg[s];
        if (!sg.out || (sg.kind >= B2KV_SEG_SOFTCAP && !(a.limit > 0.f)) || sg.end <= first || sg.kind < B2KV_SEG_STORE || sg.kind > B2KV_SEG_DECAY) return B2KV_ERR_BAD_ARG;
        // pairs of columns never straddle a boundary (the last segment may end on an odd column if it has no pairs)
        if ((sg.end & 1) && (s + 1 < a.n_seg || lin::is_pair(sg.kind))) return B2KV_ERR_BAD_ARG;
        first = sg.end;
    }
    if (o.group_x_rows) return a.path == 0 || a.path == 3 ? linear_tiled_tc(a, o, dev_status, stream) : B2KV_ERR_UNSUPPORTED;
    if (a.path == 2) return linear_rows_tc(a, dev_status, stream);
    if (a.path == 3) return linear_tiled_tc(a, o, dev_status, stream);
    if (a.path == 4) return lin::launch_thin(a, stream);
    if (a.path == 0 && a.dtype == B2KV_DTYPE_BF16) {
        int rc = lin::launch_thin(a, stream);
        if (rc != B2KV_ERR_UNSUPPORTED) return rc;
        if ((a.group_rows ? a.max_group_rows : a.rows) <= 128) {
            rc = linear_rows_tc(a, dev_status, stream);
        } else if (a.groups > 1 && a.group_rows == nullptr) {
            rc = lin::rows_in_slices(a, dev_status, stream);
        } else {
            rc = linear_tiled_tc(a, o, dev_status, stream);
        }
        if (rc != B2KV_ERR_UNSUPPORTED) return rc;
    }
    if (a.path == 0 && a.dtype == B2KV_DTYPE_F32) {
        int rc = f32_on_tensor_cores(a) ? linear_f32_tc(a, workspace, workspace_bytes, dev_status, stream) : B2KV_ERR_UNSUPPORTED;
        if (rc == B2KV_ERR_UNSUPPORTED) rc = linear_f32(a, stream);
        if (rc != B2KV_ERR_UNSUPPORTED) return rc;
    }
    return lin::launch_simt(a, stream);
}
