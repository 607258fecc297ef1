// b2kv_linear in fp32 for many rows on the tensor cores: every operand is split into three bf16 parts, x = h + m + l, which hold all
// 24 bits, and a product is h h' + (h m' + m h') + (m m' + h l' + l h'); what is dropped is below 2^-24 of it.
//
// The tensor core adds in fp32 but truncates, so a long chain of accumulations would lean towards zero by more than fp32 sums err.
// Therefore the leading products h h' are accumulated over the 64 input features of a step only; the partial sums are taken out of tensor memory
// and added up in registers, rounded to nearest.  The other five products, 2^-8 of the first and less, stay in an accumulator of
// their own until the end.  Measured against 64 bits, 2-norm of the error over that of the result: 8e-8 at 128 input features, 9e-8 at
// 768, 1.1e-7 at 3072, where sums of fp32 multiply-adds in order are off by 2.0e-7, 5.0e-7 and 9.9e-7.  693 rows, 768 -> 3072: 31 us
// against 127 of linear_f32_tile_kernel; 3072 -> 768: 39 and 130; 60 rows, 768 -> 3072: 15 and 25.
//
//   * a CTA has 128 x 128 outputs; steps of 64 input features through two stages of 96 KB;
//   * more than 256 rows, enough tiles and scratch (the rule and its times at parts_bytes): the parts are made by a kernel ahead, once for all
//     tiles (b2kv_linear_ws), and warp 8 copies them with TMA, warp 9 issues the products.  In the same kernel every row of tiles makes the parts of w and every column of tiles those of x
//     again, which takes longer than the products (693 rows, 3072 -> 768: 36.8 us, 32.5 with the kernel ahead; 3000 rows, 1024 -> 4096: 205 and 157);
//   * otherwise warps 8-15 read fp32 rows of x and w, a step ahead in registers, and write the parts as the operands the MMAs want: x K-major,
//     w as it lies (MN-major), 128-byte swizzle; a thread of warp 0 issues the products;
//   * 24 tcgen05.mma per step: 6 x 64 clocks per 16 input features, a sixth of the tensor peak, which is
//     four times what the CUDA cores have.  Issuing takes as long as the products do, so it is not for the warps that make the parts
//     (48 us with one of them), and a seventeenth warp would leave all others 96 registers (41 us, and spills);
//   * warps 0-7 take the leading sums out (two accumulators in turn), thread = row and half of the columns, warp 0 always one step
//     behind what it has issued;
//   * a product whose tiles leave SMs idle has its input features cut into ranges, one per CTA of a cluster, whose sums meet in
//     distributed shared memory, in order.
//
// What the parts cannot carry is computed again with plain multiply-adds, in order, element by element: sums that are not finite (an
// operand is not, or rounds to none in bf16, or finite operands' products overflow, where the sign of a partial product says nothing),
// and rows of x and columns of w with a number whose three parts do not add up to it (some below 2^-109, where the last part
// is below the smallest number of bf16).  The bits of every other row and column are what they are without it.  One such row among 693,
// 3072 -> 768: 137 us instead of 39; with a whole tile again, one chain of global loads per thread, it took 9.3 ms.
// Every wait is bounded; after one ran out nothing is stored and the status word is set.
#include <algorithm>

#include "linear.cuh"
#include "tc_ptx.cuh"
#include "tma_map.cuh"

namespace b2kv {
namespace linf32tc {

using namespace tc;

constexpr int kBM = 128, kBN = 128, kBK = 64, kStages = 2;
constexpr int kPartBytes = 128 * kBK * 2;           // one part of x or of w: 16 KB
constexpr int kStageBytes = 6 * kPartBytes;         // x: h, m, l; w: h, m, l
constexpr int kSumWarps = 8, kSplitWarps = 8;
constexpr int kThreads = 32 * (kSumWarps + kSplitWarps);  // 128 registers each
constexpr int kLdT = kBN + 4;                       // words per row of the tile of sums (over the stages, once they are free)
constexpr int kMinTileSteps = 900;                  // tiles x steps from which a kernel ahead makes the parts
constexpr size_t kMaxScratch = size_t{512} << 20;   // bytes of parts at most
constexpr int kMaxSplits = 8;                       // ranges of input features
constexpr int kTmemCols = 512;                      // leading sums 2 x 128, the others 128
constexpr int kColRest = 2 * kBN;
constexpr size_t kSmem = kStages * kStageBytes + 1024;
static_assert(kBM * kLdT * 4 <= kStages * kStageBytes, "the tile of sums fits the stages");

// The parts of x and w in scratch memory, [3][rows][ldx] and [3][K][ldw] bf16, and per 128 x 64 piece of x and 64 x 128 piece of w whether it has
// a number that three parts do not add up to.
struct Parts {
    uint16_t *x, *w;
    int32_t *odd_x, *odd_w;  // [tiles_m][steps], [tiles_n][steps]
    int ldx, ldw;
};
constexpr int pad8(int n) { return (n + 7) / 8 * 8; }

struct Shared {
    alignas(8) uint64_t full[kStages], empty[kStages], sum_full[2], sum_empty[2], done;
    uint32_t tmem_base;
    volatile int odd, abort_flag;
    uint32_t odd_rows[kBM / 32], odd_cols[kBN / 32];
};

// The three parts of four numbers, to `at` and one and two parts further on.  What two parts leave of a number is the third if its
// lower 16 bits are zero; they are collected in `check` (those of what is not finite are set: infinity less infinity).
template <typename Step = int>
__device__ __forceinline__ void split3(const float4& v, uint8_t* at, uint32_t& check, Step part_bytes = kPartBytes) {
    const float2 minus = make_float2(-1.f, -1.f);
    float2 r0 = make_float2(v.x, v.y), r1 = make_float2(v.z, v.w);
#pragma unroll
    for (int part = 0; part < 3; ++part) {
        const uint32_t a = pack_bf16(r0.x, r0.y), b = pack_bf16(r1.x, r1.y);
        *reinterpret_cast<uint2*>(at + part * part_bytes) = make_uint2(a, b);
        if (part == 2) break;
        r0 = __ffma2_rn(make_float2(__uint_as_float(a << 16), __uint_as_float(a & 0xffff0000u)), minus, r0);
        r1 = __ffma2_rn(make_float2(__uint_as_float(b << 16), __uint_as_float(b & 0xffff0000u)), minus, r1);
    }
    check |= (__float_as_uint(r0.x) | __float_as_uint(r0.y)) | (__float_as_uint(r1.x) | __float_as_uint(r1.y));
}
__device__ __forceinline__ bool has_no_parts(float v) {
    const float r = v - __bfloat162float(__float2bfloat16_rn(v));
    return (__float_as_uint(r - __bfloat162float(__float2bfloat16_rn(r))) & 0xffffu) != 0 || !(fabsf(v) < INFINITY);
}

// One CTA per piece of x (the first tiles_m * steps CTAs) or of w.
constexpr int kMakeThreads = 256;
__global__ void __launch_bounds__(kMakeThreads) make_parts_kernel(const __grid_constant__ b2kv_linear_args a, const __grid_constant__ Parts p, int pieces_x) {
    grid_launch_dependents();
    grid_dependency_wait();
    const int steps = (a.K + kBK - 1) / kBK;
    const bool of_x = static_cast<int>(blockIdx.x) < pieces_x;
    const int piece = of_x ? blockIdx.x : blockIdx.x - pieces_x, step = piece % steps, tile = piece / steps;
    const float* const src = static_cast<const float*>(of_x ? a.x : a.w);
    const int64_t ld = of_x ? a.ld_x : a.ld_w;
    const int row0 = of_x ? tile * kBM : step * kBK, col0 = of_x ? step * kBK : tile * kBN;
    const int n_rows = of_x ? min(kBM, a.rows - row0) : min(kBK, a.K - row0), n_cols = of_x ? min(kBK, a.K - col0) : min(kBN, a.N - col0);
    uint16_t* const out = of_x ? p.x : p.w;
    const int out_ld = of_x ? p.ldx : p.ldw, shift = of_x ? 4 : 5;  // 16-byte pieces per row of the piece: 64 / 4, 128 / 4
    const int64_t part_bytes = static_cast<int64_t>(of_x ? a.rows : a.K) * out_ld * 2;
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int e = i * kMakeThreads + threadIdx.x, r = e >> shift, c = (e & ((1 << shift) - 1)) * 4;
        v[i] = r < n_rows && c < n_cols ? *reinterpret_cast<const float4*>(src + (row0 + r) * ld + col0 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    uint32_t check = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int e = i * kMakeThreads + threadIdx.x, r = e >> shift, c = (e & ((1 << shift) - 1)) * 4;
        if (r < n_rows && c < n_cols)
            split3(v[i], reinterpret_cast<uint8_t*>(out + static_cast<int64_t>(row0 + r) * out_ld + col0 + c), check, part_bytes);
    }
    const int odd = __syncthreads_or((check & 0xffffu) != 0);
    if (threadIdx.x == 0) (of_x ? p.odd_x : p.odd_w)[piece] = odd;
}

// The sums of the input features [k_first, k_end) that need it, again: all threads, the tile of sums and the stages behind it.
__device__ __noinline__ void sums_again(const b2kv_linear_args& a, Shared& sm, float* tile, const float* x, const float* w, int row0, int col0,
                                        int k_first, int k_end) {
    constexpr int kLdX = kBK + 4;
    float* const xs = tile + kBM * kLdT;    // [row][input feature]
    float* const ws = xs + kBM * kLdX;      // [input feature][column]
    static_assert((kBM * kLdT + kBM * kLdX + kBK * kBN) * 4 <= kStages * kStageBytes, "both operands of a step fit behind the tile");
    const int tid = threadIdx.x, n_rows = min(kBM, a.rows - row0), n_cols = min(kBN, a.N - col0);
    if (tid < kBM / 32) sm.odd_rows[tid] = 0;
    if (tid < kBN / 32) sm.odd_cols[tid] = 0;
    // element i of a thread: a row of the tile per four i, so that a row is one element of 128 threads, and so is a column
    auto row_of = [&](int i) { return (tid >> 7) + 4 * i; };
    auto col_of = [&](int i) { return (tid + 37 * i) & (kBN - 1); };
    uint32_t again = 0;
    for (int pass = 0; pass < 2; ++pass) {
        for (int k0 = k_first; k0 < k_end; k0 += kBK) {
            const int kn = min(kBK, k_end - k0);
            __syncthreads();
            for (int i = tid; i < kBM * (kBK / 4); i += kThreads) {
                const int r = i / (kBK / 4), k = i % (kBK / 4) * 4;
                const float4 v = r < n_rows && k < kn ? *reinterpret_cast<const float4*>(x + static_cast<int64_t>(row0 + r) * a.ld_x + k0 + k)
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
                *reinterpret_cast<float4*>(xs + r * kLdX + k) = v;
                if (pass == 0 && (has_no_parts(v.x) || has_no_parts(v.y) || has_no_parts(v.z) || has_no_parts(v.w)))
                    atomicOr(&sm.odd_rows[r >> 5], 1u << (r & 31));
            }
            for (int i = tid; i < kBK * (kBN / 4); i += kThreads) {
                const int k = i / (kBN / 4), c = i % (kBN / 4) * 4;
                const float4 v = k < kn && c < n_cols ? *reinterpret_cast<const float4*>(w + static_cast<int64_t>(k0 + k) * a.ld_w + col0 + c)
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
                *reinterpret_cast<float4*>(ws + k * kBN + c) = v;
                if (pass == 0) {
                    const uint32_t odd = (has_no_parts(v.x) ? 1u : 0u) | (has_no_parts(v.y) ? 2u : 0u) | (has_no_parts(v.z) ? 4u : 0u) |
                                         (has_no_parts(v.w) ? 8u : 0u);
                    if (odd != 0) atomicOr(&sm.odd_cols[c >> 5], odd << (c & 31));
                }
            }
            __syncthreads();
            for (uint32_t left = again; left != 0; left &= left - 1) {
                const int i = __ffs(left) - 1, r = row_of(i), c = col_of(i);
                float sum = tile[r * kLdT + c];
#pragma unroll 8
                for (int k = 0; k < kn; ++k) sum = fmaf(xs[r * kLdX + k], ws[k * kBN + c], sum);
                tile[r * kLdT + c] = sum;
            }
        }
        __syncthreads();
        if (pass == 1) break;
        for (int i = 0; i < kBM * kBN / kThreads; ++i) {
            const int r = row_of(i), c = col_of(i);
            float& sum = tile[r * kLdT + c];
            if (r < n_rows && c < n_cols && ((sm.odd_rows[r >> 5] >> (r & 31) & 1) || (sm.odd_cols[c >> 5] >> (c & 31) & 1) || !(fabsf(sum) < INFINITY)))
                again |= 1u << i, sum = 0.f;
        }
    }
}

// One sum over all input features, in order: where the ranges' sums are infinities that are no number together.
__device__ __noinline__ float sum_in_order(const float* row, const float* col, int K, int64_t ld_w) {
    float sum = 0.f;
#pragma unroll 8
    for (int k = 0; k < K; ++k) sum = fmaf(row[k], col[static_cast<int64_t>(k) * ld_w], sum);
    return sum;
}

// After a wait that ran out: the last of `n` uses of the stages, copies (bars: full) or products (empty), end before their memory is given up.
__device__ __noinline__ void settle(uint64_t* bars, int n) {
    for (int i = max(0, n - kStages); i < n; ++i) mbar_wait(&bars[i % kStages], (i / kStages) & 1);
}

// kMade: the parts are in scratch memory.
template <bool kMade>
__global__ void __launch_bounds__(kThreads, 1)
linear_f32_tc_kernel(const __grid_constant__ b2kv_linear_args a, const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                     const __grid_constant__ Parts p, int splits, bool expire, int32_t* dev_status) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ Shared sm;
    uint8_t* const ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = blockIdx.z;
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&sm.full[s], kMade ? 1 : kSplitWarps);
            mbar_init(&sm.empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&sm.sum_full[s], 1);
            mbar_init(&sm.sum_empty[s], kSumWarps);
        }
        mbar_init(&sm.done, 1);
        sm.odd = sm.abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 0) {
        tmem_alloc(&sm.tmem_base, kTmemCols);
        tmem_relinquish();
    }
    grid_dependency_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sm.tmem_base;

    const float* const x = static_cast<const float*>(a.x) + static_cast<int64_t>(g) * a.group_x;
    const float* const w = static_cast<const float*>(a.w) + static_cast<int64_t>(g) * a.group_w;
    const int split = splits > 1 ? static_cast<int>(cluster_rank()) : 0;
    const int row0 = blockIdx.y * kBM, col0 = static_cast<int>(blockIdx.x) / splits * kBN;
    const int all_steps = (a.K + kBK - 1) / kBK;
    const int step0 = static_cast<int>(static_cast<long long>(all_steps) * split / splits);
    const int steps = static_cast<int>(static_cast<long long>(all_steps) * (split + 1) / splits) - step0;
    const int k_first = step0 * kBK, k_end = min(a.K, (step0 + steps) * kBK);

    // the products of step s, once all parts are there and the sums of the step before last are taken out
    auto issue = [&](int s) {
        constexpr uint32_t idesc = instr_desc(0, 1, kBN);
        constexpr uint64_t kPart = kPartBytes >> 4;
        const int st = s % kStages;
        if (!mbar_wait(&sm.full[st], (s / kStages) & 1) || !mbar_wait(&sm.sum_empty[s & 1], ((s >> 1) & 1) ^ 1)) return false;
        tc_fence_after();
        const uint64_t dx = smem_desc(smem_u32(ring + st * kStageBytes), 16, 1024);
        const uint64_t dw = smem_desc(smem_u32(ring + st * kStageBytes + 3 * kPartBytes), kBK * 128, 1024);
#pragma unroll
        for (int kk = 0; kk < kBK / 16; ++kk)  // 16 input features: 32 bytes of x's rows, 16 rows of w
            mma_ss(tmem + (s & 1) * kBN, dx + 2 * kk, dw + 128 * kk, idesc, kk ? 1u : 0u);
        mma_commit(&sm.sum_full[s & 1]);
#pragma unroll
        for (int kk = 0; kk < kBK / 16; ++kk) {
            const uint64_t ax = dx + 2 * kk, bw = dw + 128 * kk;
            mma_ss(tmem + kColRest, ax, bw + 2 * kPart, idesc, (s | kk) ? 1u : 0u);
            mma_ss(tmem + kColRest, ax + 2 * kPart, bw, idesc, 1u);
            mma_ss(tmem + kColRest, ax + kPart, bw + kPart, idesc, 1u);
            mma_ss(tmem + kColRest, ax, bw + kPart, idesc, 1u);
            mma_ss(tmem + kColRest, ax + kPart, bw, idesc, 1u);
        }
        mma_commit(&sm.empty[st]);
        if (s + 1 == steps) mma_commit(&sm.done);
        return true;
    };
    float acc[64];
    if (warp < kSumWarps) {
        // ------------------------------ sums: thread = row, half of the columns ------------------------------
        const uint32_t t_lane = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + (warp >> 2) * 64;
#pragma unroll
        for (int j = 0; j < 64; ++j) acc[j] = 0.f;
        auto add = [&](uint32_t at) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t r[32];
                tmem_ld32(at + half * 32, r);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 32; ++j) acc[half * 32 + j] += __uint_as_float(r[j]);
            }
        };
        auto issue_by_warp0 = [&](int s) {
            if (kMade || warp != 0 || s >= steps) return true;
            bool good = true;
            if (lane == 0) good = issue(s);
            return __all_sync(0xffffffffu, good) != 0;
        };
        bool ok = !expire && issue_by_warp0(0);  // (test hook: as if the first wait had run out)
        for (int s = 0; s < steps && ok; ++s) {
            ok = issue_by_warp0(s + 1);
            if (!ok) break;
            ok = __all_sync(0xffffffffu, mbar_wait(&sm.sum_full[s & 1], (s >> 1) & 1));
            if (!ok) break;
            tc_fence_after();
            add(t_lane + (s & 1) * kBN);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.sum_empty[s & 1]);
        }
        if (ok && steps > 0) {
            ok = __all_sync(0xffffffffu, mbar_wait(&sm.done, 0));
            tc_fence_after();
            if (ok) add(t_lane + kColRest);
        }
        if (!ok) sm.abort_flag = 1;
    } else if (kMade) {
        bool ok = true;
        if (warp == kSumWarps) {
            // ------------------------------ copies of the parts ------------------------------
            if (lane == 0) {
                int s = 0;
                for (; s < steps; ++s) {
                    const int st = s % kStages, k = k_first + s * kBK;
                    ok = mbar_wait(&sm.empty[st], ((s / kStages) & 1) ^ 1);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&sm.full[st], kStageBytes);
                    uint8_t* const to = ring + st * kStageBytes;
#pragma unroll
                    for (int part = 0; part < 3; ++part) {
                        tma_load_3d(to + part * kPartBytes, &tm_x, &sm.full[st], k, row0, part);
                        tma_load_3d(to + (3 + part) * kPartBytes, &tm_w, &sm.full[st], col0, k, part);
                        tma_load_3d(to + (3 + part) * kPartBytes + kBK * 128, &tm_w, &sm.full[st], col0 + 64, k, part);
                    }
                }
                if (!ok) settle(sm.full, s);
            }
            __syncwarp();
        } else if (warp == kSumWarps + 1) {
            if (lane == 0) {
                int s = 0;
                while (s < steps && issue(s)) ++s;
                ok = s == steps;
                if (!ok) settle(sm.empty, s);
            }
            __syncwarp();
        } else if (warp == kSumWarps + 2) {
            for (int s = lane; s < steps; s += 32)
                if (p.odd_x[blockIdx.y * all_steps + step0 + s] | p.odd_w[col0 / kBN * all_steps + step0 + s]) sm.odd = 1;
        }
        if (!ok) sm.abort_flag = 1;
    } else {
        // ------------------------------ parts of x and w ------------------------------
        const int ct = tid - 32 * kSumWarps;
        const int xc = (ct & 15) * 4, xr = ct >> 4;  // x: four input features of the rows xr, + 16, ..
        const int wc = (ct & 31) * 4, wk = ct >> 5;  // w: four columns of the input features wk, + 8, ..
        float4 xv[8], wv[8];
        // (whole tiles without a condition per piece: instructions are what the parts cost, 38 us for the first size above with one)
        const bool rows_in = row0 + kBM <= a.rows, cols_in = col0 + kBN <= a.N;

        auto read_x = [&](int k0) {
            if (rows_in && k0 + kBK <= k_end) {
                const float* p = x + static_cast<int64_t>(row0 + xr) * a.ld_x + xc + k0;
#pragma unroll
                for (int i = 0; i < 8; ++i, p += 16 * a.ld_x) xv[i] = *reinterpret_cast<const float4*>(p);
                return;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = row0 + xr + 16 * i;
                xv[i] = r < a.rows && k0 + xc < k_end ? *reinterpret_cast<const float4*>(x + static_cast<int64_t>(r) * a.ld_x + k0 + xc)
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        auto read_w = [&](int k0) {
            if (cols_in && k0 + kBK <= k_end) {
                const float* p = w + static_cast<int64_t>(k0 + wk) * a.ld_w + col0 + wc;
#pragma unroll
                for (int i = 0; i < 8; ++i, p += 8 * a.ld_w) wv[i] = *reinterpret_cast<const float4*>(p);
                return;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int k = k0 + wk + 8 * i;
                wv[i] = k < k_end && col0 + wc < a.N ? *reinterpret_cast<const float4*>(w + static_cast<int64_t>(k) * a.ld_w + col0 + wc)
                                                     : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        uint32_t check = 0;
        if (steps > 0) read_x(k_first), read_w(k_first);
        bool ok = true;
        for (int s = 0; s < steps; ++s) {
            const int st = s % kStages, next = k_first + (s + 1) * kBK;
            ok = __all_sync(0xffffffffu, mbar_wait(&sm.empty[st], ((s / kStages) & 1) ^ 1));
            if (!ok) break;
            uint8_t* const px = ring + st * kStageBytes;
            uint8_t* const pw = px + 3 * kPartBytes + (wc >> 6) * (kBK * 128);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = xr + 16 * i;
                split3(xv[i], px + r * 128 + (((xc >> 3) ^ (r & 7)) << 4) + (xc & 7) * 2, check);
            }
            if (s + 1 < steps) read_x(next);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int k = wk + 8 * i;
                split3(wv[i], pw + k * 128 + ((((wc & 63) >> 3) ^ (k & 7)) << 4) + (wc & 7) * 2, check);
            }
            if (s + 1 < steps) read_w(next);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.full[st]);
        }
        if (check & 0xffffu) sm.odd = 1;
        if (!ok) sm.abort_flag = 1;
    }
    grid_launch_dependents();
    tc_fence_before();
    __syncthreads();  // all MMAs have completed (the sums' warps have seen it): the stages are free
    float* const tile = reinterpret_cast<float*>(ring);
    if (warp < kSumWarps) {
        const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 64;
        float* const mine = tile + r * kLdT + c0;
#pragma unroll
        for (int j = 0; j < 64; j += 4) *reinterpret_cast<float4*>(mine + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
        float check[4] = {};  // become NaN
#pragma unroll
        for (int j = 0; j < 64; ++j) check[j & 3] = fmaf(acc[j], 0.f, check[j & 3]);
        if ((check[0] + check[1]) + (check[2] + check[3]) != 0.f) sm.odd = 1;
    }
    __syncthreads();
    if (sm.odd) sums_again(a, sm, tile, x, w, row0, col0, k_first, k_end);
    if (splits > 1) cluster_sync();
    const int c = (tid & 63) * 2, share = (kBM + splits - 1) / splits;
    bool complete = true;
    for (int s = 0; s < splits; ++s) complete = complete && peer_load1(peer_address(smem_u32(const_cast<int*>(&sm.abort_flag)), s)) == 0;
    if (complete && col0 + c < a.N)
        lin::finish_rows<float>(a, g, col0 + c, row0, split * share + (tid >> 6), min(min((split + 1) * share, kBM), a.rows - row0), kThreads / 64,
                                [&](int r) {
                                    float2 v = make_float2(0.f, 0.f);
                                    bool nan_x = false, nan_y = false;
                                    for (int s = 0; s < splits; ++s) {
                                        const float2 p = peer_load2(peer_address(smem_u32(tile + r * kLdT + c), s));
                                        v.x += p.x, v.y += p.y;
                                        nan_x = nan_x || p.x != p.x, nan_y = nan_y || p.y != p.y;
                                    }
                                    const float* const row = x + static_cast<int64_t>(row0 + r) * a.ld_x;
                                    if (v.x != v.x && !nan_x) v.x = sum_in_order(row, w + col0 + c, a.K, a.ld_w);
                                    if (v.y != v.y && !nan_y) v.y = sum_in_order(row, w + col0 + c + 1, a.K, a.ld_w);
                                    return v;
                                });
    __syncwarp();
    if (splits > 1) cluster_sync();  // the peers have read this CTA's part
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
    if (tid == 0 && sm.abort_flag) report_status(dev_status, B2KV_DEV_WAIT_TIMEOUT);
}

}  // namespace linf32tc

// Scratch of the parts: none where they are made in the products' kernel.
static size_t parts_bytes(const b2kv_linear_args& a, linf32tc::Parts* p, void* at) {
    using namespace linf32tc;
    // The tiles make more of the same parts the more of them there are (us in the products' kernel, and ahead): 36 tiles of 12 steps 16.2, 18.6;
    // 60 of 12 19.9, 21.3; 78 of 12 29.5, 26.0; 144 of 12 30.4, 27.6; 36 of 48 36.8, 32.5; 768 of 16 205, 157.  What the kernel ahead costs
    // is w's bytes, as parts written and read back, and what it saves is one lot of w's parts per row of tiles; by rows of tiles and MB of w's parts:
    // 2 rows, 25 MB 24.6, 25.4; 100 62, 72; 3 rows, 19 MB 30.4, 27.6; 25 37.7, 32.0; 57 49.1, 50.8; 100 106, 107; 4 rows, 57 MB 126, 116;
    // 100 151, 119; 144 203, 221; 5 rows, 100 MB 241, 175; 144 277, 273; 6 rows, 144 MB 331, 314; 384 782, 816; 24 rows, 25 MB 214, 164; 100 747, 619.
    const long long tiles_rows = (a.rows + kBM - 1) / kBM, tiles = tiles_rows * ((a.N + kBN - 1) / kBN);
    if (tiles_rows < 3 || a.groups > 1 || tiles * ((a.K + kBK - 1) / kBK) < kMinTileSteps) return 0;
    const size_t parts_w = 6 * static_cast<size_t>(a.K) * a.N;
    if (parts_w > (tiles_rows == 3 ? size_t{32} << 20 : tiles_rows == 4 ? size_t{112} << 20 : size_t{160} << 20)) return 0;
    const size_t steps = (a.K + kBK - 1) / kBK, tiles_m = (a.rows + kBM - 1) / kBM, tiles_n = (a.N + kBN - 1) / kBN;
    const size_t ldx = pad8(a.K), ldw = pad8(a.N), x = 3 * static_cast<size_t>(a.rows) * ldx, w = 3 * static_cast<size_t>(a.K) * ldw;
    if (p != nullptr) {
        p->x = static_cast<uint16_t*>(at), p->w = p->x + x;
        p->odd_x = reinterpret_cast<int32_t*>(p->w + w), p->odd_w = p->odd_x + tiles_m * steps;
        p->ldx = static_cast<int>(ldx), p->ldw = static_cast<int>(ldw);
    }
    const size_t bytes = (x + w) * 2 + (tiles_m + tiles_n) * steps * sizeof(int32_t);
    return bytes <= kMaxScratch ? bytes : 0;
}

// Three matrices of rows x cols bf16, boxes of box_rows x 64 of one of them, 128-byte swizzle; zero outside.
static bool make_parts_map(CUtensorMap* map, const uint16_t* base, int rows, int cols, int ld, int box_rows) {
    EncodeTiledFn fn = tensor_map_encoder();
    if (fn == nullptr) return false;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows), 3};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld) * 2, static_cast<cuuint64_t>(ld) * 2 * static_cast<cuuint64_t>(rows)};
    const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_rows), 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<uint16_t*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static bool f32_tc_takes(const b2kv_linear_args& a) {
    return a.dtype == B2KV_DTYPE_F32 && a.group_rows == nullptr && aligned16(a.x) && aligned16(a.w) && a.K % 4 == 0 && a.N % 4 == 0 && a.ld_x % 4 == 0 &&
           a.ld_w % 4 == 0 && a.group_x % 4 == 0 && a.group_w % 4 == 0;
}

size_t linear_f32_tc_workspace(const b2kv_linear_args& a) { return f32_tc_takes(a) ? parts_bytes(a, nullptr, nullptr) : 0; }

int linear_f32_tc(const b2kv_linear_args& a, void* workspace, size_t workspace_bytes, int32_t* dev_status, void* stream) {
    using namespace linf32tc;
    if (!f32_tc_takes(a)) return B2KV_ERR_UNSUPPORTED;
    const long long tiles_m = (a.rows + kBM - 1) / kBM, tiles_n = (a.N + kBN - 1) / kBN, tiles = tiles_m * tiles_n * a.groups;
    const int steps = (a.K + kBK - 1) / kBK;
    static bool configured[64] = {false};
    static int clusters[64][kMaxSplits + 1] = {{0}};  // that can be resident together, by size
    int dev = 0;
    B2KV_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return B2KV_ERR_UNSUPPORTED;
    if (!configured[dev]) {
        B2KV_CUDA_TRY(cudaFuncSetAttribute(linear_f32_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem)));
        B2KV_CUDA_TRY(cudaFuncSetAttribute(linear_f32_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem)));
        clusters[dev][1] = device_sm_count();
        for (int s = 2; s <= kMaxSplits; ++s) {
            OverlapLaunch most(static_cast<unsigned>(s * device_sm_count()), kThreads, kSmem, stream, s);
            most.cfg.numAttrs = 1;  // the cluster
            if (cudaOccupancyMaxActiveClusters(&clusters[dev][s], linear_f32_tc_kernel<false>, &most.cfg) != cudaSuccess) {
                (void)cudaGetLastError();
                clusters[dev][s] = 0;
            }
        }
        configured[dev] = true;
    }
    // Ranges of input features: the steps of the fullest places, where a CTA costs about four steps beside its own and the meeting of
    // a cluster two more.  (Clusters of four do not reach every SM: 36 of them are two waves.)
    int splits = 1;
    double best = 1e30;
    for (int s = 1; s <= kMaxSplits && (s == 1 || steps >= 2 * s); ++s) {
        if (clusters[dev][s] <= 0) continue;
        const double cost = static_cast<double>((tiles + clusters[dev][s] - 1) / clusters[dev][s]) * ((steps + s - 1) / s + 4 + (s > 1 ? 2 : 0));
        if (cost < best) best = cost, splits = s;
    }
    if (tune_get("matmul_splits") > 0) splits = std::min(tune_get("matmul_splits"), kMaxSplits);
    if (tiles_m > 65535 || a.groups > 65535 || tiles_n * splits > 0x7fffffffLL) return B2KV_ERR_UNSUPPORTED;
    OverlapLaunch launch(dim3(static_cast<unsigned>(tiles_n * splits), static_cast<unsigned>(tiles_m), a.groups), kThreads, kSmem, stream, splits);
    const bool expire = tune_get("linear_test_expire") != 0;
    Parts parts{};
    CUtensorMap tx{}, tw{};
    const size_t need = workspace != nullptr && aligned16(workspace) ? parts_bytes(a, &parts, workspace) : 0;
    if (need > 0 && workspace_bytes >= need && make_parts_map(&tx, parts.x, a.rows, a.K, parts.ldx, kBM) &&
        make_parts_map(&tw, parts.w, a.K, a.N, parts.ldw, kBK)) {
        const long long pieces_x = tiles_m * steps, pieces = pieces_x + tiles_n * steps;
        if (pieces > 0x7fffffffLL) return B2KV_ERR_UNSUPPORTED;
        OverlapLaunch make(static_cast<unsigned>(pieces), kMakeThreads, 0, stream);
        B2KV_CUDA_TRY(cudaLaunchKernelEx(&make.cfg, make_parts_kernel, a, parts, static_cast<int>(pieces_x)));
        B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, linear_f32_tc_kernel<true>, a, tx, tw, parts, splits, expire, dev_status));
        return B2KV_OK;
    }
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, linear_f32_tc_kernel<false>, a, tx, tw, parts, splits, expire, dev_status));
    return B2KV_OK;
}

}  // namespace b2kv
