// Causal flash-attention prefill for fp32 prompts on the Blackwell tensor cores: head_dim 128 or 64.
//
// fp32 is the reference's only storage type (simple-llm/src/gpu/gpu_buffer.py:31-39) and its kernel
// (simple-llm/src/gpu/gpu_kernels.py:499-770) is scalar fp32 arithmetic, which results here have to match
// to 1e-4.  The tensor cores have no fp32 inputs and tf32 (10 mantissa bits) cannot hold that bar, so every
// operand is split into two bfloat16 numbers, x = hi + lo with hi = bf16(x), lo = bf16(x - hi), which keeps 16
// mantissa bits, and every product is three MMAs into the same fp32 accumulator:
//
//     a * b  ~  a_hi * b_hi + a_hi * b_lo + a_lo * b_hi        (the dropped a_lo * b_lo is below 2^-16 relative)
//
//   * a first kernel writes the hi and lo halves of Q, K and V into a scratch buffer ([B*N, H*D] bfloat16 each) and, when the
//     prompt goes to a contiguous cache, the K / V rows to their places there: they pass through its registers anyway (B = 2,
//     N = 1000, H = 12, D = 64: three launches of it and the copy kernel behind the attention were 20 of 53 us);
//   * one CTA per (sequence, head, 128 query rows), at head_dim 64 in two forms: two CTAs per SM that fill each other's gaps, or one with
//     two score buffers and rings of two tiles, whose QK^T of the next step runs under the softmax of this one (the rule and both
//     times at prefill_tensor_core_f32).  What bounds the second is its products: 12 MMAs of QK^T and 24 of PV, 2900 clocks per step of
//     128 keys.  Warp 8 loads the Q tile and, step by step, a
//     128-key K tile and V tile (hi and lo: 64 KB each at head_dim 128, so the rings hold one step) with TMA tiled loads into
//     128-byte-swizzled shared memory; warp 9 issues S = Q K^T (3 x head_dim/16 tcgen05.mma, both operands in
//     shared memory) and O += P V (3 x 8, P read from tensor memory, V an MN-major shared-memory operand);
//   * warps 0 - 7: two threads per query row = TMEM lane, one for each half of a step's keys.  With one score buffer QK^T, softmax and PV
//     of the query tile follow one another, and only another CTA fills the gaps: with half a row per thread two CTAs fit the registers
//     (B = 8, N = 2048, H = 12, D = 64: 443 us with four warps and one CTA per SM, 250 so; N = 4096, H = 8, B = 4: 408 and 286;
//     one CTA per SM at D = 128, B = 2, N = 4096, H = 16: 506 and 454).  Scores in registers, the row's maximum exchanged through shared memory, running maximum
//     and sum in the log2 domain in fp32, O rescaled only when the maximum has grown by more than 2^8, P written back as hi and
//     lo halves (packed bfloat16) over the score buffer: hi in columns 0 - 63, lo in columns 64 - 127;
//   * epilogue O / max(l, 1e-8) as fp32, L and M as the reference writes them (:762-768).
//
// Tensor memory: S / P columns 0 - 127 (and 128 - 255), O behind.  Every mbarrier wait is bounded.
#include <math.h>

#include <algorithm>

#include "prefill.cuh"
#include "tc_ptx.cuh"
#include "tma_map.cuh"

namespace b2kv {

namespace tcf {

using namespace tc;

constexpr int kTileM = 128;
constexpr int kBlockN = 128;
constexpr int kHalfTileBytes = 128 * 128;  // 128 rows x 64 bf16
constexpr int kSoftmaxWarps = 8, kCopyWarp = 8, kMmaWarp = 9;
constexpr int kThreads = 320;
constexpr int kColS = 0;  // score buffers of 128 columns, then O
constexpr float kRescaleThreshold = 8.0f;

// kBuf: score buffers (2: QK^T of the next step runs under this step's softmax).  Step j uses the barriers and buffers j % kBuf: the next but
// one cannot begin before PV of this one has been issued, so that no wait by parity can be taken for an older phase.
template <int kD, int kBuf>
struct SharedStorage {
    static constexpr int kTileBytes = (kD / 64) * kHalfTileBytes;  // 128 rows x kD bf16
    static constexpr int kRing = kD == 64 ? kBuf : 1;              // tiles of K and of V that fit
    alignas(1024) uint8_t q[2][kTileBytes];  // [hi / lo]
    alignas(1024) uint8_t k[kRing][2][kTileBytes];
    alignas(1024) uint8_t v[kRing][2][kTileBytes];
    alignas(8) uint64_t q_full, k_full[kRing], k_empty[kRing], v_full[kRing], v_empty[kRing], s_full[kBuf], p_ready[kBuf], o_done[kBuf];
    float exchange[2][2][kTileM];  // [parity of the step][half of the keys][row]: maxima; sums at the end
    uint32_t tmem_base;
    volatile int abort_flag;
};

// x -> (bf16(x), bf16(x - bf16(x))) of a few rows of Q, K or V (grid: rows / per_cta, 3), and of K and V a copy in the cache.  As many rows per
// CTA as give its threads a piece each: with one row of 128 elements per CTA the CTAs' launches were what bound it (16 x 129 rows of two
// heads of 64, the whole call: 16.6 us so, 11.1 with eight).
struct SplitArgs {
    const float* src[3];
    __nv_bfloat16 *hi[3], *lo[3];
    float* cache[3];  // null: none
    int64_t stride_b, stride_t, stride_h;
    int64_t rows;
    int N, E, D, per_cta;
};
__global__ void __launch_bounds__(256) split_kernel(const __grid_constant__ SplitArgs a) {
    grid_launch_dependents();
    grid_dependency_wait();
    const int which = blockIdx.y;
    const int64_t row0 = static_cast<int64_t>(blockIdx.x) * a.per_cta;
    const int pieces = a.E / 4;  // of a row
    const float4* const x = reinterpret_cast<const float4*>(a.src[which] + row0 * a.E);
    uint2* const hi = reinterpret_cast<uint2*>(a.hi[which] + row0 * a.E);
    uint2* const lo = reinterpret_cast<uint2*>(a.lo[which] + row0 * a.E);
    const int all = static_cast<int>(min(static_cast<int64_t>(a.per_cta), a.rows - row0)) * pieces;
    for (int i = threadIdx.x; i < all; i += blockDim.x) {
        const float4 v = x[i];
        const uint32_t h0 = pack_bf16(v.x, v.y), h1 = pack_bf16(v.z, v.w);
        hi[i] = make_uint2(h0, h1);
        lo[i] = make_uint2(pack_bf16(v.x - __uint_as_float(h0 << 16), v.y - __uint_as_float(h0 & 0xffff0000u)),
                           pack_bf16(v.z - __uint_as_float(h1 << 16), v.w - __uint_as_float(h1 & 0xffff0000u)));
        if (a.cache[which] != nullptr) {
            const int r = i / pieces, e = (i - r * pieces) * 4, h = e / a.D;
            const int64_t row = row0 + r;
            *reinterpret_cast<float4*>(a.cache[which] + row / a.N * a.stride_b + row % a.N * a.stride_t + h * a.stride_h + (e - h * a.D)) = v;
        }
    }
}

template <int kD, int kBuf>
__global__ void __launch_bounds__(kThreads, kD == 64 && kBuf == 1 ? 2 : 1)
prefill_tc_f32_kernel(const __grid_constant__ CUtensorMap tm_qh, const __grid_constant__ CUtensorMap tm_ql,
                      const __grid_constant__ CUtensorMap tm_kh, const __grid_constant__ CUtensorMap tm_kl,
                      const __grid_constant__ CUtensorMap tm_vh, const __grid_constant__ CUtensorMap tm_vl,
                      const PrefillParams p) {
    extern __shared__ uint8_t smem_raw[];
    using Smem = SharedStorage<kD, kBuf>;
    constexpr int kRing = Smem::kRing, kColO = kBuf * 128, kTmemCols = kBuf == 1 ? 256 : 512;
    constexpr int kHalves = kD / 64;
    constexpr int kTileBytes = Smem::kTileBytes;
    Smem& sm = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_rb = (p.N + kTileM - 1) / kTileM;
    // Launch order: groups of `group` (sequence, head) pairs whose K / V halves together fit a quarter of L2; inside a
    // group the heaviest row blocks first.  The CTAs running together then share the K / V of few pairs, which stay
    // in L2 (with all pairs interleaved the halves were re-read from HBM five times over).
    const int n_bh = p.H * p.B;
    const int group = (p.group > 0 && p.group < n_bh) ? p.group : n_bh;
    const int per_group = group * n_rb;
    const int gi = static_cast<int>(blockIdx.x) / per_group;
    const int first_bh = gi * group;
    const int here = min(group, n_bh - first_bh);  // the last group may be smaller (and nothing follows it)
    const int within = static_cast<int>(blockIdx.x) - gi * per_group;
    const int rb = n_rb - 1 - within / here;
    const int bh = first_bh + within % here;
    const int b = bh / p.H, h = bh % p.H;
    const int q0 = rb * kTileM;
    const int n = rb + 1;  // K/V tiles 0 .. rb (the last one holds the diagonal)

    if (threadIdx.x == 0) {
        mbar_init(&sm.q_full, 1);
        for (int i = 0; i < kRing; ++i) {
            mbar_init(&sm.k_full[i], 1);
            mbar_init(&sm.k_empty[i], 1);
            mbar_init(&sm.v_full[i], 1);
            mbar_init(&sm.v_empty[i], 1);
        }
        for (int i = 0; i < kBuf; ++i) {
            mbar_init(&sm.s_full[i], 1);
            mbar_init(&sm.p_ready[i], kSoftmaxWarps);
            mbar_init(&sm.o_done[i], 1);
        }
        sm.abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == kMmaWarp) {
        tmem_alloc(&sm.tmem_base, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sm.tmem_base;

    if (warp == kCopyWarp) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0) {
            const int x0 = h * kD;
            grid_dependency_wait();  // the halves are the kernel before this one's; all else here follows from them
            mbar_arrive_expect_tx(&sm.q_full, 2 * kTileBytes);
#pragma unroll
            for (int hf = 0; hf < kHalves; ++hf) {
                tma_load_3d(sm.q[0] + hf * kHalfTileBytes, &tm_qh, &sm.q_full, x0 + hf * 64, q0, b);
                tma_load_3d(sm.q[1] + hf * kHalfTileBytes, &tm_ql, &sm.q_full, x0 + hf * 64, q0, b);
            }
            bool ok = true;
            for (int j = 0; j < n && ok; ++j) {
                const int st = j % kRing;
                const uint32_t par = ((j / kRing) & 1) ^ 1;
                ok = mbar_wait(&sm.k_empty[st], par);
                if (!ok) break;
                mbar_arrive_expect_tx(&sm.k_full[st], 2 * kTileBytes);
#pragma unroll
                for (int hf = 0; hf < kHalves; ++hf) {
                    tma_load_3d(sm.k[st][0] + hf * kHalfTileBytes, &tm_kh, &sm.k_full[st], x0 + hf * 64, j * kBlockN, b);
                    tma_load_3d(sm.k[st][1] + hf * kHalfTileBytes, &tm_kl, &sm.k_full[st], x0 + hf * 64, j * kBlockN, b);
                }
                ok = mbar_wait(&sm.v_empty[st], par);
                if (!ok) break;
                mbar_arrive_expect_tx(&sm.v_full[st], 2 * kTileBytes);
#pragma unroll
                for (int hf = 0; hf < kHalves; ++hf) {
                    tma_load_3d(sm.v[st][0] + hf * kHalfTileBytes, &tm_vh, &sm.v_full[st], x0 + hf * 64, j * kBlockN, b);
                    tma_load_3d(sm.v[st][1] + hf * kHalfTileBytes, &tm_vl, &sm.v_full[st], x0 + hf * 64, j * kBlockN, b);
                }
            }
            if (!ok) sm.abort_flag = 1;
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        // ------------------------------ MMA issuer ------------------------------
        if (lane == 0) {
            constexpr uint32_t idesc_qk = instr_desc(0, 0, kBlockN);  // S[128 x 128 keys]
            constexpr uint32_t idesc_pv = instr_desc(0, 1, kD);       // O[128 x kD]
            const uint64_t dq[2] = {smem_desc(smem_u32(sm.q[0]), 16, 1024), smem_desc(smem_u32(sm.q[1]), 16, 1024)};
            const uint64_t dk0 = smem_desc(smem_u32(sm.k[0][0]), 16, 1024), dv0 = smem_desc(smem_u32(sm.v[0][0]), kHalfTileBytes, 1024);
            constexpr uint64_t kTile16 = kTileBytes >> 4;
            const uint32_t o_tmem = tmem + kColO;
            // the three partial products of a split product: (hi, hi), (hi, lo), (lo, hi)
            auto issue_qk = [&](int j) {
                const uint32_t s_tmem = tmem + kColS + (j % kBuf) * 128;
#pragma unroll
                for (int t = 0; t < 3; ++t) {
                    const uint64_t da = dq[t == 2 ? 1 : 0], db = dk0 + (2 * (j % kRing) + (t == 1 ? 1 : 0)) * kTile16;
#pragma unroll
                    for (int kb = 0; kb < kHalves; ++kb) {
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {
                            const uint64_t off = static_cast<uint64_t>((kb * kHalfTileBytes + kk * 32) >> 4);
                            mma_ss(s_tmem, da + off, db + off, idesc_qk, (t | kb | kk) ? 1u : 0u);
                        }
                    }
                }
                mma_commit(&sm.s_full[j % kBuf]);
                mma_commit(&sm.k_empty[j % kRing]);
            };
            auto issue_pv = [&](int j) {
                const uint32_t s_tmem = tmem + kColS + (j % kBuf) * 128;
#pragma unroll
                for (int t = 0; t < 3; ++t) {
                    const uint32_t pa = s_tmem + (t == 2 ? 64 : 0);  // P hi in columns 0 - 63, P lo in 64 - 127
                    const uint64_t db = dv0 + (2 * (j % kRing) + (t == 1 ? 1 : 0)) * kTile16;
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                        mma_ts(o_tmem, pa + kk * 8, db + static_cast<uint64_t>((kk * 2048) >> 4), idesc_pv,
                               (j | t | kk) ? 1u : 0u);
                }
                mma_commit(&sm.o_done[j % kBuf]);
                mma_commit(&sm.v_empty[j % kRing]);
            };
            bool ok = mbar_wait(&sm.q_full, 0);
            for (int j = 0; j < kBuf && j < n && ok; ++j) {
                ok = mbar_wait(&sm.k_full[j % kRing], (j / kRing) & 1);
                if (!ok) break;
                tc_fence_after();
                issue_qk(j);
            }
            for (int j = 0; j < n && ok; ++j) {
                ok = mbar_wait(&sm.p_ready[j % kBuf], (j / kBuf) & 1) && mbar_wait(&sm.v_full[j % kRing], (j / kRing) & 1);
                if (!ok) break;
                tc_fence_after();
                issue_pv(j);
                const int jn = j + kBuf;
                if (jn < n) {
                    ok = mbar_wait(&sm.k_full[jn % kRing], (jn / kRing) & 1);
                    if (!ok) break;
                    tc_fence_after();
                    issue_qk(jn);  // overwrites P(j): the tensor pipe runs its MMAs in order, PV(j) has read it by then
                }
            }
            if (!ok) sm.abort_flag = 1;
        }
        __syncwarp();
    } else {
        // ------------------------------ softmax: two threads per query row ------------------------------
        const int row = threadIdx.x & (kTileM - 1), half = warp >> 2;  // row inside the tile = TMEM lane; half of the keys
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint32_t o_tmem = tmem + lane_base + kColO + half * (kD / 2);
        const float c = p.q_prescale;  // log2(e) / sqrt(D)
        float m_used = -INFINITY, m_run = -INFINITY, l = 0.f;
        bool ok = true;  // (a thread whose wait ran out goes on without waiting: its partners wait for it at the named barrier)
        for (int j = 0; j < n; ++j) {
            ok = ok && mbar_wait(&sm.s_full[j % kBuf], (j / kBuf) & 1);
            const uint32_t s_tmem = tmem + lane_base + kColS + (j % kBuf) * 128;
            __syncwarp();
            tc_fence_after();
            uint32_t r[64];
            tmem_ld32(s_tmem + half * 64, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
            tmem_ld32(s_tmem + half * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&r[32]));
            tmem_wait_ld();
            if (j == rb) {
#pragma unroll
                for (int i = 0; i < 64; ++i)
                    if (half * 64 + i > row) r[i] = 0xff800000u;  // -inf: key after the query
            }
            float mxs[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) mxs[a] = __uint_as_float(r[a]);
#pragma unroll
            for (int i = 4; i < 64; ++i) mxs[i & 3] = fmaxf(mxs[i & 3], __uint_as_float(r[i]));
            float mx = fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3]));
            sm.exchange[j & 1][half][row] = mx;
            // the four warps of the row's quarter pair up: both halves' scores are in registers behind this barrier as well,
            // so that either may write over the score columns
            tc_fence_before();
            named_barrier_sync<64>(1 + (warp & 3));
            tc_fence_after();
            mx = fmaxf(mx, sm.exchange[j & 1][half ^ 1][row]);
            m_run = fmaxf(m_run, mx * c);
            float factor = 1.f;
            bool need = false;
            if (j == 0) {
                m_used = m_run;
            } else if (m_run > m_used + kRescaleThreshold) {
                factor = ex2(m_used - m_run);
                m_used = m_run;
                need = true;
            }
            // P = exp2(s*c - m_used) in fp32, written as hi + lo: packed hi pairs over columns 0 - 63 of the score
            // buffer, packed lo pairs over columns 64 - 127
            float sums[4] = {0.f, 0.f, 0.f, 0.f};
            const float neg_m = -m_used;
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                uint32_t ph[16], pl[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float p0 = ex2(fmaf(__uint_as_float(r[cc * 32 + 2 * i]), c, neg_m));
                    const float p1 = ex2(fmaf(__uint_as_float(r[cc * 32 + 2 * i + 1]), c, neg_m));
                    sums[(2 * i) & 3] += p0;
                    sums[(2 * i + 1) & 3] += p1;
                    const uint32_t hi = pack_bf16(p0, p1);
                    ph[i] = hi;
                    pl[i] = pack_bf16(p0 - __uint_as_float(hi << 16), p1 - __uint_as_float(hi & 0xffff0000u));
                }
                tmem_st16(s_tmem + half * 32 + cc * 16, ph);
                tmem_st16(s_tmem + 64 + half * 32 + cc * 16, pl);
            }
            l = l * factor + ((sums[0] + sums[1]) + (sums[2] + sums[3]));
            if (__any_sync(0xffffffffu, need)) {
                ok = ok && mbar_wait(&sm.o_done[(j - 1) % kBuf], ((j - 1) / kBuf) & 1);
                __syncwarp();
                tc_fence_after();
#pragma unroll 1
                for (int cc = 0; cc < kD / 32; ++cc) {
                    uint32_t o[16];
                    tmem_ld16(o_tmem + cc * 16, o);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
                    tmem_st16(o_tmem + cc * 16, o);
                }
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.p_ready[j % kBuf]);
        }
        sm.exchange[n & 1][half][row] = l;
        // (the scores of the last step were complete behind PV of the step kBuf before: the parity names the last one)
        ok = ok && mbar_wait(&sm.o_done[(n - 1) % kBuf], ((n - 1) / kBuf) & 1);
        named_barrier_sync<64>(1 + (warp & 3));
        l += sm.exchange[n & 1][half ^ 1][row];
        if (__all_sync(0xffffffffu, ok)) {
            tc_fence_after();
            const int grow = q0 + row;
            const float inv = 1.f / fmaxf(l, 1e-8f);
            const int E = p.H * kD;
            float* Og = static_cast<float*>(p.O) + (static_cast<size_t>(b) * p.N + grow) * E + static_cast<size_t>(h) * kD +
                        half * (kD / 2);
#pragma unroll 1
            for (int cc = 0; cc < kD / 64; ++cc) {
                uint32_t o[32];
                tmem_ld32(o_tmem + cc * 32, o);
                tmem_wait_ld();
                if (grow < p.N) {
#pragma unroll
                    for (int v4 = 0; v4 < 8; ++v4) {
                        float4 w;
                        w.x = __uint_as_float(o[v4 * 4 + 0]) * inv;
                        w.y = __uint_as_float(o[v4 * 4 + 1]) * inv;
                        w.z = __uint_as_float(o[v4 * 4 + 2]) * inv;
                        w.w = __uint_as_float(o[v4 * 4 + 3]) * inv;
                        *reinterpret_cast<float4*>(Og + cc * 32 + v4 * 4) = w;
                    }
                }
                __syncwarp();
            }
            if (grow < p.N && half == 0) {
                const size_t sidx = (static_cast<size_t>(b) * p.N + grow) * p.H + h;
                if (p.L) p.L[sidx] = l * ex2(m_used - m_run);
                if (p.M) p.M[sidx] = m_run * 0.6931471805599453f;
            }
        } else {
            sm.abort_flag = 1;
        }
    }

    // common exit: every warp arrives here, then the allocating warp releases the tensor memory
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
    if (threadIdx.x == 0 && sm.abort_flag) report_status(p.dev_status, B2KV_DEV_WAIT_TIMEOUT);
}

// View of a [B*N, H*D] bf16 matrix as (x = column, y = row inside the sequence, z = sequence): rows past the end
// of a sequence read as zero.
static bool make_map(CUtensorMap* map, const void* base, int B, int N, int E) {
    EncodeTiledFn fn = tensor_map_encoder();
    if (fn == nullptr) return false;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(E), static_cast<cuuint64_t>(N), static_cast<cuuint64_t>(B)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(E) * 2, static_cast<cuuint64_t>(N) * E * 2};
    const cuuint32_t box[3] = {64, 128, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace tcf

size_t prefill_f32_scratch_bytes(int B, int N, int H, int D) {
    if (D != 128 && D != 64) return 0;
    return 6ull * static_cast<size_t>(B) * N * H * D * sizeof(__nv_bfloat16);
}

template <int kD, int kBuf>
static int launch_prefill_tc_f32(const PrefillParams& p_in, void* scratch, void* stream) {
    PrefillParams p = p_in;
    if (p.group == 0) {
        const long long pair_bytes = 8LL * p.N * kD;  // hi and lo halves of K and V of one (sequence, head)
        p.group = static_cast<int>(std::max<long long>(1, (32LL << 20) / pair_bytes));
    }
    const int E = p.H * kD;
    const size_t elems = static_cast<size_t>(p.B) * p.N * E;
    const long long ctas = static_cast<long long>((p.N + tcf::kTileM - 1) / tcf::kTileM) * p.H * p.B;
    if (ctas > 0x7fffffffLL) return B2KV_ERR_UNSUPPORTED;
    __nv_bfloat16* half[6];
    for (int i = 0; i < 6; ++i) half[i] = static_cast<__nv_bfloat16*>(scratch) + i * elems;
    CUtensorMap tm[6];
    for (int i = 0; i < 6; ++i)
        if (!tcf::make_map(&tm[i], half[i], p.B, p.N, E)) return B2KV_ERR_UNSUPPORTED;
    const long long rows = static_cast<long long>(p.B) * p.N;
    if (rows > 0x7fffffffLL) return B2KV_ERR_UNSUPPORTED;
    tcf::SplitArgs split{};
    const void* src[3] = {p.Q, p.K, p.V};
    void* cache[3] = {nullptr, p.k_cache, p.v_cache};
    for (int i = 0; i < 3; ++i) {
        split.src[i] = static_cast<const float*>(src[i]);
        split.hi[i] = half[2 * i], split.lo[i] = half[2 * i + 1];
        split.cache[i] = static_cast<float*>(cache[i]);
    }
    split.stride_b = p.stride_b, split.stride_t = p.stride_t, split.stride_h = p.stride_h;
    constexpr int kSplitThreads = 256;
    split.rows = rows, split.N = p.N, split.E = E, split.D = kD, split.per_cta = std::max(1, kSplitThreads / (E / 4));
    constexpr size_t smem = sizeof(tcf::SharedStorage<kD, kBuf>) + 1024;
    auto kernel = tcf::prefill_tc_f32_kernel<kD, kBuf>;
    static bool configured[64] = {false};
    int dev = 0;
    B2KV_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return B2KV_ERR_UNSUPPORTED;
    if (!configured[dev]) {
        B2KV_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        configured[dev] = true;
    }
    const unsigned split_ctas = static_cast<unsigned>((rows + split.per_cta - 1) / split.per_cta);
    OverlapLaunch first(dim3(split_ctas, 3), std::min(kSplitThreads, (split.per_cta * (E / 4) + 31) / 32 * 32), 0, stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&first.cfg, tcf::split_kernel, split));
    OverlapLaunch launch(static_cast<unsigned>(ctas), tcf::kThreads, smem, stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, kernel, tm[0], tm[1], tm[2], tm[3], tm[4], tm[5], p));
    return B2KV_OK;
}

int prefill_tensor_core_f32(const PrefillParams& p, int D, void* scratch, size_t scratch_bytes, void* stream) {
    if (scratch == nullptr || scratch_bytes < prefill_f32_scratch_bytes(p.B, p.N, p.H, D) || !aligned16(scratch))
        return B2KV_ERR_UNSUPPORTED;
    if ((static_cast<size_t>(p.B) * p.N * p.H * D) % 8 != 0) return B2KV_ERR_UNSUPPORTED;  // halves stay 16-byte aligned
    if (tensor_map_encoder() == nullptr) return B2KV_ERR_UNSUPPORTED;
    if (D == 128) return launch_prefill_tc_f32<128, 1>(p, scratch, stream);
    if (D != 64) return B2KV_ERR_UNSUPPORTED;
    // Two score buffers where a CTA is alone on its SM anyway, or nearly so and walks through several steps; else two CTAs share an SM and
    // fill each other's gaps.  One buffer and two, us: 64 CTAs of 2 steps 10.1, 8.6; 128 of 32 94.5, 63.6; 192 of 8 36.4, 26.4; 256 of
    // 16 59.2, 42.8; but 192 of 2 20.7, 22.8; 384 of 4 41.9, 42.8; 1536 of 16 250, 266.  (At head_dim 128, with one tile of K and V in
    // shared memory: 144 of 6 30.5, 31.2; 1024 of 32 457, 480.)
    const long long steps = (p.N + tcf::kTileM - 1) / tcf::kTileM, ctas = steps * p.H * p.B, sms = device_sm_count();
    if (ctas <= sms || (ctas <= 2 * sms && steps > 4)) return launch_prefill_tc_f32<64, 2>(p, scratch, stream);
    return launch_prefill_tc_f32<64, 1>(p, scratch, stream);
}

}  // namespace b2kv
