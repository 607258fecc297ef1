// Gated linear attention of fp32 runs, token after token, with the state in registers.
//
// The recurrence never mixes value columns, so a CTA takes 32 of a head's value columns for a whole run: the state is read and
// written once per run instead of once per token.  A lane owns two value columns and every eighth group of four key channels; the
// decays, keys and queries of eight tokens at a time come through a ring in shared memory, ahead of their use.  What bounds it is
// the issue of three multiply-adds per element of the state; gla_step_kernel, one CTA per head with the state streamed through L2
// for every token, took 939 us for runs of up to 400 tokens (6 heads, 64 x 128), this one 80 (100 with
// the tokens one after the other: eight at a time, their sums over the lanes run side by side).
// o goes to the output rows as it is (they are fp32); gla_norm_kernel applies the head's norm and the gate there.
#include "gla.cuh"

namespace b2kv {
namespace gla {
namespace {

constexpr int kWarps = 4, kCols = 8 * kWarps;  // value columns of a CTA
constexpr int kTok = 8, kRing = 3;

__device__ __forceinline__ void copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// kD: key channels, rounded up; kPadded: there are fewer.
template <int kD, bool kPadded>
__global__ void __launch_bounds__(32 * kWarps) gla_run_kernel(const __grid_constant__ b2kv_gla_args a, int parts, int32_t* dev_status) {
    constexpr int kGroups = (kD + 31) / 32;  // groups of four key channels per lane
    struct Stage {
        float4 alpha[kTok][kD / 4], k[kTok][kD / 4], q[kTok][kD / 4], v[kTok][kCols / 4];
    };
    __shared__ Stage ring[kRing];
    grid_launch_dependents();
    grid_dependency_wait();
    b2kv_row_segment sg;
    if (!segment_place(a, blockIdx.y, sg)) {
        if (threadIdx.x == 0) report_status(dev_status, B2KV_DEV_BAD_POSITION);
        return;
    }
    const int h = static_cast<int>(blockIdx.x) / parts, c0 = static_cast<int>(blockIdx.x) % parts * kCols;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, dg = lane >> 2, c = c0 + warp * 8 + (lane & 3) * 2;
    const bool live = c < a.vdim;
    const int d4 = a.dim / 4, v4 = min(kCols, a.vdim - c0) / 4;
    // what no copy writes (key channels and value columns that are padding) counts as zero
    for (int i = tid; i < static_cast<int>(sizeof(ring) / 16); i += 32 * kWarps) reinterpret_cast<float4*>(ring)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    float* const state = a.state + (static_cast<int64_t>(sg.slot) * a.H + h) * a.dim * a.vdim + c;
    const bool fresh = a.row_pos[sg.row0] == 0;
    float2 s[kGroups][4];
#pragma unroll
    for (int j = 0; j < kGroups; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int d = j * 32 + dg * 4 + e;
            s[j][e] = live && !fresh && d < a.dim ? *reinterpret_cast<const float2*>(state + static_cast<int64_t>(d) * a.vdim)
                                                 : make_float2(0.f, 0.f);
        }
    const float* const y = static_cast<const float*>(a.y) + static_cast<int64_t>(sg.row0) * a.ld_y;
    const float* const alpha = a.alpha + static_cast<int64_t>(sg.row0) * a.ld_alpha + static_cast<int64_t>(h) * a.dim;
    const int steps = (sg.n + kTok - 1) / kTok, per_tok = 3 * d4 + v4;
    auto request = [&](int step) {
        if (step < steps) {
            Stage& st = ring[step % kRing];
            for (int i = tid; i < kTok * per_tok; i += 32 * kWarps) {
                const int t = i / per_tok, j = i - t * per_tok, r = step * kTok + t;
                if (r >= sg.n) break;
                const float* const row = y + static_cast<int64_t>(r) * a.ld_y;
                if (j < d4) copy16(&st.alpha[t][j], alpha + static_cast<int64_t>(r) * a.ld_alpha + j * 4);
                else if (j < 2 * d4) copy16(&st.k[t][j - d4], row + a.k_col + h * a.dim + (j - d4) * 4);
                else if (j < 3 * d4) copy16(&st.q[t][j - 2 * d4], row + a.q_col + h * a.dim + (j - 2 * d4) * 4);
                else copy16(&st.v[t][j - 3 * d4], row + a.v_col + h * a.vdim + c0 + (j - 3 * d4) * 4);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    __syncthreads();  // the zeros lie under the copies
#pragma unroll
    for (int i = 0; i < kRing - 1; ++i) request(i);
    float* const out = static_cast<float*>(a.out) + static_cast<int64_t>(sg.row0) * a.ld_out + static_cast<int64_t>(h) * a.vdim + c;
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
        __syncthreads();  // this step's rows are here, and everybody has left the step before, whose place is asked for again
        request(step + kRing - 1);
        const Stage& st = ring[step % kRing];
        const int n = min(kTok, sg.n - step * kTok);
        // one token: the state moves on; this lane's part of o
        auto token = [&](int t) {
            const float2 v = reinterpret_cast<const float2*>(st.v[t])[warp * 4 + (lane & 3)];
            float2 o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < kGroups; ++j) {
                const float4 al = st.alpha[t][j * 8 + dg], kk = st.k[t][j * 8 + dg], qq = st.q[t][j * 8 + dg];
                // (a key of zero is no answer to a value that is not finite)
                const float2 vj = kPadded && j * 32 + dg * 4 >= a.dim ? make_float2(0.f, 0.f) : v;
                const float av[4] = {al.x, al.y, al.z, al.w}, kv[4] = {kk.x, kk.y, kk.z, kk.w}, qv[4] = {qq.x, qq.y, qq.z, qq.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    s[j][e] = __ffma2_rn(s[j][e], make_float2(av[e], av[e]), __fmul2_rn(make_float2(kv[e], kv[e]), vj));
                    const float q = qv[e] * a.q_scale;
                    o[e] = __ffma2_rn(make_float2(q, q), s[j][e], o[e]);
                }
            }
            return __fadd2_rn(__fadd2_rn(o[0], o[1]), __fadd2_rn(o[2], o[3]));
        };
        auto other = [](float2 x, int off) {
            return make_float2(__shfl_xor_sync(0xffffffffu, x.x, off), __shfl_xor_sync(0xffffffffu, x.y, off));
        };
        if (n == kTok) {
            // The tokens' parts of o are summed over the eight lanes that share the key channels by halving: a lane hands on what
            // the other half of the lanes sums up, and is left with one token (lane bits 4, 3, 2 = token bits 2, 1, 0).
            float2 o[kTok];
#pragma unroll
            for (int t = 0; t < kTok; ++t) o[t] = token(t);
#pragma unroll
            for (int half = kTok / 2; half > 0; half >>= 1) {
                const bool up = lane & (half * 4);
#pragma unroll
                for (int t = 0; t < half; ++t) {
                    const float2 mine = up ? o[t + half] : o[t], theirs = up ? o[t] : o[t + half];
                    o[t] = __fadd2_rn(mine, other(theirs, half * 4));
                }
            }
            if (live) *reinterpret_cast<float2*>(out + static_cast<int64_t>(step * kTok + dg) * a.ld_out) = o[0];
        } else {
            for (int t = 0; t < n; ++t) {
                float2 o = token(t);
#pragma unroll
                for (int off = 4; off < 32; off <<= 1) o = __fadd2_rn(o, other(o, off));
                if (dg == 0 && live) *reinterpret_cast<float2*>(out + static_cast<int64_t>(step * kTok + t) * a.ld_out) = o;
            }
        }
    }
    if (!live) return;
#pragma unroll
    for (int j = 0; j < kGroups; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int d = j * 32 + dg * 4 + e;
            if (d < a.dim) *reinterpret_cast<float2*>(state + static_cast<int64_t>(d) * a.vdim) = s[j][e];
        }
}

// One warp per (token, head).
constexpr int kNormWarps = 8;
__global__ void __launch_bounds__(32 * kNormWarps) gla_norm_kernel(const __grid_constant__ b2kv_gla_args a) {
    const int lane = threadIdx.x & 31, at = static_cast<int>(blockIdx.x) * kNormWarps + (threadIdx.x >> 5), t = at / a.H, h = at % a.H;
    grid_launch_dependents();
    grid_dependency_wait();
    b2kv_row_segment sg;
    if (!segment_place(a, blockIdx.y, sg) || t >= sg.n) return;
    const int64_t row = static_cast<int64_t>(sg.row0) + t;
    float* const o = static_cast<float*>(a.out) + row * a.ld_out + static_cast<int64_t>(h) * a.vdim;
    const float* const gate = static_cast<const float*>(a.y) + row * a.ld_y + a.g_col + static_cast<int64_t>(h) * a.vdim;
    float sum = 0.f;
    for (int c = lane; c < a.vdim; c += 32) sum = fmaf(o[c], o[c], sum);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const float scale = 1.0f / sqrtf(sum / static_cast<float>(a.vdim) + a.eps);
    for (int c = lane; c < a.vdim; c += 32) o[c] = o[c] * scale * a.norm[c] * silu(gate[c]);
}

}  // namespace
}  // namespace gla

int gla_run_f32(const b2kv_gla_args& a, int32_t* dev_status, void* stream) {
    using namespace gla;
    if (a.dtype != B2KV_DTYPE_F32 || a.dim > 128 || a.dim % 4 || a.vdim % 4 || a.n_segments > 65535) return B2KV_ERR_UNSUPPORTED;
    // 16-byte pieces of rows, pairs of value columns in the state and the output
    if (!aligned16(a.y) || !aligned16(a.alpha) || !aligned16(a.state) || !aligned16(a.out) || a.ld_y % 4 || a.ld_alpha % 4 || a.ld_out % 2 ||
        a.q_col % 4 || a.k_col % 4 || a.v_col % 4)
        return B2KV_ERR_UNSUPPORTED;
    const int parts = (a.vdim + kCols - 1) / kCols;
    const long long ctas = static_cast<long long>(a.H) * parts, pairs = static_cast<long long>(a.max_n) * a.H;
    if (ctas > 0x7fffffffLL || pairs > 0x7fffffffLL - kNormWarps) return B2KV_ERR_UNSUPPORTED;
    OverlapLaunch run(dim3(static_cast<unsigned>(ctas), a.n_segments), 32 * kWarps, 0, stream);
    const auto kernel = a.dim < 32    ? gla_run_kernel<32, true>
                        : a.dim == 32  ? gla_run_kernel<32, false>
                        : a.dim < 64   ? gla_run_kernel<64, true>
                        : a.dim == 64  ? gla_run_kernel<64, false>
                        : a.dim < 128  ? gla_run_kernel<128, true>
                                       : gla_run_kernel<128, false>;
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&run.cfg, kernel, a, parts, dev_status));
    OverlapLaunch norm(dim3(static_cast<unsigned>((pairs + kNormWarps - 1) / kNormWarps), a.n_segments), 32 * kNormWarps, 0, stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&norm.cfg, gla_norm_kernel, a));
    return B2KV_OK;
}

}  // namespace b2kv
