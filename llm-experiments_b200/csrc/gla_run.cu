// Gated linear attention of fp32 runs, token after token, with the state in registers.
//
// The recurrence never mixes value columns, so a CTA takes 32 of a head's value columns for a whole run: the state is read and
// written once per run instead of once per token.  A lane owns two value columns and every eighth group of four key channels; the
// decays, keys and queries of eight tokens at a time come through a ring in shared memory, ahead of their use.  What bounds it is
// the issue of three multiply-adds per element of the state; gla_step_kernel, one CTA per head with the state streamed through L2
// for every token, took 939 us for runs of up to 400 tokens (6 heads, 64 x 128), this one 80 (100 with
// the tokens one after the other: eight at a time, their sums over the lanes run side by side).
//
// 400 tokens one after the other are a chain, on half of the SMs with a warp per scheduler, so runs of more than 192 tokens over heads of up
// to 64 key channels are cut into spans of 64 where there is scratch memory.  A first pass makes every span's own part of the state from zero, and the product of its decays
// (all but the last one's); gla_spans_kernel carries the state through, S <- diag(D) S + L, and leaves what each span begins with;
// the second pass walks all spans side by side.  Two thirds more work: three prompts of 62 to 400 tokens, 6 heads of 64 x 128, 59 us in all, 124 as
// chains.  Spans begin at multiples of 64 tokens
// from the segment's first token, and the sums are in one order whatever else is in the step.
// o goes to the output rows as it is (they are fp32); gla_norm_kernel applies the head's norm and the gate there.
#include <algorithm>

#include "gla.cuh"

namespace b2kv {
namespace gla {
namespace {

constexpr int kWarps = 4, kCols = 8 * kWarps;  // value columns of a CTA
constexpr int kTok = 8, kRing = 3;
constexpr int kSpanTokens = 64;
constexpr int kMinSpanned = 193;  // tokens of a segment that is cut
constexpr int kMaxSpannedDim = 64, kMaxSpannedCtas = 32;  // CTAs: value columns of a state / 32
constexpr size_t kMaxSpanBytes = size_t{256} << 20;  // spans at a time, more only where a state per segment takes more

__host__ __device__ constexpr int spans_of(int n) { return n < kMinSpanned ? 1 : (n + kSpanTokens - 1) / kSpanTokens; }

// The spans [first, first + count) of every segment: states [segment][span][H][dim][vdim], products of decays [segment][span][H][dim].
struct Spans {
    float *states, *decays;
    int first, count;
};

enum Pass {
    kWholeRun,  // no spans
    kOwnPart,   // a span's own part of the state
    kOutputs,   // from what a span begins with
};

__device__ __forceinline__ void copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// kD: key channels, rounded up; kPadded: there are fewer.
template <int kD, bool kPadded, Pass kPass>
__global__ void __launch_bounds__(32 * kWarps)
gla_run_kernel(const __grid_constant__ b2kv_gla_args a, int parts, const Spans spans, int32_t* dev_status) {
    constexpr int kGroups = (kD + 31) / 32;  // groups of four key channels per lane
    struct Stage {
        float4 alpha[kTok][kD / 4], k[kTok][kD / 4], q[kTok][kD / 4], v[kTok][kCols / 4];
    };
    __shared__ Stage ring[kRing];
    grid_launch_dependents();
    grid_dependency_wait();
    b2kv_row_segment sg;
    if (!segment_place(a, blockIdx.y, sg)) {
        if (threadIdx.x == 0 && blockIdx.z == 0) report_status(dev_status, B2KV_DEV_BAD_POSITION);
        return;
    }
    const bool fresh = a.row_pos[sg.row0] == 0;
    const int span = spans.first + static_cast<int>(blockIdx.z), all_spans = kPass == kWholeRun ? 1 : spans_of(sg.n);
    if (kPass != kWholeRun) {
        if (span >= all_spans || (kPass == kOwnPart && span + 1 == all_spans)) return;
        if (all_spans > 1) sg.row0 += span * kSpanTokens, sg.n = min(kSpanTokens, sg.n - span * kSpanTokens);
    }
    const int h = static_cast<int>(blockIdx.x) / parts, c0 = static_cast<int>(blockIdx.x) % parts * kCols;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, dg = lane >> 2, c = c0 + warp * 8 + (lane & 3) * 2;
    const bool live = c < a.vdim;
    const int d4 = a.dim / 4, v4 = min(kCols, a.vdim - c0) / 4;
    // what no copy writes (key channels and value columns that are padding) counts as zero
    for (int i = tid; i < static_cast<int>(sizeof(ring) / 16); i += 32 * kWarps) reinterpret_cast<float4*>(ring)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    float* const state = a.state + (static_cast<int64_t>(sg.slot) * a.H + h) * a.dim * a.vdim + c;
    const int64_t place = (static_cast<int64_t>(blockIdx.y) * spans.count + blockIdx.z) * a.H + h;
    float* const scratch = all_spans > 1 ? spans.states + place * a.dim * a.vdim + c : nullptr;
    const float* const from = kPass == kOwnPart || (scratch == nullptr && fresh) ? nullptr : (scratch != nullptr ? scratch : state);
    float* const to = kPass == kOwnPart ? scratch : (span + 1 == all_spans || kPass == kWholeRun ? state : nullptr);
    const bool decays = kPass == kOwnPart && c0 == 0 && warp == 0;  // this warp multiplies them up
    float product[kGroups][4];
    float2 s[kGroups][4];
#pragma unroll
    for (int j = 0; j < kGroups; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int d = j * 32 + dg * 4 + e;
            s[j][e] = live && from != nullptr && d < a.dim ? *reinterpret_cast<const float2*>(from + static_cast<int64_t>(d) * a.vdim)
                                                           : make_float2(0.f, 0.f);
            product[j][e] = 1.f;
        }
    const float* const y = static_cast<const float*>(a.y) + static_cast<int64_t>(sg.row0) * a.ld_y;
    const float* const alpha = a.alpha + static_cast<int64_t>(sg.row0) * a.ld_alpha + static_cast<int64_t>(h) * a.dim;
    const int steps = (sg.n + kTok - 1) / kTok, rows_d4 = (kPass == kOwnPart ? 2 : 3) * d4, per_tok = rows_d4 + v4;
    auto request = [&](int step) {
        if (step < steps) {
            Stage& st = ring[step % kRing];
            for (int i = tid; i < kTok * per_tok; i += 32 * kWarps) {
                const int t = i / per_tok, j = i - t * per_tok, r = step * kTok + t;
                if (r >= sg.n) break;
                const float* const row = y + static_cast<int64_t>(r) * a.ld_y;
                if (j < d4) copy16(&st.alpha[t][j], alpha + static_cast<int64_t>(r) * a.ld_alpha + j * 4);
                else if (j < 2 * d4) copy16(&st.k[t][j - d4], row + a.k_col + h * a.dim + (j - d4) * 4);
                else if (j < rows_d4) copy16(&st.q[t][j - 2 * d4], row + a.q_col + h * a.dim + (j - 2 * d4) * 4);
                else copy16(&st.v[t][j - rows_d4], row + a.v_col + h * a.vdim + c0 + (j - rows_d4) * 4);
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
                const float4 al = st.alpha[t][j * 8 + dg], kk = st.k[t][j * 8 + dg];
                const float4 qq = kPass == kOwnPart ? make_float4(0.f, 0.f, 0.f, 0.f) : st.q[t][j * 8 + dg];
                // (a key of zero is no answer to a value that is not finite)
                const float2 vj = kPadded && j * 32 + dg * 4 >= a.dim ? make_float2(0.f, 0.f) : v;
                const float av[4] = {al.x, al.y, al.z, al.w}, kv[4] = {kk.x, kk.y, kk.z, kk.w}, qv[4] = {qq.x, qq.y, qq.z, qq.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    s[j][e] = __ffma2_rn(s[j][e], make_float2(av[e], av[e]), __fmul2_rn(make_float2(kv[e], kv[e]), vj));
                    if (kPass == kOwnPart) continue;
                    const float q = qv[e] * a.q_scale;
                    o[e] = __ffma2_rn(make_float2(q, q), s[j][e], o[e]);
                }
            }
            if (decays) {
#pragma unroll
                for (int j = 0; j < kGroups; ++j) {
                    const float4 al = st.alpha[t][j * 8 + dg];
                    product[j][0] *= al.x, product[j][1] *= al.y, product[j][2] *= al.z, product[j][3] *= al.w;
                }
            }
            return __fadd2_rn(__fadd2_rn(o[0], o[1]), __fadd2_rn(o[2], o[3]));
        };
        if (kPass == kOwnPart) {
#pragma unroll 4
            for (int t = 0; t < n; ++t) token(t);
            continue;
        }
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
    if (decays && (lane & 3) == 0) {
#pragma unroll
        for (int j = 0; j < kGroups; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int d = j * 32 + dg * 4 + e;
                if (d < a.dim) spans.decays[place * a.dim + d] = product[j][e];
            }
    }
    if (!live || to == nullptr) return;
#pragma unroll
    for (int j = 0; j < kGroups; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int d = j * 32 + dg * 4 + e;
            if (d < a.dim) *reinterpret_cast<float2*>(to + static_cast<int64_t>(d) * a.vdim) = s[j][e];
        }
}

// What every span begins with, in the place of its own part: a thread per four value columns of a key channel.  Where a span's decays
// multiply up to next to nothing, which says nothing about a large state any more, they are taken one after the other.
constexpr int kSpanRows = 4, kSpanThreads = 128;
__global__ void __launch_bounds__(kSpanThreads) gla_spans_kernel(const __grid_constant__ b2kv_gla_args a, const Spans spans) {
    grid_launch_dependents();
    grid_dependency_wait();
    b2kv_row_segment sg;
    if (!segment_place(a, blockIdx.z, sg)) return;
    const int all_spans = spans_of(sg.n), n_spans = min(spans.count, all_spans - spans.first), h = blockIdx.y, v4 = a.vdim / 4;
    if (all_spans == 1 || n_spans <= 0) return;
    const bool fresh = spans.first == 0 && a.row_pos[sg.row0] == 0, more = spans.first + n_spans < all_spans;
    const float* const alpha = a.alpha + static_cast<int64_t>(sg.row0 + spans.first * kSpanTokens) * a.ld_alpha + static_cast<int64_t>(h) * a.dim;
    const int64_t place = static_cast<int64_t>(blockIdx.z) * spans.count * a.H + h;
    for (int i = threadIdx.x; i < kSpanRows * v4; i += kSpanThreads) {
        const int d = static_cast<int>(blockIdx.x) * kSpanRows + i / v4, c = i % v4 * 4;
        if (d >= a.dim) break;
        const int64_t at = static_cast<int64_t>(d) * a.vdim + c, each = static_cast<int64_t>(a.H) * a.dim * a.vdim;
        float* const state = a.state + (static_cast<int64_t>(sg.slot) * a.H + h) * a.dim * a.vdim + at;
        float* const scratch = spans.states + place * a.dim * a.vdim + at;
        const float* const decay = spans.decays + place * a.dim + d;
        auto has_own = [&](int s) { return s + 1 < n_spans || (more && s < n_spans); };
        auto own_of = [&](int s) { return has_own(s) ? *reinterpret_cast<const float4*>(scratch + s * each) : make_float4(0.f, 0.f, 0.f, 0.f); };
        auto decay_of = [&](int s) { return has_own(s) ? decay[static_cast<int64_t>(s) * a.H * a.dim] : 1.f; };
        float4 x = fresh ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(state);
        float4 own = own_of(0), own_next = own_of(1);
        float f = decay_of(0), f_next = decay_of(1);
        for (int s = 0; s < n_spans; ++s) {
            const float4 own_far = own_of(s + 2);
            const float f_far = decay_of(s + 2);
            *reinterpret_cast<float4*>(scratch + s * each) = x;
            if (!has_own(s)) break;
            if (f >= 1e-30f) {
                x = make_float4(fmaf(x.x, f, own.x), fmaf(x.y, f, own.y), fmaf(x.z, f, own.z), fmaf(x.w, f, own.w));
            } else {
                for (int t = 0; t < kSpanTokens; ++t) {  // (a span that something follows is whole)
                    const float al = alpha[static_cast<int64_t>(s * kSpanTokens + t) * a.ld_alpha + d];
                    x.x *= al, x.y *= al, x.z *= al, x.w *= al;
                }
                x.x += own.x, x.y += own.y, x.z += own.z, x.w += own.w;
            }
            own = own_next, own_next = own_far;
            f = f_next, f_next = f_far;
        }
        if (more) *reinterpret_cast<float4*>(state) = x;
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

namespace gla {
namespace {

size_t span_floats(int H, int dim, int vdim) { return static_cast<size_t>(H) * dim * (static_cast<size_t>(vdim) + 1); }

// Spans of every segment that are walked at a time.
int span_count(const b2kv_gla_args& a) {
    const size_t each = span_floats(a.H, a.dim, a.vdim) * sizeof(float) * a.n_segments;
    return static_cast<int>(std::max<size_t>(1, std::min<size_t>({kMaxSpanBytes / each, static_cast<size_t>(spans_of(a.max_n)), size_t{65535}})));
}

template <int kD, bool kPadded>
int launch_runs(const b2kv_gla_args& a, int parts, int32_t* dev_status, void* stream) {
    const dim3 grid(static_cast<unsigned>(a.H * parts), a.n_segments);
    if constexpr (kD <= kMaxSpannedDim) {
        const size_t need = gla_run_f32_workspace(a.H, a.dim, a.vdim, a.n_segments, a.max_n);
        if (need > 0 && a.workspace != nullptr && aligned16(a.workspace) && a.workspace_bytes >= need) {
            Spans spans{};
            spans.count = span_count(a);
            spans.states = static_cast<float*>(a.workspace);
            spans.decays = spans.states + static_cast<size_t>(a.n_segments) * spans.count * a.H * a.dim * a.vdim;
            const int all = spans_of(a.max_n);
            for (; spans.first < all; spans.first += spans.count) {
                const unsigned here = std::min(spans.count, all - spans.first);
                OverlapLaunch own(dim3(grid.x, grid.y, here), 32 * kWarps, 0, stream);
                B2KV_CUDA_TRY(cudaLaunchKernelEx(&own.cfg, gla_run_kernel<kD, kPadded, kOwnPart>, a, parts, spans, dev_status));
                OverlapLaunch through(dim3((a.dim + kSpanRows - 1) / kSpanRows, a.H, a.n_segments), kSpanThreads, 0, stream);
                B2KV_CUDA_TRY(cudaLaunchKernelEx(&through.cfg, gla_spans_kernel, a, spans));
                OverlapLaunch run(dim3(grid.x, grid.y, here), 32 * kWarps, 0, stream);
                B2KV_CUDA_TRY(cudaLaunchKernelEx(&run.cfg, gla_run_kernel<kD, kPadded, kOutputs>, a, parts, spans, dev_status));
            }
            return B2KV_OK;
        }
    }
    OverlapLaunch run(grid, 32 * kWarps, 0, stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&run.cfg, gla_run_kernel<kD, kPadded, kWholeRun>, a, parts, Spans{}, dev_status));
    return B2KV_OK;
}

}  // namespace
}  // namespace gla

size_t gla_run_f32_workspace(int H, int dim, int vdim, int n_segments, int max_n) {
    using namespace gla;
    // Two passes pay where the chain is long and what they add runs on SMs that would be idle.  That is for states that few CTAs hold (32 value
    // columns each) and heads of up to 64 key channels, whose chains leave issue slots even where the segments fill the device; us as one chain
    // and in spans, 6 heads of 64 x 128 (24 CTAs): 1 run of 400 tokens 111, 45; 4 132, 69; 16 201, 173; 24 236, 251; of 200 tokens 1 47, 36; 4 77,
    // 46; 16 84, 92.  4 heads of 128 x 256 (32 CTAs): 1 run of 400 126, 58; 4 204, 110; 8 197, 189; but 16 243, 348: those stay one
    // chain.  The number of segments must not choose, a sequence's sums do not depend on its company.
    if (dim > kMaxSpannedDim || dim % 4 || vdim % 4 || max_n < kMinSpanned || H * ((vdim + kCols - 1) / kCols) > kMaxSpannedCtas) return 0;
    const size_t each = span_floats(H, dim, vdim) * sizeof(float), segments = static_cast<size_t>(n_segments);
    return std::min(each * segments * spans_of(max_n), std::max(kMaxSpanBytes, each * segments));  // (grows with segments and tokens)
}

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
    const auto runs = a.dim < 32    ? launch_runs<32, true>
                      : a.dim == 32  ? launch_runs<32, false>
                      : a.dim < 64   ? launch_runs<64, true>
                      : a.dim == 64  ? launch_runs<64, false>
                      : a.dim < 128  ? launch_runs<128, true>
                                     : launch_runs<128, false>;
    const int rc = runs(a, parts, dev_status, stream);
    if (rc != B2KV_OK) return rc;
    OverlapLaunch norm(dim3(static_cast<unsigned>((pairs + kNormWarps - 1) / kNormWarps), a.n_segments), 32 * kNormWarps, 0, stream);
    B2KV_CUDA_TRY(cudaLaunchKernelEx(&norm.cfg, gla_norm_kernel, a));
    return B2KV_OK;
}

}  // namespace b2kv
