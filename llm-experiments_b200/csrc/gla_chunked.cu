// Gated linear attention over prompt portions, sixteen tokens at a time (bf16 rows, fp32 state).
//
// With P_t the product of the decays up to token t of a chunk and R_s the product behind token s (both per key channel, both at
// most one, so nothing can overflow however strong the decay), a chunk with incoming state S is
//
//   o_t  = S^T (q_t P_t) + sum_{s <= t} A_ts v_s,   A_ts = sum_d q_td k_sd prod_{s < r <= t} alpha_rd
//   S   <- diag(P_last) S + sum_s (k_s R_s) v_s^T
//
// Three kernels.  What does not depend on the state is made for many chunks at once (gla_prepare_kernel): one CTA per chunk and
// head, thread = two key channels; A's products of decays are carried along exactly instead of being taken apart into factors that
// could overflow, and its entries are summed over the channels 32 at a time.  The result is a record per chunk and head that is
// byte for byte what the second kernel wants in shared memory.  Records are made a slice of the segments at a time, which bounds the
// workspace.
//
// gla_state_kernel has one CTA per (64 value columns of a head, segment) and walks the chunks in order.  Nothing in the recurrence
// connects value columns, and a chunk is a chain of dependent products, so what counts is how few warps share an SM's tensor pipe:
// one per scheduler here (with a whole head's 256 columns on one SM a prompt of 2048 tokens kept 8 SMs busy: two prompts of 1750 tokens, 8 heads of
// 128 x 256, took 366 us, 181 so).
//   * every warp owns 16 value columns of the state, transposed, as accumulators of mma.m16n8k16: the state never
//     leaves registers between the first and the last chunk.  As an A operand of the first product the accumulators need no
//     shuffle.  A step of the recurrence is sixteen tokens deep, one k-step of this instruction; larger tiles would have to
//     bring the state through tensor memory, decay it there and write it back as operands sixteen tokens at a time, a chain of
//     copies and waits several times as long as these products.
//   * fp32 operands (q P, k R, A and the state) are split into two bf16 halves, x = hi + lo, and lo * lo is dropped; v is
//     exact.  Accumulation, decay and state are fp32.
//   * the products of o are one chain per accumulator, in an order that no other sequence of the step has a say in; the products that
//     move the state on are independent of it and are issued in between.
//   * o leaves in fp32 for the workspace; gla_finish_kernel applies the head's norm, which needs whole rows, and the gate.
//   * copies run ahead through a ring: records with one bulk copy each, rows of v with TMA.  A thread of the first warp
//     asks for them when everybody has left the chunk before (a warp of its own would take registers from all others).
// Every wait is bounded; a thread whose wait ran out goes on without waiting (so that nobody is left at a barrier) and reports.
#include <algorithm>

#include "gla.cuh"
#include "tc_ptx.cuh"
#include "tma_map.cuh"

namespace b2kv {
namespace gla {
namespace {

constexpr int kChunk = 16;
constexpr int kPairs = kChunk * (kChunk + 1) / 2;  // entries of A on and below the diagonal
constexpr int kSlab = 16;                          // value columns per state warp
constexpr int kWarps = 4;                          // state warps of a CTA
constexpr int kMaxVdim = 256;
constexpr int kBox = 32;                           // value columns per copy of v: two warps' slabs
constexpr int kMaxRing = 6;
constexpr int kSmemLimit = 109 * 1024;     // two CTAs per SM
constexpr size_t kSliceBytes = 128u << 20;  // records and o of a slice, at most (but at least kMinSlice chunks per segment)
constexpr int kMinSlice = 8;

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Two fp32 numbers as bf16 pairs: the leading halves and what they leave.
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
    hi = tc::pack_bf16(x, y);
    lo = tc::pack_bf16(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
}
__device__ __forceinline__ void split1(float x, __nv_bfloat16& hi, __nv_bfloat16& lo) {
    hi = __float2bfloat16_rn(x);
    lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}

// What a chunk brings to a head beside v, for kD16 * 16 key channels.
template <int kD16>
struct alignas(128) Record {
    static constexpr int kD = kD16 * 16;
    static constexpr int kLd = kD + 8;  // bf16 rows an odd number of 16-byte pieces apart: no bank conflicts in ldmatrix
    static constexpr int kLa = 24;
    __nv_bfloat16 q_hi[kChunk][kLd], q_lo[kChunk][kLd], k_hi[kChunk][kLd], k_lo[kChunk][kLd];  // q P, k R
    __nv_bfloat16 a_hi[kChunk][kLa], a_lo[kChunk][kLa];
    float decay[kD];  // P_last
};

// Chunks [first, first + count) of every segment; record (segment, head, chunk) at ((segment * H + head) * count + chunk - first).
struct Slice {
    int first, count;
};

// Entries of A in a fixed order, column after column from the diagonal down, as compile-time constants.
template <int kP>
struct Entry {
    static constexpr int column(int p) {
        int c = 0;
        for (; p >= kChunk - c; ++c) p -= kChunk - c;
        return c;
    }
    static constexpr int p = kP, c = column(kP), t = kP - (c * kChunk - c * (c - 1) / 2) + c;
};
template <int kP, typename F>
__device__ __forceinline__ void each_entry(F&& fn) {
    if constexpr (kP < kPairs) {
        fn(Entry<kP>{});
        each_entry<kP + 1>(fn);
    }
}
// Lane i gets the sum over the warp of everybody's v[i].
__device__ __forceinline__ float sum_by_lane(float (&v)[32], int lane) {
#pragma unroll
    for (int h = 16; h > 0; h >>= 1) {
        const bool up = lane & h;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float mine = up ? v[i + h] : v[i], theirs = up ? v[i] : v[i + h];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, h);
        }
    }
    return v[0];
}

template <int kD16>
__global__ void __launch_bounds__(kD16 <= 4 ? 32 : 8 * kD16) gla_prepare_kernel(const __grid_constant__ b2kv_gla_args a, const Slice slice,
                                                                               int32_t* dev_status) {
    using R = Record<kD16>;
    constexpr int kD = R::kD, kThreads = kD16 <= 4 ? 32 : 8 * kD16, kWarps = kThreads / 32;
    __shared__ R out;
    __shared__ float part[kWarps][kPairs];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y, d = 2 * tid;
    grid_launch_dependents();
    if (tid == 0) grid_dependency_wait();
    __syncthreads();
    b2kv_row_segment sg;
    if (!segment_place(a, blockIdx.z, sg)) {
        if (tid == 0) report_status(dev_status, B2KV_DEV_BAD_POSITION);
        return;
    }
    const int first = (slice.first + static_cast<int>(blockIdx.x)) * kChunk;
    if (sg.n <= first) return;
    const int n = d < a.dim ? min(kChunk, sg.n - first) : 0;  // tokens of this chunk (none in channels that are padding)
    const int64_t row = sg.row0 + first;
    const float* const ra = a.alpha + row * a.ld_alpha + h * a.dim + d;
    const __nv_bfloat16* const y = static_cast<const __nv_bfloat16*>(a.y) + row * a.ld_y + h * a.dim + d;
    float2 al[kChunk], q[kChunk], k[kChunk], prod = make_float2(1.f, 1.f);
#pragma unroll
    for (int t = 0; t < kChunk; ++t) {
        al[t] = t < n ? *reinterpret_cast<const float2*>(ra + t * a.ld_alpha) : make_float2(1.f, 1.f);
        const uint32_t qb = t < n ? *reinterpret_cast<const uint32_t*>(y + t * a.ld_y + a.q_col) : 0u;
        const uint32_t kb = t < n ? *reinterpret_cast<const uint32_t*>(y + t * a.ld_y + a.k_col) : 0u;
        q[t] = make_float2(__uint_as_float(qb << 16) * a.q_scale, __uint_as_float(qb & 0xffff0000u) * a.q_scale);
        k[t] = make_float2(__uint_as_float(kb << 16), __uint_as_float(kb & 0xffff0000u));
    }
    if (d < kD) {
        auto store = [&](__nv_bfloat16* hi_at, __nv_bfloat16* lo_at, float2 v) {
            uint32_t hi, lo;
            split2(v.x, v.y, hi, lo);
            *reinterpret_cast<uint32_t*>(hi_at) = hi;
            *reinterpret_cast<uint32_t*>(lo_at) = lo;
        };
#pragma unroll
        for (int t = 0; t < kChunk; ++t) {
            prod = __fmul2_rn(prod, al[t]);
            store(&out.q_hi[t][d], &out.q_lo[t][d], __fmul2_rn(q[t], prod));
        }
        *reinterpret_cast<float2*>(&out.decay[d]) = prod;
        prod = make_float2(1.f, 1.f);
#pragma unroll
        for (int t = kChunk - 1; t >= 0; --t) {
            store(&out.k_hi[t][d], &out.k_lo[t][d], __fmul2_rn(k[t], prod));
            prod = __fmul2_rn(prod, al[t]);
        }
    }
    // these channels' part of every entry of A; 32 entries at a time are summed over the warp's channels
    float v[32];
    float2 w = make_float2(0.f, 0.f);
    each_entry<0>([&](auto entry) {
        constexpr int p = entry.p, t = entry.t, c = entry.c;
        w = t == c ? k[c] : __fmul2_rn(w, al[t]);
        const float2 z = __fmul2_rn(q[t], w);
        v[p % 32] = z.x + z.y;
        if constexpr (p % 32 == 31) part[warp][p - 31 + lane] = sum_by_lane(v, lane);
    });
#pragma unroll
    for (int i = kPairs % 32; i < 32; ++i) v[i] = 0.f;
    const float last = sum_by_lane(v, lane);
    if (lane < kPairs % 32) part[warp][kPairs / 32 * 32 + lane] = last;
    __syncthreads();
    for (int e = tid; e < kChunk * kChunk; e += kThreads) {
        const int t = e / kChunk, c = e % kChunk;
        float sum = 0.f;
        if (c <= t) {
            const int p = c * kChunk - c * (c - 1) / 2 + t - c;
#pragma unroll
            for (int i = 0; i < kWarps; ++i) sum += part[i][p];
        }
        split1(sum, out.a_hi[t][c], out.a_lo[t][c]);
    }
    __syncthreads();
    uint4* const dst = reinterpret_cast<uint4*>(reinterpret_cast<R*>(a.workspace) +
                                                (static_cast<int64_t>(blockIdx.z) * a.H + h) * slice.count + blockIdx.x);
    for (int i = tid; i < static_cast<int>(sizeof(R) / 16); i += kThreads) dst[i] = reinterpret_cast<const uint4*>(&out)[i];
}

// o of a token and head: row ((segment * count + chunk - first) * kChunk + token) * H + head of vdim floats behind the records.
__host__ __device__ inline int64_t record_count(const b2kv_gla_args& a, const Slice& slice) {
    return static_cast<int64_t>(a.n_segments) * a.H * slice.count;
}

// One place of the ring: the record, then the CTA's part of v in boxes of 32 columns (64-byte swizzle).
constexpr int kBoxBytes = kChunk * kBox * 2;
__host__ __device__ constexpr int v_offset(int record) { return (record + 1023) / 1024 * 1024; }
__host__ __device__ constexpr int place_bytes(int record) { return v_offset(record) + kWarps * kSlab / kBox * kBoxBytes; }

struct Shared {
    alignas(8) uint64_t full[kMaxRing], empty[kMaxRing];
};

template <int kD16>
__global__ void __launch_bounds__(32 * kWarps, 1) gla_state_kernel(const __grid_constant__ CUtensorMap tm_v,
                                                                  const __grid_constant__ b2kv_gla_args a, const Slice slice,
                                                                  int parts, int n_ring, int32_t* dev_status) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ Shared sm;
    using R = Record<kD16>;
    constexpr int kStride = place_bytes(sizeof(R)), kV = v_offset(sizeof(R));
    // (an offset, not a rounded pointer: the compiler has to see that all of this is shared memory)
    uint8_t* const ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int h = static_cast<int>(blockIdx.x) / parts, part = static_cast<int>(blockIdx.x) % parts;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    grid_launch_dependents();
    if (tid == 0) grid_dependency_wait();
    __syncthreads();
    b2kv_row_segment sg;
    if (!segment_place(a, blockIdx.y, sg)) return;  // (reported by the other kernel)
    const int chunks = min((sg.n + kChunk - 1) / kChunk - slice.first, slice.count);
    if (chunks <= 0) return;
    const int v0 = (part * kWarps + warp) * kSlab;  // this warp's first value column
    const int left = a.vdim - part * kWarps * kSlab;
    const int n_warps = min(kWarps, (left + kSlab - 1) / kSlab), boxes = (min(left, kWarps * kSlab) + kBox - 1) / kBox;
    if (tid == 0) {
        for (int i = 0; i < kMaxRing; ++i) {
            mbar_init(&sm.full[i], 1);
            mbar_init(&sm.empty[i], n_warps);
        }
        fence_mbar_init();
    }
    __syncthreads();
    if (warp >= n_warps) return;  // (there are no barriers of the whole CTA from here on)
    bool ok = true;
    const int row0 = sg.row0 + slice.first * kChunk, rows_left = sg.n - slice.first * kChunk;

    const R* const records = reinterpret_cast<const R*>(a.workspace) + (static_cast<int64_t>(blockIdx.y) * a.H + h) * slice.count;
    float* const o_rows = reinterpret_cast<float*>(reinterpret_cast<R*>(a.workspace) + record_count(a, slice)) +
                          ((static_cast<int64_t>(blockIdx.y) * slice.count * kChunk) * a.H + h) * a.vdim;
    auto request = [&](int ci, int slot) {
        uint8_t* const dst = ring + slot * kStride;
        uint64_t* const bar = &sm.full[slot];
        mbar_arrive_expect_tx(bar, sizeof(R) + boxes * kBoxBytes);
        bulk_g2s(dst, records + ci, sizeof(R), bar);
        for (int b = 0; b < boxes; ++b)
            tma_load_2d(dst + kV + b * kBoxBytes, &tm_v, bar, a.v_col + h * a.vdim + part * kWarps * kSlab + b * kBox, row0 + ci * kChunk);
    };
    if (tid == 0)
        for (int i = 0; i < min(n_ring, chunks); ++i) request(i, i);

    // ------------------------------ state: 16 value columns per warp ------------------------------
    const int row = lane >> 2, col = (lane & 3) * 2;  // place of this thread's first accumulator in a tile
    float* const state = a.state + (static_cast<int64_t>(sg.slot) * a.H + h) * a.dim * a.vdim;
    const bool fresh = slice.first == 0 && a.row_pos[sg.row0] == 0;
    float c[2 * kD16][4];  // [tile of 8 key channels]
    auto each_state = [&](auto&& fn) {
#pragma unroll
        for (int j = 0; j < 2 * kD16; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int v = v0 + row + (e >> 1) * 8, d = j * 8 + col + (e & 1);
                fn(c[j][e], static_cast<int64_t>(d) * a.vdim + v, v < a.vdim && d < a.dim);
            }
    };
    each_state([&](float& x, int64_t at, bool live) { x = live && !fresh ? state[at] : 0.f; });

    const int mat = lane >> 3, r8 = lane & 7;
    // ldmatrix row addresses: [token][channel] tiles as they lie (tokens 0-7 | 8-15 outermost), and transposed
    const int plain_t = r8 + 8 * (mat >> 1), plain_c = 8 * (mat & 1);
    const int trans_t = r8 + 8 * (mat & 1), trans_c = 8 * (mat >> 1);
    int slot = 0;
    uint32_t phase = 0;
    for (int ci = 0; ci < chunks; ++ci) {
        const uint8_t* const place = ring + slot * kStride;
        const R& b = *reinterpret_cast<const R*>(place);
        ok = ok && mbar_wait(&sm.full[slot], phase);
        // this warp's half of a box of v: rows of 64 bytes, 16-byte pieces exchanged by row
        const uint32_t v_addr = smem_u32(place + kV + (warp >> 1) * kBoxBytes + plain_t * 64) +
                                (((2 * (warp & 1) + (plain_c >> 3)) ^ ((plain_t >> 1) & 3)) << 4);
        const uint32_t q_addr = smem_u32(&b.q_hi[plain_t][plain_c]), k_addr = smem_u32(&b.k_hi[trans_t][trans_c]);
        constexpr uint32_t kLo = sizeof(b.q_hi);  // from a matrix of leading halves to that of what they leave
        uint32_t vf[4], q_hi[2][4], q_lo[2][4], k_hi[2][4], k_lo[2][4];  // [step of 16 key channels, even or odd]
        float o[2][4] = {};
        auto load = [&](int kk) {
            ldsm4(q_hi[kk & 1], q_addr + kk * 32);
            ldsm4(q_lo[kk & 1], q_addr + kLo + kk * 32);
            ldsm4t(k_hi[kk & 1], k_addr + kk * 32);
            ldsm4t(k_lo[kk & 1], k_addr + kLo + kk * 32);
        };
        ldsm4t(vf, v_addr);
        {
            uint32_t a_hi[4], a_lo[4];
            ldsm4(a_hi, smem_u32(&b.a_hi[plain_t][plain_c]));
            ldsm4(a_lo, smem_u32(&b.a_lo[plain_t][plain_c]));
            load(0);
#pragma unroll
            for (int n = 0; n < 2; ++n) mma16816(o[n], vf, a_hi[2 * n], a_hi[2 * n + 1]);
#pragma unroll
            for (int n = 0; n < 2; ++n) mma16816(o[n], vf, a_lo[2 * n], a_lo[2 * n + 1]);
        }
#pragma unroll
        for (int kk = 0; kk < kD16; ++kk) {
            if (kk + 1 < kD16) load(kk + 1);  // the next step's operands are on their way during this one's products
            uint32_t s_hi[4], s_lo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float(&t)[4] = c[2 * kk + (e >> 1)];
                split2(t[2 * (e & 1)], t[2 * (e & 1) + 1], s_hi[e], s_lo[e]);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float2 d = *reinterpret_cast<const float2*>(&b.decay[(2 * kk + u) * 8 + col]);
                float(&t)[4] = c[2 * kk + u];
                t[0] *= d.x, t[1] *= d.y, t[2] *= d.x, t[3] *= d.y;
            }
            const uint32_t(&qh)[4] = q_hi[kk & 1], (&ql)[4] = q_lo[kk & 1], (&kh)[4] = k_hi[kk & 1], (&kl)[4] = k_lo[kk & 1];
#pragma unroll
            for (int n = 0; n < 2; ++n) mma16816(o[n], s_hi, qh[2 * n], qh[2 * n + 1]);
#pragma unroll
            for (int u = 0; u < 2; ++u) mma16816(c[2 * kk + u], vf, kh[2 * u], kh[2 * u + 1]);
#pragma unroll
            for (int n = 0; n < 2; ++n) mma16816(o[n], s_hi, ql[2 * n], ql[2 * n + 1]);
#pragma unroll
            for (int u = 0; u < 2; ++u) mma16816(c[2 * kk + u], vf, kl[2 * u], kl[2 * u + 1]);
#pragma unroll
            for (int n = 0; n < 2; ++n) mma16816(o[n], s_lo, qh[2 * n], qh[2 * n + 1]);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = ci * kChunk + n * 8 + col + (e & 1), v = v0 + row + (e >> 1) * 8;
                if (v < a.vdim && t < rows_left) o_rows[static_cast<int64_t>(t) * a.H * a.vdim + v] = o[n][e];
            }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.empty[slot]);
        // the place of the chunk before is free when the last warp has left it (one chunk behind: nobody waits long)
        if (tid == 0 && ci > 0 && ci - 1 + n_ring < chunks) {
            const int before = slot == 0 ? n_ring - 1 : slot - 1;
            ok = ok && mbar_wait(&sm.empty[before], (ci - 1) / n_ring & 1);
            request(ci - 1 + n_ring, before);
        }
        __syncwarp();
        if (++slot == n_ring) slot = 0, phase ^= 1;
    }
    each_state([&](float& x, int64_t at, bool live) {
        if (live) state[at] = x;
    });
    if (!ok) {
        // (whoever asked for copies sees to it that they have landed before this memory is given up)
        if (tid == 0)
            for (int i = max(0, chunks - n_ring); i < chunks; ++i) mbar_wait(&sm.full[i % n_ring], (i / n_ring) & 1);
        report_status(dev_status, B2KV_DEV_WAIT_TIMEOUT);
    }
}

// The heads' norm and the gate: one warp per (token, head), eight value columns per lane.
constexpr int kFinishWarps = 8;
template <typename R>
__global__ void __launch_bounds__(32 * kFinishWarps) gla_finish_kernel(const __grid_constant__ b2kv_gla_args a, const Slice slice) {
    const int lane = threadIdx.x & 31, at = static_cast<int>(blockIdx.x) * kFinishWarps + (threadIdx.x >> 5);
    const int t = at / a.H, h = at % a.H, c = lane * 8;
    grid_launch_dependents();
    grid_dependency_wait();
    b2kv_row_segment sg;
    if (!segment_place(a, blockIdx.y, sg)) return;
    if (t >= slice.count * kChunk || slice.first * kChunk + t >= sg.n) return;
    const int64_t row = static_cast<int64_t>(sg.row0) + slice.first * kChunk + t;
    const float* const src = reinterpret_cast<const float*>(reinterpret_cast<const R*>(a.workspace) + record_count(a, slice)) +
                             ((static_cast<int64_t>(blockIdx.y) * slice.count * kChunk + t) * a.H + h) * a.vdim + c;
    const bool mine = c < a.vdim;
    float f[8], sum = 0.f;
    uint4 gate = make_uint4(0u, 0u, 0u, 0u);
    if (mine) {
        *reinterpret_cast<float4*>(f) = *reinterpret_cast<const float4*>(src);
        *reinterpret_cast<float4*>(f + 4) = *reinterpret_cast<const float4*>(src + 4);
        gate = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.y) + row * a.ld_y + a.g_col + h * a.vdim + c);
#pragma unroll
        for (int i = 0; i < 8; i += 4)
            sum = fmaf(f[i], f[i], fmaf(f[i + 1], f[i + 1], fmaf(f[i + 2], f[i + 2], fmaf(f[i + 3], f[i + 3], sum))));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if (!mine) return;
    const float scale = rsqrtf(fmaf(sum, 1.0f / static_cast<float>(a.vdim), a.eps));
    const uint32_t g[4] = {gate.x, gate.y, gate.z, gate.w};
    uint32_t out[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        out[i] = tc::pack_bf16(f[2 * i] * scale * __ldg(a.norm + c + 2 * i) * silu_fast(__uint_as_float(g[i] << 16)),
                               f[2 * i + 1] * scale * __ldg(a.norm + c + 2 * i + 1) * silu_fast(__uint_as_float(g[i] & 0xffff0000u)));
    *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(a.out) + row * a.ld_out + static_cast<int64_t>(h) * a.vdim + c) =
        make_uint4(out[0], out[1], out[2], out[3]);
}

// Row-major bf16 matrix, boxes of kChunk rows.
bool make_map(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int64_t pitch, int box, CUtensorMapSwizzle swizzle) {
    EncodeTiledFn fn = tensor_map_encoder();
    if (fn == nullptr) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(pitch) * 2};
    const cuuint32_t boxes[2] = {static_cast<cuuint32_t>(box), kChunk};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, boxes, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int record_bytes(int dim) {
    return static_cast<int>(dim <= 32 ? sizeof(Record<2>) : (dim <= 64 ? sizeof(Record<4>) : sizeof(Record<8>)));
}

size_t chunk_bytes(int H, int dim, int vdim) {
    return (static_cast<size_t>(record_bytes(dim)) + kChunk * static_cast<size_t>(vdim) * sizeof(float)) * H;
}

int slice_chunks(int H, int dim, int vdim, int n_segments, int max_n) {
    const int chunks = (max_n + kChunk - 1) / kChunk;
    const int fit = static_cast<int>(std::min<size_t>(kSliceBytes / (chunk_bytes(H, dim, vdim) * n_segments), 1u << 20));
    return std::min(chunks, std::max(kMinSlice, fit));
}

template <int kD16>
int launch_chunked(const b2kv_gla_args& a, int32_t* dev_status, void* stream) {
    using R = Record<kD16>;
    const int parts = (a.vdim + kWarps * kSlab - 1) / (kWarps * kSlab);
    const int n_ring = std::min(kMaxRing, (kSmemLimit - 1024) / place_bytes(sizeof(R)));
    const size_t smem = 1024 + static_cast<size_t>(n_ring) * place_bytes(sizeof(R));
    CUtensorMap tv;
    const int64_t cols = std::max(a.v_col, a.g_col) + static_cast<int64_t>(a.H) * a.vdim;
    if (!make_map(&tv, a.y, a.rows, cols, a.ld_y, kBox, CU_TENSOR_MAP_SWIZZLE_64B)) return B2KV_ERR_UNSUPPORTED;
    static int configured[64] = {0};
    int dev = 0;
    B2KV_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return B2KV_ERR_UNSUPPORTED;
    auto kernel = gla_state_kernel<kD16>;
    if (configured[dev] < static_cast<int>(smem)) {
        B2KV_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        configured[dev] = static_cast<int>(smem);
    }
    const int chunks = (a.max_n + kChunk - 1) / kChunk;
    Slice slice{0, slice_chunks(a.H, a.dim, a.vdim, a.n_segments, a.max_n)};
    for (; slice.first < chunks; slice.first += slice.count) {
        const unsigned here = static_cast<unsigned>(std::min(slice.count, chunks - slice.first));
        OverlapLaunch prep(dim3(here, a.H, a.n_segments), kD16 <= 4 ? 32 : 8 * kD16, 0, stream);
        B2KV_CUDA_TRY(cudaLaunchKernelEx(&prep.cfg, gla_prepare_kernel<kD16>, a, slice, dev_status));
        OverlapLaunch walk(dim3(a.H * parts, a.n_segments), 32 * kWarps, smem, stream);
        B2KV_CUDA_TRY(cudaLaunchKernelEx(&walk.cfg, kernel, tv, a, slice, parts, n_ring, dev_status));
        const unsigned pairs = here * kChunk * static_cast<unsigned>(a.H);
        OverlapLaunch finish(dim3((pairs + kFinishWarps - 1) / kFinishWarps, a.n_segments), 32 * kFinishWarps, 0, stream);
        B2KV_CUDA_TRY(cudaLaunchKernelEx(&finish.cfg, gla_finish_kernel<R>, a, slice));
    }
    return B2KV_OK;
}

bool chunked_sizes(int dim, int vdim, int dtype) {
    return dtype == B2KV_DTYPE_BF16 && dim > 0 && dim % 8 == 0 && dim <= 128 && vdim > 0 && vdim % 8 == 0 && vdim <= kMaxVdim;
}

}  // namespace
}  // namespace gla

static size_t workspace_for(int H, int dim, int vdim, int n_segments, int max_n) {
    return static_cast<size_t>(gla::slice_chunks(H, dim, vdim, n_segments, max_n)) * gla::chunk_bytes(H, dim, vdim) * n_segments;
}

// Enough for fewer segments as well: slices are of whole chunks of all segments, so that fewer segments may take a little more.
size_t gla_chunked_workspace(int H, int dim, int vdim, int n_segments, int max_n, int dtype) {
    if (!gla::chunked_sizes(dim, vdim, dtype)) return 0;
    size_t most = 0;
    for (int n = 1; n <= n_segments; ++n) most = std::max(most, workspace_for(H, dim, vdim, n, max_n));
    return most;
}

int gla_chunked(const b2kv_gla_args& a, int32_t* dev_status, void* stream) {
    using namespace gla;
    if (!chunked_sizes(a.dim, a.vdim, a.dtype) || a.n_segments > 65535 || a.H > 65535) return B2KV_ERR_UNSUPPORTED;
    // 16-byte pieces of v, gate and output rows
    if (!aligned16(a.y) || !aligned16(a.out) || a.ld_y % 8 || a.ld_out % 8 || a.v_col % 8 || a.g_col % 8) return B2KV_ERR_UNSUPPORTED;
    if (!aligned16(a.alpha) || a.ld_alpha % 2 || a.q_col % 2 || a.k_col % 2) return B2KV_ERR_UNSUPPORTED;  // pairs of channels
    if (!a.workspace || (reinterpret_cast<uintptr_t>(a.workspace) & 127) ||
        a.workspace_bytes < workspace_for(a.H, a.dim, a.vdim, a.n_segments, a.max_n))
        return B2KV_ERR_WORKSPACE;
    if (a.dim <= 32) return launch_chunked<2>(a, dev_status, stream);
    if (a.dim <= 64) return launch_chunked<4>(a, dev_status, stream);
    return launch_chunked<8>(a, dev_status, stream);
}

}  // namespace b2kv
