// Gated linear recurrences with one decay per head and key channel over a long run of tokens, sixteen tokens at a time on the tensor
// cores (linear_recurrence.cu has the definitions and the walk of a token at a time).  The chunked forms are published: gated linear attention with
// Gated Linear Attention Transformers (Yang et al., 2023), the delta rule with Parallelizing Linear Transformers with the Delta Rule (Yang et al.,
// 2024).  With G_t the products of the decays
// of tokens 0 .. t of a chunk, per key channel, S_0 the state in front of it and G_C the product of all sixteen:
//   K+ = k_t G_t,  Q+ = q_t G_t,  K- = k_t G_C / G_t                                    (formed as products, never as quotients: all <= 1)
//   L[t][i] = beta_t sum_c k_t[c] k_i[c] (decays of i + 1 .. t)[c]  for i < t,  A[t][i] the same with q_t, for i <= t
//   U = (I + L)^-1 B (V - K+ S_0)   (without the delta rule U = V),  O = Q+ S_0 + A U,  S_C = diag(G_C) S_0 + K-^T U
//   prepare   block = (chunk, head), all chunks in parallel, fp32: the three matrices, L, A, (I + L)^-1; written as MMA operands;
//   walk      block = (head, 16 or 32 value columns), chunks in order.  The chain from state to state is P = K+ S_0, U, S: two warps hold
//             sixteen value columns of the transposed state, and the accumulators of each product are the A operand of the next.  Two more
//             form O from the operands that those hand over; one fetches the terms by bulk copies, some chunks ahead.
// What enters a recurrence is fp32.  So every operand is three bf16 pieces, each rounded, and a product six of theirs (what is left
// out is below 2^-26 of it).  The tensor core does not round sums to nearest, which would pull a state that lives long towards zero: what
// a chunk adds to the state is summed from zero and added in fp32, large and small products have accumulators of their own.
// The walk holds half of the state and of the values (exact, and everything is linear in the two), so that no piece rounds up to infinity; to
// stop each one at the largest bf16 instead cost the chain 4 %.
// The walk is a chain: 1.2 us a chunk (0.8 without the delta rule), of which the MMAs of a warp, at eight clocks, are 0.45 (0.2); before, it was
// 285 ns a token on the FMA pipe.  2048 tokens, both kernels: delta rule of 32 / 16 heads of 128 583 / 581 -> 272 / 192 us (the prepare kernel 72 / 35
// of them), gated linear attention of 16 heads 224 -> 126 us.  Error against 64 bits 1.4e-7 (1.4e-7 before), with decays near one 1.7e-7 (4.0e-7).
#include "pieces_mma.cuh"
#include "typed.cuh"

namespace qd {
namespace {

constexpr int kTok = 16, kKeys = 128, kSteps = kKeys / 16;

// A chunk of a head.  Matrices as B operands of mma.sync m16n8k16: two n-tiles to a 16-byte word of a lane, three pieces one after the other.
struct LinearTerms {
    uint4 minus[kSteps][3][32];    // K-: word j for key tiles 2 j, 2 j + 1 (k = tokens)
    uint4 q[kSteps][3][32];        // Q+: word kk for keys 16 kk .. + 15 (n = tokens)
    uint4 a[3][32];                // A (n = t, k = i)
    float less[kKeys];             // G_C - 1
};
struct DeltaTerms : LinearTerms {
    uint4 plus[kSteps][3][32];     // K+, like Q+
    uint4 t[3][32];                // (I + L)^-1 B
};
template <bool DELTA> struct TermsOf { typedef LinearTerms type; };
template <> struct TermsOf<true> { typedef DeltaTerms type; };

struct ChannelParams {
    const float* q; const float* k; const float* g; const float* v; const float* beta; const float* scales;
    float* state; float* out; void* terms; unsigned int* status;
    int tokens, first, heads, kv_heads, vdim, chunks;       // tokens first .. of the run are walked; `tokens` is the end
};

// ----------------------------------------------------------------------------------- prepare
constexpr int kPad = kKeys + 8, kSmallRow = 20;

template <bool DELTA>
__global__ void __launch_bounds__(128) channel_prepare_kernel(const __grid_constant__ ChannelParams p) {
    chain_enter();
    __shared__ __align__(16) float qs[kTok][kPad], ks[kTok][kPad], ds[kTok][kPad];
    __shared__ __align__(16) float lower[kTok][kSmallRow], attend[kTok][kSmallRow], inverse[kTok][kSmallRow];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int chunk = blockIdx.x, head = blockIdx.y, kv = head / (p.heads / p.kv_heads), t0 = p.first + chunk * kTok;
    typedef typename TermsOf<DELTA>::type Terms;
    Terms* out = reinterpret_cast<Terms*>(p.terms) + (size_t)head * p.chunks + chunk;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 4 * i + warp, tok = t0 + r;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f), k = q, d = q;
        if (tok < p.tokens) {
            const size_t at = ((size_t)tok * p.kv_heads + kv) * kKeys + 4 * lane;
            q = load4(p.q + at);
            k = load4(p.k + at);
            d = load4(p.g + ((size_t)tok * p.heads + head) * kKeys + 4 * lane);
            if (DELTA) {
                const float* scale = p.scales + ((size_t)tok * p.kv_heads + kv) * 3;
                const float sk = scale[0], sq = scale[1];
                k.x *= sk; k.y *= sk; k.z *= sk; k.w *= sk;
                q.x *= sq; q.y *= sq; q.z *= sq; q.w *= sq;
            }
        }
        *reinterpret_cast<float4*>(&qs[r][4 * lane]) = q;
        *reinterpret_cast<float4*>(&ks[r][4 * lane]) = k;
        *reinterpret_cast<float4*>(&ds[r][4 * lane]) = d;
    }
    __syncthreads();
    // ---- L and A: a warp to four tokens i, a lane to four channels; the keys, decayed on, against the tokens behind them
    {
        const int first = 4 * ((warp + blockIdx.x) & 3);              // (later groups have less to do: spread over the schedulers)
        float4 w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = *reinterpret_cast<const float4*>(&ks[first + j][4 * lane]);
        for (int row = lane >> 2; row < first; row += 8) attend[row][first + (lane & 3)] = 0.f;       // exact zeros where nothing is seen
#pragma unroll 4
        for (int row = first; row < kTok; ++row) {
            const float4 q = *reinterpret_cast<const float4*>(&qs[row][4 * lane]);
            const float4 k = *reinterpret_cast<const float4*>(&ks[row][4 * lane]);
            const float4 d = *reinterpret_cast<const float4*>(&ds[row][4 * lane]);
            float sums[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float a = 0.f, l = 0.f;
                if (row > first + j) {
                    w[j].x = fmaf(w[j].x, d.x, w[j].x); w[j].y = fmaf(w[j].y, d.y, w[j].y);
                    w[j].z = fmaf(w[j].z, d.z, w[j].z); w[j].w = fmaf(w[j].w, d.w, w[j].w);
                    if (DELTA) l = fmaf(k.w, w[j].w, fmaf(k.z, w[j].z, fmaf(k.y, w[j].y, k.x * w[j].x)));
                }
                if (row >= first + j) a = fmaf(q.w, w[j].w, fmaf(q.z, w[j].z, fmaf(q.y, w[j].y, q.x * w[j].x)));
                sums[j] = a; sums[4 + j] = l;
            }
            // eight (four) sums over the warp: halves are exchanged until a lane has one, which four (eight) lanes then add up
            constexpr int kSums = DELTA ? 8 : 4;
            int lanes = 16;
#pragma unroll
            for (int n = kSums / 2; n >= 1; n >>= 1, lanes >>= 1) {
                const bool upper = lane & lanes;
#pragma unroll
                for (int j = 0; j < n; ++j)
                    sums[j] = (upper ? sums[j + n] : sums[j]) + __shfl_xor_sync(0xffffffffu, upper ? sums[j] : sums[j + n], lanes);
            }
            for (; lanes >= 1; lanes >>= 1) sums[0] += __shfl_xor_sync(0xffffffffu, sums[0], lanes);
            const int which = lane / (32 / kSums);
            if (lane % (32 / kSums) == 0) (which < 4 ? attend : lower)[row][first + (which & 3)] = sums[0];
        }
    }
    __syncthreads();
    // ---- a thread to a channel: products of the decays from the front and from behind, carried as their distance from one
    {
        float plus[kTok], kept[kTok], m = 0.f;
#pragma unroll
        for (int r = 0; r < kTok; ++r) {
            const float d = ds[r][tid];
            m += fmaf(m, d, d);
            plus[r] = fmaf(ks[r][tid], m, ks[r][tid]);
            kept[r] = fmaf(qs[r][tid], m, qs[r][tid]);
        }
        out->less[tid] = m;
        m = 0.f;
#pragma unroll
        for (int r = kTok - 1; r >= 0; --r) {
            const float d = ds[r][tid], k = ks[r][tid];
            ds[r][tid] = fmaf(k, m, k);
            m += fmaf(m, d, d);
            ks[r][tid] = plus[r];
            qs[r][tid] = kept[r];
        }
    }
    if (DELTA && warp == 0 && lane < kTok) {   // (I + L)^-1 by forward substitution, a lane to a column
        float x[kTok];
#pragma unroll
        for (int row = 0; row < kTok; ++row) {
            const float beta = t0 + row < p.tokens ? p.beta[(size_t)(t0 + row) * p.heads + head] : 0.f;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < row; ++i) sum = fmaf(lower[row][i], x[i], sum);
            x[row] = row < lane ? 0.f : (row == lane ? 1.f : 0.f) - beta * sum;
        }
        const float beta = t0 + lane < p.tokens ? p.beta[(size_t)(t0 + lane) * p.heads + head] : 0.f;
#pragma unroll
        for (int row = 0; row < kTok; ++row) inverse[row][lane] = x[row] * beta;
    }
    __syncthreads();
    // ---- operands
    auto rows_n = [&](uint4 (*dst)[32], const float* m, int ld) {     // n = rows, k = columns
        const float2 a = *reinterpret_cast<const float2*>(m + g * ld + 2 * t), b = *reinterpret_cast<const float2*>(m + g * ld + 2 * t + 8);
        const float2 c = *reinterpret_cast<const float2*>(m + (g + 8) * ld + 2 * t), d = *reinterpret_cast<const float2*>(m + (g + 8) * ld + 2 * t + 8);
        const float x[2][4] = {{a.x, a.y, b.x, b.y}, {c.x, c.y, d.x, d.y}};
        const Pieces v = split_tiles3<true>(x[0], x[1]);
        dst[0][lane] = v.p[0]; dst[1][lane] = v.p[1]; dst[2][lane] = v.p[2];
    };
#pragma unroll
    for (int i = 0; i < kSteps / 4; ++i) {
        const int kk = warp + 4 * i;
        rows_n(out->q[kk], &qs[0][16 * kk], kPad);
        if constexpr (DELTA) rows_n(out->plus[kk], &ks[0][16 * kk], kPad);
        const float* m = &ds[0][16 * kk + g];                         // n = keys, k = tokens
        float x[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int c = 0; c < 4; ++c) x[n][c] = m[(2 * t + (c & 1) + 8 * (c >> 1)) * kPad + 8 * n];
        const Pieces v = split_tiles3<true>(x[0], x[1]);
#pragma unroll
        for (int j = 0; j < 3; ++j) out->minus[kk][j][lane] = v.p[j];
    }
    if (warp == 0) rows_n(out->a, &attend[0][0], kSmallRow);
    if constexpr (DELTA)
        if (warp == 1) rows_n(out->t, &inverse[0][0], kSmallRow);
}

// -------------------------------------------------------------------------------------- walk
// A slice is sixteen value columns.  Two warps hold its state, 64 keys each: both form their part of P, add the other's and go on alike.
// (One warp with all keys took 1.8 us a chunk: its instructions wait on one another, not on the tensor cores.)  Two more form the
// results, eight tokens each.
constexpr int kHalfSteps = kSteps / 2, kVRow = 36;                    // floats of a staged row of values: 32 columns and a bank offset
template <bool DELTA> struct ChannelStage { typename TermsOf<DELTA>::type terms; float v[kTok][kVRow]; };
struct ChannelHandover { Pieces s[kSteps][32], u[32]; };
template <bool DELTA, int SLICES> struct ChannelArea {
    static constexpr int kStages = (DELTA ? 3 : 5) + (SLICES == 1);   // as many as fit
    ChannelStage<DELTA> stage[kStages];
    ChannelHandover over[SLICES][2];
    float4 pred[DELTA ? SLICES : 1][2][2][2][32];                     // [chunk & 1][half][n-tile]: a half's part of P
    uint64_t full[kStages], empty[kStages];
};
// Named barriers; a slice has seven: the exchange of P, and state, U, free for even and odd chunks.
constexpr int kBarSlice = 1, kBarState = 1, kBarU = 3, kBarFree = 5;
template <int SLICES> constexpr int walk_threads() { return 128 * SLICES + 32; }

struct Sums { float large[4], small[3][4]; };                         // of leading pieces; of the five other products
QD_DEVINL void products(Sums& s, const uint4 (&a)[3], const uint2 (&b)[3]) {
    mma_bf16(s.large, a[0], b[0].x, b[0].y);
    mma_bf16(s.small[0], a[0], b[2].x, b[2].y);
    mma_bf16(s.small[1], a[1], b[0].x, b[0].y);
    mma_bf16(s.small[2], a[1], b[1].x, b[1].y);
    mma_bf16(s.small[0], a[2], b[0].x, b[0].y);
    mma_bf16(s.small[1], a[0], b[1].x, b[1].y);
}
QD_DEVINL float total(const Sums& s, int c) { return s.large[c] + (s.small[0][c] + (s.small[1][c] + s.small[2][c])); }
// n-tile n of a B operand's word
QD_DEVINL void load_tile(uint2 (&b)[3], const uint4 (*from)[32], int lane, int n) {
#pragma unroll
    for (int j = 0; j < 3; ++j) b[j] = reinterpret_cast<const uint2*>(&from[j][lane])[n];
}
QD_DEVINL bool any_unbounded(const uint4& v) {     // a NaN among third pieces: an infinity or NaN has been split
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    bool found = false;
#pragma unroll
    for (int i = 0; i < 4; ++i) found |= (w[i] & 0x7f80u) == 0x7f80u || (w[i] & 0x7f800000u) == 0x7f800000u;
    return __any_sync(0xffffffffu, found);
}
QD_DEVINL uint4 up_to(const uint4& v, int last, int t) {              // an A operand without its k above `last`
    const auto kept = [&](uint32_t w, int k) { return (k <= last ? w & 0xffffu : 0u) | (k + 1 <= last ? w & 0xffff0000u : 0u); };
    return make_uint4(kept(v.x, 2 * t), kept(v.y, 2 * t), kept(v.z, 2 * t + 8), kept(v.w, 2 * t + 8));
}
// Rows 8 n .. + 7 of a 16 x 16 lower triangular matrix (B operand b) times sixteen tokens' vectors (A operand a, k = token), added
// to sum.  Zero times an infinity is NaN, so where a token has one every row is formed from the tokens that it sees.
QD_DEVINL void triangular(float (&sum)[4], const uint4 (&a)[3], const uint2 (&b)[3], int n, int t, bool unbounded) {
    if (!unbounded) {
        Sums s = {};
        products(s, a, b);
#pragma unroll
        for (int c = 0; c < 4; ++c) sum[c] += total(s, c);
        return;
    }
#pragma unroll 1
    for (int row = 8 * n; row < 8 * n + 8; ++row) {
        const uint4 seen[3] = {up_to(a[0], row, t), up_to(a[1], row, t), up_to(a[2], row, t)};
        Sums s = {};
        products(s, seen, b);
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (8 * n + 2 * t + (c & 1) == row) sum[c] += total(s, c);
    }
}

template <bool DELTA, int SLICES>
__global__ void __launch_bounds__(walk_threads<SLICES>(), 1) channel_walk_kernel(const __grid_constant__ ChannelParams p) {
    chain_enter();
    extern __shared__ __align__(16) unsigned char area[];
    typedef ChannelArea<DELTA, SLICES> Area;
    constexpr int kStages = Area::kStages;
    Area& s = *reinterpret_cast<Area*>(area);
    const int head = blockIdx.x, c0 = blockIdx.y * 16 * SLICES;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int slice = (warp >> 1) % SLICES, half = warp & 1, bar = kBarSlice + 7 * slice, chunks = p.chunks;
    const size_t stride = (size_t)p.heads * p.vdim;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) { mbar_init(s.full + i, 1 + 32); mbar_init(s.empty + i, 4 * SLICES); }
        mbar_fence_init();
    }
    __syncthreads();

    if (warp == 4 * SLICES) {                  // ---- copies; a wait that runs out ends the warp with none of its own in flight
        typedef typename TermsOf<DELTA>::type Terms;
        const Terms* mine = reinterpret_cast<const Terms*>(p.terms) + (size_t)head * chunks;
        constexpr uint32_t kBytes = (uint32_t)sizeof(Terms);
        const float* from = p.v + (size_t)p.first * stride + (size_t)head * p.vdim + c0;
        int issued = 0;
        bool ok = true;
#pragma unroll 1
        for (; issued < chunks; ++issued) {
            const int at = issued % kStages;
            ChannelStage<DELTA>& st = s.stage[at];
            if (issued >= kStages) ok = mbar_wait(s.empty + at, (issued / kStages - 1) & 1, p.status);
            if (!__all_sync(0xffffffffu, ok)) break;
            const int rows = min(kTok, p.tokens - (p.first + issued * kTok));
            if (lane == 0) {
                mbar_expect_tx(s.full + at, kBytes);
                bulk_load(&st.terms, mine + issued, kBytes, s.full + at);
            }
            // the values in 16-byte pieces (a bulk copy for each of their short rows kept the copy unit busy for longer than a chunk
            // takes); zeros for tokens that are not there.  The barrier counts a lane when its pieces have come.
#pragma unroll
            for (int i = 0; i < 2 * SLICES; ++i) {
                const int piece = lane + 32 * i, r = piece / (4 * SLICES), c = 4 * (piece % (4 * SLICES));
                copy16(smem_u32(&st.v[r][c]), from + (size_t)(issued * kTok + min(r, rows - 1)) * stride + c, r < rows, true);
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(s.full + at)) : "memory");
        }
        for (int i = issued > kStages ? issued - kStages : 0; i < issued; ++i)
            mbar_wait(s.full + i % kStages, (i / kStages) & 1, p.status);
        return;
    }
    bool there = true;         // after a wait that ran out (the status says so) nothing is waited for; the named barriers go on
    if (warp < 2 * SLICES) {
        float acc[8][4];                       // state: column c0 + 16 slice + g + 8 (c >> 1), key 64 half + 8 nt + 2 t + (c & 1)
        float* tile = p.state + ((size_t)head * kKeys + 64 * half) * p.vdim + c0 + 16 * slice + g;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[nt][c] = 0.5f * tile[(size_t)(8 * nt + 2 * t + (c & 1)) * p.vdim + 8 * (c >> 1)];
        bool ahead = false;                    // the next chunk's terms are there: asked for under this one's products (a look takes 200 clocks)
#pragma unroll 1
        for (int chunk = 0; chunk < chunks; ++chunk) {
            const ChannelStage<DELTA>& st = s.stage[chunk % kStages];
            const int odd = chunk & 1;
            ChannelHandover& over = s.over[slice][odd];
            if (there)
                there = __all_sync(0xffffffffu, ahead) || __all_sync(0xffffffffu, mbar_wait(s.full + chunk % kStages, (chunk / kStages) & 1, p.status));
            if (chunk >= 2) named_barrier(bar + kBarFree + odd, 128);         // the results of two chunks ago are formed
            // ---- U = V, or (I + L)^-1 B (V - K+ S_0), transposed; the state is handed over on the way
            float u[2][4];
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int c = 0; c < 4; ++c) u[n][c] = 0.5f * st.v[8 * n + 2 * t + (c & 1)][16 * slice + g + 8 * (c >> 1)];
            if constexpr (DELTA) {
                Sums sum[2] = {};
                uint2 b[2][2][3];
                load_tile(b[0][0], st.terms.plus[kHalfSteps * half], lane, 0);
                load_tile(b[0][1], st.terms.plus[kHalfSteps * half], lane, 1);
#pragma unroll
                for (int kk = 0; kk < kHalfSteps; ++kk) {
                    if (kk + 1 < kHalfSteps) {
                        load_tile(b[(kk + 1) & 1][0], st.terms.plus[kHalfSteps * half + kk + 1], lane, 0);
                        load_tile(b[(kk + 1) & 1][1], st.terms.plus[kHalfSteps * half + kk + 1], lane, 1);
                    }
                    const Pieces v = split_tiles3(acc[2 * kk], acc[2 * kk + 1]);
                    products(sum[0], v.p, b[kk & 1][0]);
                    products(sum[1], v.p, b[kk & 1][1]);
                    over.s[kHalfSteps * half + kk][lane] = v;
                }
                named_arrive(bar + kBarState + odd, 128);
                float own[2][4];
#pragma unroll
                for (int n = 0; n < 2; ++n) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) own[n][c] = total(sum[n], c);
                    s.pred[slice][odd][half][n][lane] = make_float4(own[n][0], own[n][1], own[n][2], own[n][3]);
                }
                named_barrier(bar, 64);
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    const float4 other = s.pred[slice][odd][half ^ 1][n][lane];
                    u[n][0] -= own[n][0] + other.x; u[n][1] -= own[n][1] + other.y;
                    u[n][2] -= own[n][2] + other.z; u[n][3] -= own[n][3] + other.w;
                }
                const Pieces r = split_tiles3(u[0], u[1]);
                const bool unbounded = any_unbounded(r.p[2]);
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    uint2 inverse[3];
                    load_tile(inverse, st.terms.t, lane, n);
#pragma unroll
                    for (int c = 0; c < 4; ++c) u[n][c] = 0.f;
                    triangular(u[n], r.p, inverse, n, t, unbounded);
                }
            } else {
#pragma unroll
                for (int kk = 0; kk < kHalfSteps; ++kk) over.s[kHalfSteps * half + kk][lane] = split_tiles3(acc[2 * kk], acc[2 * kk + 1]);
                named_arrive(bar + kBarState + odd, 128);
            }
            const Pieces w = split_tiles3(u[0], u[1]);
            if (half == 0) over.u[lane] = w;
            named_arrive(bar + kBarU + odd, 128);
            // ---- S = diag(G_C) S_0 + K-^T U, transposed: four key tiles at a time
            ahead = mbar_test_wait(s.full + (chunk + 1) % kStages, ((chunk + 1) / kStages) & 1);
            uint4 b[2][2][3];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int j = 0; j < 3; ++j) b[0][h][j] = st.terms.minus[kHalfSteps * half + h][j][lane];
#pragma unroll
            for (int step = 0; step < kHalfSteps / 2; ++step) {
                const uint4(&cur)[2][3] = b[step & 1];
                if (step + 1 < kHalfSteps / 2) {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int j = 0; j < 3; ++j) b[(step + 1) & 1][h][j] = st.terms.minus[kHalfSteps * half + 2 * (step + 1) + h][j][lane];
                }
                float d[4][4] = {};
                constexpr int kLeft[6] = {1, 2, 0, 1, 0, 0}, kRight[6] = {1, 0, 2, 0, 1, 0};       // small products first
#pragma unroll
                for (int i = 0; i < 6; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        mma_bf16(d[2 * h], w.p[kLeft[i]], cur[h][kRight[i]].x, cur[h][kRight[i]].y);
                        mma_bf16(d[2 * h + 1], w.p[kLeft[i]], cur[h][kRight[i]].z, cur[h][kRight[i]].w);
                    }
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    const float2 less = *reinterpret_cast<const float2*>(&st.terms.less[64 * half + 8 * (4 * step + n) + 2 * t]);
                    float(&x)[4] = acc[4 * step + n];
                    x[0] += fmaf(x[0], less.x, d[n][0]);
                    x[1] += fmaf(x[1], less.y, d[n][1]);
                    x[2] += fmaf(x[2], less.x, d[n][2]);
                    x[3] += fmaf(x[3], less.y, d[n][3]);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(s.empty + chunk % kStages);
        }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int c = 0; c < 4; ++c) tile[(size_t)(8 * nt + 2 * t + (c & 1)) * p.vdim + 8 * (c >> 1)] = 2.f * acc[nt][c];
        return;
    }
    // ---- results of tokens 8 half .. + 7 of a chunk
    float* to = p.out + (size_t)(p.first + 8 * half + 2 * t) * stride + (size_t)head * p.vdim + c0 + 16 * slice + g;
#pragma unroll 1
    for (int chunk = 0; chunk < chunks; ++chunk, to += kTok * stride) {
        const ChannelStage<DELTA>& st = s.stage[chunk % kStages];
        const int odd = chunk & 1;
        const ChannelHandover& over = s.over[slice][odd];
        if (there) there = __all_sync(0xffffffffu, mbar_wait(s.full + chunk % kStages, (chunk / kStages) & 1, p.status));
        uint2 b[2][3], attend[3];
        Pieces v[2];
        load_tile(b[0], st.terms.q[0], lane, half);
        load_tile(attend, st.terms.a, lane, half);
        named_barrier(bar + kBarState + odd, 128);
        Sums sum[2] = {};
        v[0] = over.s[0][lane];
#pragma unroll
        for (int kk = 0; kk < kSteps; ++kk) {
            if (kk + 1 < kSteps) {
                load_tile(b[(kk + 1) & 1], st.terms.q[kk + 1], lane, half);
                v[(kk + 1) & 1] = over.s[kk + 1][lane];
            }
            products(sum[kk & 1], v[kk & 1].p, b[kk & 1]);
        }
        float o[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) o[c] = total(sum[0], c) + total(sum[1], c);
        named_barrier(bar + kBarU + odd, 128);
        const Pieces u = over.u[lane];
        triangular(o, u.p, attend, half, t, any_unbounded(u.p[2]));
        if (chunk + 2 < chunks) named_arrive(bar + kBarFree + odd, 128);
        __syncwarp();
        if (lane == 0) mbar_arrive(s.empty + chunk % kStages);
        const int left = p.tokens - (p.first + chunk * kTok + 8 * half + 2 * t);
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if ((c & 1) < left) to[(c & 1) * stride + 8 * (c >> 1)] = 2.f * o[c];
    }
}

// Chunks whose terms fit the scratch area at once: 96 MB of them are still in L2 when they are walked.
int chunks_at_once(int heads) {
    const long long fit = (96ll << 20) / ((long long)heads * (long long)sizeof(DeltaTerms));
    return fit < 4 ? 4 : (int)fit;
}

template <bool DELTA, int SLICES>
int launch_walk(const ChannelParams& p, cudaStream_t stream) {
    if (!allow_smem(channel_walk_kernel<DELTA, SLICES>, sizeof(ChannelArea<DELTA, SLICES>))) return QD_ERR_LAUNCH;
    return qd_launch(channel_walk_kernel<DELTA, SLICES>, dim3(p.heads, p.vdim / (16 * SLICES)), dim3(walk_threads<SLICES>()), sizeof(ChannelArea<DELTA, SLICES>),
                     stream, 1, p);
}

template <bool DELTA>
int channel_recurrence(ChannelParams p, cudaStream_t stream) {
    const int tokens = p.tokens, at_once = chunks_at_once(p.heads);
    // two slices to a block read a head's terms half as often; one slice where that leaves SMs without a block
    const bool two = p.vdim % 32 == 0 && p.heads * (p.vdim / 16) > device_sms();
    for (p.first = 0; p.first < tokens; p.first += at_once * kTok) {
        p.tokens = tokens - p.first < at_once * kTok ? tokens : p.first + at_once * kTok;
        p.chunks = (p.tokens - p.first + kTok - 1) / kTok;
        int rc = qd_launch(channel_prepare_kernel<DELTA>, dim3(p.chunks, p.heads), dim3(128), 0, stream, 1, p);
        if (rc == QD_OK) rc = two ? launch_walk<DELTA, 2>(p, stream) : launch_walk<DELTA, 1>(p, stream);
        if (rc != QD_OK) return rc;
    }
    return QD_OK;
}

}  // namespace
}  // namespace qd

extern "C" long long qd_channel_chunk_scratch_bytes(int tokens, int heads) {
    if (tokens <= 0 || heads <= 0) return 0;
    const long long chunks = (tokens + qd::kTok - 1) / qd::kTok, most = qd::chunks_at_once(heads);
    return (chunks < most ? chunks : most) * heads * (long long)sizeof(qd::DeltaTerms);
}

extern "C" int qd_channel_recurrence_chunked(const float* q, const float* k, const float* g, const float* v, const float* beta, const float* scales,
                                             float* state, float* out, int tokens, int heads, int kv_heads, int dim, int vdim, int delta,
                                             void* scratch, unsigned int* status, void* stream) {
    QD_CHECK_ARG(q && k && g && v && state && out && scratch && tokens > 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dim > 0 && vdim > 0);
    QD_CHECK_ARG(!delta || (beta && scales));
    if (dim != qd::kKeys || vdim % 16 || heads > 65535 || tokens > (1 << 30)) return QD_ERR_UNSUPPORTED;
    if (!qd::aligned16(q) || !qd::aligned16(k) || !qd::aligned16(g) || !qd::aligned16(v) || !qd::aligned16(scratch)) return QD_ERR_UNSUPPORTED;
    const qd::ChannelParams p = {q, k, g, v, beta, scales, state, out, scratch, status, tokens, 0, heads, kv_heads, vdim, 0};
    return delta ? qd::channel_recurrence<true>(p, (cudaStream_t)stream) : qd::channel_recurrence<false>(p, (cudaStream_t)stream);
}
