// Gated delta rule over a long run of tokens, 64 tokens at a time on the tensor cores.
//
// The reference walks a prompt token by token (quickdraw/kernel/triton/delta.py:57-81: per
// token S *= decay; pred = S^T k; S += k (x) beta (v - pred); out = S^T q), and so does the
// sequence kernel of seq.cu: about 750 clocks per token whatever the width, because every token
// waits for the one before.  Within a chunk of C = 64 tokens the same recurrence has a closed
// form.  With g_t the product of the decays of tokens 0..t of the chunk, u_t = beta_t (v_t - pred_t)
// and S_0 the state at the start of the chunk:
//   (I + L) U = B (V - G K S_0),   L[t][i] = beta_t (g_t / g_i) (k_t . k_i)  for i < t
//   O = G Q S_0 + A U,              A[t][i] = (g_t / g_i) (q_t . k_i)         for i <= t
//   S_C = g_C S_0 + (K scaled by g_C / g_t)^T U
// (B = diag(beta), G = diag(g)).  Two kernels:
//   prepare     block = (chunk, key head), all chunks in parallel: K K^T and Q K^T once for the value heads that share the
//               key head, then for each of them L, A, T = (I + L)^-1 (16 x 16 diagonal blocks by forward substitution in fp32, the
//               blocks below by products) and the factors of the rows; T B and A go to a scratch area as MMA fragments;
//   recurrence  block = (value head, 32 value columns), chunks in order.  What bounds a chunk is the chain from one state to the
//               next, R = V - G K S_0, U = (T B) R, S = g_C S_0 + K^T (U scaled by g_C / g_t), so one warp holds sixteen value columns of
//               the transposed state whole and walks that chain without a block-wide barrier: the accumulators of each product
//               are, register for register, the A operand of the next (rows = value columns).  A second warp forms
//               O = G Q S_0 + A U from the same operands, handed over in shared memory.  Four warps, one to an SM sub-partition.
// Keys and queries enter as the bf16 that they are, their norms as factors of rows of the sums; every fp32 operand (S, R, U, T B, A) is
// two bf16 pieces of eight significant bits each, three products where both sides have two.  Before, all operands were rounded to
// tf32 (11 bits) and every product went through shared memory in 16 x 16 warp tiles behind five barriers a chunk.  16 key and 32 value heads of
// 128, both kernels, before and now: 64 tokens 25 -> 15 us, 511 68 -> 37, 2048 259 -> 99, 8192 1016 -> 353 us; error of the state against 64 bits
// after 2048 tokens 3.5e-4 -> 7e-6.  A chunk of the recurrence takes 2.4 us, of which the MMAs of a walking warp are 1.3 (316 at eight clocks).
#include "pieces_mma.cuh"

namespace qd {
namespace {

constexpr int kC = 64;             // tokens per chunk
constexpr int kDK = 128;           // key dimension
constexpr int kCols = 32;          // value columns per recurrence block
constexpr int kTri = 10;           // 16 x 16 blocks on and below the diagonal of a 64 x 64 matrix

// What a chunk of a value head has in the scratch area.  A block of T B or A: the B operand fragments of two n-tiles (rows of the
// matrix 0 - 7, 8 - 15 of the block), one 16-byte word a lane, the leading pieces and then the following ones.
struct ChunkTerms {
    uint4 tb[kTri][2][32];
    float pred[kC];                // g_t |k_t|^-1: rows of K S_0
    float keep[kC];                // g_C / g_t |k_t|^-1: rows of U for the state
    float end[4];                  // g_C
    uint4 a[kTri][2][32];
    float read[kC];                // g_t |q_t|^-1 128^-0.5: rows of Q S_0
};
static_assert(sizeof(ChunkTerms) % 16 == 0, "copied in 16-byte pieces");

// log of the decay of one token (<= 0)
QD_DEVINL float log_decay(float a, float a_log, float bias) { return -expf(a_log) * softplus_precise(a + bias); }

QD_DEVINL int block_of(int row, int col) { return row * (row + 1) / 2 + col; }

// A chunk's rows of one head of keys or queries -> [64][128] bf16 in shared memory, 16-byte pieces p of row r at p ^ (r & 7).
template <int THREADS>
QD_DEVINL void copy_rows(uint32_t dst, const bf16* first, int t_base, int tokens, int channels, int tid, bool wide) {
    const int piece = tid & 15;
#pragma unroll
    for (int i = 0; i < kC * 16 / THREADS; ++i) {
        const int r = tid / 16 + i * (THREADS / 16), tok = min(t_base + r, tokens - 1);
        copy16(dst + r * 256 + ((piece ^ (r & 7)) << 4), first + (size_t)tok * channels + piece * 8, t_base + r < tokens, wide);
    }
}

// ------------------------------------------------------------------------------- prepare
// Eight warps; warps 0 - 3 and 4 - 7 invert the matrices of one value head each.
constexpr int kPrepThreads = 256, kDiagRow = 20;
struct PrepareArea {
    union {
        struct { uint4 k[kC * 16], q[kC * 16]; };                     // the rows, until their products are formed
        struct {
            uint4 l[2][6][2][32];                                     // blocks of L below the diagonal, as fragments
            float diag[2][4][16][kDiagRow], inv[2][4][16][kDiagRow];  // its diagonal blocks and their inverses
        };
    };
    float kscale[kC], qscale[kC];
    float cum[2][kC], beta[2][kC];
};

__global__ void __launch_bounds__(kPrepThreads, 3)
gdn_chunk_prepare_kernel(const bf16* __restrict__ qkv, const bf16* __restrict__ a, const bf16* __restrict__ b,
                         const bf16* __restrict__ a_log, const bf16* __restrict__ dt_bias, ChunkTerms* __restrict__ terms,
                         int tokens, int hk, int hv, int dv, int wide) {
    chain_enter();
    __shared__ __align__(16) PrepareArea s;
    const int chunk = blockIdx.x, key_head = blockIdx.y, chunks = gridDim.x, share = hv / hk;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int channels = 2 * hk * kDK + hv * dv, t_base = chunk * kC;
    const uint32_t ks = smem_u32(s.k), qs = smem_u32(s.q);
    copy_rows<kPrepThreads>(ks, qkv + (size_t)(hk + key_head) * kDK, t_base, tokens, channels, tid, wide);
    copy_rows<kPrepThreads>(qs, qkv + (size_t)key_head * kDK, t_base, tokens, channels, tid, wide);
    copies_commit();
    copies_wait<0>();
    __syncthreads();
    {                                          // norms: four threads to a row
        const int r = tid >> 2;
        float kk = 0.f, qq = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 kv = s.k[r * 16 + 4 * i + (tid & 3)], qv = s.q[r * 16 + 4 * i + (tid & 3)];
            const uint32_t kw[4] = {kv.x, kv.y, kv.z, kv.w}, qw[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float k0 = __uint_as_float(kw[j] << 16), k1 = __uint_as_float(kw[j] & 0xffff0000u);
                const float q0 = __uint_as_float(qw[j] << 16), q1 = __uint_as_float(qw[j] & 0xffff0000u);
                kk += k0 * k0 + k1 * k1;
                qq += q0 * q0 + q1 * q1;
            }
        }
        kk = group_sum<4>(kk);
        qq = group_sum<4>(qq);
        if ((tid & 3) == 0) { s.kscale[r] = rsqrtf(kk + 1e-6f); s.qscale[r] = rsqrtf(qq + 1e-6f) * 0.08838834764831845f; }
    }
    // ---- K K^T and Q K^T: warp = (16 rows, two blocks of 16 columns); what lies above the diagonal is not needed
    const int mt = warp & 3, c0 = 2 * (warp >> 2);
    float g1[4][4], g2[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < 4; ++c) { g1[j][c] = 0.f; g2[j][c] = 0.f; }
    if (c0 <= mt) {
        const int sub = lane & 7;
        const uint32_t rows_a = (uint32_t)(16 * mt + (lane & 15)) * 256, rows_b = (uint32_t)(16 * c0 + 8 * (lane >> 4) + sub) * 256;
#pragma unroll
        for (int kk = 0; kk < kDK / 16; ++kk) {
            const uint32_t at_a = rows_a + (((2 * kk + (lane >> 4)) ^ sub) << 4), at_b = rows_b + (((2 * kk + ((lane >> 3) & 1)) ^ sub) << 4);
            const uint4 ka = ldsm(ks + at_a), qa = ldsm(qs + at_a);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                if (c0 + half > mt) continue;
                const uint4 kb = ldsm(ks + at_b + half * 16 * 256);
                mma_bf16(g1[2 * half], ka, kb.x, kb.y);
                mma_bf16(g1[2 * half + 1], ka, kb.z, kb.w);
                mma_bf16(g2[2 * half], qa, kb.x, kb.y);
                mma_bf16(g2[2 * half + 1], qa, kb.z, kb.w);
            }
        }
    }
    const int group = warp >> 2, column = warp & 3;
#pragma unroll 1
    for (int first = 0; first < share; first += 2) {
        const bool mine = first + group < share;                      // the same for a whole group of warps
        const int head = key_head * share + first + group;
        ChunkTerms* out = terms + ((size_t)head * chunks + chunk);
        if (mine && column == 0) {             // decays and their running sums, two tokens to a lane
            float lg[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int tok = t_base + 2 * lane + i;
                const bool there = tok < tokens;
                lg[i] = there ? log_decay(ld_bf16(a + (size_t)tok * hv + head), ld_bf16(a_log + head), ld_bf16(dt_bias + head)) : 0.f;
                s.beta[group][2 * lane + i] = there ? sigmoid_precise(ld_bf16(b + (size_t)tok * hv + head)) : 0.f;
            }
            float run = lg[0] + lg[1];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) { const float up = __shfl_up_sync(0xffffffffu, run, d); if (lane >= d) run += up; }
            s.cum[group][2 * lane] = run - lg[1];
            s.cum[group][2 * lane + 1] = run;
        }
        __syncthreads();                       // also: the rows are read (first pass), the area is free (later ones)
        if (mine && column < 2) {              // factors of the rows
            const int tok = 32 * column + lane;
            const float cum = s.cum[group][tok], total = s.cum[group][kC - 1];
            out->pred[tok] = expf(cum) * s.kscale[tok];
            out->keep[tok] = expf(total - cum) * s.kscale[tok];
            out->read[tok] = expf(cum) * s.qscale[tok];
            if (tok < 4) out->end[tok] = expf(total);
        }
        // ---- L to shared memory, A to the scratch area
#pragma unroll 1
        for (int h = 0; h < 2 && first + h < share; ++h) {
            ChunkTerms* dst = terms + ((size_t)(key_head * share + first + h) * chunks + chunk);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int kb = c0 + half;
                if (kb > mt) continue;
                float lv[2][4], av[2][4];
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int row = 16 * mt + g + 8 * (c >> 1), col = 16 * kb + 8 * j + 2 * t + (c & 1);
                        const float ratio = col <= row ? expf(s.cum[h][row] - s.cum[h][col]) * s.kscale[col] : 0.f;
                        lv[j][c] = col < row ? s.beta[h][row] * ratio * s.kscale[row] * g1[2 * half + j][c] : 0.f;
                        av[j][c] = col <= row ? ratio * s.qscale[row] * g2[2 * half + j][c] : 0.f;
                    }
                uint4 hi, lo;                  // {n-tile 0: inputs 0 - 7, 8 - 15; n-tile 1: the same}
                split_pair(av[0][0], av[0][1], hi.x, lo.x);
                split_pair(av[1][0], av[1][1], hi.y, lo.y);
                split_pair(av[0][2], av[0][3], hi.z, lo.z);
                split_pair(av[1][2], av[1][3], hi.w, lo.w);
                dst->a[block_of(mt, kb)][0][lane] = hi;
                dst->a[block_of(mt, kb)][1][lane] = lo;
                if (kb < mt) {
                    split_pair(lv[0][0], lv[0][1], hi.x, lo.x);
                    split_pair(lv[1][0], lv[1][1], hi.y, lo.y);
                    split_pair(lv[0][2], lv[0][3], hi.z, lo.z);
                    split_pair(lv[1][2], lv[1][3], hi.w, lo.w);
                    s.l[h][block_of(mt - 1, kb)][0][lane] = hi;
                    s.l[h][block_of(mt - 1, kb)][1][lane] = lo;
                } else {
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int c = 0; c < 4; ++c) s.diag[h][mt][g + 8 * (c >> 1)][8 * j + 2 * t + (c & 1)] = lv[j][c];
                }
            }
        }
        __syncthreads();
        // ---- inverses of the diagonal blocks of I + L: a thread to a column
        if (mine && column < 2) {
            const int block = 2 * column + (lane >> 4), col = lane & 15;
            float x[16];
#pragma unroll
            for (int row = 0; row < 16; ++row) {
                float sum = row == col ? 1.f : 0.f;
#pragma unroll
                for (int i = 0; i < row; i += 4) {
                    const float4 l = *reinterpret_cast<const float4*>(&s.diag[group][block][row][i]);
                    sum -= l.x * x[i];
                    if (i + 1 < row) sum -= l.y * x[i + 1];
                    if (i + 2 < row) sum -= l.z * x[i + 2];
                    if (i + 3 < row) sum -= l.w * x[i + 3];
                }
                x[row] = sum;
            }
#pragma unroll
            for (int row = 0; row < 16; ++row) s.inv[group][block][row][col] = x[row];
        }
        __syncthreads();
        // ---- the blocks below: warp = column of blocks j, transposed, T_ij' = -(sum over k of T_kj' L_ik') T_ii' for i = j + 1 .. 3
        if (mine) {
            const int j = column;
            const float* beta = s.beta[group] + 16 * j;
            uint4 thi[3], tlo[3];              // T_kj' as A operands, k = j ..
            {
                const auto& inv = s.inv[group][j];
                uint4 hi, lo;
                split_pair(inv[g][2 * t] * beta[2 * t], inv[g][2 * t + 1] * beta[2 * t + 1], hi.x, lo.x);
                split_pair(inv[g][2 * t + 8] * beta[2 * t + 8], inv[g][2 * t + 9] * beta[2 * t + 9], hi.y, lo.y);
                split_pair(inv[g + 8][2 * t] * beta[2 * t], inv[g + 8][2 * t + 1] * beta[2 * t + 1], hi.z, lo.z);
                split_pair(inv[g + 8][2 * t + 8] * beta[2 * t + 8], inv[g + 8][2 * t + 9] * beta[2 * t + 9], hi.w, lo.w);
                out->tb[block_of(j, j)][0][lane] = hi;
                out->tb[block_of(j, j)][1][lane] = lo;
                split_pair(inv[2 * t][g], inv[2 * t + 1][g], thi[0].x, tlo[0].x);
                split_pair(inv[2 * t][g + 8], inv[2 * t + 1][g + 8], thi[0].y, tlo[0].y);
                split_pair(inv[2 * t + 8][g], inv[2 * t + 9][g], thi[0].z, tlo[0].z);
                split_pair(inv[2 * t + 8][g + 8], inv[2 * t + 9][g + 8], thi[0].w, tlo[0].w);
            }
#pragma unroll
            for (int d = 1; d < 4; ++d) {
                const int i = j + d;
                if (i > 3) break;
                float x[2][4] = {}, y[2][4] = {};
#pragma unroll
                for (int e = 0; e < d; ++e) {
                    const uint4 bh = s.l[group][block_of(i - 1, j + e)][0][lane], bl = s.l[group][block_of(i - 1, j + e)][1][lane];
                    mma_bf16(x[0], thi[e], bh.x, bh.y);
                    mma_bf16(x[1], thi[e], bh.z, bh.w);
                    mma_bf16(x[0], tlo[e], bh.x, bh.y);
                    mma_bf16(x[1], tlo[e], bh.z, bh.w);
                    mma_bf16(x[0], thi[e], bl.x, bl.y);
                    mma_bf16(x[1], thi[e], bl.z, bl.w);
                }
                uint4 xh, xl, bh, bl;
                split_tiles(x[0], x[1], xh, xl);
                const auto& inv = s.inv[group][i];
                split_pair(inv[g][2 * t], inv[g][2 * t + 1], bh.x, bl.x);
                split_pair(inv[g][2 * t + 8], inv[g][2 * t + 9], bh.y, bl.y);
                split_pair(inv[g + 8][2 * t], inv[g + 8][2 * t + 1], bh.z, bl.z);
                split_pair(inv[g + 8][2 * t + 8], inv[g + 8][2 * t + 9], bh.w, bl.w);
                mma_bf16(y[0], xh, bh.x, bh.y);
                mma_bf16(y[1], xh, bh.z, bh.w);
                mma_bf16(y[0], xl, bh.x, bh.y);
                mma_bf16(y[1], xl, bh.z, bh.w);
                mma_bf16(y[0], xh, bl.x, bl.y);
                mma_bf16(y[1], xh, bl.z, bl.w);
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int c = 0; c < 4; ++c) y[n][c] = -y[n][c];
                if (d < 3) split_tiles(y[0], y[1], thi[d], tlo[d]);
                const float b_lo = beta[g], b_hi = beta[g + 8];       // rows of the transposed block are columns of T
                uint4 hi, lo;
                split_pair(y[0][0] * b_lo, y[0][1] * b_lo, hi.x, lo.x);
                split_pair(y[0][2] * b_hi, y[0][3] * b_hi, hi.y, lo.y);
                split_pair(y[1][0] * b_lo, y[1][1] * b_lo, hi.z, lo.z);
                split_pair(y[1][2] * b_hi, y[1][3] * b_hi, hi.w, lo.w);
                out->tb[block_of(i, j)][0][lane] = make_uint4(transposed(hi.x), transposed(hi.y), transposed(hi.z), transposed(hi.w));
                out->tb[block_of(i, j)][1][lane] = make_uint4(transposed(lo.x), transposed(lo.y), transposed(lo.z), transposed(lo.w));
            }
        }
        __syncthreads();                       // the next heads write over what was read
    }
}

// ---------------------------------------------------------------------------- recurrence
// Warps 0, 1 walk the states of sixteen value columns each; warps 2, 3 form their results and, having fewer MMAs, also fetch what both
// need, two chunks ahead.  Operands of the walk are read one step before their products, since nothing else hides the latency:
// a scheduler has one warp.
constexpr int kRecThreads = 128, kStages = 3;
struct Stage { uint4 k[kC * 16], q[kC * 16], v[kC * 4]; ChunkTerms terms; };
struct Handover { uint4 s[kDK / 16][2][32], u[kC / 16][2][32]; };     // A operands, leading and following pieces
struct RecurrenceArea {
    Stage stage[kStages];
    Handover over[2][2];                       // [columns][chunk & 1]
    uint4 rows[2][kC * 2];                     // results of a chunk, sixteen columns a row
};
// Named barriers; a pair of a walking and a reading warp has six: state, U, free, each for even and odd chunks.
enum { kBarFilled = 1, kBarRead = 2, kBarPair = 3 };

__global__ void __launch_bounds__(kRecThreads, 1)
gdn_chunk_recurrence_kernel(const bf16* __restrict__ qkv, float* __restrict__ state, bf16* __restrict__ out,
                            const ChunkTerms* __restrict__ terms, int tokens, int hk, int hv, int dv, int wide, int wide_out) {
    chain_enter();
    extern __shared__ __align__(16) unsigned char area[];
    RecurrenceArea& s = *reinterpret_cast<RecurrenceArea*>(area);
    const int head = blockIdx.x, c0 = blockIdx.y * kCols;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, sub = lane & 7;
    const int pair = warp & 1;
    const int key_head = head / (hv / hk), channels = 2 * hk * kDK + hv * dv;
    const int chunks = (tokens + kC - 1) / kC;
    const int bar = kBarPair + 6 * pair;
    // lanes' parts of ldmatrix addresses: rows of two n-tiles with two 8-wide pieces each (tokens are n), and the other way round (tokens are k)
    const uint32_t row_n = (uint32_t)(8 * (lane >> 4) + sub) * 256, row_k = (uint32_t)(lane & 15) * 256;
    const int piece_n = (lane >> 3) & 1, piece_k = lane >> 4;
    // tokens 0 - 63 (four pairs of n-tiles) of keys 16 kk .. + 15
    auto load_n = [&](uint4 (&b)[4], uint32_t base, int kk) {
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = ldsm(base + row_n + j * 16 * 256 + (((2 * kk + piece_n) ^ sub) << 4));
    };
    // tokens 16 (step / 2) .. + 15 of keys 64 (step & 1) .. + 63
    auto load_k = [&](uint4 (&b)[4], uint32_t base, int step) {
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = ldsm_t(base + row_k + (step >> 1) * 16 * 256 + (((8 * (step & 1) + 2 * j + piece_k) ^ sub) << 4));
    };

    if (warp < 2) {
        float acc[16][4];                      // state: column c0 + 16 pair + g + 8 (c >> 1), key 8 nt + 2 t + (c & 1)
        float* tile = state + (size_t)head * kDK * dv + c0 + 16 * pair + g;
#pragma unroll
        for (int nt = 0; nt < 16; ++nt)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[nt][c] = tile[(size_t)(8 * nt + 2 * t + (c & 1)) * dv + 8 * (c >> 1)];
#pragma unroll 1
        for (int chunk = 0; chunk < chunks; ++chunk) {
            const Stage& st = s.stage[chunk % kStages];
            const ChunkTerms& own = st.terms;
            const int odd = chunk & 1;
            Handover& over = s.over[pair][odd];
            const uint32_t ks = smem_u32(st.k), vs = smem_u32(st.v);
            named_barrier(kBarFilled, 128);
            if (chunk >= 2) named_barrier(bar + 4 + odd, 64);         // the results of two chunks ago are formed
            // ---- P = K S_0, transposed
            float p[8][4];
            uint4 b[2][4];
            load_n(b[0], ks, 0);
#pragma unroll
            for (int nt = 0; nt < 8; ++nt)
#pragma unroll
                for (int c = 0; c < 4; ++c) p[nt][c] = 0.f;
#pragma unroll
            for (int kk = 0; kk < kDK / 16; ++kk) {
                uint4 hi, lo;
                uint4(&cur)[4] = b[kk & 1];
                if (kk + 1 < kDK / 16) load_n(b[(kk + 1) & 1], ks, kk + 1);
                split_tiles(acc[2 * kk], acc[2 * kk + 1], hi, lo);
#pragma unroll
                for (int j = 0; j < 4; ++j) { mma_bf16(p[2 * j], hi, cur[j].x, cur[j].y); mma_bf16(p[2 * j + 1], hi, cur[j].z, cur[j].w); }
#pragma unroll
                for (int j = 0; j < 4; ++j) { mma_bf16(p[2 * j], lo, cur[j].x, cur[j].y); mma_bf16(p[2 * j + 1], lo, cur[j].z, cur[j].w); }
                over.s[kk][0][lane] = hi;
                over.s[kk][1][lane] = lo;
            }
            named_arrive(bar + odd, 64);
            // ---- R = V - G P
            uint4 rhi[4], rlo[4];
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {           // tokens 16 kk + 0 - 7 and 8 - 15, columns 0 - 7 and 8 - 15
                const int r = 16 * kk + 8 * (lane >> 4) + sub;
                const uint4 v = ldsm_t(vs + r * 64 + (((2 * pair + piece_n) ^ ((r >> 1) & 3)) << 4));
                const uint32_t words[2][2] = {{v.x, v.y}, {v.z, v.w}};
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    const float2 f = *reinterpret_cast<const float2*>(&own.pred[16 * kk + 8 * n + 2 * t]);
                    float(&x)[4] = p[2 * kk + n];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        x[2 * h] = __uint_as_float(words[n][h] << 16) - f.x * x[2 * h];
                        x[2 * h + 1] = __uint_as_float(words[n][h] & 0xffff0000u) - f.y * x[2 * h + 1];
                    }
                }
                split_tiles(p[2 * kk], p[2 * kk + 1], rhi[kk], rlo[kk]);
            }
            // ---- U = (T B) R: the tokens up to the block's own count
#pragma unroll
            for (int nt = 0; nt < 8; ++nt)
#pragma unroll
                for (int c = 0; c < 4; ++c) p[nt][c] = 0.f;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                uint4 bh[4], bl[4];
#pragma unroll
                for (int i = kk; i < 4; ++i) { bh[i] = own.tb[block_of(i, kk)][0][lane]; bl[i] = own.tb[block_of(i, kk)][1][lane]; }
#pragma unroll
                for (int i = kk; i < 4; ++i) { mma_bf16(p[2 * i], rhi[kk], bh[i].x, bh[i].y); mma_bf16(p[2 * i + 1], rhi[kk], bh[i].z, bh[i].w); }
#pragma unroll
                for (int i = kk; i < 4; ++i) { mma_bf16(p[2 * i], rlo[kk], bh[i].x, bh[i].y); mma_bf16(p[2 * i + 1], rlo[kk], bh[i].z, bh[i].w); }
#pragma unroll
                for (int i = kk; i < 4; ++i) { mma_bf16(p[2 * i], rhi[kk], bl[i].x, bl[i].y); mma_bf16(p[2 * i + 1], rhi[kk], bl[i].z, bl[i].w); }
            }
            load_k(b[0], ks, 0);
            // ---- U for the results; U scaled by g_C / g_t for the state
            const float end = own.end[0];
#pragma unroll
            for (int nt = 0; nt < 16; ++nt)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[nt][c] *= end;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                uint4 hi, lo;
                split_tiles(p[2 * kk], p[2 * kk + 1], hi, lo);
                over.u[kk][0][lane] = hi;
                over.u[kk][1][lane] = lo;
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    const float2 f = *reinterpret_cast<const float2*>(&own.keep[16 * kk + 8 * n + 2 * t]);
#pragma unroll
                    for (int h = 0; h < 2; ++h) { p[2 * kk + n][2 * h] *= f.x; p[2 * kk + n][2 * h + 1] *= f.y; }
                }
                split_tiles(p[2 * kk], p[2 * kk + 1], rhi[kk], rlo[kk]);
            }
            named_arrive(bar + 2 + odd, 64);
            // ---- S = g_C S_0 + K^T U, transposed
#pragma unroll
            for (int step = 0; step < 8; ++step) {
                const int kk = step >> 1, first = 8 * (step & 1);
                uint4(&cur)[4] = b[step & 1];
                if (step + 1 < 8) load_k(b[(step + 1) & 1], ks, step + 1);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    mma_bf16(acc[first + 2 * j], rhi[kk], cur[j].x, cur[j].y);
                    mma_bf16(acc[first + 2 * j + 1], rhi[kk], cur[j].z, cur[j].w);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    mma_bf16(acc[first + 2 * j], rlo[kk], cur[j].x, cur[j].y);
                    mma_bf16(acc[first + 2 * j + 1], rlo[kk], cur[j].z, cur[j].w);
                }
            }
        }
#pragma unroll
        for (int nt = 0; nt < 16; ++nt)
#pragma unroll
            for (int c = 0; c < 4; ++c) tile[(size_t)(8 * nt + 2 * t + (c & 1)) * dv + 8 * (c >> 1)] = acc[nt][c];
        return;
    }
    const int tid = threadIdx.x & 63;
    const ChunkTerms* mine = terms + (size_t)head * chunks;
    auto issue = [&](int chunk) {
        if (chunk < chunks) {
            Stage& st = s.stage[chunk % kStages];
            const int t_base = chunk * kC;
            const uint32_t v = smem_u32(st.v), dst = smem_u32(&st.terms);
            copy_rows<64>(smem_u32(st.k), qkv + (size_t)(hk + key_head) * kDK, t_base, tokens, channels, tid, wide);
            const bf16* first = qkv + (size_t)2 * hk * kDK + (size_t)head * dv + c0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {              // 16-byte pieces p of row r at p ^ (r / 2 & 3)
                const int r = tid / 4 + 16 * i, piece = tid & 3, tok = min(t_base + r, tokens - 1);
                copy16(v + r * 64 + ((piece ^ ((r >> 1) & 3)) << 4), first + (size_t)tok * channels + piece * 8, t_base + r < tokens, wide);
            }
            const char* src = reinterpret_cast<const char*>(mine + chunk);
#pragma unroll 4
            for (int i = tid; i < (int)sizeof(ChunkTerms) / 16; i += 64) copy16(dst + 16 * i, src + 16 * i, true, true);
            copy_rows<64>(smem_u32(st.q), qkv + (size_t)key_head * kDK, t_base, tokens, channels, tid, wide);
        }
        copies_commit();
    };
    issue(0);
    issue(1);
    copies_wait<1>();
    named_arrive(kBarFilled, 128);             // chunk 0, this warp's part
    uint4* rows = s.rows[pair];
#pragma unroll 1
    for (int chunk = 0; chunk < chunks; ++chunk) {
        const Stage& st = s.stage[chunk % kStages];
        const ChunkTerms& own = st.terms;
        const int odd = chunk & 1;
        const Handover& over = s.over[pair][odd];
        const uint32_t qs = smem_u32(st.q);
        float o[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[nt][c] = 0.f;
        named_barrier(bar + odd, 64);          // this pair's state is there
        named_barrier(kBarRead, 64);           // both are: nobody reads the stage of the chunk before any more
        issue(chunk + 2);
        copies_wait<1>();
        if (chunk + 1 < chunks) named_arrive(kBarFilled, 128);
        uint4 b[2][4];
        load_n(b[0], qs, 0);
#pragma unroll
        for (int kk = 0; kk < kDK / 16; ++kk) {
            const uint4 hi = over.s[kk][0][lane], lo = over.s[kk][1][lane];
            uint4(&cur)[4] = b[kk & 1];
            if (kk + 1 < kDK / 16) load_n(b[(kk + 1) & 1], qs, kk + 1);
#pragma unroll
            for (int j = 0; j < 4; ++j) { mma_bf16(o[2 * j], hi, cur[j].x, cur[j].y); mma_bf16(o[2 * j + 1], hi, cur[j].z, cur[j].w); }
#pragma unroll
            for (int j = 0; j < 4; ++j) { mma_bf16(o[2 * j], lo, cur[j].x, cur[j].y); mma_bf16(o[2 * j + 1], lo, cur[j].z, cur[j].w); }
        }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const float2 f = *reinterpret_cast<const float2*>(&own.read[8 * nt + 2 * t]);
#pragma unroll
            for (int h = 0; h < 2; ++h) { o[nt][2 * h] *= f.x; o[nt][2 * h + 1] *= f.y; }
        }
        named_barrier(bar + 2 + odd, 64);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const uint4 hi = over.u[kk][0][lane], lo = over.u[kk][1][lane];
            uint4 bh[4], bl[4];
#pragma unroll
            for (int i = kk; i < 4; ++i) { bh[i] = own.a[block_of(i, kk)][0][lane]; bl[i] = own.a[block_of(i, kk)][1][lane]; }
#pragma unroll
            for (int i = kk; i < 4; ++i) { mma_bf16(o[2 * i], hi, bh[i].x, bh[i].y); mma_bf16(o[2 * i + 1], hi, bh[i].z, bh[i].w); }
#pragma unroll
            for (int i = kk; i < 4; ++i) { mma_bf16(o[2 * i], lo, bh[i].x, bh[i].y); mma_bf16(o[2 * i + 1], lo, bh[i].z, bh[i].w); }
#pragma unroll
            for (int i = kk; i < 4; ++i) { mma_bf16(o[2 * i], hi, bl[i].x, bl[i].y); mma_bf16(o[2 * i + 1], hi, bl[i].z, bl[i].w); }
        }
        if (chunk + 2 < chunks) named_arrive(bar + 4 + odd, 64);
        // ---- [column][token] -> rows of tokens, 32 bytes each
        __syncwarp();
#pragma unroll
        for (int nt = 0; nt < 8; nt += 2) {
            uint32_t w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const __nv_bfloat162 two = __floats2bfloat162_rn(o[nt + (q >> 1)][2 * (q & 1)], o[nt + (q >> 1)][2 * (q & 1) + 1]);
                w[q] = *reinterpret_cast<const uint32_t*>(&two);
            }
            // matrices: (token tile nt, columns 0 - 7), (nt, 8 - 15), (nt + 1, 0 - 7), (nt + 1, 8 - 15)
            const int r = 8 * nt + 8 * (lane >> 4) + sub;
            asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};"
                         ::"r"(smem_u32(rows + 2 * r + (piece_n ^ ((r >> 2) & 1)))), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
        }
        __syncwarp();
        bf16* dst = out + (size_t)head * dv + c0 + 16 * pair;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 16 * i + (lane >> 1), tok = chunk * kC + r, half = lane & 1;
            const uint4 v = rows[2 * r + (half ^ ((r >> 2) & 1))];
            if (tok < tokens) {
                bf16* to = dst + (size_t)tok * hv * dv + 8 * half;
                if (wide_out) {
                    *reinterpret_cast<uint4*>(to) = v;
                } else {
                    uint32_t* words = reinterpret_cast<uint32_t*>(to);
                    words[0] = v.x; words[1] = v.y; words[2] = v.z; words[3] = v.w;
                }
            }
        }
    }
    copies_wait<0>();
}

}  // namespace
}  // namespace qd

// Bytes of the scratch area of qd_seq_gdn_recurrence_chunked for a run of `tokens` tokens.
extern "C" long long qd_seq_gdn_chunk_scratch_bytes(int tokens, int value_heads) {
    if (tokens <= 0 || value_heads <= 0) return 0;
    return (long long)((tokens + qd::kC - 1) / qd::kC) * value_heads * (long long)sizeof(qd::ChunkTerms);
}

// The contract of qd_seq_gdn_recurrence (conv_qkv [tokens, 2 key_heads 128 + value_heads value_dim]
// after the short convolution, a / b [tokens, value_heads], rec_state fp32 updated in place, out
// bf16 [tokens, value_heads value_dim]) in the chunked form.  key_dim 128, value_dim a multiple of
// 32; QD_ERR_UNSUPPORTED otherwise.  scratch: qd_seq_gdn_chunk_scratch_bytes bytes, 16-byte aligned.
extern "C" int qd_seq_gdn_recurrence_chunked(const void* conv_qkv, const void* a, const void* b, const void* a_log,
                                             const void* dt_bias, float* rec_state, void* out, int tokens, int key_heads,
                                             int value_heads, int key_dim, int value_dim, void* scratch, void* stream) {
    using namespace qd;
    QD_CHECK_ARG(conv_qkv && a && b && a_log && dt_bias && rec_state && out && scratch && tokens > 0);
    QD_CHECK_ARG(key_heads > 0 && value_heads % key_heads == 0 && value_dim > 0);
    if (key_dim != kDK || value_dim % kCols != 0 || value_heads > 65535) return QD_ERR_UNSUPPORTED;
    if (((uintptr_t)conv_qkv & 7u) || ((uintptr_t)scratch & 15u) || ((2 * key_heads * kDK + value_heads * value_dim) % 4)) return QD_ERR_UNSUPPORTED;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return QD_ERR_LAUNCH;
    static bool configured[64];
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(gdn_chunk_recurrence_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RecurrenceArea)) != cudaSuccess)
            return QD_ERR_LAUNCH;
        configured[dev] = true;
    }
    const int chunks = (tokens + kC - 1) / kC, wide = ((uintptr_t)conv_qkv & 15u) == 0, wide_out = ((uintptr_t)out & 15u) == 0;
    qd_launch(gdn_chunk_prepare_kernel, dim3(chunks, key_heads), dim3(kPrepThreads), 0, (cudaStream_t)stream, true,
        (const bf16*)conv_qkv, (const bf16*)a, (const bf16*)b, (const bf16*)a_log, (const bf16*)dt_bias, (ChunkTerms*)scratch,
        tokens, key_heads, value_heads, value_dim, wide);
    if (qd_launch_status() != QD_OK) return QD_ERR_LAUNCH;
    qd_launch(gdn_chunk_recurrence_kernel, dim3(value_heads, value_dim / kCols), dim3(kRecThreads), sizeof(RecurrenceArea), (cudaStream_t)stream, true,
        (const bf16*)conv_qkv, rec_state, (bf16*)out, (const ChunkTerms*)scratch, tokens, key_heads, value_heads, value_dim, wide, wide_out);
    return qd_launch_status();
}
