// Attention of a chunk of fp32 rows on the tensor cores.  Included by window_attention.cu.
//
// Every operand (queries, keys, probabilities, values) is three bf16 pieces, a product six of theirs (pieces_mma.cuh; what is left
// out is below 2^-26 of it), sums are fp32: the scores in three accumulators, a tile's values from zero and then onto the result, rounded to nearest.
// A block is 64 packed (token, head of the group) rows and two groups of four warps, sixteen rows a warp.  The groups take turns with the keys, 32
// at a time, each with a softmax of its own: one cuts its tile into pieces on the way into shared memory while the other multiplies.
// mma.sync, because the queries' pieces do not fit tensor memory beside the rest.
// On the FMA pipe (attn_tiles_kernel) and here: 777 tokens from position 0, window 1024, 16/4 heads of 128 385 -> 117 us, 16 heads of 192 + 128 474 -> 193,
// 300 tokens 120 -> 50, 1024 tokens behind 1024 766 -> 257; error against 64 bits 2.8e-7 -> 2.5e-7, 2.8 -> 2.7, 2.2 -> 2.3, 6.1 -> 3.1.  (One group and two
// blocks an SM: 162, 240, 65, 227 us.)  The MMAs are a third of it, the cutting and the softmax the rest.
#pragma once
#include "pieces_mma.cuh"

namespace qd {
namespace {

constexpr float kNoPieces = 3.3961775292304e38f;                    // 2^128 (1 - 2^-9): from here on the first piece rounds up to infinity
constexpr int kPieceRows = 64, kPieceKeys = 32, kPieceThreads = 256;
template <int QD, int DV> struct PieceShape {
    static constexpr int kQRow = QD + 8, kVRow = DV + 8;               // bf16 to a row: an odd number of 16-byte pieces
    static constexpr int kQPlane = kPieceRows * kQRow, kKPlane = kPieceKeys * kQRow, kVPlane = kPieceKeys * kVRow;
    static constexpr size_t kSmem = 3 * sizeof(bf16) * (kQPlane + 2 * (kKPlane + kVPlane));
    static_assert(3 * sizeof(bf16) * (kKPlane + kVPlane) >= sizeof(float) * kPieceRows * (DV + 2) && kSmem <= 227 * 1024, "");
};

// a barrier of a group's four warps; whether any of them has `found`
QD_DEVINL bool group_any(int id, bool found) {
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.cta.red.or.aligned.pred p, %2, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(any) : "r"((uint32_t)found), "r"(id) : "memory");
    return any != 0;
}
// four values as pieces into three planes
QD_DEVINL void put_planes(bf16* to, int plane, const float4& x) {
    uint2 v[3];
    split_three<false>(x.x, x.y, v[0].x, v[1].x, v[2].x);
    split_three<false>(x.z, x.w, v[0].y, v[1].y, v[2].y);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(to + i * plane) = v[i];
}

// The score of a query and a key whose pieces give no number (one of them has an infinity or a magnitude that rounds up to one, or the sum passes
// the largest number), without them and in the order of attn_tiles_kernel: an infinity that a key of weight zero may have, or NaN.
template <int QD> QD_DEVINL float plain_score(const float* q, const float* k, const float* common, int dim) {
    float sum = 0.f;
#pragma unroll 1
    for (int d0 = 0; d0 < QD; d0 += 32) {
        float part = 0.f;
#pragma unroll 1
        for (int d = d0; d < d0 + 32; d += 4) {
            const float4 a = load4(q + d), b = d < dim ? load4(k + d) : load4(common + (d - dim));
            part = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, part))));
        }
        sum += part;
    }
    return sum;
}

template <int QD, int DV>
__global__ void __launch_bounds__(kPieceThreads, 1) attn_pieces_kernel(const __grid_constant__ AttnParams p) {
    chain_enter();
    using S = PieceShape<QD, DV>;
    extern __shared__ __align__(16) bf16 tiles[];
    const int group = threadIdx.x >> 7, tid = threadIdx.x & 127, warp = tid >> 5, lane = tid & 31, g4 = lane >> 2, t4 = lane & 3;      // of the group
    bf16* qs = tiles;
    bf16* ks = qs + 3 * S::kQPlane + group * 3 * (S::kKPlane + S::kVPlane);
    bf16* vs = ks + 3 * S::kKPlane;
    const int share = p.heads / p.kv_heads, g = blockIdx.y, total = p.tokens * share, r0 = (int)(gridDim.x - 1 - blockIdx.x) * kPieceRows;   // longest first
    const int base = p.position_ptr ? *p.position_ptr : p.position;
    const int pos_first = base + r0 / share, pos_last = base + (min(r0 + kPieceRows, total) - 1) / share;
    const int key_first = lowest_key(p, pos_first), slot_first = key_first % p.capacity;
    const float* q = reinterpret_cast<const float*>(p.q_rows);
    const float* kc = reinterpret_cast<const float*>(p.k_cache) + g * p.dim;
    const float* vc = reinterpret_cast<const float*>(p.v_cache) + g * DV;
    const float* common = reinterpret_cast<const float*>(p.k_shared);
#pragma unroll 4
    for (int i = threadIdx.x; i < kPieceRows * QD / 4; i += kPieceThreads) {
        const int r = i / (QD / 4), c = i % (QD / 4) * 4, row = min(r0 + r, total - 1);
        put_planes(qs + r * S::kQRow + c, S::kQPlane, load4(q + ((size_t)(row / share) * p.heads + g * share + row % share) * QD + c));
    }
    // this lane's two rows
    int pos[2], low[2];
    float m[2], l[2], slope[2], o[DV / 8][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int row = min(r0 + warp * 16 + g4 + 8 * i, total - 1), h = g * share + row % share;
        pos[i] = base + row / share;
        low[i] = lowest_key(p, pos[i]);
        slope[i] = p.slopes ? p.slopes[h] : 0.f;
        // the sink is the first term of the first group's softmax (of the sum's four parts, one has it)
        const bool sink = p.sink_kind != QD_SINK_NONE && group == 0;
        m[i] = !sink ? -INFINITY : p.sink_kind == QD_SINK_LEARNED ? ld_bf16(as_bf16(p.sink) + h) : 0.f;
        l[i] = sink && t4 == 0 ? 1.f : 0.f;
    }
#pragma unroll
    for (int n = 0; n < DV / 8; ++n)
#pragma unroll
        for (int c = 0; c < 4; ++c) o[n][c] = 0.f;
    // lanes' parts of ldmatrix addresses: an A operand (16 rows x 16), two n-tiles of keys (n) x 16 columns (k), 16 keys (k) x two n-tiles of columns (n)
    const uint32_t qa = smem_u32(qs + (warp * 16 + (lane & 15)) * S::kQRow + (lane >> 4) * 8);
    const uint32_t kb = smem_u32(ks + ((lane & 7) + ((lane >> 4) << 3)) * S::kQRow + ((lane >> 3) & 1) * 8);
    const uint32_t vb = smem_u32(vs + (lane & 15) * S::kVRow + (lane >> 4) * 8);

    __syncthreads();                                   // the queries
    for (int j0 = key_first + group * kPieceKeys; j0 <= pos_last; j0 += 2 * kPieceKeys) {
        named_barrier(1 + group, 128);                 // the group's previous tile is used up
        const auto slot_of = [&](int j) {
            int slot = j <= pos_last ? slot_first + (j - key_first) : slot_first;
            return slot >= p.capacity ? slot - p.capacity : slot;      // what a block sees fits the ring
        };
#pragma unroll 8
        for (int i = tid; i < kPieceKeys * QD / 4; i += 128) {
            const int r = i / (QD / 4), c = i % (QD / 4) * 4, slot = slot_of(j0 + r);
            put_planes(ks + r * S::kQRow + c, S::kKPlane, c < p.dim ? load4(kc + slot * p.ld_k + c) : load4(common + slot * p.ld_shared + (c - p.dim)));
        }
        bool odd = false;
#pragma unroll 8
        for (int i = tid; i < kPieceKeys * DV / 4; i += 128) {
            const int r = i / (DV / 4), c = i % (DV / 4) * 4;
            const float4 x = j0 + r <= pos_last ? load4(vc + slot_of(j0 + r) * p.ld_v + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            odd |= !(fabsf(x.x) < kNoPieces && fabsf(x.y) < kNoPieces && fabsf(x.z) < kNoPieces && fabsf(x.w) < kNoPieces);
            put_planes(vs + r * S::kVRow + c, S::kVPlane, x);
        }
        odd = group_any(3 + group, odd);               // values without pieces, or that a product with a masked key's zero must not reach
        // ---- scores
        float s[4][4];
        {
            float large[2][4][4] = {}, small[4][4] = {};
#pragma unroll
            for (int kk = 0; kk < QD / 16; ++kk) {
                uint4 a[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) a[i] = ldsm(qa + 2 * (i * S::kQPlane + 16 * kk));
                uint4 b[3][2];
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int n = 0; n < 2; ++n) b[i][n] = ldsm(kb + 2 * (i * S::kKPlane + 16 * n * S::kQRow + 16 * kk));
                constexpr int kLeft[6] = {1, 2, 0, 1, 0, 0}, kRight[6] = {1, 0, 2, 0, 1, 0};
#pragma unroll
                for (int i = 0; i < 6; ++i)
#pragma unroll
                    for (int n = 0; n < 2; ++n) {
                        const uint4& x = b[kRight[i]][n];
                        mma_bf16(i == 5 ? large[kk & 1][2 * n] : small[2 * n], a[kLeft[i]], x.x, x.y);
                        mma_bf16(i == 5 ? large[kk & 1][2 * n + 1] : small[2 * n + 1], a[kLeft[i]], x.z, x.w);
                    }
            }
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int c = 0; c < 4; ++c) s[n][c] = (large[0][n][c] + large[1][n][c]) + small[n][c];
        }
        bool unbounded = false;
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int c = 0; c < 4; ++c) unbounded |= !(fabsf(s[n][c]) < INFINITY);
        if (__any_sync(0xffffffffu, unbounded)) {
#pragma unroll 1
            for (int e = 0; e < 16; ++e) {
                const int i = (e >> 1) & 1, key = j0 + 8 * (e >> 2) + 2 * t4 + (e & 1), row = min(r0 + warp * 16 + g4 + 8 * i, total - 1);
                if (key > (i ? pos[1] : pos[0]) || key < (i ? low[1] : low[0])) continue;
                const int slot = slot_of(key);
                const float x = plain_score<QD>(q + ((size_t)(row / share) * p.heads + g * share + row % share) * QD, kc + slot * p.ld_k,
                                                common + slot * p.ld_shared, p.dim);
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (e == 4 * n + c && !(fabsf(s[n][c]) < INFINITY)) s[n][c] = x;
            }
        }
        // ---- softmax
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float top = -INFINITY;
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int key = j0 + 8 * n + 2 * t4 + c;
                    float& x = s[n][2 * i + c];
                    x = key <= pos[i] && key >= low[i] ? x * p.scale - slope[i] * (float)(pos[i] - key) : -INFINITY;
                    top = fmaxf(top, x);
                }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(m[i], fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2)));
            const float keep = top == -INFINITY ? 1.f : expf(m[i] - top), sub = top == -INFINITY ? 0.f : top;
            m[i] = top;
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    float& x = s[n][2 * i + c];
                    x = x == -INFINITY ? 0.f : expf(x - sub);
                    sum += x;
                }
            l[i] = l[i] * keep + sum;
#pragma unroll
            for (int n = 0; n < DV / 8; ++n) { o[n][2 * i] *= keep; o[n][2 * i + 1] *= keep; }
        }
        // ---- values
        if (!odd) {
            const Pieces w[2] = {split_tiles3(s[0], s[1]), split_tiles3(s[2], s[3])};
#pragma unroll
            for (int n = 0; n < DV / 16; n += 2) {     // four n-tiles at a time
                float d[4][4] = {};
#pragma unroll
                for (int kk = 0; kk < 2; ++kk) {
                    uint4 b[3][2];
#pragma unroll
                    for (int i = 0; i < 3; ++i)
#pragma unroll
                        for (int h = 0; h < 2; ++h) b[i][h] = ldsm_t(vb + 2 * (i * S::kVPlane + 16 * kk * S::kVRow + 16 * (n + h)));
                    constexpr int kLeft[6] = {1, 2, 0, 1, 0, 0}, kRight[6] = {1, 0, 2, 0, 1, 0};
#pragma unroll
                    for (int i = 0; i < 6; ++i)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint4& x = b[kRight[i]][h];
                            mma_bf16(d[2 * h], w[kk].p[kLeft[i]], x.x, x.y);
                            mma_bf16(d[2 * h + 1], w[kk].p[kLeft[i]], x.z, x.w);
                        }
                }
#pragma unroll
                for (int h = 0; h < 4; ++h)
#pragma unroll
                    for (int c = 0; c < 4; ++c) o[2 * n + h][c] += d[h][c];
            }
        } else {                                       // key by key, each row the keys that it sees
#pragma unroll 1
            for (int t = 0; t < 4; ++t)
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int key = j0 + 8 * n + 2 * t + c;
                        const float w0 = __shfl_sync(0xffffffffu, s[n][c], (lane & ~3) | t), w1 = __shfl_sync(0xffffffffu, s[n][2 + c], (lane & ~3) | t);
                        const bool in0 = key <= pos[0] && key >= low[0], in1 = key <= pos[1] && key >= low[1];
                        if (key > pos_last) continue;
                        const float* v = vc + slot_of(key) * p.ld_v + 2 * t4;
#pragma unroll
                        for (int e = 0; e < DV / 8; ++e) {
                            const float2 x = *reinterpret_cast<const float2*>(v + 8 * e);
                            if (in0) { o[e][0] = fmaf(w0, x.x, o[e][0]); o[e][1] = fmaf(w0, x.y, o[e][1]); }
                            if (in1) { o[e][2] = fmaf(w1, x.x, o[e][2]); o[e][3] = fmaf(w1, x.y, o[e][3]); }
                        }
                    }
        }
    }
    // ---- the second group's rows to the first: maximum, sum, result
    float* other = reinterpret_cast<float*>(tiles + 3 * (S::kQPlane + S::kKPlane + S::kVPlane));
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
        if (group == 0) continue;
        float* row = other + (warp * 16 + g4 + 8 * i) * (DV + 2);
        if (i == 0) named_barrier(2, 128);             // the area held the group's last tile
        if (t4 == 0) *reinterpret_cast<float2*>(row) = make_float2(m[i], l[i]);
#pragma unroll
        for (int e = 0; e < DV / 8; ++e) *reinterpret_cast<float2*>(row + 2 + 8 * e + 2 * t4) = make_float2(o[e][2 * i], o[e][2 * i + 1]);
    }
    __syncthreads();
    if (group) return;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int row = r0 + warp * 16 + g4 + 8 * i;
        if (row >= total) continue;
        const float* from = other + (warp * 16 + g4 + 8 * i) * (DV + 2);
        const float2 ml = *reinterpret_cast<const float2*>(from);
        const float top = fmaxf(m[i], ml.x);           // (a row sees itself)
        const float own = m[i] == -INFINITY ? 0.f : expf(m[i] - top), its = ml.x == -INFINITY ? 0.f : expf(ml.x - top);
        const int t = row / share, h = g * share + row % share;
        const float* gate = reinterpret_cast<const float*>(p.gate) + (long long)t * p.ld_gate;
        const float f = (p.gate_kind == QD_GATE_HEAD ? sigmoid_precise(gate[h]) : 1.f) / (l[i] * own + ml.y * its);
        float* out = reinterpret_cast<float*>(p.out) + ((size_t)t * p.heads + h) * DV + 2 * t4;
#pragma unroll
        for (int e = 0; e < DV / 8; ++e)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const float a = own == 0.f ? 0.f : o[e][2 * i + c] * own, b = its == 0.f ? 0.f : from[2 + 8 * e + 2 * t4 + c] * its;
                out[8 * e + c] = (a + b) * f * (p.gate_kind == QD_GATE_VALUE ? sigmoid_precise(gate[h * DV + 8 * e + 2 * t4 + c]) : 1.f);
            }
    }
}

}  // namespace
}  // namespace qd
