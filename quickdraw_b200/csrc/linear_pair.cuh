// The bf16 product of many token rows on pairs of SMs (tcgen05 cta_group::2).  Included by linear.cu.
//
// linear_umma_kernel gives a block one tile: its prologue, and an epilogue in which every lane stores 8 bytes of a row of its own
// (a quarter of a 32-byte sector), lie open, 14 to 19 of the 37 us of a 256 x 256 tile of 2048 inputs.  Here a pair of blocks stays for
// many tiles of 256 tokens x 256 weight rows: each block holds half of the tokens, half of the weight rows (which an MMA of the pair reads from both)
// and the accumulators of its tokens twice, so that one tile is read out while the next is multiplied; rows leave through shared
// memory in whole 128-byte lines.  Inputs and outputs, bf16, before and now (cuBLAS): 2048 tokens 2048 -> 4160 39.1 -> 30.3 us (29.9), 2048 -> 12416
// 114 -> 77 (73), 2048 -> 16384 with gated pairs 116 -> 93, 576 -> 4096 for 3071 tokens 35.8 -> 18.2, 8192 -> 2048 56 -> 51 (48); 8192 tokens
// 2048 -> 8192 259 -> 185 (176) = 1.49 PFLOP/s.  What bounds that one is the tensor pipe, active in 90 % of the cycles (L2 49 % busy), at the clock that
// the power limit leaves.  (Tiles of 128 weight rows, which ask L2 for half as much again per product, took 305 us.)
#pragma once
#include "pair.cuh"

namespace qd {
namespace {

struct PairTile {
    static constexpr int kRows = 256;                                             // tokens of a tile, and weight rows
    static constexpr int kHalfBytes = 128 * 128, kStageBytes = 2 * kHalfBytes, kStages = 6;      // a block's rows, 64 inputs
    static constexpr int kLineBytes = 128, kStagingBytes = 32 * kLineBytes;       // of an epilogue warp
    static constexpr int kEpilogueWarps = 8, kThreads = 64 + 32 * kEpilogueWarps;
    static constexpr size_t kSmem = (size_t)kStages * kStageBytes + kEpilogueWarps * kStagingBytes + (2 * kStages + 5) * 8 + 16 + 1024;
};

QD_DEVINL void pair_umma_f16(uint32_t d_tmem, uint32_t a_low, uint32_t b_low, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n\t}"
                 ::"r"(d_tmem), "r"(a_low), "r"(b_low), "r"(idesc), "r"(accumulate), "r"(kDescHigh) : "memory");
}
// Sixteen sums of a token, the first of them output n of the matrix, finished: eight (glu) or sixteen values into `out`.
QD_DEVINL void finish16(const Finish& f, const uint32_t* v, int n, const float* bias, float (&out)[16]) {
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(v[i]);
    if (f.bias) {
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
            const float4 b = load4(bias + i);
            x[i] += b.x; x[i + 1] += b.y; x[i + 2] += b.z; x[i + 3] += b.w;
        }
    }
    if (n < f.gelu_cols) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (n + i < f.gelu_cols) x[i] = gelu_erf(x[i]);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) out[i] = x[i];
    if (f.glu) {
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = fmaxf(x[2 * i], 0.f) * x[2 * i + 1];
    }
}
// Values as 16-byte pieces of a line (piece c of lane's line at c ^ (lane & 7)), onto what is there with `add`; returns the next piece.
template <int N> QD_DEVINL int put_pieces(float (&x)[16], uint4* line, int piece, int lane, bool add, float) {
#pragma unroll
    for (int i = 0; i < N; i += 4, ++piece) {
        uint4& to = line[piece ^ (lane & 7)];
        if (add) {
            x[i] += __uint_as_float(to.x); x[i + 1] += __uint_as_float(to.y); x[i + 2] += __uint_as_float(to.z); x[i + 3] += __uint_as_float(to.w);
        }
        to = make_uint4(__float_as_uint(x[i]), __float_as_uint(x[i + 1]), __float_as_uint(x[i + 2]), __float_as_uint(x[i + 3]));
    }
    return piece;
}
template <int N> QD_DEVINL int put_pieces(float (&x)[16], uint4* line, int piece, int lane, bool add, bf16) {
#pragma unroll
    for (int i = 0; i < N; i += 8, ++piece) {
        uint4& to = line[piece ^ (lane & 7)];
        if (add) {
            float there[8];
            unpack8(to, there);
#pragma unroll
            for (int j = 0; j < 8; ++j) x[i + j] += there[j];
        }
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __nv_bfloat162 two = __floats2bfloat162_rn(x[i + 2 * j], x[i + 2 * j + 1]);
            w[j] = *reinterpret_cast<const uint32_t*>(&two);
        }
        to = make_uint4(w[0], w[1], w[2], w[3]);
    }
    return piece;
}
// An epilogue warp's 32 lines, four at a time in whole lines: from and to rows t0 .. of y, outputs first ..
template <bool STORE, typename TY>
QD_DEVINL void move_lines(uint4* lines, const LinearParams& p, int t0, int first, int out_cols, int lane) {
    constexpr int kPer = 16 / (int)sizeof(TY);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int row = 4 * r + (lane >> 3), q = lane & 7, n = first + q * kPer;
        uint4& at = lines[row * 8 + (q ^ (row & 7))];
        if (t0 + row >= p.tokens || n >= out_cols) continue;
        TY* y = reinterpret_cast<TY*>(p.y) + (long long)(t0 + row) * p.ldy + n;
        if (!STORE) at = *reinterpret_cast<const uint4*>(y);          // (outputs are multiples of eight where they are added)
        else if (n + kPer <= out_cols) *reinterpret_cast<uint4*>(y) = at;
        else *reinterpret_cast<uint2*>(y) = make_uint2(at.x, at.y);   // half of eight bf16: gated pairs of rows come in fours
    }
    __syncwarp();
}

template <typename TY>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairTile::kThreads, 1)
linear_pair_kernel(const __grid_constant__ LinearParams p, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap) {
    chain_enter();
    using Tile = PairTile;
    constexpr int kStages = Tile::kStages, TN = Tile::kRows;
    // as in linear_umma_kernel, M = 256 over the pair
    constexpr uint32_t kDesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ __align__(16) float bias[TN];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* staging = smem + kStages * Tile::kStageBytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(staging + Tile::kEpilogueWarps * Tile::kStagingBytes);       // (the first block's: both blocks' operands are there)
    uint64_t* empty = full + kStages;
    uint64_t* ready = empty + kStages;         // an accumulator holds a tile
    uint64_t* taken = ready + 2;               // (the first block's:) both blocks have read it
    uint64_t* drained = taken + 2;             // (the first block's:) every MMA has ended
    uint32_t* slot = reinterpret_cast<uint32_t*>(drained + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = (int)cluster_rank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int across = (p.tokens + 255) / 256, tiles = across * ((p.rows + TN - 1) / TN), steps = (p.width + kStepK - 1) / kStepK;

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(ready + s, 1); mbar_init(taken + s, 2 * Tile::kEpilogueWarps); }
        mbar_init(drained, 1);
        mbar_fence_init();
    }
    if (warp == 1) pair_tmem_alloc(slot, 2 * TN);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync();                            // the barriers of both blocks are there
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *slot;

    // A wait that runs out ends a role; the loads end when the MMAs have taken the last of them or 0.2 s after it (the limit of a wait), the
    // issuing warp when a commit of all MMAs has arrived, and both blocks together.
    if (warp == 0) {
        const bool leader = elect_one();
        int st = 0, n = 1;
        uint32_t parity = 1;                       // (a new barrier's phase before the first is over)
        for (int tile = pair; tile < tiles && n; tile += pairs) {
            const int t0 = (tile % across) * 256 + rank * 128, n0 = (tile / across) * TN + rank * (TN / 2);
            for (int s = 0; s < steps; s += n) {
                n = ring_ready(empty, st, parity, kStages, min(steps - s, kStages), p.status);
                if (n == 0) break;
                if (leader) {
                    for (int u = 0; u < n; ++u) {
                        const int at = st + u < kStages ? st + u : st + u - kStages;
                        uint8_t* a = smem + at * Tile::kStageBytes;
                        const uint32_t bar = of_first_block(full + at);
                        if (rank == 0) mbar_expect_tx(full + at, 2 * Tile::kStageBytes);
                        pair_tma_tile(a, &xmap, (s + u) * kStepK, t0, bar);
                        pair_tma_tile(a + Tile::kHalfBytes, &wmap, (s + u) * kStepK, n0, bar);
                    }
                }
                __syncwarp();
                st += n;
                if (st >= kStages) { st -= kStages; parity ^= 1u; }
            }
        }
        if (n) pair_loads_taken(empty, kStages, pair < tiles ? ((tiles - 1 - pair) / pairs + 1) * steps : 0, p.status);
    } else if (warp == 1) {
        if (rank == 0) {
            const bool leader = elect_one();
            const uint32_t low0 = __shfl_sync(0xffffffffu, desc_low(smem_u32(smem)), 0), to = __shfl_sync(0xffffffffu, tmem, 0);
            int st = 0, n = 1, i = 0;
            uint32_t parity = 0;
            for (int tile = pair; tile < tiles; tile += pairs, ++i) {
                const int buf = i & 1;
                if (i >= 2 && !__all_sync(0xffffffffu, mbar_wait(taken + buf, ((i >> 1) - 1) & 1, p.status))) break;
                for (int s = 0; s < steps; s += n) {
                    n = ring_ready(full, st, parity, kStages, min(steps - s, kStages), p.status);
                    if (n == 0) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (leader) {
                        for (int u = 0; u < n; ++u) {
                            const int at = st + u < kStages ? st + u : st + u - kStages;
                            const uint32_t a = low0 + at * (Tile::kStageBytes >> 4), b = a + (Tile::kHalfBytes >> 4);
#pragma unroll
                            for (int j = 0; j < kStepK / 16; ++j) pair_umma_f16(to + buf * TN, a + 2 * j, b + 2 * j, kDesc, (s | u | j) ? 1u : 0u);
                            pair_commit(empty + at);
                        }
                    }
                    __syncwarp();
                    st += n;
                    if (st >= kStages) { st -= kStages; parity ^= 1u; }
                }
                if (n == 0) break;
                if (leader) pair_commit(ready + buf);
                __syncwarp();
            }
            if (leader) pair_commit_here(drained);            // tensor memory is given back only behind the last MMA, also where a wait ran out
            mbar_wait(drained, 0, p.status);
        }
    } else {
        const int quadrant = warp & 3, half = (warp - 2) >> 2;        // lanes of tensor memory that the warp may read; columns that it takes
        uint4* lines = reinterpret_cast<uint4*>(staging + (warp - 2) * Tile::kStagingBytes);
        uint4* line = lines + lane * 8;
        const int out_cols = p.f.glu ? p.rows / 2 : p.rows;
        bool ok = true;
        int i = 0;
        for (int tile = pair; tile < tiles; tile += pairs, ++i) {
            const int buf = i & 1, t0 = (tile % across) * 256 + rank * 128 + quadrant * 32, n0 = (tile / across) * TN;
            if (p.f.bias) {
                named_barrier(1, 32 * Tile::kEpilogueWarps);          // the tile before is read out
                for (int c = tid - 64; c < TN; c += 32 * Tile::kEpilogueWarps) bias[c] = n0 + c < p.rows ? p.f.bias[n0 + c] : 0.f;
                named_barrier(1, 32 * Tile::kEpilogueWarps);
            }
            // behind a wait that ran out nothing is waited for nor stored, but the warps still meet for the bias
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(ready + buf, (i >> 1) & 1, p.status));
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            int piece = 0, first = p.f.glu ? (n0 + half * (TN / 2)) / 2 : n0 + half * (TN / 2);      // pieces of the line that are filled; its first output
            if (ok && t0 < p.tokens) {
#pragma unroll 1
                for (int c = half * (TN / 2); c < (half + 1) * (TN / 2); c += 32) {
                    if (p.f.add && piece == 0) move_lines<false, TY>(lines, p, t0, first, out_cols, lane);
                    uint32_t v[32];
                    tmem_ld32(tmem + ((uint32_t)(quadrant * 32) << 16) + buf * TN + c, v);
#pragma unroll
                    for (int h = 0; h < 32; h += 16) {
                        float x[16];
                        finish16(p.f, v + h, n0 + c + h, bias + c + h, x);
                        piece = p.f.glu ? put_pieces<8>(x, line, piece, lane, p.f.add, TY()) : put_pieces<16>(x, line, piece, lane, p.f.add, TY());
                    }
                    if (piece < 8) continue;
                    move_lines<true, TY>(lines, p, t0, first, out_cols, lane);
                    piece = 0;
                    first += 128 / (int)sizeof(TY);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_at(of_first_block(taken + buf));
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1) pair_tmem_dealloc(tmem, 2 * TN);
}

}  // namespace
}  // namespace qd
