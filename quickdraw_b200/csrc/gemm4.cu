// Block-scaled FP4 x FP4 product on the 5th generation tensor cores (tcgen05.mma
// kind::mxf4nvf4, scale_vec::4X): Y[T, N] = X[T, K] . W[N, K]^T with BOTH operands NVFP4, and
// the activation quantiser that produces X in that format.
//
// The reference multiplies bf16 activations with dequantised NVFP4 weights
// (quickdraw/kernel/triton/matvec.py:118-163); its notes (todo.md:13) name "W4A4 activation
// quantisation" as the step to validate separately from that W4A16 path.  This file is that
// step: qd_nvfp4_quantize_act writes the activations of a chunk of tokens as E2M1 codes, one
// E4M3 scale per sixteen inputs and one fp32 scale per tensor (the weight format of
// quickdraw/models/weights.py:29-47, so the same container describes both operands), and
// qd_nvfp4_matmul_w4a4 multiplies the two without expanding anything: codes travel HBM -> shared
// memory as tiled TMA loads in the layout the MMA reads, block scales travel the same way and
// are moved into tensor memory, the accumulator lives in tensor memory.  The result differs from
// the W4A16 product by the activation rounding only; the exact path stays qd_nvfp4_matmul.
//
// Small products, nvfp4_gemm_w4a4_kernel: 128 tokens x 128 weight rows per block, K in stages of 256 inputs (a 128-byte row of
// codes, sixteen scales).  Two blocks share an SM (3 stages of 36 KB and 256 columns of tensor
// memory each), so one block's epilogue overlaps the other's K loop.
//   warp 0      TMA: per stage four boxes (codes and scales of both operands)
//   warp 1      allocates tensor memory, issues 4 MMAs of 128 x 128 x 64 per stage
//   warps 2..5  move the stage's block scales shared memory -> tensor memory (every warp fills
//               its own 32-lane quarter), then run the epilogue: one token per lane
// Large ones, w4a4_pair_kernel: 256 x 256 tiles on pairs of SMs, see there.
// Every wait is bounded; a wait that runs out sets the status word and the block leaves.
#include <algorithm>

#include "pair.cuh"
#include "umma.cuh"

namespace qd {
namespace {

constexpr int kTile = 128;                    // tokens and weight rows per block
constexpr int kStages4 = 3;
constexpr int kCodeBytes = kTile * 128;       // 128 rows x 256 inputs
constexpr int kScaleBytes = kTile * 16;       // 128 rows x 16 scales
constexpr int kStage4Bytes = 2 * (kCodeBytes + kScaleBytes);
constexpr int kThreads4 = 6 * 32;
constexpr uint32_t kCols4 = 256, kColAcc = 0, kColSf = 128;
// scale columns of a stage: 16 for the 128 tokens (four per 64-input step: rows l, l + 32, l + 64,
// l + 96 of lane l), then as many for the weight rows
constexpr uint32_t kSfCols = 32;
constexpr uint32_t desc_of(int m, int n) { return (1u << 7) | (1u << 10) | (((uint32_t)n >> 3) << 17) | (((uint32_t)m >> 4) << 24); }

struct Gemm4Params {
    const float* x_global; const float* w_global; bf16* y;
    int tokens, out_features, in_features;
    unsigned int* status;
};

struct Bars4 { uint64_t full[kStages4], empty[kStages4], sf_ready[kStages4], done; };

// the scale words of rows l, l + 32, l + 64, l + 96 of lane l (rows of sixteen bytes from `from` on): four columns per 64-input step
QD_DEVINL void scales_of_128(uint32_t to, const uint8_t* from, int lane) {
    uint32_t w[16];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        const uint4 v = *reinterpret_cast<const uint4*>(from + (lane + 32 * g) * 16);
        w[0 + g] = v.x; w[4 + g] = v.y; w[8 + g] = v.z; w[12 + g] = v.w;
    }
    tmem_store16(to, w);
}

__global__ void __launch_bounds__(kThreads4, 2)
nvfp4_gemm_w4a4_kernel(const __grid_constant__ Gemm4Params p, const __grid_constant__ CUtensorMap x_codes,
                       const __grid_constant__ CUtensorMap x_scales, const __grid_constant__ CUtensorMap w_codes,
                       const __grid_constant__ CUtensorMap w_scales) {
    grid_dependency_wait();       // before the tensor memory: a block that waits for its predecessor must not hold what that one needs
    extern __shared__ __align__(1024) uint8_t gemm4_smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gemm4_smem_raw) + 1023) & ~uintptr_t(1023));
    Bars4* bars = reinterpret_cast<Bars4*>(smem + kStages4 * kStage4Bytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int t0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
    const int chunks = p.in_features / 256;

    if (tid == 0) {
        for (int s = 0; s < kStages4; ++s) { mbar_init(bars->full + s, 1); mbar_init(bars->empty + s, 1); mbar_init(bars->sf_ready + s, 4); }
        mbar_init(&bars->done, 1);
        mbar_fence_init();
    }
    if (warp == 1) { tmem_alloc(tmem_slot, kCols4); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    auto stage = [&](int st) { return smem + (size_t)st * kStage4Bytes; };

    if (warp == 0) {
        const bool leader = elect_one();
        if (leader) { tma_prefetch_map(&x_codes); tma_prefetch_map(&x_scales); tma_prefetch_map(&w_codes); tma_prefetch_map(&w_scales); }
        int st = 0, n = 1;
        uint32_t parity = 1;                       // (a new barrier's phase before the first is over)
        for (int c = 0; c < chunks; c += n) {
            n = ring_ready(bars->empty, st, parity, kStages4, min(chunks - c, kStages4), p.status);
            if (n == 0) break;
            if (leader) {
                for (int u = 0; u < n; ++u) {
                    const int at = st + u < kStages4 ? st + u : st + u - kStages4;
                    // rows past the end of a matrix arrive as zeros; a box always counts in full
                    mbar_expect_tx(bars->full + at, kStage4Bytes);
                    uint8_t* base = stage(at);
                    // codes: tokens, then the weight rows; scales in the same order
                    uint8_t* sc = base + 2 * kCodeBytes;
                    tma_load_2d(base, &x_codes, (c + u) * 128, t0, bars->full + at);
                    tma_load_2d(sc, &x_scales, (c + u) * 16, t0, bars->full + at);
                    tma_load_2d(base + kCodeBytes, &w_codes, (c + u) * 128, n0, bars->full + at);
                    tma_load_2d(sc + kScaleBytes, &w_scales, (c + u) * 16, n0, bars->full + at);
                }
            }
            __syncwarp();
            st += n;
            if (st >= kStages4) { st -= kStages4; parity ^= 1u; }
        }
    } else if (warp == 1) {
        const bool leader = elect_one();
        const uint32_t low0 = __shfl_sync(0xffffffffu, desc_lo_sw128(smem_u32(stage(0))), 0), to = __shfl_sync(0xffffffffu, tmem, 0);
        int st = 0, n = 1;
        uint32_t parity = 0;
        for (int c = 0; c < chunks; c += n) {
            n = ring_ready(bars->full, st, parity, kStages4, min(chunks - c, kStages4), p.status);
            if (n) n = ring_ready(bars->sf_ready, st, parity, kStages4, n, p.status);
            if (n == 0) break;
            tc_fence_after();
            if (leader) {
                for (int u = 0; u < n; ++u) {
                    const int at = st + u < kStages4 ? st + u : st + u - kStages4;
                    const uint32_t a_lo = low0 + at * (kStage4Bytes >> 4), b_lo = a_lo + (kCodeBytes >> 4);
                    const uint32_t sfa = to + kColSf + at * kSfCols, sfb = sfa + 16;
#pragma unroll
                    for (int j = 0; j < 4; ++j)       // a 64-input step: 32 bytes further in both operands
                        umma_nvfp4_lo(to + kColAcc, a_lo + 2 * j, b_lo + 2 * j, desc_of(128, 128), sfa + j * 4, sfb + j * 4, (c | u | j) ? 1u : 0u);
                    umma_commit(bars->empty + at);    // the stage (and its scale columns) is free once these MMAs are done
                }
            }
            __syncwarp();
            st += n;
            if (st >= kStages4) { st -= kStages4; parity ^= 1u; }
        }
        if (n && leader) umma_commit(&bars->done);
    } else {
        // ---- block scales of every stage into tensor memory: lane l of a quarter holds, per
        //      64-input step, the scale words of rows l, l + 32, l + 64, l + 96 in four columns
        const uint32_t quarter = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        bool ok = true;
        for (int c = 0; c < chunks && ok; ++c) {
            const int st = c % kStages4;
            if (!mbar_wait(bars->full + st, (c / kStages4) & 1, p.status)) { ok = false; break; }
            const uint8_t* sc = stage(st) + 2 * kCodeBytes;
            scales_of_128(quarter + kColSf + st * kSfCols, sc, lane);
            scales_of_128(quarter + kColSf + st * kSfCols + 16, sc + kScaleBytes, lane);
            tmem_store_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars->sf_ready + st);
        }
        // ---- epilogue: this lane's token, 128 outputs, both tensor scales after the sum
        if (ok && mbar_wait(&bars->done, 0, p.status)) {
            tc_fence_after();
            const float scale = p.x_global[0] * p.w_global[0];
            const int token = t0 + (warp & 3) * 32 + lane;
            bf16* out = p.y + (size_t)token * p.out_features + n0;
#pragma unroll 1
            for (int col = 0; col < kTile; col += 16) {
                uint32_t v[16];
                tmem_load16(quarter + kColAcc + col, v);
                tmem_load_wait();
                if (token < p.tokens) {
                    uint32_t packed[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const __nv_bfloat162 two = __floats2bfloat162_rn(__uint_as_float(v[2 * q]) * scale, __uint_as_float(v[2 * q + 1]) * scale);
                        packed[q] = *reinterpret_cast<const uint32_t*>(&two);
                    }
                    *reinterpret_cast<uint4*>(out + col) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                    *reinterpret_cast<uint4*>(out + col + 8) = make_uint4(packed[4], packed[5], packed[6], packed[7]);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, kCols4);
}

// ---- large products
// Tiles of 256 tokens x 256 weight rows on a pair of SMs that stays for many of them (tcgen05 cta_group::2): each block holds the codes of
// half of the tokens and half of the weight rows, the scales of its tokens and of all the weight rows, and 256 columns of sums.  With one
// 128 x 256 tile to a block, operands came from L2 at 54 KB a stage and block, where an SM gets some 40 bytes a clock (the MMAs would need 89), and
// the prologue and an epilogue of scattered 16-byte stores lay open.  Here it is 38 KB, loads run on through the end of a tile, and the
// sums wait only for a pass of eight warps from tensor memory into registers (tensor memory holds no second set beside the scales).
//   warp 0      TMA: codes count at the first block, scales in their own
//   warp 1      of the first block: 4 MMAs of 256 x 256 x 64 per stage
//   warps 2-13  scales to tensor memory, as above, four warps a group, a stage of the ring always the same group's (below); the weight rows' in
//               eight columns per 64-input step
//   the last 8  sums, 32 tokens x 128 outputs each, as bf16 through shared memory in whole 128-byte lines
// What bounded both forms was the way of the scales, some 1000 clocks a stage for its four warps from the wait to the hand-over: 8192 x 8192 x
// 2048 127 us before, here 141 with one group of four warps, 111 with two, 105 with three (102 before a stage had a group of its own).  Its
// counters there: L2 40 % busy, tensor pipe 32 %, issue 20 %.  2048 x 8192 x 2048 37 -> 33 us.
struct Pair4 {
    static constexpr int kStages = 5, kStageBytes = 2 * kCodeBytes + 3 * kScaleBytes, kEpilogueWarps = 8, kStagingBytes = 32 * 128;
    static constexpr int kScaleGroups = 3, kFirst = 2 + 4 * kScaleGroups, kThreads = 32 * (kFirst + kEpilogueWarps);
    static constexpr uint32_t kColSf = 256, kSfCols = 48;
    struct Bars { uint64_t full[kStages], scales[kStages], sf_ready[kStages], empty[kStages], ready, taken, drained; };
    static constexpr size_t kSmem = (size_t)kStages * kStageBytes + kEpilogueWarps * kStagingBytes + sizeof(Bars) + 64 + 1024;
    static_assert(kColSf + kStages * kSfCols <= 512 && kStageBytes % 1024 == 0 && kSmem <= 227 * 1024, "");
};
// The step of the loads (one stage each) that a group of scale warps takes after step `it`; group g begins with step g.  A stage has the same
// group in every round of the ring.  Copies end in any order, so a group that met a stage only every third round could ask for a round while the
// copy of the one before, which another group waits for, is still on its way: the parity of a phase that is over would let it pass.  Two
// of the groups have two of the five stages, 2.5 steps of time for each.
constexpr int next_scale_step(int it) {
    constexpr int S = Pair4::kStages, G = Pair4::kScaleGroups;
    return it % S + G < S ? it + G : it / S * S + S + it % S % G;
}

QD_DEVINL void pair_umma_nvfp4(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %7, 0;\n\t"
                 "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
                 "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%0], da, db, %4, [%5], [%6], p;\n\t}"
                 ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(kDescHiSw128), "r"(idesc), "r"(sfa_tmem), "r"(sfb_tmem), "r"(accumulate) : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Pair4::kThreads, 1)
w4a4_pair_kernel(const __grid_constant__ Gemm4Params p, const __grid_constant__ CUtensorMap x_codes, const __grid_constant__ CUtensorMap x_scales,
                 const __grid_constant__ CUtensorMap w_codes, const __grid_constant__ CUtensorMap w_scales) {
    grid_dependency_wait();       // before the tensor memory, as above
    extern __shared__ __align__(1024) uint8_t gemm4_smem_raw[];
    using T = Pair4;
    constexpr int kStages = T::kStages;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gemm4_smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* staging = smem + kStages * T::kStageBytes;
    T::Bars* bars = reinterpret_cast<T::Bars*>(staging + T::kEpilogueWarps * T::kStagingBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = (int)cluster_rank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1, chunks = p.in_features / 256;
    const int across = (p.tokens + 255) / 256, tiles = across * ((p.out_features + 255) / 256);
    const auto steps_of_pair = [&] { return pair < tiles ? ((tiles - 1 - pair) / pairs + 1) * chunks : 0; };       // (its value held throughout costs spills)

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(bars->full + s, 1); mbar_init(bars->scales + s, 1); mbar_init(bars->sf_ready + s, 2 * 4); mbar_init(bars->empty + s, 1);
        }
        mbar_init(&bars->ready, 1);
        mbar_init(&bars->taken, 2 * T::kEpilogueWarps);
        mbar_init(&bars->drained, 1);
        mbar_fence_init();
    }
    if (warp == 1) pair_tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    cluster_sync();               // the barriers of both blocks are there
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // A wait that runs out ends a role; the loads end when the MMAs have taken the last of them or 0.2 s after it (the limit of a wait), the
    // issuing warp when a commit of all MMAs has arrived, and both blocks together.
    if (warp == 0) {
        const bool leader = elect_one();
        int st = 0, n = 1;
        uint32_t parity = 1;                       // (a new barrier's phase before the first is over)
        for (int tile = pair; tile < tiles && n; tile += pairs) {
            const int t0 = (tile % across) * 256 + rank * 128, n0 = (tile / across) * 256;
            for (int c = 0; c < chunks; c += n) {
                n = ring_ready(bars->empty, st, parity, kStages, min(chunks - c, kStages), p.status);
                if (n == 0) break;
                if (leader) {
                    for (int u = 0; u < n; ++u) {
                        const int at = st + u < kStages ? st + u : st + u - kStages;
                        uint8_t* base = smem + at * T::kStageBytes;
                        uint8_t* sc = base + 2 * kCodeBytes;
                        const uint32_t bar = of_first_block(bars->full + at);
                        if (rank == 0) mbar_expect_tx(bars->full + at, 4 * kCodeBytes);
                        pair_tma_tile(base, &x_codes, (c + u) * 128, t0, bar);
                        pair_tma_tile(base + kCodeBytes, &w_codes, (c + u) * 128, n0 + rank * 128, bar);
                        mbar_expect_tx(bars->scales + at, 3 * kScaleBytes);
                        tma_load_2d(sc, &x_scales, (c + u) * 16, t0, bars->scales + at);
                        tma_load_2d(sc + kScaleBytes, &w_scales, (c + u) * 16, n0, bars->scales + at);
                        tma_load_2d(sc + 2 * kScaleBytes, &w_scales, (c + u) * 16, n0 + 128, bars->scales + at);
                    }
                }
                __syncwarp();
                st += n;
                if (st >= kStages) { st -= kStages; parity ^= 1u; }
            }
        }
        if (n) pair_loads_taken(bars->empty, kStages, steps_of_pair(), p.status);
    } else if (warp == 1) {
        if (rank == 0) {
            const bool leader = elect_one();
            const uint32_t low0 = __shfl_sync(0xffffffffu, desc_lo_sw128(smem_u32(smem)), 0), to = __shfl_sync(0xffffffffu, tmem, 0);
            int st = 0, n = 1, i = 0;
            uint32_t parity = 0;
            for (int tile = pair; tile < tiles; tile += pairs, ++i) {
                if (i && !__all_sync(0xffffffffu, mbar_wait(&bars->taken, (i - 1) & 1, p.status))) break;
                for (int c = 0; c < chunks; c += n) {
                    n = ring_ready(bars->full, st, parity, kStages, min(chunks - c, kStages), p.status);
                    if (n) n = ring_ready(bars->sf_ready, st, parity, kStages, n, p.status);
                    if (n == 0) break;
                    tc_fence_after();
                    if (leader) {
                        for (int u = 0; u < n; ++u) {
                            const int at = st + u < kStages ? st + u : st + u - kStages;
                            const uint32_t a_lo = low0 + at * (T::kStageBytes >> 4), b_lo = a_lo + (kCodeBytes >> 4);
                            const uint32_t sfa = to + T::kColSf + at * T::kSfCols, sfb = sfa + 16;
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                pair_umma_nvfp4(to, a_lo + 2 * j, b_lo + 2 * j, desc_of(256, 256), sfa + j * 4, sfb + j * 8, (c | u | j) ? 1u : 0u);
                            pair_commit(bars->empty + at);
                        }
                    }
                    __syncwarp();
                    st += n;
                    if (st >= kStages) { st -= kStages; parity ^= 1u; }
                }
                if (n == 0) break;
                if (leader) pair_commit(&bars->ready);
                __syncwarp();
            }
            if (leader) pair_commit_here(&bars->drained);     // tensor memory is given back only behind the last MMA, also where a wait ran out
            mbar_wait(&bars->drained, 0, p.status);
        }
    } else if (warp < T::kFirst) {
        const uint32_t quarter = tmem + ((uint32_t)((warp & 3) * 32) << 16) + T::kColSf;
        const int group = (warp - 2) >> 2, steps = steps_of_pair();
        bool ok = true;
        for (int it = group; it < steps; it = next_scale_step(it)) {
            const int st = it % kStages;
            ok = __all_sync(0xffffffffu, mbar_wait(bars->scales + st, (it / kStages) & 1, p.status));
            if (!ok) break;
            const uint8_t* sc = smem + st * T::kStageBytes + 2 * kCodeBytes;
            scales_of_128(quarter + st * T::kSfCols, sc, lane);
#pragma unroll
            for (int half = 0; half < 2; ++half) {                    // 64-input steps 2 half, 2 half + 1: row l + 32 g in column g
                uint32_t w[16];
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    const uint2 v = *reinterpret_cast<const uint2*>(sc + kScaleBytes + (lane + 32 * g) * 16 + half * 8);
                    w[g] = v.x; w[8 + g] = v.y;
                }
                tmem_store16(quarter + st * T::kSfCols + 16 + half * 16, w);
            }
            tmem_store_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_at(of_first_block(bars->sf_ready + st));
        }
    } else {
        const int quadrant = warp & 3, half = (warp - T::kFirst) >> 2;
        uint4* lines = reinterpret_cast<uint4*>(staging + (warp - T::kFirst) * T::kStagingBytes);
        const float scale = p.x_global[0] * p.w_global[0];
        bool ok = true;
        int i = 0;
        for (int tile = pair; tile < tiles && ok; tile += pairs, ++i) {
            const int t0 = (tile % across) * 256 + rank * 128 + quadrant * 32, n0 = (tile / across) * 256 + half * 128;
            ok = __all_sync(0xffffffffu, mbar_wait(&bars->ready, i & 1, p.status));
            if (!ok) break;
            tc_fence_after();
            uint32_t packed[64];
#pragma unroll
            for (int c = 0; c < 128; c += 16) {
                uint32_t v[16];
                tmem_load16(tmem + ((uint32_t)(quadrant * 32) << 16) + half * 128 + c, v);
                tmem_load_wait();
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const __nv_bfloat162 two = __floats2bfloat162_rn(__uint_as_float(v[2 * q]) * scale, __uint_as_float(v[2 * q + 1]) * scale);
                    packed[c / 2 + q] = *reinterpret_cast<const uint32_t*>(&two);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_at(of_first_block(&bars->taken));
#pragma unroll
            for (int part = 0; part < 2; ++part) {                    // 64 outputs: a 128-byte line, pieces q of line l at q ^ (l & 7)
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const uint32_t* w = packed + part * 32 + q * 4;
                    lines[lane * 8 + (q ^ (lane & 7))] = make_uint4(w[0], w[1], w[2], w[3]);
                }
                __syncwarp();
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const int row = 4 * r + (lane >> 3), q = lane & 7, n = n0 + part * 64 + q * 8;
                    const uint4 w = lines[row * 8 + (q ^ (row & 7))];
                    if (t0 + row < p.tokens && n < p.out_features) *reinterpret_cast<uint4*>(p.y + (size_t)(t0 + row) * p.out_features + n) = w;
                }
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    cluster_sync();
    tc_fence_after();
    if (warp == 1) pair_tmem_dealloc(tmem, 512);
}

// ---- activation quantiser --------------------------------------------------------------
// Largest magnitude of the chunk (bf16 magnitudes order like their bit patterns).  Four pieces of a thread in flight and one atomic
// a block: 8192 x 2048 in 11.8 us, 13.8 with one piece and an atomic a warp.
__global__ void __launch_bounds__(256) act_amax_kernel(const uint4* __restrict__ x, long long n8, unsigned int* __restrict__ amax_bits) {
    __shared__ uint32_t warps[8];
    const long long step = (long long)gridDim.x * blockDim.x;
    uint32_t m = 0u;                                  // a pair of magnitudes
    const auto take = [&](const uint4& v) {
        m = __vmaxu2(m, __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu)));
    };
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 3 * step < n8; i += 4 * step) {
        const uint4 a = x[i], b = x[i + step], c = x[i + 2 * step], d = x[i + 3 * step];
        take(a); take(b); take(c); take(d);
    }
    for (; i < n8; i += step) take(x[i]);
    m = max(m & 0xffffu, m >> 16);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < 8 ? warps[threadIdx.x] : 0u;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0 && m) atomicMax(amax_bits, m);
    }
}

// Eight values -> eight E2M1 codes, round to nearest even, saturating; value 2i in the low
// nibble of byte i (the checkpoint's nibble order).
QD_DEVINL uint32_t e2m1x8(const float (&v)[16], int first) {
    uint32_t r;
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
        "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
        : "=r"(r)
        : "f"(v[first]), "f"(v[first + 1]), "f"(v[first + 2]), "f"(v[first + 3]), "f"(v[first + 4]), "f"(v[first + 5]),
          "f"(v[first + 6]), "f"(v[first + 7]));
    return r;
}
QD_DEVINL uint32_t e4m3_of(float v) {                 // round to nearest even, saturating
    unsigned short r;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(0.f), "f"(v));
    return (uint32_t)r & 0xffu;
}

// One thread per block of sixteen inputs: tensor scale g = amax / (6 * 448) (1 for a zero chunk),
// block scale s = e4m3(block amax / (6 g)), codes = e2m1(x / (s g)), everything round to
// nearest even; a block whose scale rounds to zero gets zero codes.  The result has the layout of a weight, which some
// products fetch before they wait for the kernel in front of them: nobody is released before the stores are visible.
__global__ void act_quantize_kernel(const bf16* __restrict__ x, long long blocks, const unsigned int* __restrict__ amax_bits,
                                    uint8_t* __restrict__ codes, uint8_t* __restrict__ scales, float* __restrict__ global) {
    grid_dependency_wait();
    const float amax = __uint_as_float(*amax_bits << 16);
    const float g = amax > 0.f ? amax / (6.f * 448.f) : 1.f;
    if (blockIdx.x == 0 && threadIdx.x == 0) *global = g;
    const long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= blocks) return;
    const uint4 lo = reinterpret_cast<const uint4*>(x)[2 * b], hi = reinterpret_cast<const uint4*>(x)[2 * b + 1];
    const uint32_t raw[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    float v[16], top = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        v[2 * i] = __uint_as_float(raw[i] << 16);
        v[2 * i + 1] = __uint_as_float(raw[i] & 0xffff0000u);
        top = fmaxf(top, fmaxf(fabsf(v[2 * i]), fabsf(v[2 * i + 1])));
    }
    const uint32_t sbits = e4m3_of(top / (6.f * g));
    const float s = e4m3_to_float((uint8_t)sbits) * g;
    const float inv = s > 0.f ? 1.f / s : 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] *= inv;
    reinterpret_cast<uint2*>(codes)[b] = make_uint2(e2m1x8(v, 0), e2m1x8(v, 8));
    scales[b] = (uint8_t)sbits;
    __threadfence();
}

int scale_map_of(CUtensorMap* map, const void* base, long long rows, long long row_bytes) {
    EncodeTiledFn encode = umma_encode_fn();
    if (!encode) return QD_ERR_UNSUPPORTED;
    const cuuint64_t dims[2] = {(cuuint64_t)row_bytes, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)row_bytes};
    const cuuint32_t box[2] = {16, (cuuint32_t)kTile};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, elem,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? QD_OK : QD_ERR_LAUNCH;
}

}  // namespace
}  // namespace qd

extern "C" int qd_nvfp4_quantize_act(const void* x, int tokens, int in_features, void* codes, void* scales,
                                     float* global, unsigned int* amax_scratch, void* stream) {
    using namespace qd;
    QD_CHECK_ARG(x && codes && scales && global && amax_scratch && tokens > 0 && in_features > 0 && in_features % 16 == 0);
    QD_CHECK_ARG(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(codes)) & 15u) == 0);
    cudaStream_t s = (cudaStream_t)stream;
    const long long n = (long long)tokens * in_features;
    if (cudaMemsetAsync(amax_scratch, 0, 4, s) != cudaSuccess) return QD_ERR_LAUNCH;
    const int grid = (int)std::min<long long>((n / 8 + 255) / 256, 148 * 8);
    act_amax_kernel<<<grid, 256, 0, s>>>(reinterpret_cast<const uint4*>(x), n / 8, amax_scratch);
    const long long blocks = n / 16;
    if (qd_launch_status() != QD_OK) return QD_ERR_LAUNCH;
    return qd_launch(act_quantize_kernel, dim3((unsigned)((blocks + 255) / 256)), dim3(256), 0, s, 3, reinterpret_cast<const bf16*>(x), blocks,
                     (const unsigned int*)amax_scratch, reinterpret_cast<uint8_t*>(codes), reinterpret_cast<uint8_t*>(scales), global);
}

extern "C" int qd_nvfp4_matmul_w4a4(const void* x_codes, const void* x_scales, const float* x_global, const void* w_codes,
                                    const void* w_scales, const float* w_global, void* y, int tokens, int out_features,
                                    int in_features, int wide_tiles, unsigned int* status, void* stream) {
    using namespace qd;
    QD_CHECK_ARG(x_codes && x_scales && x_global && w_codes && w_scales && w_global && y && tokens > 0);
    QD_CHECK_ARG(in_features > 0 && in_features % 256 == 0 && out_features > 0 && out_features % 128 == 0);
    QD_CHECK_ARG(((reinterpret_cast<uintptr_t>(x_codes) | reinterpret_cast<uintptr_t>(x_scales) | reinterpret_cast<uintptr_t>(w_codes) |
                   reinterpret_cast<uintptr_t>(w_scales) | reinterpret_cast<uintptr_t>(y)) & 15u) == 0);
    alignas(64) CUtensorMap xc, xs, wc, ws;
    int rc = umma_make_map(&xc, x_codes, tokens, in_features / 2, 128, kTile);
    if (rc == QD_OK) rc = umma_make_map(&wc, w_codes, out_features, in_features / 2, 128, kTile);
    if (rc == QD_OK) rc = scale_map_of(&xs, x_scales, tokens, in_features / 16);
    if (rc == QD_OK) rc = scale_map_of(&ws, w_scales, out_features, in_features / 16);
    if (rc != QD_OK) return rc;
    Gemm4Params p = {};
    p.x_global = x_global; p.w_global = w_global; p.y = reinterpret_cast<bf16*>(y);
    p.tokens = tokens; p.out_features = out_features; p.in_features = in_features; p.status = status;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return QD_ERR_LAUNCH;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long token_tiles = (tokens + kTile - 1) / kTile, tiles = (long long)((tokens + 255) / 256) * ((out_features + 255) / 256);
    // a pair needs two tiles or more to hide its start (256 tiles 33 us against 38 of the small form, 128 tiles 20.0 / 20.2, 100 tiles 18 / 16)
    const bool wide = wide_tiles >= 0 ? wide_tiles != 0 : tiles >= sms;
    constexpr size_t smem = (size_t)kStages4 * kStage4Bytes + sizeof(Bars4) + 64 + 1024;
    static bool configured[2][64];
    if (!configured[wide][dev]) {
        if ((wide ? cudaFuncSetAttribute(w4a4_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Pair4::kSmem)
                  : cudaFuncSetAttribute(nvfp4_gemm_w4a4_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess)
            return QD_ERR_LAUNCH;
        configured[wide][dev] = true;
    }
    if (wide)
        return qd_launch(w4a4_pair_kernel, dim3((unsigned)(2 * std::min<long long>(tiles, sms / 2))), dim3(Pair4::kThreads), Pair4::kSmem, (cudaStream_t)stream, 3, p,
                         xc, xs, wc, ws);
    return qd_launch(nvfp4_gemm_w4a4_kernel, dim3((unsigned)(out_features / kTile), (unsigned)token_tiles), dim3(kThreads4), smem, (cudaStream_t)stream, 3, p, xc, xs,
                     wc, ws);
}
