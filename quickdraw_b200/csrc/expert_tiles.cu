// Grouped NVFP4 product of the routed experts with the weights decoded into TENSOR MEMORY (tcgen05.mma with its A operand
// there): 128 weight rows are the lanes of the A operand, up to 80 routes of an expert the columns of the accumulator.
//
// Arithmetic as in the other forms (quickdraw/kernel/triton/moe.py:99-151, quickdraw/models/qwen.py:176-191): weights
// expanded exactly to bf16(e2m1 * block scale), bf16 activations, fp32 accumulation on the tensor cores, the fp32 global
// scale on the finished sum, one bf16 rounding; the routed form rounds the sum and the scaled routing weight to bf16 first.
// The SwiGLU form multiplies the gate and up banks in one pass and writes bf16(bf16(silu(gate)) * up).
//
// Why this split.  An expert of a prompt chunk has few routes (8 of 256 experts a token: 64 in a 2048-token chunk), so a
// bank is read once from HBM (151 MB for 256 x 512 x 2048: 23 us) and decoded once, and both are the work; the MMAs are a
// fraction of it.  Tiles with the tokens as the A operand (gemm.cu) keep decoded weights in shared memory, written and read
// at 128 bytes a clock, and 256-token tiles are three quarters empty.  Here a decoded row goes from the registers of the
// lane that owns it to tensor memory, and shared memory carries only the routes' rows and the raw codes.
//   warps 0..15  decode: warp w takes lanes 32 (w mod 4) of row tile (w / 4) mod 2 and the steps of parity w / 8: 64 inputs
//                a step, 32 bytes of codes a lane (128-byte swizzled: conflict-free), hardware convert to f16, the mixed
//                multiply-add with the block scale to f32, one 32-column store to tensor memory
//   warps 16..19 epilogue of the previous item (two accumulator sets of 2 x 80 columns)
//   warp 20      issues 2 x 4 MMAs of 128 x n x 16 per step, n the item's routes rounded up to sixteen
//   warp 21      codes and scales of 256 inputs x 2 row tiles by tiled TMA, four stages of 36 KB (144 KB in flight)
//   warps 22..27 rows of the routes by cp.async, a stage of 10 KB each
// An item is (expert, at most 80 routes, 2 x 128 weight rows); blocks take items in turn, so the loads of the next item run
// under the decoding of this one.  Every wait is bounded.
//
// Measured (256 experts, gate and up of 512 x 2048 with the SwiGLU | down of 2048 x 512, cold L2, beside the faster of the
// other two forms): 512 tokens 115 | 68 us against 198 | 97; 2048 tokens 145 | 98 against 292 | 172; 8192 tokens 428 | 295
// against 597 | 481.  Bound by issue slots (the decoding) and by the hand-over of a step between the warps, 700 clocks of
// which 420 are issue; the floor of the three banks is 68 us of HBM.
#include <algorithm>

#include "expert_tiles.cuh"
#include "umma.cuh"

namespace qd {
namespace {

constexpr int kTileRoutes = 80;                         // routes of an item at most = columns of an accumulator
constexpr int kDecodeWarps = 16, kEpilogueWarps = 4;
constexpr int kMmaWarp = kDecodeWarps + kEpilogueWarps, kWeightWarp = kMmaWarp + 1, kRowsWarp = kMmaWarp + 2, kRowsWarps = 6;
constexpr int kTileThreads = 32 * (kRowsWarp + kRowsWarps);
constexpr int kWStages = 4, kBStages = kRowsWarps, kAStages = 3, kItemSlots = 4;
static_assert(kBStages == 2 * kAStages, "a step's tensor-memory stage follows from its barrier");
constexpr int kCodeTile = 128 * 128, kScaleTile = 128 * 16;                  // 128 rows x 256 inputs
constexpr int kWStageBytes = 2 * (kCodeTile + kScaleTile);
constexpr int kBStageBytes = kTileRoutes * 128;                             // 80 rows x 64 inputs
constexpr int kMaxExperts = 1024;
// tensor memory: three stages of (two tiles x 32 columns of decoded weights), then two sets of two accumulators
constexpr uint32_t kColA = 0, kColD = kAStages * 64, kSetCols = 2 * kTileRoutes, kTileCols = 512;

struct TileBars { uint64_t w_full[kWStages], w_empty[kWStages], full[kBStages], empty[kBStages], item_full[kItemSlots], item_empty[kItemSlots], d_full[2], d_empty[2], drained; };

struct TileParams {
    const bf16* x;
    const float* global; const float* global2;           // SwiGLU form: gate, up
    const int32_t* order; const int32_t* boundaries; const float* routing;
    bf16* y;
    int experts, topk, out_features, in_features, by_token, scatter, global_per_expert;
    unsigned int* status;
};

struct TileItem { int expert, t0, count, rows; };        // rows: which pair of row tiles
// and of its routes the input rows, the output rows and the factors of the sums (past the end: the last one again)
struct ItemSlot { TileItem item; int src[kTileRoutes]; int2 out[kTileRoutes]; };

// Item i: `row_tiles` consecutive items share the routes (their rows then come from L2).  An expert's routes are cut into
// equal parts of at most 80, rounded up to sixteen.
QD_DEVINL TileItem item_of(int i, const int* bounds, const int* before, int experts, int row_tiles) {
    const int tile = i / row_tiles;
    int lo = 0, hi = experts;                            // before[lo] <= tile < before[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (before[mid] <= tile) lo = mid; else hi = mid;
    }
    const int n = bounds[lo + 1] - bounds[lo], tiles = before[lo + 1] - before[lo];
    const int part = ((n + tiles - 1) / tiles + 15) & ~15, at = (tile - before[lo]) * part;
    return TileItem{lo, bounds[lo] + at, min(part, n - at), i - tile * row_tiles};
}

// D[tensor memory] (+)= A[tensor memory] B[shared memory]; the descriptor's upper half is the same for every tile.
QD_DEVINL void umma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 db, {%2, %3};\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
                 ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(kDescHiSw128), "r"(idesc), "r"(accumulate) : "memory");
}
QD_DEVINL void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
QD_DEVINL void copy16_async(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
QD_DEVINL void tmem_store32(uint32_t addr, const uint32_t (&v)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
                 "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                   "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
                   "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
                   "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]) : "memory");
}
// Sixteen columns of two accumulators.  The wait names the registers, so that no arithmetic on them moves in front of it.
QD_DEVINL void tmem_load16x2(uint32_t addr0, uint32_t addr1, uint32_t (&u)[16], uint32_t (&v)[16]) {
    tmem_load16(addr0, u);
    tmem_load16(addr1, v);
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(u[0]), "+r"(u[1]), "+r"(u[2]), "+r"(u[3]), "+r"(u[4]), "+r"(u[5]), "+r"(u[6]), "+r"(u[7]), "+r"(u[8]), "+r"(u[9]),
                   "+r"(u[10]), "+r"(u[11]), "+r"(u[12]), "+r"(u[13]), "+r"(u[14]), "+r"(u[15])
                 :: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) asm volatile("" : "+r"(v[j]));
}

// Eight codes times a block scale (the half SIDE of `scales`) as four bf16 pairs.  The product has at most six significant
// bits, so the f32 from the mixed multiply-add is exact and its upper half is the bf16.
template <int SIDE>
QD_DEVINL void decode8(uint32_t word, uint32_t scales, uint32_t* out) {
    uint32_t h[4];
    e2m1x8_to_f16x2(word, h);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float lo, hi;
        asm("{\n\t.reg .b16 a0, a1, s0, s1;\n\tmov.b32 {a0, a1}, %2;\n\tmov.b32 {s0, s1}, %3;\n\t"
            "fma.rn.f32.f16 %0, a0, s%5, %4;\n\tfma.rn.f32.f16 %1, a1, s%5, %4;\n\t}"
            : "=f"(lo), "=f"(hi) : "r"(h[i]), "r"(scales), "f"(-0.f), "n"(SIDE));
        out[i] = __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
    }
}
QD_DEVINL uint32_t e4m3x2_to_f16x2(uint32_t two) {
    const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)two, __NV_E4M3);
    return *reinterpret_cast<const uint32_t*>(&h);
}

template <bool SWIGLU>
__global__ void __launch_bounds__(kTileThreads, 1)
expert_tiles_kernel(const __grid_constant__ TileParams p, const __grid_constant__ CUtensorMap codes_map, const __grid_constant__ CUtensorMap scales_map,
                    const __grid_constant__ CUtensorMap codes2_map, const __grid_constant__ CUtensorMap scales2_map) {
    chain_enter();
    extern __shared__ __align__(1024) uint8_t tiles_smem_raw[];
    uint8_t* smem = tiles_smem_raw + ((1024u - (smem_u32(tiles_smem_raw) & 1023u)) & 1023u);
    uint8_t* b_ring = smem + kWStages * kWStageBytes;
    TileBars* bars = reinterpret_cast<TileBars*>(b_ring + kBStages * kBStageBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 1);
    ItemSlot* slots = reinterpret_cast<ItemSlot*>(tmem_slot + 2);
    int* bounds = reinterpret_cast<int*>(slots + kItemSlots);         // experts + 1 boundaries, then the tiles before each expert
    int* before = bounds + p.experts + 1;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        for (int s = 0; s < kWStages; ++s) { mbar_init(bars->w_full + s, 1); mbar_init(bars->w_empty + s, kDecodeWarps); }
        // a step's operands share a barrier: its rows in shared memory and its decoded weights (eight warps) in tensor memory
        for (int s = 0; s < kBStages; ++s) { mbar_init(bars->full + s, 1 + 8); mbar_init(bars->empty + s, 1); }
        for (int s = 0; s < kItemSlots; ++s) { mbar_init(bars->item_full + s, 1); mbar_init(bars->item_empty + s, kRowsWarps + 1 + kEpilogueWarps); }
        for (int s = 0; s < 2; ++s) { mbar_init(bars->d_full + s, 1); mbar_init(bars->d_empty + s, kEpilogueWarps); }
        mbar_init(&bars->drained, 1);
        mbar_fence_init();
    }
    if (warp == kMmaWarp) { tmem_alloc(tmem_slot, kTileCols); tmem_relinquish(); }
    for (int e = tid; e <= p.experts; e += kTileThreads) bounds[e] = p.boundaries[e];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // all 512 columns, so the allocation starts at column 0: tensor-memory addresses are constants below
    constexpr uint32_t tmem = 0;
    if (warp == 0) {
        int total = 0;
        for (int e0 = 0; e0 < p.experts; e0 += 32) {
            const int e = e0 + lane;
            const int tiles = e < p.experts ? (bounds[e + 1] - bounds[e] + kTileRoutes - 1) / kTileRoutes : 0;
            int sum = tiles;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += up;
            }
            if (e < p.experts) before[e] = total + sum - tiles;
            total += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) before[p.experts] = total;
    }
    __syncthreads();
    // a pair of row tiles: rows r .. r + 127 of the gate and of the up bank, or 256 neighbouring rows of one
    const int row_tiles = p.out_features / (SWIGLU ? 128 : 256), K = p.in_features, chunks = K / 256;
    const int items = before[p.experts] * row_tiles;

    if (warp == kWeightWarp) {
        // Also writes what the other warps need to know of an item, ahead of them by the chunks in flight: the search and the
        // look-up of the rows are 2000 clocks that nobody waits for.
        int fill = 0, turn = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x, ++turn) {
            const TileItem it = item_of(i, bounds, before, p.experts, row_tiles);
            const int slot = turn % kItemSlots;
            ok = __all_sync(0xffffffffu, mbar_wait(bars->item_empty + slot, ((turn / kItemSlots) & 1) ^ 1, p.status));
            if (!ok) break;
            const float g = p.global[p.global_per_expert ? it.expert : 0];
            for (int r = lane; r < kTileRoutes; r += 32) {
                const int t = it.t0 + min(r, it.count - 1), route = p.order[t];
                slots[slot].src[r] = p.by_token ? route / p.topk : t;
                slots[slot].out[r] = make_int2(p.scatter ? route : t, __float_as_int(p.routing ? round_bf16(g * p.routing[route]) : g));
            }
            if (lane == 0) slots[slot].item = it;
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(bars->item_full + slot);
                const int row = it.expert * p.out_features + it.rows * (SWIGLU ? 128 : 256);
                for (int c = 0; c < chunks; ++c, ++fill) {
                    const int st = fill % kWStages;
                    ok = mbar_wait(bars->w_empty + st, ((fill / kWStages) & 1) ^ 1, p.status);
                    if (!ok) break;
                    uint8_t* base = smem + st * kWStageBytes;
                    mbar_expect_tx(bars->w_full + st, kWStageBytes);
                    tma_load_2d(base, &codes_map, c * 128, row, bars->w_full + st);
                    tma_load_2d(base + kCodeTile, SWIGLU ? &codes2_map : &codes_map, c * 128, SWIGLU ? row : row + 128, bars->w_full + st);
                    tma_load_2d(base + 2 * kCodeTile, &scales_map, c * 16, row, bars->w_full + st);
                    tma_load_2d(base + 2 * kCodeTile + kScaleTile, SWIGLU ? &scales2_map : &scales_map, c * 16, SWIGLU ? row : row + 128, bars->w_full + st);
                }
            }
            ok = __shfl_sync(0xffffffffu, ok, 0);
        }
        if (lane == 0)
            for (int f = max(0, fill - kWStages); f < fill; ++f)            // no copy outlives the block
                mbar_wait(bars->w_full + f % kWStages, (f / kWStages) & 1, p.status);
    } else if (warp >= kRowsWarp) {
        // A warp fills one stage: every kBStages-th step, pieces of sixteen bytes, eight lanes a row, handed over once they have
        // arrived.  (TMA gathers four rows an instruction, one lane at a time: 640 clocks a step of 64 rows.  Two warps that
        // fill every step and hand it over some steps later take 700, most of it for the fence.)
        const int st = warp - kRowsWarp, row0 = lane >> 3, piece = lane & 7;
        const uint32_t dst = smem_u32(b_ring) + st * kBStageBytes + row0 * 128;
        int step = 0, use = 0, turn = 0;                                      // steps of the items before this one; uses of the stage
        bool ok = true;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x, step += 4 * chunks, ++turn) {
            const int slot = turn % kItemSlots;
            ok = __all_sync(0xffffffffu, mbar_wait(bars->item_full + slot, (turn / kItemSlots) & 1, p.status));
            if (!ok) break;
            const int passes = ((slots[slot].item.count + 15) & ~15) / 4;
            int src[kTileRoutes / 4];                                         // rows row0 + 4 k
#pragma unroll
            for (int k = 0; k < kTileRoutes / 4; ++k) src[k] = slots[slot].src[row0 + 4 * k];
            __syncwarp();
            if (lane == 0) mbar_arrive(bars->item_empty + slot);
            for (int s = (st + kBStages - step % kBStages) % kBStages; s < 4 * chunks; s += kBStages, ++use) {
                ok = mbar_wait(bars->empty + st, (use & 1) ^ 1, p.status);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                const bf16* from = p.x + s * 64 + piece * 8;
#pragma unroll
                for (int k = 0; k < kTileRoutes / 4; ++k)
                    if (k < passes) copy16_async(dst + k * 512 + ((piece ^ ((row0 + 4 * k) & 7)) << 4), from + (size_t)src[k] * K);
                asm volatile("cp.async.wait_all;" ::: "memory");
                fence_async_proxy();
                __syncwarp();
                if (lane == 0) mbar_arrive(bars->full + st);
            }
        }
    } else if (warp == kMmaWarp) {
        // The whole warp walks the steps so that the operands stay in uniform registers; one lane issues.  (With the loop in
        // one lane an MMA took 90 clocks to issue between the decoding warps.)
        const bool leader = elect_one();
        const uint32_t b0 = desc_lo_sw128(smem_u32(b_ring));
        int bs = 0, phase = 0, as = 0, turn = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x, ++turn) {
            const int slot = turn % kItemSlots;
            ok = __all_sync(0xffffffffu, mbar_wait(bars->item_full + slot, (turn / kItemSlots) & 1, p.status));
            if (!ok) break;
            const uint32_t n = (slots[slot].item.count + 15) & ~15;
            __syncwarp();
            if (lane == 0) mbar_arrive(bars->item_empty + slot);
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
            const uint32_t d = kColD + (turn & 1) * kSetCols;
            ok = __all_sync(0xffffffffu, mbar_wait(bars->d_empty + (turn & 1), ((turn >> 1) & 1) ^ 1, p.status));
            for (int s = 0, m; s < 4 * chunks && ok; s += m) {
                m = ring_ready(bars->full, bs, phase, kBStages, min(4 * chunks - s, kBStages), p.status);
                ok = m > 0;
                if (ok) {
                    tc_fence_after();
                    if (leader) {
                        for (int k = 0; k < m; ++k) {
                            const int at = bs + k < kBStages ? bs + k : bs + k - kBStages;
                            const uint32_t b = b0 + at * (kBStageBytes >> 4), a = kColA + (as + k) % kAStages * 64;
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                umma_bf16_ts(d, a + j * 8, b + 2 * j, idesc, (s | k | j) ? 1u : 0u);
                                umma_bf16_ts(d + kTileRoutes, a + 32 + j * 8, b + 2 * j, idesc, (s | k | j) ? 1u : 0u);
                            }
                            umma_commit(bars->empty + at);
                        }
                    }
                    __syncwarp();
                }
                if ((bs += m) >= kBStages) { bs -= kBStages; phase ^= 1; }
                as = (as + m) % kAStages;
            }
            if (ok && leader) umma_commit(bars->d_full + (turn & 1));
            __syncwarp();
        }
        if (leader) umma_commit(&bars->drained);                          // tensor memory is given back only behind the last MMA
        mbar_wait(&bars->drained, 0, p.status);
    } else if (warp < kDecodeWarps) {
        const int tile = (warp >> 2) & 1, group = warp >> 3, row = (warp & 3) * 32 + lane;
        const uint32_t a = tmem + ((uint32_t)((warp & 3) * 32) << 16) + kColA + tile * 32;
        int fill = 0, slot = group, phase = 0;                              // of the group's next step
        bool ok = true, there = mbar_test_wait(bars->w_full, 0);
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
            for (int c = 0; c < chunks && ok; ++c, ++fill) {
                const int st = fill % kWStages;
                // (a look at a barrier takes some 200 clocks: it is asked for ahead of its use, and again only if it came too early)
                ok = __all_sync(0xffffffffu, there) || __all_sync(0xffffffffu, mbar_wait(bars->w_full + st, (fill / kWStages) & 1, p.status));
                if (!ok) break;
                const uint8_t* codes = smem + st * kWStageBytes + tile * kCodeTile + row * 128;
                const uint4 sc = lds128(smem + st * kWStageBytes + 2 * kCodeTile + tile * kScaleTile + row * 16);
                const uint32_t sw[2] = {group ? sc.y : sc.x, group ? sc.w : sc.z};            // of the two steps of this group
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int piece = 2 * (2 * half + group);
                    const uint4 c0 = lds128(codes + ((piece ^ (row & 7)) << 4)), c1 = lds128(codes + (((piece + 1) ^ (row & 7)) << 4));
                    if (half == 1) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bars->w_empty + st);
                        there = mbar_test_wait(bars->w_full + (fill + 1) % kWStages, ((fill + 1) / kWStages) & 1);
                    }
                    // whether the step kAStages before this one has been multiplied
                    uint64_t* const before_it = bars->empty + (slot >= kAStages ? slot - kAStages : slot + kAStages);
                    const int its_phase = slot >= kAStages ? phase : phase ^ 1;
                    const bool freed = mbar_test_wait(before_it, its_phase);
                    const uint32_t words[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
                    uint32_t v[32];
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const uint32_t scales = e4m3x2_to_f16x2((sw[half] >> (16 * q)) & 0xffffu);
                        decode8<0>(words[4 * q], scales, v + 16 * q);
                        decode8<0>(words[4 * q + 1], scales, v + 16 * q + 4);
                        decode8<1>(words[4 * q + 2], scales, v + 16 * q + 8);
                        decode8<1>(words[4 * q + 3], scales, v + 16 * q + 12);
                    }
                    ok = __all_sync(0xffffffffu, freed) || __all_sync(0xffffffffu, mbar_wait(before_it, its_phase, p.status));
                    if (!ok) break;
                    tc_fence_after();
                    tmem_store32(a + (slot >= kAStages ? slot - kAStages : slot) * 64, v);
                    tmem_store_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bars->full + slot);
                    if ((slot += 2) >= kBStages) { slot -= kBStages; phase ^= 1; }
                }
            }
        }
    } else {
        const int quadrant = warp & 3;
        int turn = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x, ++turn) {
            const int slot = turn % kItemSlots;
            ok = __all_sync(0xffffffffu, mbar_wait(bars->item_full + slot, (turn / kItemSlots) & 1, p.status));
            if (!ok) break;
            const TileItem it = slots[slot].item;
            const int set = turn & 1, n = (it.count + 15) & ~15;
            const float g2 = SWIGLU ? p.global2[p.global_per_expert ? it.expert : 0] : 0.f;
            ok = __all_sync(0xffffffffu, mbar_wait(bars->d_full + set, (turn >> 1) & 1, p.status));
            if (!ok) break;
            tc_fence_after();
            const uint32_t d = tmem + ((uint32_t)(quadrant * 32) << 16) + kColD + set * kSetCols;
            // Neighbouring lanes (weight rows) swap halves of two routes' results, so that a lane stores two rows of one route
            const int odd = lane & 1;
            bf16* out = p.y + (size_t)it.rows * (SWIGLU ? 128 : 256) + quadrant * 32 + (lane & ~1);
            auto swapped = [&](uint32_t mine) {
                const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 1);
                return odd ? __byte_perm(other, mine, 0x7632) : __byte_perm(mine, other, 0x5410);
            };
            auto packed = [](float a, float b) { const __nv_bfloat162 v = __floats2bfloat162_rn(a, b); return *reinterpret_cast<const uint32_t*>(&v); };
            auto lower = [](uint32_t v) { return __uint_as_float(v << 16); };
            auto upper = [](uint32_t v) { return __uint_as_float(v & 0xffff0000u); };
            for (int c = 0; c < n; c += 16) {
                uint32_t u[16], v[16];
                tmem_load16x2(d + c, d + kTileRoutes + c, u, v);
                if (c + 16 >= n) {                                            // both accumulators are in registers
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bars->d_empty + set);
                }
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    const int2 to = slots[slot].out[c + j + odd];             // of the route this lane stores
                    const float f = __int_as_float(to.y);
                    bf16* at = out + (size_t)to.x * p.out_features;
                    if (SWIGLU) {
                        float h[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e)                           // (one gate factor for all routes of an expert)
                            h[e] = round_bf16(silu_precise(round_bf16(__uint_as_float(u[j + e]) * f))) * round_bf16(__uint_as_float(v[j + e]) * g2);
                        const uint32_t two = swapped(packed(h[0], h[1]));
                        if (c + j + odd < it.count) *reinterpret_cast<uint32_t*>(at) = two;
                    } else {
                        uint32_t two[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float a0 = __uint_as_float(e ? v[j] : u[j]), a1 = __uint_as_float(e ? v[j + 1] : u[j + 1]);
                            if (p.routing) {
                                const uint32_t sums = swapped(packed(a0, a1));
                                two[e] = packed(lower(sums) * f, upper(sums) * f);
                            } else {
                                two[e] = swapped(packed(a0 * f, a1 * f));     // one factor for all routes of an expert
                            }
                        }
                        if (c + j + odd < it.count) { *reinterpret_cast<uint32_t*>(at) = two[0]; *reinterpret_cast<uint32_t*>(at + 128) = two[1]; }
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bars->item_empty + slot);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) tmem_dealloc(*tmem_slot, kTileCols);
}

// Block scales: boxes of sixteen bytes (256 inputs) x 128 rows.
int scale_map(CUtensorMap* map, const void* base, long long rows, long long row_bytes) {
    EncodeTiledFn encode = umma_encode_fn();
    if (!encode) return QD_ERR_UNSUPPORTED;
    const cuuint64_t dims[2] = {(cuuint64_t)row_bytes, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)row_bytes};
    const cuuint32_t box[2] = {16, 128}, elem[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? QD_OK : QD_ERR_LAUNCH;
}

template <bool SWIGLU>
int launch_tiles(const TileParams& p, int routes, const void* codes, const void* scales, const void* codes2, const void* scales2, cudaStream_t stream) {
    const long long bank_rows = (long long)p.experts * p.out_features;
    alignas(64) CUtensorMap maps[4];
    const void* banks[4] = {codes, scales, SWIGLU ? codes2 : codes, SWIGLU ? scales2 : scales};
    int rc = QD_OK;
    for (int b = 0; b < 4 && rc == QD_OK; ++b)
        rc = b & 1 ? scale_map(maps + b, banks[b], bank_rows, p.in_features / 16) : umma_make_map(maps + b, banks[b], bank_rows, p.in_features / 2, 128, 128);
    if (rc != QD_OK) return rc;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return QD_ERR_LAUNCH;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    constexpr size_t fixed = kWStages * kWStageBytes + kBStages * kBStageBytes + sizeof(TileBars) + 16 + kItemSlots * sizeof(ItemSlot) + 1024;
    static bool configured[64];
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(expert_tiles_kernel<SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(fixed + (2 * kMaxExperts + 2) * 4)) != cudaSuccess)
            return QD_ERR_LAUNCH;
        configured[dev] = true;
    }
    const long long tiles = std::min(p.experts, routes) + routes / kTileRoutes;
    const long long items = tiles * (p.out_features / (SWIGLU ? 128 : 256));
    const dim3 grid((unsigned)std::max(1ll, std::min<long long>(items, sms > 0 ? sms : 148)));
    return qd_launch(expert_tiles_kernel<SWIGLU>, grid, dim3(kTileThreads), fixed + (2 * p.experts + 2) * 4, stream, 1, p, maps[0], maps[1], maps[2], maps[3]);
}

}  // namespace

bool expert_tiles_cover(int experts, int out_features, int in_features, int out_multiple, const void* x, const void* codes, const void* scales) {
    const uintptr_t align = (uintptr_t)x | (uintptr_t)codes | (uintptr_t)scales;
    return experts <= kMaxExperts && in_features % 256 == 0 && out_features % out_multiple == 0 &&
           (long long)experts * out_features < (1ll << 31) && !(align & 15u);
}

int expert_tiles_matmul(const ExpertTilesArgs& a, cudaStream_t stream) {
    TileParams p = {};
    p.x = (const bf16*)a.x; p.global = a.global; p.order = a.order; p.boundaries = a.boundaries; p.routing = a.routing; p.y = a.y;
    p.experts = a.experts; p.topk = a.topk; p.out_features = a.out_features; p.in_features = a.in_features; p.by_token = a.by_token;
    p.scatter = a.scatter; p.global_per_expert = a.global_per_expert; p.status = a.status;
    return launch_tiles<false>(p, a.routes, a.codes, a.scales, nullptr, nullptr, stream);
}

}  // namespace qd

// h[r] = bf16(bf16(silu(gate(x))) * up(x)) of the routes in sorted order: the gate and up products of the routed experts
// (quickdraw/models/qwen.py:176-191) and their SwiGLU in one launch.
extern "C" int qd_nvfp4_expert_swiglu(const void* x, const void* gate_codes, const void* gate_scales, const float* gate_global,
                                      const void* up_codes, const void* up_scales, const float* up_global, const int32_t* order,
                                      const int32_t* boundaries, void* h, int routes, int experts, int topk, int out_features,
                                      int in_features, int group_size, int global_per_expert, unsigned int* status, void* stream) {
    using namespace qd;
    QD_CHECK_ARG(x && gate_codes && gate_scales && gate_global && up_codes && up_scales && up_global && order && boundaries && h);
    QD_CHECK_ARG(routes > 0 && experts > 0 && topk > 0 && out_features > 0 && in_features > 0);
    if (group_size != 16 || !expert_tiles_cover(experts, out_features, in_features, 128, x, gate_codes, gate_scales) ||
        (((uintptr_t)up_codes | (uintptr_t)up_scales | (uintptr_t)h) & 15u))
        return QD_ERR_UNSUPPORTED;
    TileParams p = {};
    p.x = (const bf16*)x; p.global = gate_global; p.global2 = up_global; p.order = order; p.boundaries = boundaries; p.y = (bf16*)h;
    p.experts = experts; p.topk = topk; p.out_features = out_features; p.in_features = in_features; p.by_token = 1;
    p.global_per_expert = global_per_expert; p.status = status;
    return launch_tiles<true>(p, routes, gate_codes, gate_scales, up_codes, up_scales, (cudaStream_t)stream);
}
