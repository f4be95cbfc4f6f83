// Softmax attention of a prompt chunk on tcgen05.mma: scores and results in tensor memory, probabilities written back there
// as the A operand of the value product.
//
// A block owns TILES x 128 packed (token, head of the group) rows of one key/value head and walks the positions they see in
// tiles of 64.  Per tile and 128 rows: S = Q K^T (both from shared memory), a thread per row takes the softmax in registers,
// P goes over S as two bf16 pieces (sixteen bits), O += P V.  The result is rescaled only when a row's maximum
// has grown by more than 2^8 since the last time (P stays below 2^8 and the sum in fp32, so the quotient is the same to
// rounding): after the first tiles a warp hardly ever reads O before the end.  (Conditional rescaling is published with
// FlashAttention-4.)
//   warps 0 .. 4 TILES - 1   softmax, one row a thread; then the epilogue, for one row tile together with the loading warps
//   warps 4 TILES .. 5 TILES - 1   issue the MMAs of a row tile each: S of key tile i + 1 before O of tile i, so that softmax and products overlap
//   the rest                 keys and values into the 128-byte swizzled layout, two stages of each: by tiled TMA where a tile's 64
//                            rows lie together, else (the last tile, the ring's end) row by row with cp.async, zeros past the end
// Values are read as they lie (rows of a key, the result's columns innermost): a B operand with the columns as the major
// dimension.  Every wait is bounded; a block whose wait ran out writes NaN.
//
// Measured (2048 tokens, with the launch gap; before: mma.sync, eight or sixteen rows a warp).  Head dimension 256, 16/2 heads:
// behind 0 / 2048 / 6144 positions 106 / 193 / 365 us (2000 positions by mma.sync 1017), 128 and 16 tokens behind 500 positions 36 and 33 us.  128 columns, window
// 1024: 16/4 heads 48 us (243), 16 heads with 64 shared key columns 64 us (293).  With one warp issuing for both row tiles, and a descriptor built
// for every MMA, these were 110 / 207 / 402, 38 and 35, 55 and 73: that warp took 4200 clocks for a key tile, 90 an MMA.  Now a key tile takes
// 2300 clocks at 192 + 128 columns, of which the tensor core has 2180 (a product of S is bound by shared memory: 48 clocks for 64 columns).
// One piece, eight bits, took 120 / 199 / 1290 us there where two took 129 / 225 / 1611 (before the epilogue was shared), but since the largest P is not one here (the reference lags behind the
// maximum) its rounding reaches the result: 2.04e-3 from 64 bits with sharp scores, where the result's own rounding is 1.65e-3
// and mma.sync with the exact maximum had 1.72e-3.  Two pieces: 1.65e-3.
#pragma once
#include <cuda.h>

#include <type_traits>

#include "common.cuh"

namespace qd {
namespace flash {

constexpr int kKeys = 64;

struct In {
    const bf16* q;                         // [tokens, heads, QD]
    const bf16* k; const bf16* v;          // rows of a position; head g's columns at g * dim, g * DV
    const bf16* common;                    // key columns dim .. QD - 1, shared by the heads; rows as of k
    const int* position_ptr;
    const float* slopes;                   // per head, off the scaled scores per position of distance; NULL: none
    long long ld_k, ld_v, ld_common;
    float scale;                           // times log2 e
    int position, tokens, heads, kv_heads, dim, capacity, span, chunked;        // span 0: everything up to a row's own position
    int boxes;                             // the maps below hold; set by launch
};
struct Maps { CUtensorMap k, v, common; };     // boxes of 64 columns x 64 rows

QD_DEVINL int lowest(const In& p, int position) {
    if (p.span == 0) return 0;
    if (p.chunked) return position - position % p.span;
    return max(0, position - p.span + 1);
}

// Shared-memory descriptors, lower words; the upper one is the same for all: 1024 bytes between groups of eight rows, 128-byte swizzle.
// The products walk by adding to them (16-byte units): a descriptor built anew for every MMA made the issuing warp the bound (90 clocks an MMA).
constexpr uint32_t kDescHigh = (1024u >> 4) | (1u << 14) | (1u << 30);
QD_DEVINL uint32_t desc_k(uint32_t addr) { return ((addr >> 4) & 0x3fffu) | (1u << 16); }          // K-major
// MN-major: 64 columns innermost; `apart` bytes to the next 64 columns
QD_DEVINL uint32_t desc_mn(uint32_t addr, uint32_t apart) { return ((addr >> 4) & 0x3fffu) | ((apart >> 4) << 16); }
constexpr uint32_t idesc(int n, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}
QD_DEVINL void mma_ss(uint32_t d, uint32_t a, uint32_t b, uint32_t i, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 da, {%1, %4};\n\tmov.b64 db, {%2, %4};\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "r"(b), "r"(i), "r"(kDescHigh), "r"(accumulate) : "memory");
}
QD_DEVINL void mma_ts(uint32_t d, uint32_t a, uint32_t b, uint32_t i, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 db, {%2, %4};\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "r"(b), "r"(i), "r"(kDescHigh), "r"(accumulate) : "memory");
}
QD_DEVINL void commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
QD_DEVINL void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
QD_DEVINL void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
QD_DEVINL void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
QD_DEVINL bool elected() {
    uint32_t leader;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(leader));
    return leader != 0;
}
// 32 columns of this warp's lanes.  The wait names the registers, so that no arithmetic on them moves in front of it.
QD_DEVINL void load32(uint32_t addr, float (&v)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]),
                   "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]),
                   "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]),
                   "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
                 : "r"(addr) : "memory");
}
QD_DEVINL void loaded(float (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]), "+f"(v[8]), "+f"(v[9]),
                   "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15])
                 :: "memory");
#pragma unroll
    for (int j = 16; j < 32; ++j) asm volatile("" : "+f"(v[j]));
}
template <typename T>
QD_DEVINL void store32(uint32_t addr, const T (&v)[32]) {
    const auto bits = [&](int i) { return *reinterpret_cast<const uint32_t*>(&v[i]); };
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
                 "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(addr), "r"(bits(0)), "r"(bits(1)), "r"(bits(2)), "r"(bits(3)), "r"(bits(4)), "r"(bits(5)), "r"(bits(6)), "r"(bits(7)),
                   "r"(bits(8)), "r"(bits(9)), "r"(bits(10)), "r"(bits(11)), "r"(bits(12)), "r"(bits(13)), "r"(bits(14)), "r"(bits(15)),
                   "r"(bits(16)), "r"(bits(17)), "r"(bits(18)), "r"(bits(19)), "r"(bits(20)), "r"(bits(21)), "r"(bits(22)), "r"(bits(23)),
                   "r"(bits(24)), "r"(bits(25)), "r"(bits(26)), "r"(bits(27)), "r"(bits(28)), "r"(bits(29)), "r"(bits(30)), "r"(bits(31)) : "memory");
}
QD_DEVINL void stored() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
QD_DEVINL void copy16(uint32_t dst, const void* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
QD_DEVINL void load_box(uint32_t dst, const CUtensorMap* map, int column, int row, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(column), "r"(row), "r"(smem_u32(bar)) : "memory");
}
QD_DEVINL float exp2_fast(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
QD_DEVINL uint32_t pair(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

template <int QD, int DV, int TILES>
struct Shape {
    static constexpr int kLoaders = 12 - 4 * TILES, kPerStage = kLoaders / 4;            // loader warps; of one stage of keys or values
    static constexpr int kThreads = 32 * (5 * TILES + kLoaders);
    static constexpr int kScores = TILES == 1 ? 3 : 2;                                  // score buffers of a row tile
    static constexpr int kTileCols = DV + kScores * kKeys;
    static constexpr int kQBytes = TILES * 128 * QD * 2, kKBytes = kKeys * QD * 2, kVBytes = kKeys * DV * 2;
    // A block of one row tile has eight loading warps that are free at its end: a row's columns are shared by three warps then.  (Alone
    // a softmax warp takes 1.4 us for 32 columns, most of it the gates: 16 tokens behind 500 positions 46 us, 35 shared.)
    static constexpr int kSharers = TILES == 1 ? 1 + kLoaders / 4 : 1;
    static constexpr int kStatsBytes = TILES == 1 ? 128 * 8 : 0;
    static constexpr size_t kSmem = kQBytes + 2 * (kKBytes + kVBytes) + 512 + kStatsBytes + 1024;
    static_assert(TILES * kTileCols <= 512 && QD % 64 == 0 && DV % 64 == 0 && DV <= 256 && kLoaders % 4 == 0 && kSmem <= 227 * 1024, "");
};

template <int TILES>
struct Bars {
    uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[TILES][3], p_full[TILES][3], o_done[TILES][2], q_full, stats_full, drained;
};

// Columns `column` .. + 31 of the rows of the warp's lanes `rows` once more, summed in fp32 over the keys that a row sees and no
// others; a lane's row, `m` and `l` are as for Out.  For results that are not finite although their rows' probabilities are: a value
// that is not finite makes NaN of its products with the zeros of the keys that a row does not see, and with pieces of a
// probability that are zero.
template <int QD, int DV, typename Out>
__device__ __noinline__ void plain_columns(const In& p, const Out& out, unsigned rows, int row, float m, float l, int column) {
    const int lane = threadIdx.x & 31, share = p.heads / p.kv_heads, g = blockIdx.x;
    for (; rows; rows &= rows - 1) {
        const int from = __ffs(rows) - 1, r = __shfl_sync(0xffffffffu, row, from), head = g * share + r % share;
        const float reference = __shfl_sync(0xffffffffu, m, from);
        const int pos = (p.position_ptr ? *p.position_ptr : p.position) + r / share;
        const bf16* q = p.q + ((size_t)(r / share) * p.heads + head) * QD;
        const float slope = p.slopes ? p.slopes[head] * 1.4426950408889634f : 0.f;
        float sum = 0.f;
#pragma unroll 1
        for (int j = lowest(p, pos); j <= pos; ++j) {
            const long long slot = j % p.capacity;
            const bf16* own = p.k + slot * p.ld_k + g * p.dim;
            float score = 0.f;
#pragma unroll 1
            for (int d = lane; d < QD; d += 32)
                score = fmaf(ld_bf16(q + d), ld_bf16(d < p.dim ? own + d : p.common + slot * p.ld_common + (d - p.dim)), score);
            const float w = exp2f(fmaf(warp_sum(score), p.scale, slope * (float)(j - pos)) - reference);
            sum = fmaf(w, ld_bf16(p.v + slot * p.ld_v + g * DV + column + lane), sum);
        }
        float o[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] = __shfl_sync(0xffffffffu, sum, e);
        if (lane == from) out(row / share, head, column, o, m, l);
        __syncwarp();
    }
}

// Out: called per row and 32 columns as out(token, head, c0, o, m, l) with the unnormalised columns c0 .. c0 + 31 and the row's
// softmax state (log2 of the reference, the sum relative to it); l NaN marks a failed wait.
template <int QD, int DV, int TILES, typename Out>
__global__ void __launch_bounds__(Shape<QD, DV, TILES>::kThreads, 1) flash_umma_kernel(const __grid_constant__ In p, const __grid_constant__ Maps maps, const __grid_constant__ Out out) {
    chain_enter();
    using S = Shape<QD, DV, TILES>;
    extern __shared__ __align__(16) uint8_t flash_raw[];        // (the largest alignment of a file holds for all its kernels)
    uint8_t* smem = flash_raw + ((1024u - (smem_u32(flash_raw) & 1023u)) & 1023u);
    uint8_t* ks = smem + S::kQBytes;
    uint8_t* vs = ks + 2 * S::kKBytes;
    Bars<TILES>* bars = reinterpret_cast<Bars<TILES>*>(vs + 2 * S::kVBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 1);
    static_assert(sizeof(Bars<TILES>) + 8 <= 512, "");
    float2* stats = reinterpret_cast<float2*>(reinterpret_cast<uint8_t*>(bars) + 512);        // of the rows, for those who share the epilogue
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int kMma = 4 * TILES, kRows = 128 * TILES;
    const int share = p.heads / p.kv_heads, g = blockIdx.x, total = p.tokens * share;
    const int r0 = (int)(gridDim.y - 1 - blockIdx.y) * kRows;                 // the longest rows first
    const int base = p.position_ptr ? *p.position_ptr : p.position;
    const int pos_first = base + r0 / share, pos_last = base + (min(r0 + kRows, total) - 1) / share;
    const int key_first = lowest(p, pos_first), tiles = (pos_last - key_first) / kKeys + 1;

    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(bars->k_full + s, S::kPerStage); mbar_init(bars->v_full + s, S::kPerStage);
            mbar_init(bars->k_empty + s, TILES); mbar_init(bars->v_empty + s, TILES);
            for (int t = 0; t < TILES; ++t) mbar_init(&bars->o_done[t][s], 1);
        }
        for (int t = 0; t < TILES; ++t)
            for (int s = 0; s < 3; ++s) { mbar_init(&bars->s_full[t][s], 1); mbar_init(&bars->p_full[t][s], 4); }
        mbar_init(&bars->q_full, 4 * TILES);
        mbar_init(&bars->stats_full, 4);
        mbar_init(&bars->drained, TILES);
        mbar_fence_init();
    }
    if (warp == kMma) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    constexpr uint32_t tmem = 0;               // all 512 columns, so the allocation starts at column 0
    // the result of a row of tile t, 32 columns of every kSharers * 32, from the first-th 32 on
    const auto finish = [&](int t, int row, float m, float l, int first) {
        const uint32_t o_at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + t * S::kTileCols;
#pragma unroll 1
        for (int c = first * 32; c < DV; c += S::kSharers * 32) {
            float o[32];
            load32(o_at + c, o);
            loaded(o);
            bool odd = false;
#pragma unroll
            for (int e = 0; e < 32; ++e) odd |= !(fabsf(o[e]) < INFINITY);
            if (row < total) out(row / share, g * share + row % share, c, o, m, l);
            const unsigned rows = __ballot_sync(0xffffffffu, odd && row < total && l < INFINITY);      // (and the whole warp goes on)
            if (rows) plain_columns<QD, DV>(p, out, rows, row, m, l, c);
        }
    };

    if (warp >= kMma + TILES) {
        // ---- keys and values: warps of (matrix, stage) take every second tile
        const int w = warp - kMma - TILES, part = w >> 2, stage = w & 1, values = (w >> 1) & 1;
        constexpr int kRowsEach = kKeys / S::kPerStage;
        const uint32_t dst = smem_u32(values ? vs + stage * S::kVBytes : ks + stage * S::kKBytes);
        uint64_t* full = (values ? bars->v_full : bars->k_full) + stage;
        uint64_t* empty = (values ? bars->v_empty : bars->k_empty) + stage;
        const int slot_first = key_first % p.capacity, ld_own = (int)(values ? p.ld_v : p.ld_k), ld_common = (int)p.ld_common;
        const bf16* own = values ? p.v + g * DV : p.k + g * p.dim;
        bool ok = true;
        int issued = -1;                                                     // the last tile whose copies this warp has started
        const auto fill = [&](auto pieces, int tile) {
            constexpr int kPieces = decltype(pieces)::value, kBatch = 8;
            static_assert(kRowsEach * kPieces % (32 * kBatch) == 0, "");
#pragma unroll 1
            for (int i0 = lane; i0 < kRowsEach * kPieces; i0 += 32 * kBatch) {
                // addresses of a batch first: computed between the copies they are one long chain (150 clocks a copy)
                const bf16* src[kBatch];
                uint32_t to[kBatch];
                bool inside[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const int i = i0 + 32 * u, r = part * kRowsEach + i / kPieces, c = i % kPieces, ahead = tile * kKeys + r;
                    inside[u] = key_first + ahead <= pos_last;
                    int slot = inside[u] ? slot_first + ahead : 0;
                    if (slot >= p.capacity) slot -= p.capacity;              // what a block sees fits the ring
                    src[u] = values || c * 8 < p.dim ? own + (long long)slot * ld_own + c * 8 : p.common + (long long)slot * ld_common + (c * 8 - p.dim);
                    to[u] = dst + (c >> 3) * (kKeys * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4);
                }
#pragma unroll
                for (int u = 0; u < kBatch; ++u) copy16(to[u], src[u], inside[u]);
            }
        };
        for (int tile = stage; tile < tiles && ok; tile += 2) {
            ok = __all_sync(0xffffffffu, mbar_wait(empty, ((tile >> 1) & 1) ^ 1, nullptr));
            if (!ok) break;
            issued = tile;
            // Boxes where the tile is whole: row by row an SM copies 18 bytes a clock, by TMA what L2 gives.
            const int slot = (int)((slot_first + (long long)tile * kKeys) % p.capacity);
            if (p.boxes && key_first + (tile + 1) * kKeys - 1 <= pos_last && slot + kKeys <= p.capacity) {
                if (lane == 0) {
                    if (part) {
                        mbar_arrive(full);
                    } else {
                        mbar_expect_tx(full, values ? S::kVBytes : S::kKBytes);
                        for (int c = 0; c < (values ? DV : QD); c += 64) {
                            const bool shared = !values && c >= p.dim;
                            load_box(dst + (c >> 6) * (kKeys * 128), values ? &maps.v : shared ? &maps.common : &maps.k,
                                     values ? g * DV + c : shared ? c - p.dim : g * p.dim + c, slot, full);
                        }
                    }
                }
                __syncwarp();
                continue;
            }
            if (values) fill(std::integral_constant<int, DV / 8>{}, tile);
            else fill(std::integral_constant<int, QD / 8>{}, tile);
            asm volatile("cp.async.wait_all;" ::: "memory");
            fence_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(full);
        }
        if (issued >= 0) mbar_wait(full, (issued >> 1) & 1, nullptr);        // no copy outlives the block, also where a wait ran out
        if constexpr (S::kSharers > 1) {
            __syncwarp();
            const int r = (warp & 3) * 32 + lane;
            // behind the statistics the last product has ended: its barrier is in its last phase
            const bool done = __all_sync(0xffffffffu, mbar_wait(&bars->stats_full, 0, nullptr) &&
                                                      mbar_wait(&bars->o_done[0][(tiles - 1) & 1], ((tiles - 1) >> 1) & 1, nullptr));
            const float2 ml = done ? stats[r] : make_float2(0.f, NAN);
            fence_after();
            finish(0, r0 + r, ml.x, ml.y, 1 + (w >> 2));
        }
    } else if (warp >= kMma) {
        const int t = warp - kMma;
        const bool leader = elected();
        const uint32_t qa = desc_k(smem_u32(smem) + t * (128 * QD * 2)), ka = desc_k(smem_u32(ks)), va = desc_mn(smem_u32(vs), kKeys * 128);
        const uint32_t o_at = tmem + t * S::kTileCols;
        bool ok = true;
        const auto scores = [&](int i) {                                     // S of key tile i
            const uint32_t d = o_at + DV + (i % S::kScores) * kKeys, b = ka + (i & 1) * (S::kKBytes >> 4);
#pragma unroll
            for (int j = 0; j < QD / 16; ++j)
                mma_ss(d, qa + (j >> 2) * (16384 >> 4) + (j & 3) * 2, b + (j >> 2) * (kKeys * 128 >> 4) + (j & 3) * 2, idesc(kKeys, 0), j ? 1u : 0u);
            commit(&bars->s_full[t][i % S::kScores]);
            commit(bars->k_empty + (i & 1));
        };
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->q_full, 0, nullptr) && mbar_wait(bars->k_full, 0, nullptr));
        if (ok) {
            fence_after();
            if (leader) scores(0);
            __syncwarp();
        }
        for (int i = 0; i < tiles && ok; ++i) {
            if (i + 1 < tiles) {
                const int before = i + 1 - S::kScores;                        // the probabilities that lie where these scores go are read
                ok = __all_sync(0xffffffffu, mbar_wait(bars->k_full + ((i + 1) & 1), ((i + 1) >> 1) & 1, nullptr) &&
                                                 (before < 0 || mbar_wait(&bars->o_done[t][before & 1], (before >> 1) & 1, nullptr)));
                fence_after();
                if (ok && leader) scores(i + 1);
                __syncwarp();
            }
            if (ok)
                ok = __all_sync(0xffffffffu, mbar_wait(bars->v_full + (i & 1), (i >> 1) & 1, nullptr) &&
                                                 mbar_wait(&bars->p_full[t][i % S::kScores], (i / S::kScores) & 1, nullptr));
            if (ok) {
                fence_after();
                if (leader) {
                    const uint32_t a = o_at + DV + (i % S::kScores) * kKeys, b = va + (i & 1) * (S::kVBytes >> 4);
#pragma unroll
                    for (int j = 0; j < kKeys / 16; ++j) {
                        mma_ts(o_at, a + j * 8, b + j * (2048 >> 4), idesc(DV, 1), (i | j) ? 1u : 0u);
                        mma_ts(o_at, a + 32 + j * 8, b + j * (2048 >> 4), idesc(DV, 1), 1u);
                    }
                    commit(&bars->o_done[t][i & 1]);
                    commit(bars->v_empty + (i & 1));
                }
                __syncwarp();
            }
        }
        if (leader) commit(&bars->drained);                 // tensor memory is given back only behind the last MMA
        mbar_wait(&bars->drained, 0, nullptr);
    } else {
        {   // the queries: [row tile][64 columns][128 rows][128 bytes]
            constexpr int kPieces = QD / 8;
#pragma unroll 8
            for (int i = tid; i < kRows * kPieces; i += kRows) {
                const int r = i / kPieces, c = i % kPieces, query = r0 + r;
                const bool inside = query < total;
                const bf16* src = p.q + (inside ? ((size_t)(query / share) * p.heads + g * share + query % share) * QD + c * 8 : 0);
                copy16(smem_u32(smem) + (r >> 7) * (128 * QD * 2) + (c >> 3) * 16384 + (r & 127) * 128 + (((c & 7) ^ (r & 7)) << 4), src, inside);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            fence_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->q_full);
        }
        const int t = warp >> 2, row = r0 + tid, tile_last = base + (min(r0 + (t + 1) * 128, total) - 1) / share;
        const int pos = base + row / share, low = lowest(p, pos), tile_first = base + (r0 + t * 128) / share, low_last = lowest(p, max(tile_last, tile_first));
        const int head = g * share + row % share;
        const uint32_t o_at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + t * S::kTileCols, s_at = o_at + DV;
        const float slope = p.slopes ? p.slopes[head] * 1.4426950408889634f : 0.f;
        const bool plain = !p.slopes && p.scale > 0.f;
        float m = -INFINITY, l = 0.f;
        bool ok = true;
        for (int i = 0; i < tiles; ++i) {
            const int b = i % S::kScores, j0 = key_first + i * kKeys;
            ok = __all_sync(0xffffffffu, mbar_wait(&bars->s_full[t][b], (i / S::kScores) & 1, nullptr));
            if (!ok) break;
            fence_after();
            float s[2][32];
            load32(s_at + b * kKeys, s[0]);
            load32(s_at + b * kKeys + 32, s[1]);
            loaded(s[0]);
            loaded(s[1]);
            const bool inside = j0 + kKeys - 1 <= tile_first && j0 >= low_last;
            float factor = p.scale, top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            if (!(inside && plain)) {
                factor = 1.f;
#pragma unroll
                for (int c = 0; c < kKeys; ++c) {
                    const int j = j0 + c;
                    const float x = fmaf(s[c >> 5][c & 31], p.scale, slope * (float)(j - pos));
                    s[c >> 5][c & 31] = (j <= pos && j >= low) ? x : -INFINITY;
                }
            }
#pragma unroll
            for (int c = 0; c < kKeys; ++c) top[c & 3] = fmaxf(top[c & 3], s[c >> 5][c & 31]);
            const float mx = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])) * factor;
            const bool grown = mx > m + 8.f;                                  // (also from -inf)
            if (__any_sync(0xffffffffu, grown)) {
                const float keep = grown ? (m == -INFINITY ? 0.f : exp2_fast(m - mx)) : 1.f;
                if (grown) { m = mx; l *= keep; }
                if (i > 0) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&bars->o_done[t][(i - 1) & 1], ((i - 1) >> 1) & 1, nullptr));
                    if (!ok) break;
                    fence_after();
#pragma unroll 1
                    for (int c = 0; c < DV; c += 32) {
                        float o[32];
                        load32(o_at + c, o);
                        loaded(o);
#pragma unroll
                        for (int e = 0; e < 32; ++e) o[e] *= keep;
                        store32(o_at + c, o);
                    }
                }
            }
            const float sub = m == -INFINITY ? 0.f : m;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < kKeys; ++c) {
                const float e = exp2_fast(fmaf(s[c >> 5][c & 31], factor, -sub));
                s[c >> 5][c & 31] = e;
                sum[c & 3] += e;
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            uint32_t hi[32];
#pragma unroll
            for (int c = 0; c < 32; ++c) hi[c] = pair(s[c >> 4][(2 * c) & 31], s[c >> 4][(2 * c + 1) & 31]);
            store32(s_at + b * kKeys, hi);
            uint32_t lo[32];
#pragma unroll
            for (int c = 0; c < 32; ++c)
                lo[c] = pair(s[c >> 4][(2 * c) & 31] - __uint_as_float(hi[c] << 16), s[c >> 4][(2 * c + 1) & 31] - __uint_as_float(hi[c] & 0xffff0000u));
            store32(s_at + b * kKeys + 32, lo);
            stored();
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->p_full[t][b]);
        }
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&bars->o_done[t][(tiles - 1) & 1], ((tiles - 1) >> 1) & 1, nullptr));
        fence_after();
        if (!ok) l = NAN;
        if constexpr (S::kSharers > 1) {
            stats[tid] = make_float2(m, l);
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->stats_full);
        }
        finish(t, row, m, l, 0);
    }
    fence_before();
    __syncthreads();
    if (warp == kMma) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*tmem_slot), "r"(512) : "memory");
}

// false where TMA does not take the matrix (its rows are then copied one by one)
inline bool map_of(CUtensorMap* map, const void* base, long long columns, long long ld, long long rows) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult result;
        const bool found = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &result) == cudaSuccess;
        return reinterpret_cast<Encode>(found && result == cudaDriverEntryPointSuccess ? f : nullptr);
    }();
    const cuuint64_t dims[2] = {(cuuint64_t)columns, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * sizeof(bf16)};
    const cuuint32_t box[2] = {64, kKeys}, elem[2] = {1, 1};
    return encode && encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int QD, int DV, int TILES, typename Out>
int launch(In p, const Out& out, cudaStream_t stream) {
    alignas(64) Maps maps = {};
    p.boxes = p.dim % 64 == 0 && p.capacity >= kKeys && map_of(&maps.k, p.k, (long long)p.kv_heads * p.dim, p.ld_k, p.capacity) &&
              map_of(&maps.v, p.v, (long long)p.kv_heads * DV, p.ld_v, p.capacity) &&
              (p.dim == QD || map_of(&maps.common, p.common, QD - p.dim, p.ld_common, p.capacity));
    constexpr size_t smem = Shape<QD, DV, TILES>::kSmem;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return QD_ERR_LAUNCH;
    static bool configured[64];
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(flash_umma_kernel<QD, DV, TILES, Out>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
            return QD_ERR_LAUNCH;
        configured[dev] = true;
    }
    const long long rows = (long long)p.tokens * (p.heads / p.kv_heads);
    const dim3 grid(p.kv_heads, (unsigned)((rows + 128 * TILES - 1) / (128 * TILES)));
    return qd_launch(flash_umma_kernel<QD, DV, TILES, Out>, grid, dim3(Shape<QD, DV, TILES>::kThreads), smem, stream, 1, p, maps, out);
}

}  // namespace flash
}  // namespace qd
