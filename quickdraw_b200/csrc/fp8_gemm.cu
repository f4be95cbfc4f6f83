// Static-FP8 projection of a chunk of tokens: y[t] = W q(x[t]) for an E4M3 matrix with scalar
// weight and activation scales (FP8Linear: quickdraw/models/weights.py:58-74; arithmetic of
// fp8_gemv, quickdraw/models/qwen.py:25-33: q(x) = e4m3(clamp(x / input_scale, +-448)), products
// exact, fp32 sum, both scales on the sum, one bf16 rounding).  The one-launch step takes such
// mixers token by token; this is the form for prompt chunks and decode batches.
//
//   quantiser   x bf16 [tokens, K] -> E4M3 bytes [tokens, K] (round to nearest even, saturating)
//   product     tcgen05.mma kind::f8f6f4, both operands by tiled TMA (128-byte swizzle), persistent
//               blocks with two accumulators in tensor memory, so that one tile's results are
//               scaled and stored while the next is multiplied.  Tile = 128 tokens x 32 .. 256
//               weight rows.  Bound by the operands' way from L2 (a 128 x 256 tile: 170 operations
//               per byte): 8192 x 8192 x 2048 in 122 us = 2 240 TFLOP/s, 2047 x 2048 x 4096 in 16.5 us; on
//               mma.sync.m16n8k32, as before, 845 us (325 TFLOP/s) and 118 us.
#include "umma.cuh"

namespace qd {
namespace {

constexpr int kF8Tokens = 128, kF8Chunk = 128;      // inputs per stage: one swizzled row of 128 bytes
template <int TN> struct F8Tile {
    static constexpr int kABytes = kF8Tokens * kF8Chunk, kStageBytes = kABytes + TN * kF8Chunk;
    static constexpr int kStages = TN == 256 ? 4 : TN == 128 ? 6 : 8;
    static constexpr size_t kSmem = (size_t)kStages * kStageBytes + (2 * kStages + 5) * 8 + 16 + 1024;
    // fp32 accumulator, E4M3 A and B (format 0), K-major, N >> 3 at 17, M >> 4 at 24
    static constexpr uint32_t kDesc = (1u << 4) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(kF8Tokens >> 4) << 24);
};
constexpr int kF8Threads = 192;      // TMA, MMA, four warps of 32 tokens each

__global__ void __launch_bounds__(256) fp8_quantize_rows_kernel(const uint4* __restrict__ x, const float* __restrict__ in_scale,
                                                                uint2* __restrict__ q, long long n8) {
    chain_enter();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n8) return;
    const float s = *in_scale;
    const uint4 v = x[i];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t out[2] = {0u, 0u};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t lo = __nv_cvt_float_to_fp8(__fdiv_rn(__uint_as_float(w[k] << 16), s), __NV_SATFINITE, __NV_E4M3);
        const uint32_t hi = __nv_cvt_float_to_fp8(__fdiv_rn(__uint_as_float(w[k] & 0xffff0000u), s), __NV_SATFINITE, __NV_E4M3);
        out[k >> 1] |= (lo | (hi << 8)) << (16 * (k & 1));
    }
    q[i] = make_uint2(out[0], out[1]);
}

QD_DEVINL void umma_e4m3(uint32_t d_tmem, uint32_t a_low, uint32_t b_low, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
                 "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], da, db, %3, p;\n\t}"
                 ::"r"(d_tmem), "r"(a_low), "r"(b_low), "r"(idesc), "r"(accumulate), "r"(kDescHiSw128) : "memory");
}

struct F8Params { const float* w_scale; const float* in_scale; bf16* y; int tokens, rows, chunks, across, tiles; };

template <int TN>
__global__ void __launch_bounds__(kF8Threads, 1)
fp8_gemm_kernel(const __grid_constant__ F8Params p, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap) {
    chain_enter();
    using Tile = F8Tile<TN>;
    constexpr int kStages = Tile::kStages;
    extern __shared__ __align__(1024) uint8_t f8_smem_raw[];
    uint8_t* smem = f8_smem_raw + ((1024u - (smem_u32(f8_smem_raw) & 1023u)) & 1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * Tile::kStageBytes);
    uint64_t* empty = full + kStages;
    uint64_t* ready = empty + kStages;         // an accumulator holds a whole tile
    uint64_t* taken = ready + 2;               // it has been read
    uint64_t* drained = taken + 2;             // every MMA has ended
    uint32_t* slot = reinterpret_cast<uint32_t*>(drained + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(ready + s, 1); mbar_init(taken + s, 4); }
        mbar_init(drained, 1);
        mbar_fence_init();
    }
    if (warp == 1) { tmem_alloc(slot, 2 * TN); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *slot;
    const int mine = (p.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x, steps = mine * p.chunks;

    if (warp == 0) {
        const bool leader = elect_one();
        int issued = 0, st = 0, n = 1, c = 0, tile = blockIdx.x;
        uint32_t parity = 1;                       // (a new barrier's phase before the first is over)
        for (; issued < steps; issued += n) {
            n = ring_ready(empty, st, parity, kStages, min(steps - issued, kStages), nullptr);
            if (n == 0) break;
            for (int u = 0; u < n; ++u, ++c) {
                if (c == p.chunks) { c = 0; tile += gridDim.x; }
                const int at = st + u < kStages ? st + u : st + u - kStages;
                if (leader) {
                    uint8_t* a = smem + at * Tile::kStageBytes;
                    mbar_expect_tx(full + at, Tile::kStageBytes);          // rows past a matrix's end arrive as zeros and count in full
                    tma_load_2d(a, &xmap, c * kF8Chunk, tile / p.across * kF8Tokens, full + at);
                    tma_load_2d(a + Tile::kABytes, &wmap, c * kF8Chunk, tile % p.across * TN, full + at);
                }
            }
            __syncwarp();
            st += n;
            if (st >= kStages) { st -= kStages; parity ^= 1u; }
        }
        if (n == 0)             // leave no copy in flight behind
            for (int s = issued > kStages ? issued - kStages : 0; s < issued; ++s)
                mbar_wait(full + s % kStages, (s / kStages) & 1, nullptr);
    } else if (warp == 1) {
        const bool leader = elect_one();
        const uint32_t low0 = __shfl_sync(0xffffffffu, desc_lo_sw128(smem_u32(smem)), 0), to = __shfl_sync(0xffffffffu, tmem, 0);
        int st = 0, n = 1;
        uint32_t parity = 0;
        for (int k = 0; k < mine && n; ++k) {
            if (k >= 2 && !__all_sync(0xffffffffu, mbar_wait(taken + (k & 1), ((k >> 1) - 1) & 1, nullptr))) break;
            tc_fence_after();
            for (int c = 0; c < p.chunks; c += n) {
                n = ring_ready(full, st, parity, kStages, min(p.chunks - c, kStages), nullptr);
                if (n == 0) break;
                tc_fence_after();
                if (leader) {
                    for (int u = 0; u < n; ++u) {
                        const int at = st + u < kStages ? st + u : st + u - kStages;
                        const uint32_t a = low0 + at * (Tile::kStageBytes >> 4), b = a + (Tile::kABytes >> 4);
#pragma unroll
                        for (int j = 0; j < kF8Chunk / 32; ++j) umma_e4m3(to + (k & 1) * TN, a + 2 * j, b + 2 * j, Tile::kDesc, (c | u | j) ? 1u : 0u);
                        umma_commit(empty + at);
                    }
                }
                __syncwarp();
                st += n;
                if (st >= kStages) { st -= kStages; parity ^= 1u; }
            }
            if (n && leader) umma_commit(ready + (k & 1));
            __syncwarp();
        }
        if (leader) umma_commit(drained);             // tensor memory is given back only behind the last MMA, also where a wait ran out
        mbar_wait(drained, 0, nullptr);
    } else {
        const int quadrant = warp & 3;
        const float s_in = *p.in_scale, s_w = *p.w_scale;
        const bool vectors = p.rows % 8 == 0 && ((uintptr_t)p.y & 15u) == 0;
        bool ok = true;
        for (int k = 0; k < mine; ++k) {
            const int tile = blockIdx.x + k * gridDim.x;
            const int token = tile / p.across * kF8Tokens + quadrant * 32 + lane, n0 = tile % p.across * TN;
            ok = __all_sync(0xffffffffu, ok && mbar_wait(ready + (k & 1), (k >> 1) & 1, nullptr));
            tc_fence_after();
            bf16* out = p.y + (size_t)token * p.rows;
#pragma unroll 1
            for (int c = 0; c < TN; c += 16) {
                if (n0 + c >= p.rows) break;
                uint32_t v[16];
                if (ok) {
                    tmem_load16(tmem + ((uint32_t)(quadrant * 32) << 16) + (k & 1) * TN + c, v);
                    tmem_load_wait();
                } else {        // a wait ran out (no status word here): the results say so
#pragma unroll
                    for (int q = 0; q < 16; ++q) v[q] = 0x7fc00000u;
                }
                if (token < p.tokens) {
                    uint32_t packed[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const __nv_bfloat162 two = __floats2bfloat162_rn((__uint_as_float(v[2 * q]) * s_in) * s_w, (__uint_as_float(v[2 * q + 1]) * s_in) * s_w);
                        packed[q] = *reinterpret_cast<const uint32_t*>(&two);
                    }
                    if (vectors && n0 + c + 16 <= p.rows) {
                        *reinterpret_cast<uint4*>(out + n0 + c) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                        *reinterpret_cast<uint4*>(out + n0 + c + 8) = make_uint4(packed[4], packed[5], packed[6], packed[7]);
                    } else {        // rows is even and y on a four-byte boundary
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            if (n0 + c + 2 * q < p.rows) *reinterpret_cast<uint32_t*>(out + n0 + c + 2 * q) = packed[q];
                    }
                }
                __syncwarp();       // the next read of tensor memory is the whole warp's
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(taken + (k & 1));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 2 * TN);
}

template <int TN>
int launch_f8(const void* q, const void* w, F8Params p, int in_features, int sms, cudaStream_t stream) {
    using Tile = F8Tile<TN>;
    if (cudaFuncSetAttribute(fp8_gemm_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Tile::kSmem) != cudaSuccess) return QD_ERR_LAUNCH;
    alignas(64) CUtensorMap xmap = {}, wmap = {};
    int rc = umma_make_map(&xmap, q, p.tokens, in_features, kF8Chunk, kF8Tokens);
    if (rc == QD_OK) rc = umma_make_map(&wmap, w, p.rows, in_features, kF8Chunk, TN);
    if (rc != QD_OK) return rc;
    p.across = (p.rows + TN - 1) / TN;
    p.tiles = p.across * ((p.tokens + kF8Tokens - 1) / kF8Tokens);
    const unsigned grid = (unsigned)(p.tiles < sms ? p.tiles : sms);
    qd_launch(fp8_gemm_kernel<TN>, dim3(grid), dim3(kF8Threads), Tile::kSmem, stream, true, p, xmap, wmap);
    return qd_launch_status();
}

}  // namespace
}  // namespace qd

// y [tokens, out_features] = q(x) W^T for a static-FP8 projection (see above).  q_scratch: tokens *
// in_features bytes, 16-byte aligned, receives the quantised rows; convert = 0 reuses what the
// previous call left there (projections that share input and input scale).  in_features a multiple
// of 128, out_features even; QD_ERR_UNSUPPORTED otherwise.
extern "C" int qd_fp8_matmul(const void* x, const void* w, const float* w_scale, const float* in_scale, void* y,
                             int tokens, int out_features, int in_features, void* q_scratch, int convert, void* stream) {
    using namespace qd;
    QD_CHECK_ARG(x && w && w_scale && in_scale && y && q_scratch && tokens > 0 && out_features > 0 && in_features > 0);
    if (in_features % kF8Chunk != 0 || out_features % 2 != 0 || (tokens + kF8Tokens - 1) / kF8Tokens > 65535) return QD_ERR_UNSUPPORTED;
    if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)q_scratch) & 15u || ((uintptr_t)y & 3u)) return QD_ERR_UNSUPPORTED;
    if (convert) {
        const long long n8 = (long long)tokens * in_features / 8;
        qd_launch(fp8_quantize_rows_kernel, dim3((unsigned)((n8 + 255) / 256)), dim3(256), 0, (cudaStream_t)stream, true, 
            (const uint4*)x, in_scale, (uint2*)q_scratch, n8);
        if (qd_launch_status() != QD_OK) return QD_ERR_LAUNCH;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return QD_ERR_LAUNCH;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return QD_ERR_LAUNCH;
    const F8Params p = {w_scale, in_scale, (bf16*)y, tokens, out_features, in_features / kF8Chunk, 0, 0};
    const long long token_tiles = (tokens + kF8Tokens - 1) / kF8Tokens;
    const auto busy = [&](int tn) { return token_tiles * ((out_features + tn - 1) / tn) * 4 >= 3ll * sms; };
    // the widest tile that still gives most SMs one: a wider one reads the tokens fewer times
    if (busy(256)) return launch_f8<256>(q_scratch, w, p, in_features, sms, (cudaStream_t)stream);
    if (busy(128)) return launch_f8<128>(q_scratch, w, p, in_features, sms, (cudaStream_t)stream);
    if (busy(64)) return launch_f8<64>(q_scratch, w, p, in_features, sms, (cudaStream_t)stream);
    return launch_f8<32>(q_scratch, w, p, in_features, sms, (cudaStream_t)stream);
}
