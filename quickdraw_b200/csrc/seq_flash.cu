// Causal attention of a prompt chunk of the NVFP4 model: head dimension 256, a sigmoid gate per value column
// (quickdraw/kernel/triton/attention.py:53-100), the cache rows prepared by seq_attn_prepare_kernel.
#include "seq_flash.cuh"

#include "flash_umma.cuh"

namespace {

// bf16(attended) * bf16(sigmoid(gate)), as in the decode kernels
struct GatedOut {
    const bf16* qg; bf16* out;
    int heads, wide;                       // wide: rows of both on 16-byte boundaries
    QD_DEVINL void operator()(int token, int head, int c0, const float (&o)[32], float, float l) const {
        const bf16* gate = qg + ((size_t)token * heads + head) * 512 + 256 + c0;
        bf16* dst = out + ((size_t)token * heads + head) * 256 + c0;
        const float f = 1.f / l;
        uint32_t v[16];
        uint32_t z[16];
        if (wide) {
#pragma unroll
            for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(z + 4 * i) = reinterpret_cast<const uint4*>(gate)[i];
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) z[i] = (uint32_t)__bfloat16_as_ushort(gate[2 * i]) | ((uint32_t)__bfloat16_as_ushort(gate[2 * i + 1]) << 16);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float g0 = round_bf16(sigmoid_precise(__uint_as_float(z[i] << 16))), g1 = round_bf16(sigmoid_precise(__uint_as_float(z[i] & 0xffff0000u)));
            v[i] = qd::flash::pair(round_bf16(o[2 * i] * f) * g0, round_bf16(o[2 * i + 1] * f) * g1);
        }
        if (wide) {
#pragma unroll
            for (int i = 0; i < 4; ++i) reinterpret_cast<uint4*>(dst)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) reinterpret_cast<uint32_t*>(dst)[i] = v[i];
        }
    }
};

}  // namespace

int seq_flash_attention(const bf16* q, const bf16* qg, const bf16* k_cache, const bf16* v_cache, bf16* out, int tokens, int position0,
                        int capacity, int q_heads, int kv_heads, cudaStream_t stream) {
    qd::flash::In p = {};
    p.q = q; p.k = k_cache; p.v = v_cache; p.ld_k = p.ld_v = (long long)kv_heads * 256;
    p.scale = 0.0625f * 1.4426950408889634f;                 // 1 / sqrt(256)
    p.position = position0; p.tokens = tokens; p.heads = q_heads; p.kv_heads = kv_heads; p.dim = 256; p.capacity = capacity;
    const GatedOut store = {qg, out, q_heads, (((uintptr_t)out | (uintptr_t)qg) & 15u) == 0};
    return qd::flash::launch<256, 256, 1>(p, store, stream);
}
