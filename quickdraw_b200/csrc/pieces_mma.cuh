// What the chunked recurrences share: mma.sync operands in bf16 pieces, ldmatrix, copies in the background, named barriers.
#pragma once
#include "common.cuh"

namespace qd {

QD_DEVINL void mma_bf16(float (&d)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

QD_DEVINL uint32_t upper_halves(float x0, float x1) { return __byte_perm(__float_as_uint(x0), __float_as_uint(x1), 0x7632); }
QD_DEVINL float upper_half(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
// x0, x1 as two bf16 pieces each (cut off, then the rest rounded), packed as MMA operands take them.
QD_DEVINL void split_pair(float x0, float x1, uint32_t& hi, uint32_t& lo) {
    hi = upper_halves(x0, x1);
    const __nv_bfloat162 rest = __floats2bfloat162_rn(x0 - upper_half(x0), x1 - upper_half(x1));
    lo = *reinterpret_cast<const uint32_t*>(&rest);
}
// Accumulators of two neighbouring n-tiles (16 rows x 16 columns) as the A operand of the next product, in two pieces.
QD_DEVINL void split_tiles(const float (&l)[4], const float (&r)[4], uint4& hi, uint4& lo) {
    split_pair(l[0], l[1], hi.x, lo.x);
    split_pair(l[2], l[3], hi.y, lo.y);
    split_pair(r[0], r[1], hi.z, lo.z);
    split_pair(r[2], r[3], hi.w, lo.w);
}
QD_DEVINL float rounded_up(float x) { return __uint_as_float(__float_as_uint(x) + 0x8000u); }
QD_DEVINL float kept_finite(float x) { return fminf(fmaxf(x, -3.38953139e38f), 3.38953139e38f); }      // to the largest bf16, 2^128 (1 - 2^-8)
// x0, x1 as three bf16 pieces each, the first two rounded (half away from zero; in integer instructions, because the conversion of a pair
// takes longer: 64 values of a lane 281 against 124 clocks): together they are x to its last bit or the one before.  Where x is an
// infinity or NaN the third is NaN (the others need not be: a NaN's bits can run over).  From 2^128 (1 - 2^-9) on the first piece would round up to
// infinity: with BOUND it stops at the largest bf16, else these magnitudes count as infinite.
template <bool BOUND> QD_DEVINL void split_three(float x0, float x1, uint32_t& a, uint32_t& b, uint32_t& c) {
    float u = rounded_up(BOUND ? kept_finite(x0) : x0), v = rounded_up(BOUND ? kept_finite(x1) : x1);
    a = upper_halves(u, v);
    x0 -= upper_half(u); x1 -= upper_half(v);
    u = rounded_up(x0); v = rounded_up(x1);
    b = upper_halves(u, v);
    c = upper_halves(x0 - upper_half(u), x1 - upper_half(v));
}
struct Pieces { uint4 p[3]; };
template <bool BOUND = false> QD_DEVINL Pieces split_tiles3(const float (&l)[4], const float (&r)[4]) {
    Pieces v;
    split_three<BOUND>(l[0], l[1], v.p[0].x, v.p[1].x, v.p[2].x);
    split_three<BOUND>(l[2], l[3], v.p[0].y, v.p[1].y, v.p[2].y);
    split_three<BOUND>(r[0], r[1], v.p[0].z, v.p[1].z, v.p[2].z);
    split_three<BOUND>(r[2], r[3], v.p[0].w, v.p[1].w, v.p[2].w);
    return v;
}

QD_DEVINL uint4 ldsm(uint32_t addr) {
    uint4 v;
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
QD_DEVINL uint4 ldsm_t(uint32_t addr) {
    uint4 v;
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
QD_DEVINL uint32_t transposed(uint32_t v) {        // an 8 x 8 matrix of 16-bit values across the warp
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}

// Sixteen bytes global -> shared in the background; zeros where there is nothing.  wide: the source is 16-byte aligned (else 8).
QD_DEVINL void copy16(uint32_t dst, const void* src, bool there, bool wide) {
    const uint32_t bytes = there ? 16u : 0u;
    if (wide) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
    } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes / 2) : "memory");
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + 8), "l"((const char*)src + 8), "r"(bytes / 2) : "memory");
    }
}
QD_DEVINL void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> QD_DEVINL void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }
QD_DEVINL void named_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

}  // namespace qd
