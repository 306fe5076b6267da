// visg_math.cuh — float3 arithmetic with one IEEE-754 rounding per operation.
//
// Every operation is written with the round-to-nearest intrinsics so that the
// compiler never contracts a multiply and an add into an FMA, whatever the build
// flags.  This reproduces the reference's GLM 0.9.9.8 expressions operation by
// operation (dot = (x*x' + y*y') + z*z', normalize(v) = v * (1/sqrt(dot(v,v))),
// vector / scalar divides each component), which is what makes the Morton codes,
// boxes and positions bit-identical to the reference's own kernels compiled
// without contraction.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace visg {

struct f3 {
    float x, y, z;
};

__device__ __forceinline__ f3 mk3(float x, float y, float z) { return f3{x, y, z}; }
__device__ __forceinline__ f3 add(f3 a, f3 b) {
    return f3{__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z)};
}
__device__ __forceinline__ f3 sub(f3 a, f3 b) {
    return f3{__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)};
}
__device__ __forceinline__ f3 mul(f3 a, float s) {
    return f3{__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s)};
}
__device__ __forceinline__ f3 mul(float s, f3 a) {
    return f3{__fmul_rn(s, a.x), __fmul_rn(s, a.y), __fmul_rn(s, a.z)};
}
__device__ __forceinline__ f3 divs(f3 a, float s) {
    return f3{__fdiv_rn(a.x, s), __fdiv_rn(a.y, s), __fdiv_rn(a.z, s)};
}
__device__ __forceinline__ f3 divv(f3 a, f3 b) {
    return f3{__fdiv_rn(a.x, b.x), __fdiv_rn(a.y, b.y), __fdiv_rn(a.z, b.z)};
}
__device__ __forceinline__ float dot(f3 a, f3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ f3 cross(f3 a, f3 b) {
    return f3{__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(b.y, a.z)),
              __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(b.z, a.x)),
              __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(b.x, a.y))};
}
__device__ __forceinline__ float length(f3 v) { return __fsqrt_rn(dot(v, v)); }
// 1/sqrt(x) correctly rounded twice, as GLM's inversesqrt = 1 / sqrt(x)
__device__ __forceinline__ f3 normalize(f3 v) { return mul(v, __frcp_rn(__fsqrt_rn(dot(v, v)))); }

__device__ __forceinline__ f3 xyz(float4 v) { return f3{v.x, v.y, v.z}; }

// ---- 32-byte records: one 256-bit access (sm_100+) per record -----------------------------
// A record of two float4 (state, leaf, box, one side of a node) is one sector; as two
// 16-byte accesses each warp touches every sector twice.  Addresses are 32-byte aligned.
struct f4x2 {
    float4 a, b;
};
#define VISG_LD8(name, op, vol)                                                                                  \
    __device__ __forceinline__ f4x2 name(const float4* p) {                                                     \
        f4x2 r;                                                                                                 \
        asm vol(op ".v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"                                            \
                : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y), "=f"(r.b.z),    \
                  "=f"(r.b.w)                                                                                   \
                : "l"(p));                                                                                      \
        return r;                                                                                               \
    }
VISG_LD8(ld8_nc, "ld.global.nc", )           // data no one writes during the launch
VISG_LD8(ld8, "ld.global", volatile)
VISG_LD8(ld8_cg, "ld.global.cg", volatile)   // through L2: data another CTA wrote earlier in the launch
#undef VISG_LD8
__device__ __forceinline__ float4 ld4(const float4* p) {  // 16 bytes, not merged with an earlier load
    float4 r;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(p));
    return r;
}
__device__ __forceinline__ void st8(float4* p, float4 a, float4 b) {
    asm volatile("st.global.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};" ::"f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
                 "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w), "l"(p)
                 : "memory");
}

// ---- packed pairs (sm_100+ f32x2 instructions) -----------------------------------------
// Two floats in one 64-bit register pair; every packed operation rounds each lane
// to nearest on its own, so a lane gets exactly the bits the scalar intrinsic
// (__fadd_rn, __fmul_rn, __fmaf_rn) gives, in half the instructions.
typedef unsigned long long fp2;
__device__ __forceinline__ fp2 pk2(float lo, float hi) {
    fp2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo2(fp2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a;
}
__device__ __forceinline__ float hi2(fp2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return b;
}
// Not for a sum with a packed product: the assembler contracts mul.f32x2 and add.f32x2 into
// one FMA in spite of their .rn (seen against the scalar intrinsics).  Sums of products take
// scalar additions of the product's lanes, which it leaves alone (add_lanes).
__device__ __forceinline__ fp2 add2(fp2 a, fp2 b) {
    fp2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ fp2 add_lanes(fp2 a, fp2 b) {
    return pk2(__fadd_rn(lo2(a), lo2(b)), __fadd_rn(hi2(a), hi2(b)));
}
__device__ __forceinline__ fp2 mul2(fp2 a, fp2 b) {
    fp2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ fp2 fma2(fp2 a, fp2 b, fp2 c) {  // a * b + c, one rounding per lane
    fp2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ fp2 splat2(float v) { return pk2(v, v); }

// ---- correctly rounded square root and reciprocal, two lanes at once -------------------
// For s in [2^-100, 2^100):  q = RN(sqrt(s))  and  nr = -RN(1 / q), bit for bit what
// __fsqrt_rn(s) and -__frcp_rn(__fsqrt_rn(s)) return (checked against them on every
// float of that range by visg_selftest_exact_math).  Method: Markstein's correction
// of a hardware approximation by one Newton step whose residual an FMA forms with a
// single rounding (P. W. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Develop. 34(1), 1990; the square-root form is
// the one of M. Cornea, J. Harrison, P. T. P. Tang, "Scientific Computing on
// Itanium-based Systems", Intel Press, 2002, ch. 8):
//   y ~ 1/sqrt(s) (rsqrt.approx), g = s y, h = y/2;  d = s - g^2 (one FMA);  q = g + d h.
//   z ~ 1/q (rcp.approx);  e = 1 - q z (one FMA);  r = z + z e.
// The reciprocal comes negated because rcp.approx takes -q at no cost and the packed FMA,
// which has no negated operands, then needs no extra product for the residuals.
// The caller sees to the range (PairRange): below 2^-100 the remainder s - g^2 can
// fall among the subnormals and lose the bits the last correction needs.
constexpr uint32_t kExactLo = 27u << 23;                     // 2^-100
constexpr uint32_t kExactSpan = (227u << 23) - (27u << 23);  // up to 2^100

__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void sqrt_rcp_pair(fp2 s, fp2& q, fp2& nr) {
    const fp2 y = pk2(rsqrt_approx(lo2(s)), rsqrt_approx(hi2(s)));
    const fp2 nh = mul2(y, splat2(-0.5f));  // -h
    const fp2 g = mul2(s, y);
    const fp2 dn = fma2(g, g, mul2(s, splat2(-1.0f)));  // g^2 - s
    q = fma2(dn, nh, g);                                // g + (s - g^2) h
    const fp2 nz = pk2(rcp_approx(-lo2(q)), rcp_approx(-hi2(q)));
    const fp2 e = fma2(q, nz, splat2(1.0f));
    nr = fma2(nz, e, nz);
}

// -g / q in both lanes, rounded as __fdiv_rn rounds, given q and nr = -RN(1 / q) as
// sqrt_rcp_pair returns them: two corrections of g r by an FMA's exact residual (the same
// sources).  The first brings the quotient within one unit in the last place of g / q,
// from where, with r correctly rounded, the second is correctly rounded (Markstein's
// theorem; visg_selftest_exact_math runs 1.3e10 pairs, over every significand of q).  The caller
// sees to it that |g| >= 2^-60 or g = 0, so that no residual underflows, and that the
// quotient does not overflow.  A zero numerator gives a zero, of either sign.
__device__ __forceinline__ fp2 div_pair(fp2 g, fp2 q, fp2 nr) {
    fp2 nd = mul2(g, nr);
    nd = fma2(fma2(q, nd, g), nr, nd);
    return fma2(fma2(q, nd, g), nr, nd);
}
constexpr uint32_t kDivLo = (127u - 60u) << 23;  // 2^-60
// orders |g| as a uint32 with the sign gone and zero last
__device__ __forceinline__ uint32_t div_order(float g) { return 2u * __float_as_uint(g) - 1u; }

// Order-preserving map float -> uint32 (for atomicMin/atomicMax on floats).
__device__ __forceinline__ uint32_t f2ord(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ __forceinline__ float ord2f(uint32_t u) {
    uint32_t v = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
#ifdef __CUDA_ARCH__
    return __uint_as_float(v);
#else
    float f;
    __builtin_memcpy(&f, &v, 4);
    return f;
#endif
}

}  // namespace visg
