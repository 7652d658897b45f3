// 64-bit fixed-point arithmetic of the FP64 step (fixed_kernels.cuh).
//
// GB300 issues one FP64 instruction for about 60 FP32 or integer ones (measured
// per SM and clock: 2.1 DFMA lanes, 134 IADD lanes, 27 IMAD.WIDE lanes), so a
// 64-bit integer addition is 30 times and a 64 x 64 -> high 64 product (three
// IMAD.WIDE) four times cheaper than the FP64 operation it stands for.
// Distribution values are held as integers scaled 2^62 (|x| < 2): a resolution of
// 2.2e-19, sixteen times finer than the last bit of an FP64 value near 1/36 (the
// smallest lattice weight) and 256 times finer than that of 1/3, so sums and
// products round less than their FP64 counterparts.  The scaling holds for states
// near unit density; fixed_kernels.cuh states the range and what happens outside.
//
// Host and device: the same integer operations, tested on the CPU against
// quadruple precision (tests/fixed_check.cpp).
#pragma once
#include <cstdint>
#include <cstring>

#include <cmath>

#ifdef __CUDACC__
#define DG_FX __host__ __device__ __forceinline__
#else
#define DG_FX inline
#endif
#ifdef __CUDA_ARCH__
#define DG_UNROLL _Pragma("unroll")
#else
#define DG_UNROLL
#endif

namespace dg {

using i64 = long long;
using u64 = unsigned long long;

// A multiplier m: the integer M = m 2^s (s fixed by the use) as two signed limbs,
// M = h 2^32 + l with -2^31 <= l < 2^31.  |M| < 2^63 - 2^31.
struct FxMul {
    int h, l;
};
DG_FX FxMul fx_split(i64 M) { return FxMul{int(M >> 32) + int(unsigned(M) >> 31), int(unsigned(M))}; }

// a b and a b + c of 32-bit factors as one IMAD.WIDE each (written as PTX: from C the
// compiler turns these products into twice the instructions)
DG_FX i64 fx_wide(int a, int b)
{
#ifdef __CUDA_ARCH__
    i64 d;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
    return d;
#else
    return i64(a) * b;
#endif
}
DG_FX i64 fx_wide(int a, int b, i64 c)
{
#ifdef __CUDA_ARCH__
    i64 d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
#else
    return i64(a) * b + c;
#endif
}

// acc + a M / 2^64: three 32 x 32 -> 64 products (a in the same signed limbs; the
// l x l product, below a quarter of the last place, is left out), rounded down.
// |a| < 2^63 - 2^31.  Nine instructions and 17 clocks of a warp's scheduler with
// the subtraction of fx_lerp, 7.4 lanes per SM and clock measured.
DG_FX i64 fx_mad(i64 a, FxMul m, i64 acc)
{
    const FxMul x = fx_split(a);
    const i64 q = fx_wide(x.h, m.l, fx_wide(x.l, m.h));
    return fx_wide(x.h, m.h, acc) + (q >> 32);
}
DG_FX i64 fx_mul(i64 a, FxMul m)
{
    const FxMul x = fx_split(a);
    const i64 q = fx_wide(x.h, m.l, fx_wide(x.l, m.h));
    return fx_wide(x.h, m.h) + (q >> 32);
}

// fx_mad rounded to nearest: the update of f-tilde, whose rounding adds up step
// after step (face values and fluxes are rounded down, the same on both sides of a
// face)
DG_FX i64 fx_madr(i64 a, FxMul m, i64 acc)
{
    const FxMul x = fx_split(a);
    const i64 q = fx_wide(x.h, m.l, fx_wide(x.l, m.h, 0x80000000ll));
    return fx_wide(x.h, m.h, acc) + (q >> 32);
}

// a^2 / 2^64, rounded down
DG_FX i64 fx_sq(i64 a)
{
    const FxMul x = fx_split(a);
    return fx_wide(x.h, x.h) + (fx_wide(x.h, x.l) >> 31);
}

// a + m (b - a)
DG_FX i64 fx_lerp(i64 a, i64 b, FxMul m) { return fx_mad(b - a, m, a); }

// An FP64 value in [2^-10, 2) as an integer scaled 2^62 (exact): the 53-bit
// significand shifted by the exponent.
DG_FX i64 fx_from_double(double x)
{
#ifdef __CUDA_ARCH__
    const i64 b = __double_as_longlong(x);
#else
    i64 b;
    std::memcpy(&b, &x, 8);
#endif
    const int e = int(b >> 52) - 1013;
    const i64 m = (b & 0xfffffffffffffll) | 0x10000000000000ll;
    return m << e;
}

// The FP64 value nearest to v / 2^s, any v: one conversion and an exponent
// adjustment (zero has no exponent to adjust).
DG_FX double fx_to_double(i64 v, int s = 62)
{
#ifdef __CUDA_ARCH__
    const double d = __ll2double_rn(v);
    const int hi = __double2hiint(d);
    return __hiloint2double(v ? hi - (s << 20) : 0, __double2loint(d));
#else
    return std::ldexp(double(v), -s);
#endif
}

// Multiplier M / 2^64 = 3 / (16 rho) for a density scaled 2^62, 0.39 < rho < 2:
// a single-precision reciprocal X / 2^28 (relative error below 2^-21) and one
// second-order Newton step on its residual r = 1 - rho X (|r| < 2^-20, kept to
// 2^-58), (3/16) X (1 + r + r^2); the cubic term is below 2^-60.
DG_FX FxMul fx_recip3(i64 rho)
{
    const unsigned rh = unsigned(u64(rho) >> 32), rl = unsigned(rho);
#ifdef __CUDA_ARCH__
    float x;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(__uint2float_rn(rh)));
    const unsigned X = __float2uint_rn(x * 0x1p58f);
#else
    const unsigned X = unsigned(std::lrint(0x1p58f / float(rh)));
#endif
    const i64 r = (1ll << 58) - i64(u64(rh) * X) - i64(u64(rl) * X >> 32);
    const int rs = int(r >> 8);
    const i64 t = r + ((i64(rs) * rs) >> 42);  // r + r^2, scaled 2^58
    const unsigned X3 = 3u * X;                 // below 2^31
    const i64 M = (i64(X3) << 32) + i64(u64(X3) * unsigned(t) >> 26) + (i64(int(X3)) * int(t >> 32)) * 64;
    return fx_split(M);
}

}  // namespace dg
