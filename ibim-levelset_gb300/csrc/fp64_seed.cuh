// Seeds of 1 / x and 1 / sqrt(x) in FP64, to 2^-44, without the FP64 pipe.
//
// GB300's FP64 pipe takes a warp instruction in 16 cycles of an SM, which has some 60 issue slots of the other pipes
// beside each: in the kernels that pipe bounds, FP32 and integer instructions cost next to nothing.  The operand's
// head (24 bits) goes through the hardware's approximation, the residual against the whole operand is formed by
// FP32 multiply-adds (exact where it cancels), and y + y residual is assembled in units of 2^-53 in integers.  One
// FP64 correction y + y e then is good to an ulp, where an FP32 seed (2^-22) needs a cubic one.
#pragma once

namespace ibim {

// y 2^-k for y in [1/2, 2), y's FP32 value and a correction in units of 2^-50 (|inc| < 2^29).
__device__ __forceinline__ double seed_assemble(float y, int inc, int k) {
    const int b = __float_as_int(y);
    const long long Y = ((long long)((b & 0x7fffff) | 0x800000) << ((b >> 23) - 97)) + ((long long)inc << 3);
    const int c = (int)(Y >> 53) & 1;  // y >= 1
    return __longlong_as_double((Y >> c) + ((long long)(1021 + c - k) << 52));
}

// x = head + tail, head its upper 24 bits at exponent 0 (odd: 1).
__device__ __forceinline__ float seed_head(double x, int odd) {
    return __uint_as_float(((127u + odd) << 23) | (((unsigned)__double2hiint(x) & 0xfffffu) << 3) |
                           ((unsigned)__double2loint(x) >> 29));
}
__device__ __forceinline__ float seed_tail(double x, int odd) {
    return (float)((unsigned)__double2loint(x) & 0x1fffffffu) * __int_as_float((127 - 52 + odd) << 23);
}

// 1 / sqrt(x) for normal x > 0; r: sqrt(x) to FP32 (at most 2^121).
__device__ __forceinline__ double rsqrt_seed(double x, float &r) {
    const int E = (__double2hiint(x) >> 20) - 1023, odd = E & 1, E2 = E >> 1;
    const float a = seed_head(x, odd), rho = seed_tail(x, odd);  // x = 4^E2 (a + rho), a in [1, 4)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
    r = __int_as_float(__float_as_int(a * y) + (min(E2, 120) << 23));
    const float ph = y * y, pl = fmaf(y, y, -ph);
    const float res = fmaf(-rho, ph, fmaf(-a, pl, fmaf(-a, ph, 1.f)));
    return seed_assemble(y, __float2int_rn(y * res * 0x1p49f), E2);  // y (1 + residual / 2)
}

// 1 / x for normal x in (0, 2^1020).
__device__ __forceinline__ double rcp_seed(double x) {
    const int E = (__double2hiint(x) >> 20) - 1023;
    const float a = seed_head(x, 0), rho = seed_tail(x, 0);  // x = 2^E (a + rho), a in [1, 2)
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
    const float res = fmaf(-rho, y, fmaf(-a, y, 1.f));
    return seed_assemble(y, __float2int_rn(y * res * 0x1p50f), E);
}

// Exact halves by the exponent (x normal, not below 2^-1021).
__device__ __forceinline__ double half_of(double x) {
    return __hiloint2double(__double2hiint(x) - 0x00100000, __double2loint(x));
}

}  // namespace ibim
