// quotient.cuh -- FP64 to FP32 conversions and quotients in few FP64 instructions.
#pragma once

namespace nbx {

// (double)f in integer operations: FP64 instructions and conversions run at a
// small fraction of the FP32 rate on this part (a warp instruction holds the
// pipe for tens of cycles), and the moments are bound by them.
__device__ __forceinline__ double widen(float f) {
    const unsigned u = __float_as_uint(f);
    const unsigned e = (u >> 23) & 255u;
    if (e - 1u >= 254u && (u << 1) != 0u) return (double)f;  // subnormal, infinity, NaN
    const unsigned hi = (u & 0x80000000u) | ((u << 1) ? ((u >> 3) & 0x0fffffffu) + 0x38000000u : 0u);
    return __hiloint2double((int)hi, (int)(u << 29));
}

// The float nearest to the double nearest to s / m, with one FP64 instruction
// instead of a division: an FP32 quotient q, the exact remainder s - q m (one
// fused product) and its FP32 quotient d give s / m to about 2^-41 of itself;
// q + d then rounds like s / m unless it lies that close to the middle of two
// floats (or is a power of two, zero, or out of the plain range): then divide.
__device__ __forceinline__ float narrow(double v) {  // towards zero, in integer operations
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    return __uint_as_float((hi & 0x80000000u) | ((((hi & 0x7fffffffu) - 0x38000000u) << 3) | (lo >> 29)));
}
__device__ __forceinline__ bool plain_range(double v) {  // 2^-60 <= |v| < 2^61
    return (((unsigned)__double2hiint(v) & 0x7fffffffu) >> 20) - (1023u - 60u) <= 120u;
}
__device__ __forceinline__ float quotient32(double s, double m) {
    if (plain_range(s) && plain_range(m)) {
        float ri;
        const float mf = narrow(m);
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ri) : "f"(mf));
        const float q0 = narrow(s) * ri;  // within 2^-21; its exponent is within (-122, 122)
        const double r = __fma_rn(-widen(q0), m, s);
        const unsigned re = ((unsigned)__double2hiint(r) & 0x7fffffffu) >> 20;
        if (re - (1023u - 100u) <= 200u) {  // (a zero or tiny remainder divides)
            const float d = __fmul_rn(narrow(r), ri);
            const float q = __fadd_rn(q0, d);
            const float e = __fsub_rn(d, __fsub_rn(q, q0));  // exact: q + e = q0 + d
            const unsigned qb = __float_as_uint(q);
            const unsigned qe = (qb >> 23) & 255u;
            if (qe - 60u <= 135u && (qb & 0x7fffffu) != 0u) {
                const float half = __uint_as_float((qe - 24u) << 23);   // half a unit in the last place of q
                const float tol = __uint_as_float((qe - 38u) << 23);    // 2^-38 of q's binade
                if (half - fabsf(e) > tol) return q;
            }
        }
    }
    return (float)(s / m);
}

}  // namespace nbx
