// exp() of a difference of two floats in double precision, for sweeps that take it of every logit of a row.
//
// Tang's table method ("Table-driven implementation of the exponential function in IEEE floating-point
// arithmetic", ACM TOMS 15, 1989): d = n * ln2/512 + r, exp(d) = 2^(n / 512) * 2^((n % 512) / 512) * exp(r).  With
// |r| <= ln2/1024 (and a little, n is rounded in single precision) the Taylor series to r^4 / 24 ends below
// 2e-18; the rounding of ln2/512, n times, adds at most |d| * 2^-53 -- what the rounding of the reference's own
// argument (double)x - (double)max (src/generation.cpp:46) may do as well.  Relative error (4 + |d|) * 2^-53 at most.
// Nine double-precision operations, against the twenty-odd of the general function, which has to take any argument.
#pragma once

#include <stdint.h>

namespace psx {

constexpr int kExpTable = 512;

struct ExpTable {
    double power[kExpTable];  // 2^(j / 512)
    constexpr ExpTable() : power() {
        for (int j = 0; j < kExpTable; ++j) {
            const double x = (double)j / kExpTable * 0.693147180559945309417232121458;  // 2^t = e^(t ln 2), t in [0, 1)
            double sum = 1.0;
            for (int k = 24; k >= 1; --k) sum = 1.0 + sum * x / k;
            power[j] = sum;
        }
    }
};
static __device__ constexpr ExpTable kExpPowers{};

// The table in shared memory (4 KB): every thread of the block calls this, and the block meets before the first use.
__device__ __forceinline__ void load_exp_table(double* table) {
    for (int j = threadIdx.x; j < kExpTable; j += blockDim.x) table[j] = kExpPowers.power[j];
}

// A float as a double by its bits (the conversion instruction runs at a quarter of the double-precision rate).  A zero or
// subnormal comes out below 2^-126 in magnitude, which moves no exponential here.  Finite x only.
__device__ __forceinline__ double double_of_float(float x) {
    const uint32_t u = __float_as_uint(x);
    return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7FFFFFFFu) >> 3) + (896u << 20))), (int)(u << 29));
}

constexpr float kExpFloor = -700.0f;  // exp(-700) = 1e-304: what lies below counts as nothing

// exp(x - top) for finite x <= top (x_d, top_d: the same two as doubles); 0 below kExpFloor and for x = -inf.
__device__ __forceinline__ double exp_below(float x, double x_d, float top, double top_d, const double* table) {
    const float gap = __fsub_rn(x, top);
    const float rounded = __fmaf_rn(fmaxf(gap, kExpFloor), 738.65986f, 12582912.0f);  // + 1.5 * 2^23: n in the low bits
    const int n = (int)(__float_as_uint(rounded) - 0x4B400000u);
    const double whole = __hiloint2double(0x43300000, n ^ (int)0x80000000) - 4503601774854144.0;  // n: 2^52 + 2^31 + n, less the offset
    const double r = fma(whole, -0.001353803087031143182455531, x_d - top_d);                              // - ln2 / 512
    const double tail = fma(r * r, fma(r, fma(r, 1.0 / 24.0, 1.0 / 6.0), 0.5), r);
    const double p = table[n & (kExpTable - 1)];
    const double y = fma(p, tail, p);
    const double scaled = __hiloint2double(__double2hiint(y) + ((n >> 9) << 20), __double2loint(y));
    return gap >= kExpFloor ? scaled : 0.0;
}

}  // namespace psx
