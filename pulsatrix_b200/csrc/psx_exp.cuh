// exp() of a difference of two floats in double precision, for sweeps that take it of every logit of a row.
//
// Tang's table method ("Table-driven implementation of the exponential function in IEEE floating-point
// arithmetic", ACM TOMS 15, 1989): d = n * ln2/32 + r, exp(d) = 2^(n / 32) * 2^((n % 32) / 32) * exp(r).  With
// |r| <= ln2/64 the Taylor series to r^6 / 720 ends below 4e-18; the rounding of ln2/32, n times, adds at most
// |d| * 2^-53 -- what the rounding of the reference's own argument (double)x - (double)max (src/generation.cpp:46)
// may do as well.  Relative error (4 + |d|) * 2^-53 at most.  Twelve double-precision operations, against the
// twenty-odd of the general function, which has to take any argument.
//
// The table's 32 powers lie one in each lane, and a look-up is two shuffles: nothing to load ahead of the sweep, no
// shared memory, no two lanes in one another's way.  (A table of 512 in shared memory saves two operations of the
// series, but its random look-ups queue six deep at the banks; sixteen copies of 64 entries do not, but every CTA then
// writes 8 KB before it starts.)
#pragma once

#include <stdint.h>

namespace psx {

struct ExpPowers {
    double power[32];  // 2^(j / 32)
    constexpr ExpPowers() : power() {
        for (int j = 0; j < 32; ++j) {
            const double x = (double)j / 32 * 0.693147180559945309417232121458;  // 2^t = e^(t ln 2), t in [0, 1)
            double sum = 1.0;
            for (int k = 24; k >= 1; --k) sum = 1.0 + sum * x / k;
            power[j] = sum;
        }
    }
};
static __device__ constexpr ExpPowers kExpPowers{};
__device__ __forceinline__ double exp_power_of_lane() { return kExpPowers.power[threadIdx.x & 31]; }

// exp(d) for -705 <= d <= 0, by a whole warp; `power` is exp_power_of_lane().
__device__ __forceinline__ double exp_of_gap(double d, double power) {
    const double shifted = fma(d, 46.166241308446828, 6755399441055744.0);  // 32 / ln2; + 1.5 * 2^52: n in the low word
    const int n = __double2loint(shifted);
    const double r = fma(shifted - 6755399441055744.0, -0.021660849392498290919288503568, d);  // ln2 / 32
    const double r2 = r * r;
    const double high = fma(r2, 1.0 / 720.0, fma(r, 1.0 / 120.0, 1.0 / 24.0));
    const double tail = fma(r2, fma(r2, high, fma(r, 1.0 / 6.0, 0.5)), r);
    const double p = __hiloint2double(__shfl_sync(0xFFFFFFFFu, __double2hiint(power), n), __shfl_sync(0xFFFFFFFFu, __double2loint(power), n));
    const double y = fma(p, tail, p);
    return __hiloint2double(__double2hiint(y) + ((n & ~31) << 15), __double2loint(y));
}

constexpr float kExpFloor = -700.0f;  // exp(-700) = 1e-304: what lies below counts as nothing

// exp(x - top) for finite x <= top by a thread of its own; 0 below kExpFloor and for x = -inf.
__device__ __forceinline__ double exp_below(float x, float top) { return x - top >= kExpFloor ? exp((double)x - (double)top) : 0.0; }

}  // namespace psx
