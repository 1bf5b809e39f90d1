// exp_of_gap (pulsatrix_b200/csrc/psx_exp.cuh) compiled for the host, one lane at a time, against the 64-bit-mantissa expl: the relative
// error stays below (4 + |d|) * 2^-53 over the whole range, at whole multiples of ln2 / 32 and just beside the points where the rounding of
// d * 32 / ln2 changes.  A warp's shuffle becomes a look into the table that the lanes hold: the value handed in is lane 0's, 1.0.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <random>

#define __device__
#define __forceinline__ inline

static struct { unsigned x; } threadIdx{0};

static uint64_t bits_of(double v) { uint64_t b; std::memcpy(&b, &v, 8); return b; }
static int __double2loint(double v) { return (int)(uint32_t)bits_of(v); }
static int __double2hiint(double v) { return (int)(uint32_t)(bits_of(v) >> 32); }
static double __hiloint2double(int hi, int lo) {
    const uint64_t b = ((uint64_t)(uint32_t)hi << 32) | (uint32_t)lo;
    double v;
    std::memcpy(&v, &b, 8);
    return v;
}
static int __shfl_sync(unsigned mask, int value, int lane);
using std::exp;
using std::fma;

#include "../../pulsatrix_b200/csrc/psx_exp.cuh"

static int __shfl_sync(unsigned, int value, int lane) {  // (lane 0's halves: 0x3FF00000 and 0)
    const double power = psx::kExpPowers.power[lane & 31];
    return value != 0 ? __double2hiint(power) : __double2loint(power);
}

int main() {
    double worst = 0.0, at = 0.0;
    const double power = psx::exp_power_of_lane();
    auto look = [&](double d) {
        if (!(d <= 0.0 && d >= -705.0)) return;
        const long double want = expl((long double)d);
        const double error = (double)(fabsl((long double)psx::exp_of_gap(d, power) - want) / want) / ((4.0 + std::fabs(d)) * 0x1p-53);
        if (error > worst) { worst = error; at = d; }
    };
    std::mt19937_64 random(7);
    std::uniform_real_distribution<double> whole(-705.0, 0.0), exponent(-40.0, 9.4);
    std::normal_distribution<float> logit(0.0f, 30.0f);
    for (int i = 0; i < 2000000; ++i) {
        look(whole(random));
        look(-std::exp2(exponent(random)));
        look(-std::fabs((double)logit(random) - (double)logit(random)));  // what the sweeps hand in: differences of floats
    }
    const double step = 0.693147180559945309417232121458 / 32;
    for (int n = 0; n <= 32545; ++n) {
        for (double around : {n * step, (n + 0.5) * step}) {
            for (int ulp = -2; ulp <= 2; ++ulp) look(-around * (1.0 + ulp * 0x1p-52));
        }
    }
    look(-0.0); look(0.0); look(-705.0);
    std::printf("worst error %.3f of the bound, at %.17g\n", worst, at);
    return worst < 1.0 && psx::exp_of_gap(0.0, power) == 1.0 ? 0 : 1;
}
