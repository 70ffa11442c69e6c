// Host check of the FP64 path's quotient (rcp_f64, quot_f64) against the exact
// one, for reciprocals as rough as the hardware's approximation may be (20
// bits of the operand and of the result: 2^-19 relative, either way).  Built
// for the host only; no GPU.
//
// One Newton step leaves r within 2^-38 of 1 / d relative and q = num r within
// 2^-37; the remainder num - d q, rounded once, is a 2^-37th of num, so the
// corrected q is within 2^-74 of the quotient before its own rounding: half an
// ulp but for 2^-21 of one.  Measured against long double (64 bits or more),
// whose own rounding is 2^-12 of an ulp: at most 0.5 + 2^-10 ulp.
#include "../adeco_gb300/csrc/kernels.cuh"

#include <cmath>
#include <cstdio>
#include <random>

using namespace adeco;

int main()
{
    std::mt19937_64 rng(17);
    std::uniform_real_distribution<double> U(0.0, 1.0), E(-1.0, 1.0);
    double worst = 0.0;
    for (int i = 0; i < 2000000; ++i) {
        // a crossing edge: ends on either side of a face, up to 4096 cells away
        const double plane = (double)(i & 1), s = (i & 2) ? 1.0 : -1.0;
        const double in = plane + s * std::exp2(-40.0 + 52.0 * U(rng)), out = plane - s * std::exp2(-40.0 + 52.0 * U(rng));
        const double num = plane - in, d = out - in;
        const double r = rcp_f64(d, (double)(float)((1.0 + E(rng) * 0x1p-19) / d));
        const double q = quot_f64(num, d, r);
        const long double exact = (long double)num / (long double)d;
        const double ulp = std::ldexp(1.0, std::ilogb((double)exact) - 52);
        worst = std::fmax(worst, (double)std::fabs((long double)q - exact) / ulp);
    }
    const bool ok = worst <= 0.5 + 0x1p-10;
    std::printf("FP64 quotient: %s (worst %.6f ulp)\n", ok ? "ok" : "FAIL", worst);
    return ok ? 0 : 1;
}
