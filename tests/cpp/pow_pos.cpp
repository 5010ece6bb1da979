// pow_pos (pow_pos.cuh) as host code, against powers in 113 bits.
//   pow_pos errors SEED COUNT   largest error in units in the last place over random arguments
//   pow_pos ends                arguments that it hands to pow()
//   pow_pos table               the rows of its table
#include <quadmath.h>

#include <cstdio>
#include <cstdlib>
#include <limits>
#include <random>
#include <string>

#include "pow_pos.cuh"

static double error(double x, double b) {
    const double y = umapb::pow_pos(x, b);
    const __float128 want = powq(x, b);
    int e;
    frexp(static_cast<double>(want), &e);
    return static_cast<double>(fabsq(y - want) / scalbnq(1, e - 53));
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "errors") {
        std::mt19937_64 rng(std::atoi(argv[2]));
        auto uniform = [&](double lo, double hi) { return lo + (hi - lo) * (rng() >> 11) * 0x1p-53; };
        double worst = 0;
        for (int i = 0, n = std::atoi(argv[3]); i < n; ++i) {
            double x = std::exp2(uniform(-52, 40));
            if (i % 4 == 1) x = 1 + uniform(-0x1p-6, 0x1p-6);                                            // near 1
            if (i % 4 == 2) x = std::ldexp(1 + (rng() % 64) / 64.0, int(rng() % 60) - 40) * (1 + uniform(-2, 2) * 0x1p-52);   // edges of the table's parts
            const double err = error(x, uniform(0.3, 1.8));
            worst = err > worst ? err : worst;
        }
        std::printf("%.4f\n", worst);
        return 0;
    }
    if (what == "ends") {
        const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
        for (double x : {0.0, 0x1p-1074, 0x1p-1030, 0x1p-1022, 0x1.8p-1001, 0x1p1001, 0x1.fffffffffffffp1023, inf, nan, -1.0, 0x1p-900, 0x1p900})
            for (double b : {0.0, 0.3, 0.895, 1.0, 1.8, 40.0, -2.0, inf, nan}) {
                const double y = umapb::pow_pos(x, b), want = std::pow(x, b);
                const bool handed = !(x >= 0x1p-1000 && x <= 0x1p1000 && std::fabs(std::log2(x) * b) < 999);
                if (std::isnan(want) ? !std::isnan(y) : handed ? y != want : !(std::fabs(y - want) <= 0x1p-51 * want)) {
                    std::printf("pow(%a, %a) = %a, not %a\n", x, b, want, y);
                    return 1;
                }
            }
        return 0;
    }
    for (const umapb::PowRow& r : umapb::POW_TABLE) std::printf("%a %a %a %a\n", r.inv, r.log_hi, r.log_lo, r.exp2);
    return 0;
}
