// The largest error of ral_sf_sin and ral_sf_cos (softfp.cuh) in ulp of the exact value, taken from the host's long
// double functions (at least 64 bits: 2^-11 ulp of their own), over one kind of argument after the other:
// "name arguments max_error first_x" a line.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "softfp.cuh"

namespace {

struct Worst {
    const char* name;
    long n = 0;
    double err = 0, at = 0;
    void take(double got, long double exact, double x) {
        int e = -1074;
        if (exact != 0) e = std::fmax(std::ilogb(exact) - 52, -1074);
        const double d = (double)(std::fabs((long double)got - exact) / std::ldexp(1.0L, e));
        if (!(d <= err)) err = d, at = x;
    }
    void check(double x) {
        n++;
        take(ral_sf_sin(x), sinl((long double)x), x);
        take(ral_sf_cos(x), cosl((long double)x), x);
    }
    void neighbours(double b, int k) {  // b's 2 k + 1 neighbours, of either sign
        double up = b, down = b;
        check(b);
        for (int i = 0; i < k; i++) {
            up = std::nextafter(up, HUGE_VAL);
            down = std::nextafter(down, -HUGE_VAL);
            check(up);
            check(-up);
            check(down);
            check(-down);
        }
    }
    void report() const { std::printf("%s %ld %.6f %a\n", name, n, err, at); }
};

}  // namespace

int main(int argc, char** argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 100000;
    std::mt19937_64 rng(20261205);
    auto unit = [&] { return std::ldexp((double)(rng() >> 11), -53); };
    const double pi2 = 1.5707963267948966;
    Worst bounds{"bounds"}, quarters{"quarters"}, spread{"spread"}, small{"small"}, plain{"plain"};
    // the reduction's bounds (1/2, 2^-27 and its power-of-two neighbours), pi/4 and where a result changes binade
    for (const double b : {0.5, 1.0, 0x1p-27, 0x1p-26, 0x1p-28, pi2 / 2, pi2, pi2 / 3, 2 * pi2 / 3, 0x1p51, 0x1.fp51}) bounds.neighbours(b, 5000);
    for (long i = 0; i < n / 8; i++) quarters.neighbours(std::rint(std::ldexp(1 + unit(), (int)(rng() % 50) - 1)) * pi2, 2);
    for (long i = 0; i < n; i++) {
        spread.check(std::ldexp(1 + unit(), (int)(rng() % 53) - 1) * ((rng() & 1) ? 1 : -1));
        small.check(std::ldexp(1 + unit(), -(int)(rng() % 60)));
        plain.check(unit() * 2000 - 1000);
    }
    for (const Worst* w : {&bounds, &quarters, &spread, &small, &plain}) w->report();
}
