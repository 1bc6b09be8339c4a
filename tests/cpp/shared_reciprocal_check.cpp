// The FP64 pair kernel's shared root and reciprocal (kernels_pairs.cu,
// ref_terms), restated with std::fma: the root against std::sqrt and every
// quotient against the division operator, bit for bit, over random operands,
// operands with few bits or runs of ones (quotients near the middle of two
// doubles), and seeds anywhere within the FP32 seed's error.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

static uint64_t bits(double x) { uint64_t b; std::memcpy(&b, &x, 8); return b; }
static double from(uint64_t b) { double x; std::memcpy(&x, &b, 8); return x; }
static int ef(double x) { return (int)((bits(x) >> 52) & 0x7FF); }

int main(int argc, char** argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    auto mant = [&]() -> uint64_t {
        uint64_t m = g() & ((1ull << 52) - 1);
        switch (g() % 5) {
            case 0: return m & ~((1ull << (g() % 52)) - 1);           // few bits
            case 1: return m | ((1ull << (g() % 52)) - 1);            // trailing ones
            case 2: return ((1ull << 52) - 1) & ~(1ull << (g() % 52)); // nearly all ones
            default: return m;
        }
    };
    auto num = [&](int lo, int hi) {
        return from((uint64_t)(1023 + lo + (int)(g() % (uint64_t)(hi - lo + 1))) << 52 | mant() | (g() & 1) << 63);
    };
    long fallback = 0;
    for (long k = 0; k < n; ++k) {
        const double a = std::fabs(num(-12, 12));
        const double y0 = (double)(float)(1.0 / std::sqrt(a)) * (1.0 + U(g) * 2.4e-7);
        const double e = std::fma(-(a * y0), y0, 1.0);
        double y = std::fma(y0 * e, std::fma(0.375, e, 0.5), y0);
        const double gg = a * y, h = y * 0.5;
        const double r = std::fma(std::fma(-gg, gg, a), h, gg);
        const double rem = std::fma(-r, r, a);
        const double lim = std::ldexp(r, ef(r) - 1023 - 52);
        bool ok = std::fabs(rem) < lim || rem == lim;
        ok = ok && (bits(r) & 0xFFFFFFFFFFFFFull) < 0xFFFFFFFFFFF00ull;
        if (!ok) { ++fallback; continue; }   // the kernel takes the library's root
        if (r != std::sqrt(a)) { std::printf("root of %a: %a\n", a, r); return 1; }
        y = std::fma(std::fma(-r, y, 1.0), y, y);
        const double yl = std::fma(-r, y, 1.0) * y;
        for (int q = 0; q < 3; ++q) {
            const double x = num(-40, 10);
            const double q0 = std::fma(x, y, x * yl);
            const double d = std::fma(std::fma(-r, q0, x), y, q0);
            if (d != x / r) { std::printf("%a / %a: %a, not %a\n", x, r, d, x / r); return 1; }
        }
    }
    std::printf("ok %ld roots, %ld left to the library\n", n, fallback);
    return 0;
}
