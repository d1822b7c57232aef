// ReciprocalDivisor (adjoint.cuh) against the division it stands for, on the CPU: the same bits for
// quotients and reciprocals in the normal range, the same infinities and NaN, equal zeros (the sign
// of a zero is not kept), and subnormal quotients within one unit of the last place.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>

#include "adjoint.cuh"

namespace {

uint64_t state = 88172645463325252ull;
uint64_t next() {
    state ^= state << 13;
    state ^= state >> 7;
    return state ^= state << 17;
}
double of_bits(uint64_t b) {
    double d;
    std::memcpy(&d, &b, sizeof(d));
    return d;
}
uint64_t bits_of(double d) {
    uint64_t b;
    std::memcpy(&b, &d, sizeof(b));
    return b;
}

// 0: as stated above
int check(double a, double x) {
    const double want = a / x;
    const double got = mkb::ReciprocalDivisor<double>(x).div(a);
    const double r = std::fabs(1.0 / x), q = std::fabs(want);
    const double tiny = std::numeric_limits<double>::min();
    bool ok;
    if (std::isnan(want)) ok = std::isnan(got);
    else if (std::isinf(r) && x != 0.0) return 0;  // a subnormal divisor: no reciprocal
    else if (want == 0.0 && a == 0.0) ok = got == 0.0;
    else if (std::isinf(x) || std::isinf(a) || x == 0.0) ok = bits_of(got) == bits_of(want);
    else if (r < tiny) ok = std::fabs(got - want) <= q * 2.3e-16;  // a subnormal reciprocal
    else if (std::isinf(want) || q > 1e308) return 0;  // a * (1 / x) may round past the largest
    else if (q < tiny * 4.0) ok = std::fabs(got - want) <= 2.0 * std::numeric_limits<double>::denorm_min();
    else if (std::fabs(a) < std::ldexp(tiny, 108)) ok = std::fabs(got - want) <= q * 2.3e-16;
    else ok = bits_of(got) == bits_of(want);
    if (!ok) std::printf("%a / %a: %a, not %a\n", a, x, got, want);
    return ok ? 0 : 1;
}

}  // namespace

int main() {
    int bad = 0;
    const double inf = std::numeric_limits<double>::infinity();
    const double edges[] = {0.0, 1.0, 3.0, 1.0 / 3.0, std::nextafter(1.0, 0.0),
                            std::nextafter(1.0, 2.0), std::nextafter(2.0, 0.0), 0x1p-1022, 0x1p-1021,
                            0x1p-1074, 0x1p-1030, 0x1p-500, 0x1p500, 0x1p1022, 0x1p1023, 1.7e308,
                            inf, std::numeric_limits<double>::quiet_NaN()};
    for (double a : edges)
        for (double x : edges)
            for (int s = 0; s < 4; ++s) bad += check(s & 1 ? -a : a, s & 2 ? -x : x);
    for (int i = 0; i < 20000000; ++i) {
        // mantissas of all kinds (random, few bits set, near a power of two), exponents around 1
        // and, in every fourth pair, over the whole range
        auto draw = [&](bool wide) {
            uint64_t m = next() & 0xFFFFFFFFFFFFFull;
            const uint64_t kind = next() & 3;
            if (kind == 1) m &= ~0ull << (next() % 52);
            if (kind == 2) m = (0ull - (next() & 63)) & 0xFFFFFFFFFFFFFull;
            if (kind == 3) m = next() & 63;
            const uint64_t e = wide ? next() % 2047 : 1023 - 20 + next() % 41;
            return of_bits((next() & 1) << 63 | e << 52 | m);
        };
        bad += check(draw(i % 4 == 0), draw(i % 4 == 0));
        if (bad > 20) break;
    }
    if (bad == 0) std::printf("divisor checks passed\n");
    return bad == 0 ? 0 : 1;
}
