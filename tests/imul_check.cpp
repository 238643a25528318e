/* Checks the integer-pipe product of the exact FP64 step (mul_int, fp64_imul.cuh) bit for bit
 * against IEEE multiplication: random significands, all-ones and sparse ones (exact halves,
 * carries into the next power of two), exponents over the accepted window, signed zeros; and that
 * operands outside the window are reported.  Usage: imul_check N -> prints "N mismatches". */
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include <limits>

#include "../mpdugks_gb300/csrc/fp64_imul.cuh"

static uint64_t state = 0x9E3779B97F4A7C15ULL;
static uint64_t next() {
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    return state;
}
static double of_bits(uint64_t b) { return dugks::double_of((uint32_t)(b >> 32), (uint32_t)b); }
static uint64_t bits(double d) {
    uint64_t v;
    std::memcpy(&v, &d, 8);
    return v;
}
static double operand(int kind) {
    uint64_t m = next() & ((1ULL << 52) - 1);
    if (kind == 1) m |= (1ULL << 40) - 1;
    if (kind == 2) m &= ~((1ULL << (next() % 53)) - 1);
    if (kind == 3) m = ((1ULL << 52) - 1) ^ (next() & 3);
    const uint64_t e = 768 + next() % 512;  // the window: 2^-255 .. 2^256
    const uint64_t b = ((next() & 1) << 63) | (e << 52) | m;
    return kind == 4 ? of_bits((next() & 1) << 63) : of_bits(b);
}
int main(int argc, char **argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
    long wrong = 0;
    for (long i = 0; i < n; ++i) {
        const double a = operand((int)(i % 5)), b = operand((int)(next() % 5));
        uint32_t bad = 0;
        const double r = dugks::mul_int(a, b, bad);
        if (bad || bits(r) != bits(a * b)) ++wrong;
    }
    const double outside[] = {5e-324, 1e-310, 0x1p-256, 0x1p257, std::numeric_limits<double>::infinity(),
                              std::numeric_limits<double>::quiet_NaN()};
    for (double x : outside)
        for (double y : {1.5, 0.0, -2.0}) {
            uint32_t p = 0, q = 0;
            dugks::mul_int(x, y, p);
            dugks::mul_int(y, -x, q);
            if (!p || !q) ++wrong;
        }
    std::printf("%ld products, %ld mismatches\n", n, wrong);
    return wrong ? 1 : 0;
}
