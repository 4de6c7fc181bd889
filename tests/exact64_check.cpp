// Host check of csrc/ts_exact64.cuh against the hardware's division and square
// root: reads operand pairs (doubles) from stdin, prints the number of
// quotients, roots and halves that differ in any bit, and of operands refused.
#include <cmath>
#include <cstdio>

#include "ts_exact64.cuh"

using namespace ts::x64;

int main() {
    double p[2];
    long quo = 0, rt = 0, hf = 0, refused = 0;
    while (std::fread(p, 8, 2, stdin) == 2) {
        bool bad = false;
        const double q = div(p[0], p[1], bad);
        if (bad) ++refused;
        else if (bits_of(q) != bits_of(p[0] / p[1])) ++quo;
        bad = false;
        const double r = root(std::fabs(p[1]), bad);
        if (bad) ++refused;
        else if (bits_of(r) != bits_of(std::sqrt(std::fabs(p[1])))) ++rt;
        bad = false;
        const double h = half(p[0], bad);
        if (bad) ++refused;
        else if (bits_of(h) != bits_of(p[0] * 0.5)) ++hf;
    }
    std::printf("%ld %ld %ld %ld\n", quo, rt, hf, refused);
    return 0;
}
