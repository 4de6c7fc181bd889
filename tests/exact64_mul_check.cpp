// Host check of ts::x64::mul against the hardware's product: reads operand
// pairs (doubles) from stdin, prints the number of products that differ in
// any bit and the number refused.
#include <cstdio>

#include "ts_exact64.cuh"

using namespace ts::x64;

int main() {
    double p[2];
    long wrong = 0, refused = 0;
    while (std::fread(p, 8, 2, stdin) == 2) {
        bool rare;
        const double m = mul(p[0], p[1], rare);
        if (rare) ++refused;
        else if (bits_of(m) != bits_of(p[0] * p[1])) ++wrong;
    }
    std::printf("%ld %ld\n", wrong, refused);
    return 0;
}
