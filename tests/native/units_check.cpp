// Prints up_bits for n full shares times `terms` (arguments: pairs n terms).
#include <cstdio>
#include <cstdlib>

#include "../../chimes_lsq-myllfork_gb300/csrc/units.h"

int main(int argc, char** argv) {
    for (int i = 1; i + 1 < argc; i += 2) {
        const unsigned long long n = std::strtoull(argv[i], nullptr, 10);
        unsigned long long sum = n * cgd::share16(0, 0);
        std::printf("%d\n", cgd::up_bits(sum, std::atoi(argv[i + 1])));
    }
    std::printf("%u %u %u\n", cgd::share16(-3, 0), cgd::share16(-16, 0), cgd::share16(-900, 12));
    return 0;
}
