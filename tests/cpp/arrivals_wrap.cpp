// The barrier rule of csrc/arrivals.cuh in a simulation: T CTAs arrive and look in
// random order, over barriers that take the 32-bit count through its wrap. argv: T,
// the count's start, barriers, seed. Prints "ok", or what went wrong.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "arrivals.cuh"

int main(int argc, char **argv) {
    if (argc != 5) return 2;
    const unsigned T = (unsigned)std::atoi(argv[1]), start = (unsigned)std::strtoul(argv[2], nullptr, 0);
    const long barriers = std::atol(argv[3]);
    std::mt19937 rng((unsigned)std::atoi(argv[4]));
    struct Cta {
        long done = 0;  // barriers passed
        bool in = false;
        unsigned target;
    };
    std::vector<Cta> c(T);
    for (Cta &x : c) x.target = start;
    unsigned count = start;
    std::vector<long> arrived(T, 0);
    long left = T, idle = 0;
    while (left) {
        const unsigned i = rng() % T;
        Cta &x = c[i];
        if (x.done == barriers) continue;
        if (!x.in) {
            ++count;
            ++arrived[i];
            x.target += T;
            x.in = true;
            idle = 0;
        } else if (gbg::all_arrived(count, x.target)) {
            for (unsigned k = 0; k < T; ++k)
                if (arrived[k] <= x.done) return std::printf("CTA %u passed barrier %ld before CTA %u came\n", i, x.done, k), 1;
            x.in = false;
            if (++x.done == barriers) --left;
            idle = 0;
        } else if (++idle > 1000L * T) {
            return std::printf("nobody passes barrier %ld\n", x.done), 1;
        }
    }
    std::puts("ok");
    return 0;
}
