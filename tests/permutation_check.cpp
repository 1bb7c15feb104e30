// permute() against permute_index() for every length and seed given; prints the number of positions compared.
#include <cstdio>
#include <cstdlib>

#include "layout.cuh"

int main(int argc, char** argv) {
    unsigned long long compared = 0;
    for (int a = 1; a + 1 < argc; a += 2) {
        const unsigned long long n = std::strtoull(argv[a], nullptr, 0), seed = std::strtoull(argv[a + 1], nullptr, 0), step = n / 50000 + 1;
        const mascot::Permutation p = mascot::make_permutation(n, seed);
        for (unsigned long long j = 0; j < n; j = j + 1 < n && j + step >= n ? n - 1 : j + step, compared++)
            if (mascot::permute(p, (uint32_t)j) != mascot::permute_index(j, n, seed)) { std::printf("n %llu seed %llu position %llu\n", n, seed, j); return 1; }
    }
    std::printf("%llu\n", compared);
    return 0;
}
