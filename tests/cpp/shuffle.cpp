// The order in which a training call visits its rows: std::shuffle of 0 .. n - 1 with mt19937(seed), once an
// epoch with the same generator.
#include <algorithm>
#include <cstdint>
#include <numeric>
#include <random>
#include <vector>

extern "C" void epochs_order(uint32_t n, uint32_t epochs, uint32_t seed, int32_t* out) {
    std::mt19937 rng(seed);
    for (uint32_t e = 0; e < epochs; ++e, out += n) {
        std::vector<int32_t> perm(n);
        std::iota(perm.begin(), perm.end(), 0);
        std::shuffle(perm.begin(), perm.end(), rng);
        std::copy(perm.begin(), perm.end(), out);
    }
}
