// Prints the first logical slot of each block and the array size that the library uses
// (am_chunks.hpp) for the block slot counts given as arguments.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "am_chunks.hpp"

int main(int argc, char** argv) {
    std::vector<int64_t> counts;
    for (int k = 1; k < argc; ++k) counts.push_back(std::atoll(argv[k]));
    for (int64_t b : am::slot_bases(counts)) std::printf("%lld\n", static_cast<long long>(b));
    return 0;
}
