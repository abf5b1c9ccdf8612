// The work chunk that the library takes for a configured chunk, a photon count and a number of
// multiprocessors, one line each (read by test_chunk_rule.py; host code only).
#include <cstdio>
#include <cstdlib>

#include "../shapefromcaustics_b200/csrc/pds_internal.h"

int main(int argc, char** argv) {
    for (int k = 1; k + 2 < argc; k += 3)
        std::printf("%d\n", int(pds::effective_chunk(std::atoi(argv[k]), std::atoll(argv[k + 1]),
                                                     std::atoll(argv[k + 2]))));
    return 0;
}
