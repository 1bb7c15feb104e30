// Prints the quota that csrc/host_cores.h finds under the root argv[1], and the threads it allows.
#include "host_cores.h"

int main(int, char** argv) {
    std::printf("%g %d\n", mascot::quota_cores(argv[1]), mascot::usable_cores(argv[1]));
    return 0;
}
