// persistent_grid on the host: prints one line per argument set read from the command line
// (n ppb resident limit one_round), the blocks it gives.
#include <cstdio>
#include <cstdlib>
#include "sph_persistent.cuh"

int main(int argc, char** argv) {
    for (int k = 1; k + 4 < argc; k += 5)
        printf("%d\n", wsph::persistent_grid(atoll(argv[k]), atoi(argv[k + 1]), atoll(argv[k + 2]), atoll(argv[k + 3]), atoi(argv[k + 4]) != 0));
    return 0;
}
