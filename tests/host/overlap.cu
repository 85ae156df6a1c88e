// Prints overlap_pays(blocks, slots per SM, SMs) for the numbers given.
#include <cstdio>
#include <cstdlib>

#include "lbm_fused.cuh"

int main(int argc, char** argv) {
  for (int i = 1; i + 2 < argc; i += 3)
    std::printf("%d\n", (int)lbm::overlap_pays(atoll(argv[i]), atoi(argv[i + 1]), atoi(argv[i + 2])));
  return 0;
}
