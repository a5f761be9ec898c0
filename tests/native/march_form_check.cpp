/* The forms march_form (plume_b200/csrc/march_plan.cuh, compiled here as it is) gives the calls of its arguments:
 * n0 n1 n2 dt set, five at a time. */
#include <stdio.h>
#include <stdlib.h>

#include "march_plan.cuh"

int main(int argc, char** argv) {
  for (int a = 1; a + 4 < argc; a += 5) {
    const int dims[3] = {atoi(argv[a]), atoi(argv[a + 1]), atoi(argv[a + 2])};
    printf("%d\n", plume::mac::march_form(dims, strtof(argv[a + 3], nullptr), atoi(argv[a + 4])));
  }
  return 0;
}
