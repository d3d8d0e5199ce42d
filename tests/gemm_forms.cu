// Prints the tokens of a wide unit (0: another form) for every product m n k of the arguments.
#include <cstdio>
#include <cstdlib>

#include "q8_gemm_tc.cuh"

int main(int argc, char** argv) {
  for (int i = 1; i + 2 < argc; i += 3) printf("%d\n", logos::gemm_wide_tokens(atoll(argv[i]), atoll(argv[i + 1]), atoll(argv[i + 2]), 0));
  return 0;
}
