// Prints k2_limit(R) of csrc/ts_radius.h for every radius given on the command line.
#include <cstdio>
#include <cstdlib>

#include "ts_radius.h"

int main(int argc, char** argv) {
  for (int i = 1; i < argc; ++i) printf("%.17g\n", ts::k2_limit(strtod(argv[i], nullptr)));
  return 0;
}
