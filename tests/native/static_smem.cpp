// The shared memory of a register-kernel CTA of the model whose headers are
// in the include path: {row table, static bytes with it, largest dynamic
// share, what a CTA may have}.
#include <cstdio>

#include "engine_types.hpp"

using namespace dense_b200;

int main() {
  std::printf("%d %d %d %d\n", kRowTables ? 1 : 0, kStepStatic + (kRowTables ? kTableBytes : 0), kStepSmem1, kCtaSmem);
  return 0;
}
