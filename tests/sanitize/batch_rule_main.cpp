// csrc/batch_rule.h: which kernel a batch runs on.
#include <cstdio>

#include "../../mpi-cst-fem-solver_b200/csrc/batch_rule.h"

using namespace cstg;

static int wrong = 0;
static void check(const char* what, bool got, bool want) {
  if (got == want) return;
  std::printf("%s\n", what);
  ++wrong;
}

int main() {
  const unsigned smem = 222 * 1024;
  check("both fit", batch_shape_runs({18, 18}), true);
  check("the halo kernel cannot be resident: the other one runs the batch", batch_shape_runs({1, 0}), true);
  check("nothing fits", batch_shape_runs({0, 0}), false);
  check("small plates", batch_halo_runs({18, 18}, 20301, 8, 4, smem), true);
  check("small plates, no room for the halo kernel", batch_halo_runs({18, 0}, 20301, 8, 4, smem), false);
  check("a large plate", batch_halo_runs({18, 18}, 80601, 8, 4, smem), false);
  check("a large plate, one load case", batch_halo_runs({18, 18}, 80601, 16, 1, smem), true);
  std::printf("%s\n", wrong ? "wrong" : "ok");
  return wrong != 0;
}
