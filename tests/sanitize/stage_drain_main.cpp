// csrc/stage_drain.cuh against a model of the barriers: two producers that stop at any two tiles a pipeline allows.
#include <cstdio>
#include <initializer_list>

#define __device__
#define __forceinline__ inline
#include "../../mpi-cst-fem-solver_b200/csrc/stage_drain.cuh"

struct Barrier {  // two arrivals a phase
  int pending = 2, phases = 0;
  void arrive() {
    if (--pending == 0) {
      pending = 2;
      ++phases;
    }
  }
  bool done(unsigned parity) const { return (unsigned)(phases & 1) != parity; }  // what a wait for this parity sees
};

int main() {
  int wrong = 0, cases = 0;
  for (int stages : {2, 3, 4})
    for (int a = 0; a < 40; ++a)
      for (int b = 0; b < 40; ++b) {
        // tile j needs tile j - stages consumed, for which both have arrived
        if (a > b + stages || b > a + stages) continue;
        ++cases;
        Barrier bar[4];
        for (int j = 0; j < (a > b ? a : b); ++j) {
          if (j < a) bar[j % stages].arrive();
          if (j < b) bar[j % stages].arrive();
        }
        for (int s = 0; s < stages; ++s) {
          const cstg::StageDrain d = cstg::stage_drain(s, stages, a, b);
          int newest = -1;
          for (int j = s; j < (a > b ? a : b); j += stages) newest = j;
          if (d.arrive) bar[s].arrive();
          if (d.wait != (newest >= 0)) ++wrong;
          // every phase that copies were issued for has ended, and no arrival is left over
          if (bar[s].pending != 2 || bar[s].phases != (newest < 0 ? 0 : newest / stages + 1)) ++wrong;
          if (d.wait && !bar[s].done(d.parity)) ++wrong;
        }
      }
  std::printf("%s\n", wrong || cases < 300 ? "wrong" : "ok");
  return wrong != 0;
}
