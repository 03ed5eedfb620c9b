// What is left to wait for on a stage's barrier that two producers arrive on, when they may have stopped at different
// tiles. Tile j goes to stage j % stages and is that barrier's phase j / stages; a producer takes a stage's next tile
// only after the stage's last one has been consumed, so at most the newest tile of a stage is pending.
#pragma once

namespace cstg {

struct StageDrain {
  bool wait;        // the phase of the stage's newest tile
  bool arrive;      // in place of the producer that stopped before that tile
  unsigned parity;
};

// a, b: tiles that each producer has arrived for (0 .. a - 1 and 0 .. b - 1)
__device__ __forceinline__ StageDrain stage_drain(int s, int stages, int a, int b) {
  const int la = a > s ? s + (a - 1 - s) / stages * stages : -1, lb = b > s ? s + (b - 1 - s) / stages * stages : -1;
  const int newest = la > lb ? la : lb;
  return StageDrain{newest >= 0, la != lb, newest >= 0 ? (unsigned)(newest / stages) & 1u : 0u};
}

}  // namespace cstg
