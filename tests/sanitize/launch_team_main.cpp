// csrc/teams.h against a fake of the launch: which team a solve ends on when the device refuses some.
#include <cstdio>
#include <vector>

#include "../../mpi-cst-fem-solver_b200/csrc/teams.h"

using namespace cstg;

static int cleared = 0;
extern "C" cudaError_t cudaGetLastError(void) {
  ++cleared;
  return cudaSuccess;
}

static int wrong = 0;
static void check(const char* what, std::vector<cudaError_t> answers, PcgTeam from, PcgTeam want, cudaError_t err,
                  int launches) {
  int calls = 0;
  cleared = 0;
  PcgTeam team = from;
  const cudaError_t e = launch_first_team(
      team, [&](PcgTeam t) { return ++calls, answers[(int)t]; }, [](PcgTeam t) { return (PcgTeam)((int)t + 1); });
  const int refused = launches - (team == PcgTeam::kNone ? 0 : 1);
  if (team != want || e != err || calls != launches || cleared != refused) {
    std::printf("%s: team %d error %d calls %d cleared %d\n", what, (int)team, (int)e, calls, cleared);
    ++wrong;
  }
}

int main() {
  const cudaError_t ok = cudaSuccess, coop = cudaErrorCooperativeLaunchTooLarge, cl = cudaErrorInvalidClusterSize,
                    res = cudaErrorLaunchOutOfResources, bad = cudaErrorInvalidValue;
  check("taken", {ok, ok, ok, ok, ok}, PcgTeam::kCluster, PcgTeam::kCluster, ok, 1);
  check("no cluster", {cl, ok, ok, ok, ok}, PcgTeam::kCluster, PcgTeam::kResident, ok, 2);
  check("no grid team", {res, coop, coop, coop, ok}, PcgTeam::kCluster, PcgTeam::kGrid, ok, 5);
  check("none", {cl, coop, coop, coop, coop}, PcgTeam::kResident, PcgTeam::kNone, ok, 4);
  check("another error", {bad, ok, ok, ok, ok}, PcgTeam::kCluster, PcgTeam::kCluster, bad, 1);
  check("then another error", {cl, bad, ok, ok, ok}, PcgTeam::kCluster, PcgTeam::kResident, bad, 2);
  check("not asked", {ok, ok, ok, ok, ok}, PcgTeam::kNone, PcgTeam::kNone, ok, 0);
  std::printf("%s\n", wrong ? "wrong" : "ok");
  return wrong != 0;
}
