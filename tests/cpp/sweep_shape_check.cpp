// Prints the default sweep shape ("words threads slots", or "none") of a .ckt
// file's circuit in `smem` bytes of shared memory for tiles of `words`
// pattern words, and the likely shapes after it.  Usage: sweep_shape_check
// <.ckt file> <smem> <words>.
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <iterator>
#include <string>
#include <vector>

#include "../../lsim_b200/csrc/fsimb_internal.h"

using namespace fsimb;

int main(int argc, char** argv) {
  if (argc < 4) return 2;
  std::ifstream f(argv[1]);
  const std::string text((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
  const size_t smem = (size_t)std::atoll(argv[2]);
  const uint32_t words = (uint32_t)std::atoi(argv[3]);
  Netlist nl;
  parse_ckt(text.data(), text.size(), nl);
  std::vector<Fault> faults;
  for (uint32_t e = 0; e < nl.N; ++e) faults.push_back(Fault{e, 0, 0});
  Plan P;
  build_plan(nl, faults, P);
  Schedule S[9];
  auto sched_at = [&](int m) -> const Schedule& {
    if (!S[m].G) build_schedule(nl, P, 16u / (uint32_t)m, S[m]);
    return S[m];
  };
  int M = 0, T = 0;
  if (default_sweep_shape(P, sched_at, words, smem, smem + 1024, M, T))
    std::printf("%d %d %u\n", M, T, S[M].max_live);
  else
    std::printf("none\n");
  for (const SweepShape& s : likely_shapes(P, words, smem, smem + 1024, 10)) std::printf("%d %d\n", s.M, s.threads);
  return 0;
}
