// Builds a circuit's sweep schedules and packs them: for each residue group
// size (16, 8, 4, 2: one, two, four, eight words per item) prints the size, the slots, and
// the records of the packed stream or "refused".  Usage: sweep_limits_check
// <.ckt file>; faults: every output stuck at 0.
#include <cstdio>
#include <fstream>
#include <iterator>
#include <string>
#include <vector>

#include "../../lsim_b200/csrc/fsimb_netlist.h"
#include "../../lsim_b200/csrc/fsimb_plan.h"

using namespace fsimb;

int main(int argc, char** argv) {
  if (argc < 2) return 2;
  std::ifstream f(argv[1]);
  const std::string text((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
  Netlist nl;
  parse_ckt(text.data(), text.size(), nl);
  std::vector<Fault> faults;
  for (uint32_t e = 0; e < nl.N; ++e) faults.push_back(Fault{e, 0, 0});
  Plan P;
  build_plan(nl, faults, P);
  std::printf("live %u\n", P.max_live);
  for (uint32_t G : {16u, 8u, 4u, 2u}) {
    Schedule S;
    build_schedule(nl, P, G, S);
    std::printf("%u %u ", G, S.max_live);
    try {
      pack_schedule(S, 64);
      std::printf("%u\n", S.stream_recs);
    } catch (const LimitError&) {
      std::printf("refused\n");
    }
  }
  return 0;
}
