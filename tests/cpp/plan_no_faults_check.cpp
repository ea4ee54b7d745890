// The plan of a circuit without faults holds what the good machine reads and
// nothing that only sweeps and tracing need.  Usage: plan_no_faults_check
// <.ckt file>; prints the time of a plan without and with faults, in us.
#include <algorithm>
#include <chrono>
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
  std::vector<Fault> one(1);
  one[0] = Fault{(uint32_t)nl.n_pi, 0, 0};
  auto us = [&](const std::vector<Fault>& faults, Plan& P) {
    double best = 1e30;
    for (int k = 0; k < 5; ++k) {
      const auto t0 = std::chrono::steady_clock::now();
      build_plan(nl, faults, P);
      best = std::min(best, std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0).count());
    }
    return best;
  };
  Plan none, some;
  const double a = us({}, none), b = us(one, some);
  std::printf("%.0f %.0f\n", a, b);
  const bool same = none.N == some.N && none.n_levels == some.n_levels && none.level_off == some.level_off &&
                    none.max_gate_level == some.max_gate_level && none.net.gates == some.net.gates;
  const bool bare = none.gate_fo.empty() && none.po_drv.empty() && none.nfp_prefix.empty() && none.sweeps.empty() &&
                    none.net.live.empty();
  Schedule S;
  build_schedule(nl, none, 2, S);
  pack_schedule(S, 64);
  return same && bare && S.stream_recs == 0 ? 0 : 1;
}
