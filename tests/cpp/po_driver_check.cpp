// Sweep schedules of a circuit whose PO drivers, or folded gates' inputs,
// outnumber its gates' live values: the slots of every residue group size,
// and some sweeps run on the CPU record by record, forwards and backwards,
// against a plain evaluation of the netlist.  Usage: po_driver_check <.ckt
// file> <sweeps per schedule>; prints the gates' live values, the drivers
// compared by their own records, the folded gates, and per group size the
// slots and the sweeps compared.
#define main sweep_net_check_main
#include "sweep_net_check.cpp"
#undef main

#include <fstream>
#include <iterator>

// A record, a direct PO record among them.
static void run_any(const Schedule& S, const std::array<uint32_t, 4>& w, const Words& good, Words& vals,
                    uint64_t& diff) {
  if (((w[1] >> kRecKindShift) & 7u) == kRecPo && (w[0] & kPoDirect)) {
    const uint32_t* d = &S.blob.at(4 * (size_t)(w[0] & ~kPoDirect));
    uint64_t in[4] = {0, 0, 0, 0};
    const uint32_t n = (d[5] >> 4) & 15u;
    for (uint32_t k = 0; k < n; ++k) in[k] = vals.at(d[k]);
    diff |= gate(d[5] & 15u, in, n) ^ good.at(d[4]);
    return;
  }
  run_record(S, w, good, vals, diff);
}

static uint64_t run_sweep(const Netlist& nl, const Plan& P, const Schedule& S, const Words& good, const InjRec& inj,
                          uint64_t fv, bool backwards) {
  const uint32_t x = inj.stored, L0 = inj.level, nw = S.rec_words();
  Words vals(S.max_live, 0xDEADDEADDEADDEADull);
  uint64_t diff = inj.mode & kInjReachesPo ? fv ^ good[x] : 0;
  if (L0 > P.max_gate_level) return diff;
  for (uint32_t i = S.lvl[L0][1]; i < S.lvl[L0][2]; ++i)
    vals.at(S.li[2 * i + 1]) = S.li[2 * i] == x ? fv : good[S.li[2 * i]];
  size_t fix = inj.fix ? 4 * (size_t)S.fix0 + 8 * (inj.fix - 1) : 0;
  if (fix) vals.at(S.max_live - 1) = fv ^ (inj.mode & kInjAliasInv ? ~0ull : 0ull);
  for (uint32_t at = S.lvl[L0][0]; at < S.stream_recs;) {
    uint32_t end = at;
    while (!(S.blob.at((size_t)end * nw + 1) & kRecEnd)) end += S.T;
    end += S.T;
    for (uint32_t p = at; p < end; ++p)
      run_any(S, record(S, (size_t)(backwards ? end - 1 - (p - at) : p) * nw, nw), good, vals, diff);
    if (fix && S.blob.at(fix + 4) == end - S.T) {
      const uint32_t n = S.blob[fix + 5];
      for (uint32_t i = 0; i < n; ++i) run_any(S, record(S, fix + 8 * i, 4), good, vals, diff);
      fix += 8 * n;
    }
    at = end;
  }
  return diff;
}

int main(int argc, char** argv) {
  if (argc < 3) return 2;
  std::ifstream f(argv[1]);
  const std::string text((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
  Netlist nl;
  parse_ckt(text.data(), text.size(), nl);
  std::vector<Fault> faults;
  for (uint32_t e = 0; e < nl.N; ++e)
    for (uint32_t pin = 0; pin <= nl.fanin_count(e); ++pin) faults.push_back(Fault{e, (uint8_t)pin, (uint8_t)(e & 1)});
  Plan P;
  build_plan(nl, faults, P);
  size_t direct = 0, folded = 0;
  for (uint32_t e = 0; e < nl.N; ++e) {
    direct += P.net.direct[e];
    folded += P.net.lev_up[e] >> 31;
  }
  std::printf("%u %zu %zu\n", P.max_live, direct, folded);
  std::mt19937_64 rng(7);
  Words good(nl.N);
  for (uint32_t e = 0; e < nl.N; ++e) good[e] = nl.type[e] == G_PI ? rng() : eval(nl, e, good);
  const size_t per = std::max<size_t>(1, P.sweeps.size() / std::atoi(argv[2]));
  for (uint32_t G : {2u, 4u, 8u, 16u}) {
    Schedule S;
    build_schedule(nl, P, G, S);
    pack_schedule(S, 32 * (1 + rng() % 8));
    size_t compared = 0;
    for (size_t si = rng() % per; si < P.sweeps.size(); si += per, ++compared) {
      const InjRec& s = P.sweeps[si];
      const uint64_t sv = s.mode & kInjValue ? ~0ull : 0ull;
      const uint32_t pin = s.mode >> kInjPinShift;
      Words bad(good);
      uint64_t want = 0;
      for (uint32_t e = s.elem; e < nl.N; ++e) {
        if (nl.type[e] != G_PI) bad[e] = eval(nl, e, bad);
        if (e == s.elem) {
          uint64_t in[4] = {0, 0, 0, 0};
          for (uint32_t k = 0; k < nl.fanin_count(e); ++k)
            in[k] = k + 1 == pin ? sv : bad[nl.fi_idx[nl.fi_off[e] + k]];
          bad[e] = !(s.mode & kInjStuck) ? ~good[e] : pin ? gate(nl.type[e], in, nl.fanin_count(e)) : sv;
        }
        if (nl.type[e] == G_PO) want |= bad[e] ^ good[e];
      }
      for (bool backwards : {false, true})
        if (run_sweep(nl, P, S, good, s, bad[s.stored], backwards) != want)
          return std::fprintf(stderr, "G %u, sweep of element %u (stored %u): differs\n", G, s.elem, s.stored), 1;
    }
    std::printf("%u %u %zu\n", G, S.max_live, compared);
  }
  return 0;
}
