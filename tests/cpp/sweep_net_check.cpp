// Runs sweep schedules on the CPU, record by record as the kernels read
// them, and compares the PO differences of every injection with a plain
// evaluation of the netlist.  Usage: sweep_net_check <seed> <gates> <max
// inputs> <mux 0/1> <window> <near>: every gate's first input is one of the
// `near` elements before it, the others one of the last `window`; prints the
// number of sweeps compared.
#include <array>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <string>
#include <vector>

#include "../../lsim_b200/csrc/fsimb_netlist.h"
#include "../../lsim_b200/csrc/fsimb_plan.h"

using namespace fsimb;
using Words = std::vector<uint64_t>;

static uint64_t gate(uint8_t t, const uint64_t* in, uint32_t n) {
  if (t == G_MUX) return (in[2] & in[1]) | (in[0] & (uint64_t)(in[2] == 0));
  uint64_t r = in[0];
  if (t == G_INV || t == G_CLKBUF || t == G_PO) n = 1;
  for (uint32_t k = 1; k < n; ++k)
    r = t == G_AND || t == G_NAND ? r & in[k] : t == G_OR || t == G_NOR ? r | in[k] : r ^ in[k];
  return t == G_INV || t == G_NAND || t == G_NOR || t == G_XNOR ? ~r : r;
}

static uint64_t eval(const Netlist& nl, uint32_t e, const Words& v) {
  uint64_t in[4] = {0, 0, 0, 0};
  const uint32_t n = nl.fanin_count(e);
  for (uint32_t k = 0; k < n && k < 4; ++k) in[k] = v[nl.fi_idx[nl.fi_off[e] + k]];
  return gate(nl.type[e], in, n);
}

// The record at word `i` of the blob, four words.
static std::array<uint32_t, 4> record(const Schedule& S, size_t i, uint32_t words) {
  std::array<uint32_t, 4> w{0, 0, 0, 0};
  for (uint32_t k = 0; k < words; ++k) w[k] = S.blob.at(i + k);
  return w;
}

// One record on the slot values.
static void run_record(const Schedule& S, const std::array<uint32_t, 4>& w, const Words& good, Words& vals,
                       uint64_t& diff) {
  auto at = [&](uint32_t k) -> uint64_t& {  // slot k of the record
    const uint32_t sh = 14 * (k & 1u);
    return vals.at(((w[k / 2] >> sh) & kRecSlot) | ((w[2 + k / 2] >> sh) & kRecSlot) << 14);
  };
  auto inv = [&](uint32_t k) { return (w[0] >> (31 - k)) & 1u ? ~0ull : 0ull; };
  const uint32_t kind = (w[1] >> kRecKindShift) & 7u;
  if (kind == kRecNop) return;
  if (kind == kRecWide) {
    const uint32_t* d = &S.blob.at(4 * (size_t)w[0]);
    uint64_t in[4] = {0, 0, 0, 0};
    const uint32_t n = (d[5] >> 4) & 15u;
    for (uint32_t k = 0; k < n; ++k) in[k] = vals.at(d[k]);
    vals.at(d[4]) = gate(d[5] & 15u, in, n);
    return;
  }
  if (kind == kRecPo) {
    diff |= at(3) ^ good.at(w[0]);
    return;
  }
  if (kind == kRecMux) {
    const uint64_t in[3] = {at(0), at(1), at(2)};
    at(3) = gate(G_MUX, in, 3);
    return;
  }
  const bool third = kind == kRecAnd3 || kind == kRecXor3, is_xor = kind >= kRecXor2;
  uint64_t x[3];
  for (int k = 0; k < 3; ++k) x[k] = (k < 2 || third ? at(k) : 0ull) ^ inv(k);
  at(3) = (is_xor ? x[0] ^ x[1] ^ x[2] : x[0] & x[1] & x[2]) ^ inv(3);
}

// The record stream of one sweep: PO differences of `fv` on element x.  A
// level's records run in stream order or backwards: they are independent.
static uint64_t run_schedule(const Netlist& nl, const Plan& P, const Schedule& S, const Words& good,
                             const InjRec& inj, uint64_t fv, bool backwards) {
  const uint32_t x = inj.stored;
  Words vals(S.max_live, 0xDEADDEADDEADDEADull);
  const uint32_t L0 = inj.level;
  if (L0 != P.net.lev_up[x] + 1) std::abort();
  uint64_t diff = nl.type[x] == G_PO || P.po_drv[x] ? fv ^ good[x] : 0;
  if (L0 > P.max_gate_level) return diff;
  for (uint32_t i = S.lvl[L0][1]; i < S.lvl[L0][2]; ++i)
    vals[S.li[2 * i + 1]] = S.li[2 * i] == x ? fv : good[S.li[2 * i]];
  size_t fix = inj.fix ? 4 * (size_t)S.fix0 + 8 * (inj.fix - 1) : 0;
  if (fix) vals.at(S.max_live - 1) = fv ^ (inj.mode & kInjAliasInv ? ~0ull : 0ull);
  const uint32_t nw = S.rec_words();
  auto ends = [&](uint32_t i) { return S.blob.at((size_t)i * nw + 1) & kRecEnd; };
  for (uint32_t at = S.lvl[L0][0]; at < S.stream_recs;) {
    uint32_t end = at;  // whole rounds, the last one marked on every record
    for (;; end += S.T) {
      for (uint32_t i = 1; i < S.T; ++i)
        if (ends(end) != ends(end + i)) std::abort();
      if (ends(end)) break;
    }
    end += S.T;
    for (uint32_t p = at; p < end; ++p)
      run_record(S, record(S, (size_t)(backwards ? end - 1 - (p - at) : p) * nw, nw), good, vals, diff);
    if (fix && S.blob.at(fix + 4) == end - S.T) {
      const uint32_t n = S.blob[fix + 5];
      for (uint32_t i = 0; i < n; ++i) run_record(S, record(S, fix + 8 * (backwards ? n - 1 - i : i), 4), good, vals, diff);
      fix += 8 * n;
    }
    at = end;
  }
  if (fix && S.blob.at(fix + 4) != ~0u) std::abort();  // every fix level was met
  return diff;
}

int main(int argc, char** argv) {
  if (argc < 7) return 2;
  std::mt19937_64 rng(std::atoi(argv[1]));
  const uint32_t n_gates = std::atoi(argv[2]), max_in = std::atoi(argv[3]), mux = std::atoi(argv[4]),
                 window = std::atoi(argv[5]), near = std::atoi(argv[6]), n_pi = 12,
                 n_po = n_gates > 1000 ? n_gates / 2 : 7, po_near = n_gates > 1000 ? n_gates : 30;
  // A random netlist: ids PIs, POs, gates; every gate reads 1..max_in of the
  // `window` elements before it, sometimes the same one twice.
  const uint32_t g0 = n_pi + n_po;
  std::vector<std::vector<std::pair<uint32_t, uint32_t>>> sinks(g0 + n_gates);
  std::string types;
  auto element = [&](uint32_t i) { return i < n_pi ? i : i - n_pi + g0; };  // i-th PI or gate
  for (uint32_t g = 0; g < n_gates; ++g) {
    uint32_t t = rng() % (mux ? 9 : 8);
    if (!mux && t == G_MUX) t = G_CLKBUF;
    uint32_t n = 1 + rng() % max_in;
    if (t == G_MUX) n = 3;
    if (t == G_INV || t == G_CLKBUF) n = rng() % 8 ? 1 : std::min<uint32_t>(2, max_in);
    for (uint32_t k = 1; k <= n; ++k) {
      const uint32_t hi = n_pi + g, lo = hi > window ? hi - window : 0;
      sinks[element(k == 1 ? hi - 1 - rng() % std::min<uint32_t>(hi, near) : lo + rng() % (hi - lo))]
          .emplace_back(g0 + g, k);
    }
    types += " " + std::to_string(t);
  }
  for (uint32_t o = 0; o < n_po; ++o)
    sinks[element(n_pi + n_gates - 1 - rng() % std::min(n_gates, po_near))].emplace_back(n_pi + o, 1);
  std::string text;
  uint32_t n_wires = 0;
  for (uint32_t e = 0; e < sinks.size(); ++e) {
    if (sinks[e].empty()) continue;
    ++n_wires;
    text += std::to_string(e) + " 0 " + std::to_string(sinks[e].size());
    for (auto& s : sinks[e]) text += " " + std::to_string(s.first) + " " + std::to_string(s.second);
    text += "\n";
  }
  text = std::to_string(n_pi) + " " + std::to_string(n_po) + " " + std::to_string(n_gates) + " " +
         std::to_string(n_wires) + "\n" + text + types + "\n";
  Netlist nl;
  parse_ckt(text.data(), text.size(), nl);
  // Every output and pin fault, twice: the plan's sweeps cover stems and exact faults.
  std::vector<Fault> faults;
  for (uint32_t e = 0; e < nl.N; ++e)
    for (uint32_t pin = 0; pin <= nl.fanin_count(e); ++pin)
      for (uint8_t v = 0; v < 2; ++v) faults.push_back(Fault{e, (uint8_t)pin, v});
  Plan P;
  build_plan(nl, faults, P);
  Words good(nl.N);
  for (uint32_t e = 0; e < nl.N; ++e) good[e] = nl.type[e] == G_PI ? rng() : eval(nl, e, good);
  uint64_t compared = 0;
  for (uint32_t G : {2u, 4u, 8u, 16u}) {
    Schedule S;
    build_schedule(nl, P, G, S);
    const uint32_t T = 32 * (1 + rng() % 4);
    pack_schedule(S, T);
    if (S.blob.size() != (S.stream_recs + (size_t)kPrefetch * T) * S.rec_words() + 8 * (S.wides.size() + S.fixes.size()) || S.stream_recs % T)
      return std::fprintf(stderr, "stream size\n"), 1;
    if (S.max_live < P.net_live) return std::fprintf(stderr, "fewer slots than live values\n"), 1;
    if (n_gates > 1000 && !S.split) return std::fprintf(stderr, "levels are not split: %zu records, %u levels\n", S.recs.size(), nl.n_levels), 1;
    for (size_t si = rng() % (1 + n_gates / 300); si < P.sweeps.size(); si += 1 + n_gates / 300) {
      const InjRec& s = P.sweeps[si];
      // the whole netlist with the injection
      const bool stuck = s.mode & kInjStuck;
      const uint64_t sv = s.mode & kInjValue ? ~0ull : 0ull;
      const uint32_t pin = s.mode >> kInjPinShift;
      Words bad(nl.N);
      for (uint32_t e = 0; e < nl.N; ++e) {
        bad[e] = nl.type[e] == G_PI ? good[e] : eval(nl, e, bad);
        if (e != s.elem) continue;
        if (!stuck) {
          bad[e] = ~good[e];
        } else if (pin == 0) {
          bad[e] = sv;
        } else {
          uint64_t in[4] = {0, 0, 0, 0};
          for (uint32_t k = 0; k < nl.fanin_count(e); ++k) in[k] = k + 1 == pin ? sv : bad[nl.fi_idx[nl.fi_off[e] + k]];
          bad[e] = gate(nl.type[e], in, nl.fanin_count(e));
        }
      }
      uint64_t want = 0;
      for (uint32_t e = (uint32_t)(nl.N - nl.n_po); e < nl.N; ++e) want |= bad[e] ^ good[e];
      if (nl.type[s.elem] == G_PO) want = bad[s.elem] ^ good[s.elem];
      if (run_schedule(nl, P, S, good, s, bad[s.stored], false) != want ||
          run_schedule(nl, P, S, good, s, bad[s.stored], true) != want)
        return std::fprintf(stderr, "G %u, sweep of element %u (stored %u): differs\n", G, s.elem, s.stored), 1;
      ++compared;
    }
  }
  // an element that no PO is reached from has no sweep; flipping it changes none
  for (uint32_t e = 0; e < nl.N; ++e) {
    if (P.net.live[e]) continue;
    Words bad(good);
    bad[e] = ~good[e];
    for (uint32_t k = e + 1; k < nl.N; ++k) bad[k] = nl.type[k] == G_PI ? good[k] : eval(nl, k, bad);
    for (uint32_t k = (uint32_t)(nl.N - nl.n_po); k < nl.N; ++k)
      if (bad[k] != good[k]) return std::fprintf(stderr, "element %u reaches a PO\n", e), 1;
  }
  std::printf("%llu %zu %zu %zu\n", (unsigned long long)compared, P.net.clusters.size(), P.net.fixes.size(),
              (size_t)n_gates);
  return 0;
}
