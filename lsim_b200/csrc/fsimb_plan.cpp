// Netlist + fault list -> device plan (see fsimb_plan.h).
#include "fsimb_plan.h"

#include <algorithm>
#include <array>

namespace fsimb {

namespace {

// Inputs an element's evaluation reads: INV, CLKBUF and PO use their first
// input only (fsim/simulation.cpp:979-983, 1062-1067, 1074-1077).
uint32_t eff_fanin(const Netlist& nl, uint32_t e) {
  uint32_t nf = nl.fanin_count(e);
  const uint8_t t = nl.type[e];
  if (t == G_INV || t == G_CLKBUF || t == G_PO) nf = std::min<uint32_t>(nf, 1);
  return nf;
}

}  // namespace

uint32_t gate_family(uint8_t t) {
  switch (t) {
    case G_XOR:
    case G_XNOR: return 1;
    case G_MUX: return 2;
    default: return 0;
  }
}

namespace {

constexpr uint32_t kInvLit = 0x80000000u;

// A cluster while clusters are formed, over netlist elements.
struct Form {
  uint32_t lit[3];
  uint8_t n, is_xor, inv, pad;
};

inline void add_literal(Form& c, uint32_t lit) {
  if (c.is_xor) {  // its inversion turns the output
    c.inv ^= (uint8_t)(lit >> 31);
    lit &= ~kInvLit;
  }
  c.lit[c.n++] = lit;
}

// Adds the literals of `t`, inverted by `inv`, to cluster c.  False if the
// result is not one AND or XOR of three literals.
bool add_term(Form& c, const Form& t, uint32_t inv) {
  const uint32_t tinv = t.inv ^ inv;
  if (c.n + t.n > 3) return false;
  if (t.n == 1) {  // a literal (its inversion is in the literal)
    add_literal(c, t.lit[0] ^ (tinv ? kInvLit : 0u));
    return true;
  }
  if (t.is_xor != c.is_xor || (!c.is_xor && tinv)) return false;
  for (uint32_t k = 0; k < t.n; ++k) c.lit[c.n++] = t.lit[k];
  if (c.is_xor) c.inv ^= (uint8_t)tinv;
  return true;
}

}  // namespace

static void build_gate_recs(const Netlist& nl, std::vector<GateRec>& gates) {
  gates.resize(nl.N);
  for (uint32_t e = 0; e < nl.N; ++e) {
    const uint32_t nf = std::min<uint32_t>(eff_fanin(nl, e), 4);
    for (uint32_t k = 0; k < 4; ++k)
      gates[e][k] = (k < nf ? nl.fi_idx[nl.fi_off[e] + k] : kNoInput) | (nl.type[e] >> k & 1u) << 31;
  }
}

void build_sweep_net(const Netlist& nl, const Plan& P, NetForm net_form, SweepNet& net) {
  const uint32_t N = nl.N;
  const bool fold = net_form != kNetPlain;
  // A PO is reached: the element is a PO, or a live element reads it.
  net.live.assign(N, 0);
  for (int64_t e = (int64_t)N - 1; e >= 0; --e) {
    if (nl.type[e] == G_PO) net.live[e] = 1;
    if (!net.live[e]) continue;
    const uint32_t nf = eff_fanin(nl, (uint32_t)e);
    for (uint32_t k = 0; k < nf; ++k) net.live[nl.fi_idx[nl.fi_off[e] + k]] = 1;
  }
  const uint32_t g1 = P.n_pi + P.n_gates;
  // PO drivers that no gate's record reads.
  net.direct.assign(N, 0);
  for (uint32_t e = P.n_pi; e < g1 && net_form != kNetFolded; ++e) {
    if (!P.po_drv[e]) continue;
    bool read = false;
    for (uint32_t k = nl.fo_off[e]; k < nl.fo_off[e + 1] && !read; ++k) {
      const uint32_t c = nl.fo_idx[k];
      read = nl.type[c] != G_PO && net.live[c] && nl.fo_pin[k] < eff_fanin(nl, c);
    }
    net.direct[e] = !read;
  }
  // Clusters of the gates that have one, bottom up.
  std::vector<Form> form(N, Form{});  // n == 0: no cluster form
  net.lev_up = nl.level;
  for (uint32_t e = P.n_pi; e < g1; ++e) {
    const uint32_t nf = eff_fanin(nl, e);
    const uint8_t t = nl.type[e];
    if (!net.live[e] || net.direct[e] || t == G_MUX || nf < 1 || nf > 3) continue;
    const uint32_t ii = nf > 1 && (t == G_OR || t == G_NOR);
    const bool inverts = t == G_INV || t == G_NAND || t == G_NOR || t == G_XNOR;
    const uint32_t io = inverts != (bool)ii;  // OR and NOR are ANDs of inverted inputs
    const uint32_t* in = &nl.fi_idx[nl.fi_off[e]];
    const Form empty{{0, 0, 0}, 0, (uint8_t)(gate_family(t) == 1 && nf > 1), (uint8_t)io, 0};
    uint32_t may = 0;  // inputs that can be folded in
    for (uint32_t k = 0; k < nf; ++k)
      if (fold && form[in[k]].n && nl.fo_off[in[k] + 1] - nl.fo_off[in[k]] == 1) may |= 1u << k;
    // The subset of them that folds the most gates; of those one with the
    // fewest literals.
    Form best = empty;
    int best_score = -1;
    uint32_t best_set = 0;
    for (uint32_t set = may; set; set = (set - 1) & may) {
      Form c = empty;
      bool ok = true;
      if (nf == 1) {  // BUF / INV of a folded gate: that gate's form
        c = form[in[0]];
        c.inv ^= (uint8_t)io;
      } else {
        for (uint32_t k = 0; k < nf && ok; ++k) {
          if ((set >> k) & 1u)
            ok = add_term(c, form[in[k]], ii);
          else if ((ok = c.n < 3))
            add_literal(c, in[k] | ii << 31);
        }
      }
      const int score = __builtin_popcount(set) * 4 + 3 - c.n;
      if (ok && score > best_score) {
        best = c;
        best_score = score;
        best_set = set;
      }
    }
    if (!best_set)
      for (uint32_t k = 0; k < nf; ++k) add_literal(best, in[k] | ii << 31);
    if (best.n == 1 && best.inv) {  // one literal takes the inversion
      best.lit[0] ^= kInvLit;
      best.inv = 0;
    }
    form[e] = best;
    for (uint32_t k = 0; k < nf; ++k)
      if ((best_set >> k) & 1u) net.lev_up[in[k]] = kFolded | e;
  }
  // Aliases: one literal, not folded away, and read by clusters only (every
  // record a reader is folded into is a cluster's).
  net.alias.assign(N, kNoSlot);
  net.alias_of.assign(N, kNoSlot);
  for (uint32_t e = P.n_pi; e < g1 && fold; ++e) {
    if (form[e].n != 1 || (net.lev_up[e] & kFolded)) continue;
    bool clusters_only = true;
    for (uint32_t k = nl.fo_off[e]; k < nl.fo_off[e + 1] && clusters_only; ++k) {
      const uint32_t c = nl.fo_idx[k];
      clusters_only = form[c].n || !net.live[c] || nl.fo_pin[k] >= eff_fanin(nl, c);
    }
    if (!clusters_only) continue;
    const uint32_t x = form[e].lit[0] & ~kInvLit, src = net.alias[x];
    net.alias[e] = (src == kNoSlot ? x : src) ^ (form[e].lit[0] & kInvLit);
    net.alias_of[e] = x;
  }
  // Records of the live elements that are neither folded away nor aliases.
  net.cluster.assign(N, kNoSlot);
  net.use_level.assign(N, 0);
  net.fix_first.assign(N, kNoSlot);
  std::vector<std::pair<uint32_t, uint32_t>> via;  // (alias, element whose record reads it), once each
  std::vector<uint32_t> last_via(N, kNoSlot);
  net.clusters.reserve(P.n_gates);
  for (uint32_t e = P.n_pi; e < g1; ++e) {
    if (!net.live[e] || (net.lev_up[e] & kFolded) || net.alias[e] != kNoSlot) continue;
    const uint32_t L = nl.level[e];
    auto read = [&](uint32_t x) { net.use_level[x] = std::max(net.use_level[x], L); };
    if (P.po_drv[e] && !net.direct[e]) net.use_level[e] = L + 1;  // its PO record
    const Form& f = form[e];
    if (f.n) {
      net.cluster[e] = (uint32_t)net.clusters.size();
      net.clusters.push_back(Cluster{{f.lit[0], f.lit[1], f.lit[2]}, {0, 0, 0}, f.n, f.is_xor, f.inv});
      Cluster& c = net.clusters.back();
      for (uint32_t k = 0; k < c.n; ++k) {
        const uint32_t x = c.lit[k] & ~kInvLit;
        c.via[k] = x;
        if (net.alias[x] != kNoSlot) {
          c.lit[k] = net.alias[x] ^ (c.lit[k] & kInvLit);
          if (c.is_xor) {  // the alias's inversion goes to the output
            c.inv ^= (uint8_t)(c.lit[k] >> 31);
            c.lit[k] &= ~kInvLit;
          }
          for (uint32_t y = x; net.alias[y] != kNoSlot; y = net.alias_of[y])
            if (last_via[y] != e) {
              last_via[y] = e;
              via.emplace_back(y, e);
            }
        }
        read(c.lit[k] & ~kInvLit);
      }
    } else {
      const uint32_t nf = std::min<uint32_t>(eff_fanin(nl, e), 4);
      for (uint32_t k = 0; k < nf; ++k) read(nl.fi_idx[nl.fi_off[e] + k]);
    }
  }
  net.level_recs.assign(nl.n_levels, 0);
  for (uint32_t e = P.n_pi; e < g1; ++e)
    if (net.live[e] && !(net.lev_up[e] & kFolded) && net.alias[e] == kNoSlot) net.level_recs[nl.level[e]]++;
  for (uint32_t e = 0; e < g1; ++e)
    if (P.po_drv[e] && net.use_level[e]) net.level_recs[nl.level[e] + 1]++;
  // Fix lists: by alias, elements ascending and so by level.
  std::vector<uint32_t> count(N, 0);
  for (const auto& v : via) ++count[v.first];
  uint32_t at = 0;
  for (uint32_t e = 0; e < N; ++e)
    if (count[e]) {
      net.fix_first[e] = at;
      at += count[e] + 1;
    }
  net.fixes.assign(at, kNoSlot);
  for (const auto& v : via) net.fixes[net.fix_first[v.first]++] = v.second;
  for (uint32_t e = 0; e < N; ++e)
    if (count[e]) net.fix_first[e] -= count[e];
}

void build_circuit_plan(const Netlist& nl, CircuitPlan& C, bool sweeps) {
  C = CircuitPlan();
  Plan& P = C.base;
  const uint32_t N = nl.N;
  P.N = N;
  P.n_pi = (uint32_t)nl.n_pi;
  P.n_gates = (uint32_t)nl.n_gates;
  P.n_po = (uint32_t)nl.n_po;
  P.n_levels = nl.n_levels;
  P.level_off = nl.level_off;
  const uint32_t po_begin = P.n_pi + P.n_gates;
  P.max_gate_level = P.n_gates ? nl.level[po_begin - 1] : 0;
  for (uint32_t l = 0; l < nl.n_levels; ++l)
    P.max_level_width = std::max<uint32_t>(P.max_level_width, nl.level_off[l + 1] - nl.level_off[l]);

  build_gate_recs(nl, P.net.gates);
  if (!sweeps) return;

  // Per-element fanout facts.
  C.mux_below.assign(N, 0);
  P.po_drv.assign(N, 0);
  P.gate_fo.assign(N, 0);
  std::vector<uint32_t> maxfo_level(N, 0);  // highest non-PO consumer level (0 if none)
  for (uint32_t e = 0; e < N; ++e) {
    for (uint32_t k = nl.fo_off[e]; k < nl.fo_off[e + 1]; ++k) {
      uint32_t c = nl.fo_idx[k];
      if (nl.type[c] == G_PO) {
        P.po_drv[e] = 1;
      } else {
        P.gate_fo[e] = 1;
        maxfo_level[e] = std::max(maxfo_level[e], nl.level[c]);
      }
    }
    P.has_mux |= nl.type[e] == G_MUX;
  }
  for (int64_t e = (int64_t)N - 1; e >= 0; --e) {
    uint8_t hb = 0;
    for (uint32_t k = nl.fo_off[e]; k < nl.fo_off[e + 1]; ++k) {
      uint32_t c = nl.fo_idx[k];
      hb |= (nl.type[c] == G_MUX) | C.mux_below[c];
    }
    C.mux_below[e] = hb;
  }

  // What sweeps evaluate, and the peak number of live values (interval graph
  // of [level, highest reading level]), over all gates and over the stored
  // ones; a schedule may need a few more slots to honour residues.
  {
    auto peak = [&](const std::vector<uint32_t>& last) {
      std::vector<int64_t> delta(nl.n_levels + 2, 0);
      for (uint32_t e = 0; e < N; ++e)
        if (last[e]) {
          delta[nl.level[e]]++;
          delta[last[e] + 1]--;
        }
      int64_t live = 0, most = 0;
      for (uint32_t l = 0; l < nl.n_levels; ++l) most = std::max(most, live += delta[l]);
      return (uint32_t)most;
    };
    P.max_live = peak(maxfo_level);
    for (NetForm f : {kNetFolded, kNetDirectPos, kNetPlain}) {
      build_sweep_net(nl, P, f, P.net);
      P.net_live = peak(P.net.use_level);
      if (P.net_live + !P.net.fixes.empty() <= std::max(P.max_live, kAnyShapeSlots)) break;
    }
  }

  // FFR roots: an element with exactly one consumer belongs to the FFR of that
  // consumer; the members of each FFR, element-descending (consumer first).
  C.root.resize(N);
  for (int64_t e = (int64_t)N - 1; e >= 0; --e) {
    uint32_t fo = nl.fo_off[e + 1] - nl.fo_off[e];
    if (nl.type[e] == G_PO || fo != 1)
      C.root[e] = (uint32_t)e;
    else
      C.root[e] = C.root[nl.fo_idx[nl.fo_off[e]]];
  }
  C.ffr_off.assign(N + 1, 0);
  for (uint32_t e = 0; e < N; ++e)
    if (C.root[e] != e) C.ffr_off[C.root[e] + 1]++;
  for (uint32_t r = 0; r < N; ++r) C.ffr_off[r + 1] += C.ffr_off[r];
  C.ffr_mem.resize(C.ffr_off[N]);
  C.ffr_local.assign(N, 0);
  {
    std::vector<uint32_t> fill(C.ffr_off.begin(), C.ffr_off.end() - 1);
    for (int64_t e = (int64_t)N - 1; e >= 0; --e) {
      const uint32_t r = C.root[e];
      if (r == (uint32_t)e) continue;
      const uint32_t k = nl.fo_off[e];
      C.ffr_local[e] = fill[r] - C.ffr_off[r];
      C.ffr_mem[fill[r]++] = MemberRec{(uint32_t)e, nl.fo_idx[k], nl.fo_pin[k], 0};
    }
  }

  // Algorithmic bytes of one gate-word evaluation: its fanin words read and
  // its output word written, 8 * (fanin + 1).  A sweep evaluates the gates
  // that feed a gate or a PO; gates that feed nothing cannot change a PO.
  P.nfp_prefix.assign(N + 1, 0);
  P.eval_prefix.assign(N + 1, 0);
  for (uint32_t e = 0; e < N; ++e) {
    const bool ev = e >= P.n_pi && (P.gate_fo[e] || P.po_drv[e]);
    const uint32_t nf = ev ? eff_fanin(nl, e) : 0;
    P.nfp_prefix[e + 1] = P.nfp_prefix[e] + (ev ? 8ull * (nf + 1) : 0);
    P.eval_prefix[e + 1] = P.eval_prefix[e] + (ev ? 1 : 0);
  }
}

void build_fault_plan(const Netlist& nl, const CircuitPlan& C, const std::vector<Fault>& faults,
                      Plan& P) {
  const Plan& B = C.base;
  P = Plan();
  P.N = B.N;
  P.n_pi = B.n_pi;
  P.n_gates = B.n_gates;
  P.n_po = B.n_po;
  P.n_levels = B.n_levels;
  P.level_off = B.level_off;
  P.max_gate_level = B.max_gate_level;
  P.max_level_width = B.max_level_width;
  P.max_live = B.max_live;
  P.net_live = B.net_live;
  P.has_mux = B.has_mux;
  auto reaches_po = [&](uint32_t x) {
    return (nl.type[x] == G_PO || B.po_drv[x]) ? kInjReachesPo : 0u;
  };
  auto stored = [&](uint32_t x) {
    while (B.net.lev_up[x] & kFolded) x = B.net.lev_up[x] & ~kFolded;
    return x;
  };
  auto inject = [&](uint32_t x, uint32_t v, uint32_t mode) {
    const uint32_t a = B.net.alias[v];
    const uint32_t L = nl.level[v] + 1;
    if (a == kNoSlot) return InjRec{x, v, mode, 0, L, {0, 0, 0}};
    return InjRec{x, v, mode | ((a & kInvLit) ? kInjAliasInv : 0u), B.net.fix_first[v] + 1, L, {0, 0, 0}};
  };
  auto is_exact = [&](const Fault& ft) {
    return ft.pin == 0 ? (bool)C.mux_below[ft.site]
                       : (nl.type[ft.site] == G_MUX || C.mux_below[ft.site]);
  };

  // Traced faults grouped by FFR root (fault order within a root), roots in
  // topological order so neighbouring warps touch neighbouring data.
  std::vector<std::pair<uint32_t, uint32_t>> rf;  // (root, fault)
  rf.reserve(faults.size());
  for (uint32_t f = 0; f < faults.size(); ++f)
    if (!is_exact(faults[f])) rf.emplace_back(C.root[faults[f].site], f);
  std::stable_sort(rf.begin(), rf.end(),
                   [](const std::pair<uint32_t, uint32_t>& a, const std::pair<uint32_t, uint32_t>& b) {
                     return a.first < b.first;
                   });
  for (size_t i = 0; i < rf.size();) {
    const uint32_t r = rf[i].first;
    RootRec rr{};
    rr.root = r;
    if (nl.type[r] == G_PO || B.po_drv[r])
      rr.obs = kObsOne;
    else if (!B.net.live[r])
      rr.obs = kObsZero;
    else {
      rr.obs = (uint32_t)P.sweeps.size();
      P.sweeps.push_back(inject(r, r, reaches_po(r)));
      P.sweep_root.push_back((uint32_t)P.roots.size());
    }
    rr.mem_begin = (uint32_t)P.members.size();
    // a member's slot is its index in members; its consumer is the root
    // (patched below, once the number of members is known) or a member of
    // the same FFR listed before it
    for (uint32_t k = C.ffr_off[r]; k < C.ffr_off[r + 1]; ++k) {
      MemberRec m = C.ffr_mem[k];
      m.p_slot = m.p == r ? kNoSlot : rr.mem_begin + C.ffr_local[m.p];
      P.members.push_back(m);
    }
    rr.mem_end = (uint32_t)P.members.size();
    rr.flt_begin = (uint32_t)P.traced.size();
    for (; i < rf.size() && rf[i].first == r; ++i) {
      const Fault& ft = faults[rf[i].second];
      P.traced.push_back(TracedRec{rf[i].second, ft.site, ft.pin, ft.value});
      P.traced_slot.push_back(ft.site == r ? kNoSlot : rr.mem_begin + C.ffr_local[ft.site]);
    }
    rr.flt_end = (uint32_t)P.traced.size();
    P.roots.push_back(rr);
  }
  // root slots follow the members
  const uint32_t n_mem = (uint32_t)P.members.size();
  for (uint32_t ri = 0; ri < P.roots.size(); ++ri) {
    RootRec& rr = P.roots[ri];
    rr.slot = n_mem + ri;
    for (uint32_t k = rr.mem_begin; k < rr.mem_end; ++k)
      if (P.members[k].p_slot == kNoSlot) P.members[k].p_slot = rr.slot;
    for (uint32_t k = rr.flt_begin; k < rr.flt_end; ++k)
      if (P.traced_slot[k] == kNoSlot) P.traced_slot[k] = rr.slot;
  }
  P.n_stem_sweeps = (uint32_t)P.sweeps.size();
  for (uint32_t f = 0; f < faults.size(); ++f) {
    const Fault& ft = faults[f];
    if (!is_exact(ft)) continue;
    const uint32_t v = stored(ft.site);
    P.sweeps.push_back(inject(ft.site, v,
                              kInjStuck | reaches_po(v) | (ft.value ? kInjValue : 0u) |
                                  ((uint32_t)ft.pin << kInjPinShift)));
    P.exact_fault.push_back(f);
  }

  const uint32_t gates_end = nl.level_off[std::min(P.max_gate_level + 1, nl.n_levels)];
  for (auto& s : P.sweeps) {
    uint32_t L0 = nl.level[s.stored] + 1;
    if (L0 <= P.max_gate_level) {
      P.dense_sweep_gates += B.eval_prefix[gates_end] - B.eval_prefix[nl.level_off[L0]];
      P.dense_sweep_bytes += B.nfp_prefix[gates_end] - B.nfp_prefix[nl.level_off[L0]];
    }
  }
}

void build_plan(const Netlist& nl, const std::vector<Fault>& faults, Plan& P) {
  CircuitPlan C;
  build_circuit_plan(nl, C, !faults.empty());
  build_fault_plan(nl, C, faults, P);
  P.net = std::move(C.base.net);
  P.gate_fo = std::move(C.base.gate_fo);
  P.po_drv = std::move(C.base.po_drv);
  P.nfp_prefix = std::move(C.base.nfp_prefix);
  P.eval_prefix = std::move(C.base.eval_prefix);
}

// ---------------------------------------------------------------- schedule
namespace {

// Slots by residue mod G, in blocks of one of each residue; at `cap` slots a
// free one of another residue is taken instead of a new block.
struct SlotPool {
  uint32_t G, cap;
  uint32_t n = 0;  // slots so far
  std::vector<std::vector<uint32_t>> free;  // per residue
  SlotPool(uint32_t g, uint32_t most) : G(g), cap(most), free(g) {}
  uint32_t alloc(uint32_t r) {
    if (free[r].empty())
      for (uint32_t q = 0; q < G && n < cap; ++q, ++n) free[n % G].push_back(n);
    for (uint32_t q = 0; q < G && free[r].empty(); ++q) r = (r + 1) % G;
    if (free[r].empty()) {  // more live values than the cap
      r = n % G;
      free[r].push_back(n++);
    }
    uint32_t s = free[r].back();
    free[r].pop_back();
    return s;
  }
  void release(uint32_t s) { free[s % G].push_back(s); }
};

}  // namespace

void build_schedule(const Netlist& nl, const Plan& P, uint32_t G, Schedule& S) {
  S = Schedule();
  S.G = G;
  const uint32_t N = nl.N;
  const SweepNet& net = P.net;
  S.rec_off.assign(nl.n_levels + 1, 0);
  S.li_off.assign(nl.n_levels + 1, 0);
  if (net.use_level.empty()) return;  // no fault will be simulated: no sweeps
  std::vector<uint32_t> slot(N, kNoSlot);
  const uint32_t inj_slots = net.fixes.empty() ? 0 : 1;
  SlotPool pool(G, P.slot_cap(G) - inj_slots);
  std::vector<std::vector<uint32_t>> release(nl.n_levels + 2);
  // PIs: residues round robin.
  uint32_t rr = 0;
  for (uint32_t e = nl.level_off[0]; e < nl.level_off[1]; ++e) {
    if (!net.use_level[e]) continue;
    slot[e] = pool.alloc(rr++ % G);
    release[net.use_level[e] + 1].push_back(slot[e]);
  }
  // A record's literals, and its kind.
  auto has_record = [&](uint32_t e) {
    return net.live[e] && !(net.lev_up[e] & kFolded) && net.alias[e] == kNoSlot;
  };
  uint64_t n_recs = 0, n_lev = 0;
  for (uint32_t n : net.level_recs) {
    n_recs += n;
    n_lev += n > 0;
  }
  // Levels with fewer records than kSplitRecords on average are not ordered
  // by kind: a warp would run several bodies on most of its rounds, so there
  // the sweep runs one body for all ANDs and XORs.
  S.split = n_recs >= kSplitRecords * n_lev;
  auto order_key = [&](uint32_t kind) { return S.split || kind >= kRecMux ? kind : (uint32_t)kRecAnd2; };
  struct Rec {
    uint32_t e, kind, n;
    uint32_t lit[4], via[4];
    uint8_t res[4];   // slot residues
    bool taken;
  };
  auto rec_of = [&](uint32_t e) {
    Rec r{};
    r.e = e;
    if (net.cluster[e] != kNoSlot) {
      const Cluster& c = net.clusters[net.cluster[e]];
      r.n = std::max<uint32_t>(c.n, 2);
      r.kind = (c.is_xor ? kRecXor2 : kRecAnd2) + r.n - 2;
      for (uint32_t k = 0; k < r.n; ++k) {
        r.lit[k] = c.lit[k % c.n];
        r.via[k] = c.via[k % c.n];
      }
    } else {
      r.n = std::min<uint32_t>(eff_fanin(nl, e), 4);
      r.kind = net.direct[e] ? kRecPo : nl.type[e] == G_MUX && r.n == 3 ? kRecMux : kRecWide;
      for (uint32_t k = 0; k < r.n; ++k) r.lit[k] = nl.fi_idx[nl.fi_off[e] + k];
    }
    for (uint32_t k = 0; k < r.n; ++k) r.res[k] = (uint8_t)(slot[r.lit[k] & ~kInvLit] % G);
    return r;
  };
  auto po_rec = [&](uint32_t e) {
    Rec r{};
    r.e = e;
    r.kind = kRecPo;
    r.n = 1;
    r.lit[0] = e;
    r.res[0] = (uint8_t)(slot[e] % G);
    return r;
  };
  // Permutations of 1 to 4 literals; the order of a MUX's is fixed.
  std::vector<std::array<uint8_t, 4>> perms[5];
  for (uint32_t n = 1; n <= 4; ++n) {
    std::array<uint8_t, 4> a{0, 1, 2, 3};
    do perms[n].push_back(a);
    while (std::next_permutation(a.begin(), a.begin() + n));
  }
  // Orders a level's records in groups of G consecutive positions.  Each
  // member is the candidate (with its best literal order) adding the fewest
  // repeated residues per literal position to the group, none if possible,
  // among the next 256 of the first one's kind; a group that runs out of a
  // kind's candidates goes on with the next kind's.
  std::vector<Rec> recs, order;
  auto make_groups = [&] {
    order.clear();
    size_t first = 0, left = recs.size();
    while (left > 0) {
      uint32_t used[4] = {0, 0, 0, 0};
      for (size_t n_grp = 0; n_grp < G && left > 0; ++n_grp) {
        while (recs[first].taken) ++first;
        size_t best = first, scanned = 0;
        int best_cost = 1 << 30;
        const std::array<uint8_t, 4>* best_perm = &perms[1][0];
        for (size_t c = first; c < recs.size() && scanned < 256 &&
                               order_key(recs[c].kind) == order_key(recs[first].kind); ++c) {
          const Rec& r = recs[c];
          if (r.taken) continue;
          ++scanned;
          for (const auto& q : perms[r.n]) {
            int cost = 0;
            for (uint32_t k = 0; k < r.n; ++k) cost += (used[k] >> r.res[q[k]]) & 1u;
            if (cost < best_cost) {
              best_cost = cost;
              best = c;
              best_perm = &q;
            }
            if (best_cost == 0 || r.kind >= kRecMux) break;
          }
          if (best_cost == 0) break;
        }
        Rec& b = recs[best];
        b.taken = true;
        --left;
        Rec o = b;
        for (uint32_t k = 0; k < b.n; ++k) {
          o.lit[k] = b.lit[(*best_perm)[k]];
          o.via[k] = b.via[(*best_perm)[k]];
          used[k] |= 1u << b.res[(*best_perm)[k]];
        }
        order.push_back(o);
      }
    }
  };
  // A slot at bit 14 * (k & 1) of word k / 2, its high bits in word 2 + k / 2.
  auto put_slot = [](std::array<uint32_t, 4>& w, uint32_t k, uint32_t sl) {
    const uint32_t sh = 14 * (k & 1u);
    w[k / 2] = (w[k / 2] & ~(kRecSlot << sh)) | (sl & kRecSlot) << sh;
    w[2 + k / 2] = (w[2 + k / 2] & ~(kRecSlot << sh)) | (sl >> 14) << sh;
  };
  std::vector<std::array<uint32_t, 4>> fix_rec(net.fixes.empty() ? 0 : N);  // per element: record index, via
  std::vector<std::array<uint32_t, 5>> pos_slot;
  for (uint32_t L = 1; L <= P.max_gate_level + 1 && L < nl.n_levels; ++L) {
    for (uint32_t s : release[L]) pool.release(s);
    recs.clear();
    for (uint32_t e = nl.level_off[L]; e < nl.level_off[L + 1] && nl.type[e] != G_PO; ++e)
      if (has_record(e)) recs.push_back(rec_of(e));
    for (uint32_t e = nl.level_off[L - 1]; e < nl.level_off[L]; ++e)
      if (P.po_drv[e] && slot[e] != kNoSlot) recs.push_back(po_rec(e));
    std::stable_sort(recs.begin(), recs.end(), [&](const Rec& a, const Rec& b) { return order_key(a.kind) > order_key(b.kind); });
    make_groups();
    // Output slots (residue = position mod G) and records.
    S.rec_off[L] = (uint32_t)S.recs.size();
    pos_slot.assign(order.size(), std::array<uint32_t, 5>{kNoSlot, kNoSlot, kNoSlot, kNoSlot, kNoSlot});
    for (uint32_t pos = 0; pos < order.size(); ++pos) {
      const Rec& r = order[pos];
      const uint32_t e = r.e;
      for (uint32_t k = 0; k < r.n; ++k) pos_slot[pos][k] = slot[r.lit[k] & ~kInvLit];
      if (r.kind == kRecPo && !net.direct[e]) {
        std::array<uint32_t, 4> w{0, (uint32_t)kRecPo << kRecKindShift, 0, 0};
        put_slot(w, 3, slot[e]);
        w[0] = e;
        S.recs.push_back(w);
        continue;
      }
      uint32_t out = e;
      if (!net.direct[e]) {
        out = slot[e] = pool.alloc(pos % G);  // every such record is read
        release[net.use_level[e] + 1].push_back(out);
        pos_slot[pos][4] = out;
      }
      if (r.kind == kRecWide || r.kind == kRecPo) {
        std::array<uint32_t, 8> d{0, 0, 0, 0, out, (uint32_t)nl.type[e] | r.n << 4, 0, 0};
        for (uint32_t k = 0; k < r.n; ++k) d[k] = pos_slot[pos][k];
        S.recs.push_back({(uint32_t)S.wides.size() | (net.direct[e] ? kPoDirect : 0u), r.kind << kRecKindShift, 0, 0});
        S.wides.push_back(d);
        S.direct |= r.kind == kRecPo;
        continue;
      }
      std::array<uint32_t, 4> w{0, r.kind << kRecKindShift, 0, 0};
      for (uint32_t k = 0; k < r.n; ++k) {
        put_slot(w, k, pos_slot[pos][k]);
        w[0] |= (r.lit[k] >> 31) << (31 - k);
      }
      put_slot(w, 3, out);
      if (r.kind == kRecAnd2) w[0] |= 1u << 29;  // an absent literal reads as inverted zeros
      if (r.kind != kRecMux) w[0] |= (uint32_t)net.clusters[net.cluster[e]].inv << 28;
      if (!fix_rec.empty()) fix_rec[e] = {(uint32_t)S.recs.size(), r.via[0], r.via[1], r.via[2]};
      S.recs.push_back(w);
    }
    // Bank-conflict accounting per aligned group of G positions.
    for (uint32_t g0 = 0; g0 < order.size(); g0 += G) {
      const uint32_t g_end = std::min<uint32_t>(g0 + G, (uint32_t)order.size());
      for (uint32_t k = 0; k < 5; ++k) {
        uint32_t seen = 0, any = 0;
        bool conflict = false;
        for (uint32_t o = g0; o < g_end; ++o) {
          const uint32_t sl = pos_slot[o][k];
          if (sl == kNoSlot) continue;
          any = 1;
          conflict |= (seen >> (sl % G)) & 1u;
          seen |= 1u << (sl % G);
        }
        S.access_groups += any;
        S.conflict_groups += conflict;
      }
    }
  }
  for (uint32_t L = std::min(P.max_gate_level + 2, nl.n_levels); L <= nl.n_levels; ++L)
    S.rec_off[L] = (uint32_t)S.recs.size();
  S.max_live = pool.n + inj_slots;
  if (S.max_live > max_slots(G)) {
    S.recs.clear();
    S.wides.clear();
    S.rec_off.assign(nl.n_levels + 1, 0);
    return;
  }
  // Fix entries: the record of a reader of alias y, with the literals that
  // name y, or an alias of y, on the injection slot.
  S.fixes.resize(net.fixes.size(), std::array<uint32_t, 4>{0, 0, 0, 0});
  S.fix_level.assign(net.fixes.size(), kNoSlot);
  for (uint32_t y = 0; y < N && !net.fixes.empty(); ++y) {
    if (net.fix_first[y] == kNoSlot) continue;
    for (uint32_t i = net.fix_first[y]; net.fixes[i] != kNoSlot; ++i) {
      const auto& fr = fix_rec[net.fixes[i]];
      std::array<uint32_t, 4> w = S.recs[fr[0]];
      const uint32_t n = std::max<uint32_t>(net.clusters[net.cluster[net.fixes[i]]].n, 2);
      for (uint32_t k = 0; k < n; ++k) {
        uint32_t x = fr[1 + k];
        while (x != y && net.alias[x] != kNoSlot) x = net.alias_of[x];
        if (x == y) put_slot(w, k, S.max_live - 1);
      }
      S.fixes[i] = w;
      S.fix_level[i] = nl.level[net.fixes[i]];
    }
  }
  // Live-in sets as (element, slot) pairs.
  std::vector<uint32_t> cnt(nl.n_levels + 2, 0);
  for (uint32_t e = 0; e < N; ++e)
    if (slot[e] != kNoSlot)
      for (uint32_t l = nl.level[e] + 1; l <= net.use_level[e]; ++l) cnt[l]++;
  for (uint32_t l = 0; l < nl.n_levels; ++l) S.li_off[l + 1] = S.li_off[l] + cnt[l];
  S.li.assign(2ull * S.li_off[nl.n_levels], 0);
  std::vector<uint32_t> fill(S.li_off.begin(), S.li_off.end() - 1);
  for (uint32_t e = 0; e < N; ++e)
    if (slot[e] != kNoSlot)
      for (uint32_t l = nl.level[e] + 1; l <= net.use_level[e]; ++l) {
        const uint32_t i = fill[l]++;
        S.li[2 * i] = e;
        S.li[2 * i + 1] = slot[e];
      }
}

void pack_schedule(Schedule& S, uint32_t T) {
  if (S.T == T) return;
  if (S.max_live > max_slots(S.G))
    throw LimitError{"a sweep needs " + std::to_string(S.max_live) + " live values; a schedule of this word count holds " +
                     std::to_string(max_slots(S.G))};
  S.T = T;
  S.blob.clear();
  const uint32_t n_levels = (uint32_t)S.rec_off.size() - 1, nw = S.rec_words();
  S.lvl.assign(n_levels + 1, std::array<uint32_t, 4>{0, 0, 0, 0});
  // Lane l of a shared-memory phase (8 lanes; 16 at one word per item, where
  // a phase is one group) takes position (l % C) * G + l / C of the phase's
  // groups, C = 16-byte chunks per slot: with chunk (l % C) ^ i at step i the
  // phase's chunks lie in different banks wherever the group's slots do.
  const uint32_t C = 8 / S.G ? 8 / S.G : 1, ph = S.G == 16 ? 16 : 8;
  uint32_t n = 0;  // records so far
  std::vector<uint32_t> wide_at;
  for (uint32_t L = 0; L < n_levels; ++L) {
    S.lvl[L] = {n, S.li_off[L], S.li_off[L + 1], 0};
    const uint32_t lo = S.rec_off[L], n_lev = S.rec_off[L + 1] - lo;
    const uint32_t rounds = (n_lev + T - 1) / T;
    S.blob.resize((size_t)(n + rounds * T) * nw, 0);
    for (uint32_t i = 0; i < rounds * T; ++i) {
      const uint32_t l = i % ph;
      const uint32_t pos = i - l + (S.G == 16 ? l : (l % C) * S.G + l / C);
      uint32_t* w = &S.blob[(size_t)(n + i) * nw];
      if (pos < n_lev) {
        std::copy_n(S.recs[lo + pos].begin(), nw, w);
        const uint32_t kind = (w[1] >> kRecKindShift) & 7u;
        if (kind == kRecWide || (kind == kRecPo && (w[0] & kPoDirect))) wide_at.push_back(n + i);
      }
      if (i >= (rounds - 1) * T) w[1] |= kRecEnd;
    }
    n += rounds * T;
  }
  S.lvl[n_levels][0] = S.stream_recs = n;
  S.blob.resize((size_t)(n + kPrefetch * T) * nw, 0);
  const uint32_t wide0 = (uint32_t)(S.blob.size() / 4);
  for (uint32_t i : wide_at) {
    uint32_t& w = S.blob[(size_t)i * nw];
    w = (w & kPoDirect) | (wide0 + 2 * (w & ~kPoDirect));
  }
  for (const auto& d : S.wides) S.blob.insert(S.blob.end(), d.begin(), d.end());
  S.fix0 = (uint32_t)(S.blob.size() / 4);
  for (size_t i = 0; i < S.fixes.size(); ++i) {
    uint32_t at = kNoSlot, same = 0;
    if (S.fix_level[i] != kNoSlot) {
      at = S.lvl[S.fix_level[i] + 1][0] - T;
      while (S.fix_level[i + same] == S.fix_level[i]) ++same;  // a list ends with kNoSlot
    }
    S.blob.insert(S.blob.end(), S.fixes[i].begin(), S.fixes[i].end());
    S.blob.insert(S.blob.end(), {at, same, 0u, 0u});
  }
}

}  // namespace fsimb
