// Host-side compilation of a netlist + fault list into the device data layout
// used by the B200 kernels.
//
// Layout in HBM (all arrays indexed by the reference's topological index):
//   type[N]            u8 gate type
//   gates[N]           inputs and type of each gate in one record (GateRec)
//   fi_off[N+1], fi_idx[E]   fanin CSR in pin order (good-machine kernel)
//   blob[]             the sweep's record stream, 8 bytes a record, level
//                      after level in order of evaluation.  A record is a
//                      cluster: a gate together with single-consumer gates
//                      folded into it, an AND or XOR of up to three literals
//                      in all.  The inner values are never stored, because a
//                      sweep flips multi-consumer elements only.  MUX gates
//                      have records of their own kind; gates of four inputs
//                      ("wide" records) are described in 32 bytes each
//                      behind the stream.  A PO driver's value is compared
//                      with the good one by a record one level above it, or,
//                      where the kept values would need more slots than the
//                      gates alone, by a PO record that evaluates it.
//                      Elements from which no PO is reached are left out.
//                      A level is padded to rounds of T records, T the sweep
//                      CTA's threads: thread t of round r reads record
//                      r * T + t, and the last round of a level carries
//                      kRecEnd, so a sweep needs no other table of levels.
//                      Within a level the order is by kind, and every
//                      group of G consecutive positions has pairwise
//                      different slot residues mod G for each literal and
//                      for the output wherever the host found such groups,
//                      so the group's shared-memory accesses hit distinct
//                      banks
//   lvl[L]             of a sweep that starts at level L: record offset in the
//                      stream of its first round, and its range in li
//   level[e]           level of a stored element; kFolded | consumer for an
//                      element folded into its consumer's cluster
//   li[]               (element, slot) pairs live when a sweep starts at
//                      level L (read from the good values at start)
//   good[tile][N][32]  u64 good-machine words, 32 words (2048 patterns) per tile
//
// Fault handling:
//   * fanout-free regions (FFRs): every element with exactly one consumer
//     belongs to the FFR of that consumer; all others are FFR roots;
//   * faults whose downstream logic is bitwise (no MUX) are "traced": their
//     detection word is  sens(line -> root) & (good(line) ^ stuck) & obs(root)
//     where sens is computed by backward critical-path tracing inside the
//     FFR and obs(root) by one sweep per root that flips the root's value;
//   * faults with a MUX downstream are "exact": one sweep per fault with the
//     stuck value injected, since the reference's MUX uses a word-level
//     logical not (fsim/simulation.cpp:1056) that is not bitwise.
#pragma once

#include <array>
#include <cstdint>
#include <string>
#include <vector>

#include "fsimb_netlist.h"

namespace fsimb {

// Thrown where a size is beyond what the code can hold; FSIMB_ERR_LIMIT at
// the C ABI.
struct LimitError {
  std::string msg;
};

constexpr uint32_t kTileWords = 32;  // words per tile = lanes of a warp
constexpr uint32_t kNoSlot = 0xFFFFFFFFu;
// Slots a schedule may have: the documented limit, at one word per item more
// than shared memory holds; the width of a record's slot field at more.
constexpr uint32_t kMaxSlots = 32767;
constexpr uint32_t max_slots(uint32_t G) { return G == 16 ? kMaxSlots : 1u << 14; }

constexpr uint32_t kFolded = 0x80000000u;  // level[]: the element is folded; low bits: its consumer

// A record is two 32-bit words.  Word 0: slots of literals 0 and 1 in bits
// 0-13 and 14-27; word 1: slots of literal 2 and of the output.  The top four
// bits of word 0 are inversions (literals 0, 1, 2 from bit 31 down, then the
// output's), those of word 1 the end-of-level bit and the kind.  At one word
// per item, where up to 28,000 slots fit shared memory, a record is four
// words, one slot each in bits 0-13 and 14-27 (low and high half): word 2 the
// high halves of literals 0 and 1, word 3 those of literal 2 and the output.
// A cluster of one literal is the AND of it with itself.  A MUX record has
// its three inputs in pin order.  A wide record's word 0 is the offset of its
// description from the stream's start, in 16-byte units.  A PO record has the
// driver's slot in the output's place and the driver in word 0.
enum RecKind : uint32_t {
  kRecNop = 0,  // padding
  kRecAnd2, kRecAnd3, kRecXor2, kRecXor3,
  kRecMux,
  kRecWide,
  kRecPo
};
constexpr int kRecKindShift = 28;  // word 1, three bits
constexpr uint32_t kRecEnd = 1u << 31;  // word 1: the last round of the level
constexpr uint32_t kRecSlot = 0x3FFFu;
// A wide record's description, eight words: slots of up to four inputs, of
// the output, and type | fan-in << 4.  A direct PO record has kPoDirect and
// the offset of such a description in word 0, the description the driver in
// the output's place: the record evaluates the driver and compares it.
constexpr uint32_t kPoDirect = 1u << 31;

// InjRec::mode bit fields
constexpr uint32_t kInjStuck = 1u;      // 0: flip the element's word, 1: stuck value
constexpr uint32_t kInjReachesPo = 2u;  // the stored element is, or drives, a PO
constexpr uint32_t kInjValue = 4u;      // the stuck value
constexpr uint32_t kInjAliasInv = 8u;   // the stored element is an inverting alias
constexpr int kInjPinShift = 4;         // exact faults: 0 output, k input; flips: 0

// Observability source of an FFR root.
constexpr uint32_t kObsZero = 0xFFFFFFFEu;  // root reaches no PO
constexpr uint32_t kObsOne = 0xFFFFFFFFu;   // root is / drives a PO

struct RootRec {
  uint32_t root;
  uint32_t obs;        // sweep index, kObsZero or kObsOne
  uint32_t mem_begin;  // into members
  uint32_t mem_end;
  uint32_t flt_begin;  // into traced faults
  uint32_t flt_end;
  uint32_t slot;       // compact sensitivity slot of the root: members.size() + root index
  uint32_t pad;
};

struct MemberRec {  // internal FFR element e, its consumer p and pin position
  uint32_t e;
  uint32_t p;
  uint32_t pin;
  uint32_t p_slot;  // compact sensitivity slot of p (a member's slot is its index in members)
};

struct TracedRec {  // one traced fault
  uint32_t fault;   // index into the caller's fault list
  uint32_t elem;    // output fault: the element; pin fault: the gate
  uint32_t pin;     // 0 = output, k = k-th input
  uint32_t value;   // 0 / 1
};

struct InjRec {     // sweep injection: flip (stem) or stuck (exact fault)
  uint32_t elem;
  uint32_t stored;  // the stored element whose word the sweep replaces: elem, or the
                    // element whose cluster it is folded into
  uint32_t mode;    // kInjStuck | kInjReachesPo | kInjValue | kInjAliasInv | pin << kInjPinShift
  uint32_t fix;     // stored is an alias: its first fix entry + 1; else 0
  uint32_t level;   // the sweep's first level: one above stored
  uint32_t pad[3];
};

// What a sweep evaluates and stores (independent of the fault list).
struct Cluster {
  uint32_t lit[3];  // stored element | inversion << 31
  uint32_t via[3];  // the element the literal names in the netlist: the same, or an alias of it
  uint8_t n;        // literals
  uint8_t is_xor;
  uint8_t inv;      // the output inverted
};
// A gate for the good machine, one 16-byte load: its inputs' indices, the
// bits of the type in the top bits (bit k of the type in word k); an input
// it does not have, or does not read, is kNoInput.
using GateRec = std::array<uint32_t, 4>;
constexpr uint32_t kNoInput = 0x7FFFFFFFu;

struct SweepNet {
  std::vector<GateRec> gates;       // [N]
  std::vector<uint32_t> lev_up;     // [N] level, or kFolded | consumer
  std::vector<uint32_t> use_level;  // [N] highest level of a record that reads it (0: none, no slot)
  std::vector<uint32_t> cluster;    // [N] index into clusters; kNoSlot: no cluster record
  // BUF and INV gates that only clusters read have no record and no slot:
  // their readers take the source's slot, inverted or not.  A sweep that
  // injects at such an alias runs the level as it is and then evaluates the
  // records that read it again, on an extra slot with the faulty value.
  std::vector<uint32_t> alias;      // [N] stored source | inversion << 31; kNoSlot: not an alias
  std::vector<uint32_t> alias_of;   // [N] an alias's direct source, maybe an alias itself
  std::vector<uint32_t> fix_first;  // [N] an alias's first entry in fixes; kNoSlot: none
  std::vector<uint32_t> fixes;      // per alias, by level: elements whose records read it, then kNoSlot
  std::vector<uint8_t> live;        // [N] a PO is reached from it
  std::vector<uint8_t> direct;      // [N] a PO driver compared by its own record: no slot
  std::vector<Cluster> clusters;
  std::vector<uint32_t> level_recs; // [n_levels] records a sweep evaluates on each level
};

// Forms of a sweep net, in the order they are tried.  What a circuit may ask
// of shared memory is stated by its gates' live values (Plan::max_live), but
// folding a gate keeps its inputs alive instead, and a PO driver that no gate
// reads lives to the next level.  So a net that would keep more values than
// the gates alone (and than kAnyShapeSlots) gives such PO drivers direct
// records, and if that is not enough folds nothing and has no aliases, which
// keeps at most the gates' live values.  Generated circuits of 400 to 200,000
// gates keep 10 to 25 % less than their gates; 40,000 PO drivers on a level
// kept 40,500 values against 927, and 930 slots with direct records.
enum NetForm { kNetFolded, kNetDirectPos, kNetPlain };
// Slots that every launch shape has room for (8 words an item, 8 CTAs an SM:
// 431): below this, fewer slots allow nothing more.
constexpr uint32_t kAnyShapeSlots = 384;

struct Plan {
  uint32_t N = 0, n_pi = 0, n_gates = 0, n_po = 0;
  uint32_t n_levels = 0;
  uint32_t max_gate_level = 0;       // highest level holding a non-PO element
  // Peak of live gate outputs, every gate counted: the documented limit of
  // the shared-memory sweep and of explicit shapes.
  uint32_t max_live = 0;
  uint32_t net_live = 0;             // peak of stored values: slots needed without residue constraints
  uint32_t max_level_width = 0;
  uint64_t dense_sweep_gates = 0;    // sum over sweeps of gates evaluated
  uint64_t dense_sweep_bytes = 0;    // sum over sweeps of 8*(fanin+1) per evaluated gate, per word
  // [N+1] prefix sums of 8*(effective fanin+1) over the elements a sweep
  // evaluates (gates that feed a gate or a PO)
  std::vector<uint64_t> nfp_prefix;
  std::vector<uint32_t> eval_prefix; // [N+1] prefix counts of those elements
  std::vector<uint32_t> level_off;   // [n_levels+1]
  SweepNet net;
  std::vector<uint8_t> gate_fo;      // [N] has a non-PO consumer
  std::vector<uint8_t> po_drv;       // [N] drives a PO
  // traced faults
  std::vector<RootRec> roots;
  std::vector<MemberRec> members;
  std::vector<TracedRec> traced;
  std::vector<uint32_t> traced_slot;  // compact sensitivity slot of each traced fault's element
  // sweeps: first n_stem_sweeps are root flips, the rest exact faults
  std::vector<InjRec> sweeps;
  uint32_t n_stem_sweeps = 0;
  std::vector<uint32_t> exact_fault;  // fault index of each exact sweep
  std::vector<uint32_t> sweep_root;   // root record of each stem sweep
  bool has_mux = false;
  // The most slots a schedule of residue groups of G has: the gates' live
  // values, rounded up to whole groups.
  uint32_t slot_cap(uint32_t G) const {
    const uint32_t n = max_live > kAnyShapeSlots ? max_live : kAnyShapeSlots;
    return (n + G - 1) / G * G;
  }
};

// The fault-independent part of a plan, built once per circuit: `base` holds
// the circuit fields of Plan (sizes, levels, fanout facts, live-value peak,
// byte prefix sums; no roots or sweeps), plus what classifying a fault list
// needs: MUX-below flags, the FFR root of every element and the members of
// every FFR (element-descending, consumer first).
struct CircuitPlan {
  Plan base;
  std::vector<uint8_t> mux_below;   // [N] some consumer path reaches a MUX
  std::vector<uint32_t> root;       // [N] FFR root
  std::vector<uint32_t> ffr_off;    // [N+1] members of the FFR rooted at r
  std::vector<MemberRec> ffr_mem;
  std::vector<uint32_t> ffr_local;  // [N] position of a member within its FFR's list
};

// Evaluation order and shared-memory slots for one residue group size G
// (16 / words per item), and the record stream packed for a CTA size.
struct Schedule {
  uint32_t G = 0;
  uint32_t max_live = 0;             // slots, the injection slot among them
  bool split = false;                // levels are ordered by kind
  bool direct = false;               // it has direct PO records
  std::vector<std::array<uint32_t, 4>> recs;  // records in position order, level after level
                                     // (a wide one's word 0: its index in wides)
  std::vector<std::array<uint32_t, 8>> wides;
  std::vector<uint32_t> rec_off;     // [n_levels+1] first record of each level
  std::vector<uint32_t> li_off;      // [n_levels+1] first pair of each level in li
  std::vector<uint32_t> li;          // pairs (element, slot)
  std::vector<std::array<uint32_t, 4>> fixes;  // per net.fixes entry: its record, reading the
                                     // injection slot (the last one) in the alias's place
  std::vector<uint32_t> fix_level;   // level of each entry; kNoSlot ends a list
  uint64_t conflict_groups = 0;      // group accesses whose slots repeat a residue
  uint64_t access_groups = 0;        // group accesses (fanin loads + stores)
  // pack_schedule
  uint32_t T = 0;                    // CTA threads the stream is packed for
  uint32_t stream_recs = 0;          // records of all rounds
  uint32_t fix0 = 0;                 // offset of the fix entries in blob, 16-byte units
  // The rounds (rec_words() words a record), kPrefetch rounds of padding, the
  // wide descriptions, and eight words per fix entry: the record (four
  // words), then stream offset of its level's last round and entries of the
  // list on that level; ~0 ends a list.
  std::vector<uint32_t> blob;
  uint32_t rec_words() const { return G == 16 ? 4 : 2; }
  std::vector<std::array<uint32_t, 4>> lvl;  // [n_levels+1] first record, li begin, li end, 0
  uint64_t bytes() const { return blob.size() * 4 + lvl.size() * 16 + li.size() * 4; }
};
constexpr uint32_t kPrefetch = 3;  // rounds a sweep reads ahead at most
constexpr uint64_t kSplitRecords = 256;  // records a level from which ANDs and XORs have kinds of their own

// 0: AND family (AND, NAND, OR, NOR, INV, CLKBUF, PO), 1: XOR family, 2: MUX.
uint32_t gate_family(uint8_t type);
void build_plan(const Netlist& nl, const std::vector<Fault>& faults, Plan& plan);
// Without `sweeps` (no fault will be simulated) it holds the sizes, the
// levels and the gate records only: what the good machine reads (200,000 gates:
// 13 ms with the fanout facts and FFRs, 2 without).
void build_circuit_plan(const Netlist& nl, CircuitPlan& cplan, bool sweeps = true);
// Roots, members, traced faults and sweeps of a fault list; the circuit's
// per-element vectors (net, gate_fo, po_drv, nfp_prefix) stay in
// cplan.base and are left empty in `plan`.  Costs O(faults log faults +
// members of the FFRs the faults touch).
void build_fault_plan(const Netlist& nl, const CircuitPlan& cplan, const std::vector<Fault>& faults,
                      Plan& plan);
// Folds single-consumer gates into their consumers, as `form` has it
// (net.gates is left as it is).
void build_sweep_net(const Netlist& nl, const Plan& plan, NetForm form, SweepNet& net);
// G in {2, 4, 8, 16}.  A schedule that needs more than max_slots(G) slots
// reports its max_live and holds no records, fix entries or live-in pairs.
void build_schedule(const Netlist& nl, const Plan& plan, uint32_t G, Schedule& out);
// Packs the schedule's records into the stream of a T-thread CTA (T a
// multiple of 32); nothing to do if it is packed for T already.  LimitError
// for a schedule of more than max_slots(G) slots.
void pack_schedule(Schedule& s, uint32_t T);

}  // namespace fsimb
