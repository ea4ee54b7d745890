// Device kernels of the B200 stuck-at fault simulator.  All arithmetic is
// bitwise on 64-bit words (64 patterns per word); no tensor cores are
// involved because gate evaluation is not a contraction.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "fsimb_plan.h"

namespace fsimb {

struct GoodView {
  const uint4* gates;         // GateRec per element
  const uint32_t* level_off;  // [n_levels + 1]
  const uint64_t* pwords;     // [W][n_pi]
  uint64_t* good;             // [tiles][N][32]; words at and beyond W are left as they are
  uint32_t n_pi, N, n_levels;
  uint32_t W;
};

struct SweepArgs {
  const uint4* blob;       // record stream for the launch's CTA size (see fsimb_plan.h)
  const uint4* lvl;        // per level: its first record in the stream, its range in li
  const uint32_t* level;   // element -> level, or kFolded | consumer
  const uint32_t* li;      // (element, slot) pairs
  const uint32_t* fi_off;
  const uint32_t* fi_idx;
  const uint8_t* type;
  const InjRec* inj;
  const uint32_t* list;    // sweep indices to run (nullptr: 0..n_list-1)
  uint32_t n_list;
  uint32_t n_tiles, n_sweeps;
  uint32_t n_words;        // pattern words of the last tile (1..32): the others are not swept
  uint32_t max_gate_level;
  uint32_t N;
  const uint64_t* good;    // first tile: [n_tiles][N][32]
  uint64_t* out;           // [n_tiles][n_sweeps][32] OR of PO differences
  int* queue;              // work counter for this launch
  uint32_t stream_recs;    // records of the stream's rounds
  uint32_t fix0, inj_slot; // fix entries in blob; the injection slot
  uint32_t split;          // levels are ordered by record kind
  int* err;                // set to 1 if a bounded wait gave up
  uint64_t wait_ns;        // time limit of that wait
  uint32_t wait_test;      // 1: the first CTA waits on a barrier nothing completes (test hook)
};

// Sweep of circuits whose live values do not fit in shared memory.
struct SweepWideArgs {
  const uint32_t* level;     // element -> level
  const uint32_t* level_off; // element offsets per level
  const uint32_t* fi_off;
  const uint32_t* fi_idx;
  const uint8_t* type;
  const uint8_t* eflag;      // bit 0: evaluated in sweeps, bit 1: drives a PO
  const InjRec* inj;
  const uint32_t* list;      // sweep indices to run (nullptr: 0..n_list-1)
  uint32_t n_list;
  uint32_t n_words;          // pattern words of this tile (1..32)
  uint32_t max_gate_level;
  uint32_t N;
  const uint64_t* good;      // this tile: [N][32]
  uint64_t* out;             // this tile: [n_sweeps][32]
  int* queue;
  uint64_t* gvals;           // [blocks][N][M] values of each CTA's item
};

struct FfrArgs {
  const RootRec* roots;
  const uint32_t* list;    // root indices to process (nullptr: all)
  uint32_t n_list;
  const MemberRec* members;
  const TracedRec* traced;
  const uint32_t* traced_slot;
  const uint32_t* fi_off;
  const uint32_t* fi_idx;
  const uint8_t* type;
  const uint64_t* good;    // first tile: [n_tiles][N][32]
  const uint64_t* obs;     // [n_tiles][n_sweeps][32]
  uint64_t* sens;          // scratch [n_tiles][n_slots][32]: members, then roots
  uint32_t N, n_sweeps, n_slots;
  uint32_t n_tiles;
  uint32_t tile, W;        // first tile
  uint64_t P;
  int drop;                // skip faults whose count reached n_detect in an earlier tile
  uint32_t n_detect;       // >= 1
  unsigned long long* count;
  unsigned long long* first;
  uint8_t* lastflag;
};

struct ExactArgs {
  const uint32_t* exact_fault;
  const uint32_t* list;    // exact indices to process (nullptr: all)
  uint32_t n_exact;
  uint32_t first_sweep;    // index of the first exact sweep
  const uint64_t* out;     // [n_tiles][n_sweeps][32]
  uint32_t n_sweeps, n_tiles;
  uint32_t tile, W;        // first tile
  uint64_t P;
  int drop;
  uint32_t n_detect;
  unsigned long long* count;
  unsigned long long* first;
  uint8_t* lastflag;
};

struct ResultArgs {
  const unsigned long long* count;
  const unsigned long long* first;
  const uint8_t* lastflag;
  const int* err;
  ulonglong2* out;           // [F] records of two, then the error word
  unsigned long long last_rd;
  uint32_t F, any_rounds;    // 0: no pattern rounds
};

// Threads [0, n_in_pad) handle roots, the rest exact faults.
struct DropArgs {
  const RootRec* roots;
  const uint32_t* in_list;   // current live roots (nullptr: all)
  uint32_t n_in, n_in_pad;
  const TracedRec* traced;
  const uint32_t* exact_fault;
  const uint32_t* exact_in;  // current live exact indices (nullptr: all)
  uint32_t n_exact_in;
  uint32_t first_exact_sweep;
  const unsigned long long* count;
  uint32_t n_detect;         // a fault survives while its count is below this
  uint32_t* out_roots;       // surviving root indices
  uint32_t* out_sweeps;      // sweeps still needed (stem flips and exact faults)
  uint32_t* out_exact;       // surviving exact indices
  uint32_t* n_out;           // [3]: roots, sweeps, exact
};

// ---------------------------------------------------------------- batches
// One circuit of a batch: device pointers into the batch's concatenated
// arrays and the circuit's sizes.
struct BatchCirc {
  const uint4* blob;
  const uint4* lvl;
  const uint32_t* level;
  const uint32_t* level_off;
  const uint4* gates;
  const uint32_t* li;
  const uint32_t* fi_off;
  const uint32_t* fi_idx;
  const uint8_t* type;
  const InjRec* inj;
  const RootRec* roots;
  const MemberRec* members;
  const TracedRec* traced;
  const uint32_t* traced_slot;
  const uint32_t* exact_fault;
  const uint64_t* pwords;        // [W][n_pi]
  uint64_t* good;                // [tiles][N][32]
  uint64_t* out;                 // [tiles][n_sweeps][32]
  uint64_t* sens;                // [tiles][n_slots][32]: members, then roots
  unsigned long long* count;     // per fault
  unsigned long long* first;
  uint8_t* lastflag;
  uint64_t P;
  uint32_t N, n_pi, W, tiles;
  uint32_t n_sweeps, n_stem_sweeps, n_roots, n_exact;
  uint32_t max_gate_level, n_levels;
  uint32_t n_slots;              // sensitivity slots per tile
  uint32_t stream_recs, fix0, inj_slot, split;  // see SweepArgs
};

// What the batched sweep reads of one circuit.  A launch carries these in
// its parameters, so the compiler sees them as warp-uniform values.
struct SweepCirc {
  const uint4* blob;
  const uint4* lvl;
  const uint32_t* level;
  const uint32_t* li;
  const uint32_t* fi_off;
  const uint32_t* fi_idx;
  const uint8_t* type;
  const InjRec* inj;
  const uint64_t* good;  // [tiles][N][32]
  uint64_t* out;         // [tiles][n_sweeps][32]
  uint32_t N, n_sweeps, max_gate_level;
  uint32_t n_items;      // (tile, sweep, subtile), tile-major: n_sweeps * (32 / M) per tile,
                         // n_sweeps * last_sub for the last one
  uint32_t tiles, last_sub, stream_recs, fix0, inj_slot, split;
};

constexpr int kSweepCircsPerLaunch = 240;

struct BatchSweepParams {
  SweepCirc c[kSweepCircsPerLaunch];
  unsigned long long* queue;  // [n_circ] work counters, zero before the launch
  uint32_t n_circ;
};
static_assert(sizeof(BatchSweepParams) <= 32000, "kernel parameters are limited to 32,764 bytes");

constexpr int kGoodBatchWords = 4;  // words per CTA of the batched good machine

// Units of the batched kernels: one warp per (circuit, tile, root) or
// (circuit, tile, exact fault), one CTA per (circuit, words); prefix over
// circuits.
struct BatchUnits {
  const BatchCirc* circs;
  const unsigned long long* unit_prefix;  // [n_circ + 1]
  uint32_t n_circ;
};

void launch_good_batch(const BatchUnits& u, unsigned long long n_units, cudaStream_t s);
cudaError_t launch_sweep_batch(int M, bool direct, int threads, int blocks, size_t smem, const BatchSweepParams& p,
                               cudaStream_t s);
// Lets launches take up to `smem` bytes of dynamic shared memory.  The limit
// is the kernel's, shared by all threads and handles: every caller sets the
// largest CTA's, so that none lowers it between another's setting and launch.
cudaError_t sweep_batch_set_smem(int M, bool direct, size_t smem);
cudaError_t sweep_batch_occupancy(int M, bool direct, int threads, size_t smem, int* blocks_per_sm);
void launch_ffr_batch(const BatchUnits& u, unsigned long long n_units, cudaStream_t s);
void launch_exact_batch(const BatchUnits& u, unsigned long long n_units, cudaStream_t s);
void launch_init_results_batch(unsigned long long* count, unsigned long long* first, uint8_t* lastflag,
                               uint64_t F, cudaStream_t s);

// The good machine of all words; level_off is the host's copy.  Returns the
// kernels launched.
uint32_t launch_good(const GoodView& a, const uint32_t* level_off, int n_sms, cudaStream_t s);
// direct: the schedule (any of the launch's) has direct PO records.  Returns
// cudaErrorInvalidValue when M is unsupported.
cudaError_t launch_sweep(int M, bool direct, int threads, int blocks, size_t smem, const SweepArgs& a,
                         cudaStream_t s);
cudaError_t sweep_set_smem(int M, bool direct, size_t smem);  // as sweep_batch_set_smem
cudaError_t sweep_occupancy(int M, bool direct, int threads, size_t smem, int* blocks_per_sm);
// M in {1, 2}; threads a multiple of 32, at most 1,024.
cudaError_t launch_sweep_wide(int M, int threads, int blocks, const SweepWideArgs& a, cudaStream_t s);
cudaError_t sweep_wide_occupancy(int M, int threads, int* blocks_per_sm);
// Time limit of the wait test's wait.
constexpr uint64_t kWaitTestNs = 20000000ull;
void launch_ffr(const FfrArgs& a, cudaStream_t s);
void launch_exact(const ExactArgs& a, cudaStream_t s);
// Also zeroes n_zero control words.
void launch_init_results(unsigned long long* count, unsigned long long* first, uint8_t* lastflag,
                         uint32_t F, int* zero, uint32_t n_zero, cudaStream_t s);
void launch_results(const ResultArgs& a, cudaStream_t s);
// good: the round's word of element 0 in its tile.
void launch_round(const uint64_t* good, uint32_t N, uint64_t mask, uint64_t* out, cudaStream_t s);
void launch_drop(const DropArgs& a, cudaStream_t s);

}  // namespace fsimb
