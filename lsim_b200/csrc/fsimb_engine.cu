// Handle, device memory and run orchestration behind the C ABI (include/fsimb.h).
//
// One run:
//   1. upload the compiled plan (once per circuit + fault list) and patterns;
//   2. good machine for all words (launch_good);
//   3. per group of 2,048-pattern tiles: stem / exact sweeps (k_sweep<M>), FFR
//      tracing and per-fault accumulation (k_ffr, k_exact); in drop mode a
//      group is one tile, followed by the compaction of what is still
//      undetected (k_drop);
//   4. per-fault records back to the host (k_results).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <functional>
#include <cstdio>
#include <cstddef>
#include <cstring>
#include <fstream>
#include <mutex>
#include <new>
#include <sstream>
#include <string>
#include <vector>

#include "../../include/fsimb.h"
#include "fsimb_gen.h"
#include "fsimb_internal.h"
#include "fsimb_kernels.cuh"
#include "fsimb_netlist.h"
#include "fsimb_plan.h"

using namespace fsimb;

namespace fsimb {
uint64_t next_generation() {
  static std::atomic<uint64_t> g{0};
  return ++g;
}
}  // namespace fsimb

namespace {

thread_local std::string g_create_error;

std::string read_file(const char* path) {
  std::ifstream f(path, std::ios::binary);
  if (!f) throw IoError{std::string("cannot open ") + path};
  std::ostringstream ss;
  ss << f.rdbuf();
  return ss.str();
}

}  // namespace

// --------------------------------------------------------------------------
static int m_slot(int M) { return M == 1 ? 0 : M == 2 ? 1 : M == 4 ? 2 : 3; }

Schedule& fsimb_handle::cached_schedule(int M) {
  const int sl = m_slot(M);
  if (sched_cache_gen[sl] != plan_gen) {
    build_schedule(nl, plan, 16u / (uint32_t)M, sched_cache[sl]);
    sched_cache_gen[sl] = plan_gen;
  }
  return sched_cache[sl];
}

const Schedule& fsimb_handle::use_schedule(int M, int T, cudaStream_t s) {
  Schedule& sc = cached_schedule(M);
  if (sched_M == M && sched_T == T) return sc;
  sched_M = 0;
  pack_schedule(sc, (uint32_t)T);
  upload(d_recs, sc.blob, s);
  upload(d_lvl, sc.lvl, s);
  upload(d_li, sc.li, s);
  sched_M = M;
  sched_T = T;
  return sc;
}

namespace fsimb {

// A model of one SM's time per pattern word.  A level of a CTA's sweep takes
// a latency (barrier, record, operands, store) of kLevel cycles plus kRound
// for each further round, and the shared-memory and issue time of all the
// SM's CTAs: a number of cycles by M for a warp's records, kPad for a warp of
// padding.  A CTA alone on its SM has nothing to fill its barriers with: a
// fifth more.  Fitted to shape sweeps on a B200; best of the nine cheapest
// against the model's choice: 2,000 gates 0.113 / 0.113 ms, 6,586 gates 2.25 /
// 2.25, 20,000 gates with MUX 8.14 / 8.04, 30,000 gates 2.84 / 2.84, 60,000
// gates 6.12 / 6.12; two CTAs of 512 threads and 4 words against one of 1,024
// and 8: 50,000 gates 52.7 / 54.6 ms, 100,000 gates 11.8 / 12.3, 200,000 gates
// 342 / 344.
double sweep_shape_cost(const SweepNet& net, int m, uint32_t t, size_t vals, size_t smem_per_sm, uint32_t words) {
  constexpr double kLevel = 1100, kRound = 300, kPad = 4;
  const uint32_t w = std::max<uint32_t>(1, std::min<uint32_t>(words, kTileWords));
  const double warp = m == 8 ? 61 : m == 4 ? 30 : m == 2 ? 18 : 15;
  const uint32_t ctas = (uint32_t)std::min<size_t>({smem_per_sm / (vals + 1024 + 256), 1024 / t, 32});
  if (ctas < 1) return 1e300;
  double cycles = 0;
  for (uint32_t n : net.level_recs) {
    if (!n) continue;
    const uint32_t rounds = (n + t - 1) / t, full = (n + 31) / 32, all = rounds * (t / 32);
    cycles += kLevel + kRound * (rounds - 1) + ctas * (full * warp + (all - full) * kPad);
  }
  return (ctas == 1 ? 1.2 : 1.0) * cycles / ctas * ((w + m - 1) / m);
}

std::vector<SweepShape> likely_shapes(const Plan& plan, uint32_t words, size_t smem_optin, size_t smem_per_sm,
                                      size_t most) {
  struct Priced {
    double cost;
    SweepShape s;
  };
  std::vector<Priced> all;
  for (int m : {8, 4, 2, 1}) {
    const size_t vals = sweep_vals_bytes(plan.net_live, m);
    if (plan.net_live > kMaxSlots || vals > sweep_smem_share(smem_optin, smem_per_sm, 1)) continue;
    for (uint32_t t : {32, 64, 96, 128, 192, 256, 320, 384, 448, 512, 640, 768, 1024})
      all.push_back({sweep_shape_cost(plan.net, m, t, vals, smem_per_sm, words), {m, (int)t}});
  }
  std::stable_sort(all.begin(), all.end(), [](const Priced& a, const Priced& b) { return a.cost < b.cost; });
  std::vector<SweepShape> out;
  for (const Priced& p : all)
    if (out.size() < most && p.cost < 1.5 * all[0].cost) out.push_back(p.s);
  return out;
}

bool default_sweep_shape(const Plan& plan, const std::function<const Schedule&(int)>& sched_at,
                         uint32_t words, size_t smem_optin, size_t smem_per_sm, int& M, int& threads) {
  const size_t share1 = sweep_smem_share(smem_optin, smem_per_sm, 1);
  // Slots are about the peak of live values until a schedule says more, and
  // at most the plan's cap.
  size_t vals[4] = {0, 0, 0, 0};
  bool exact[4] = {false, false, false, false};
  for (int i = 0; i < 4; ++i) {
    const uint32_t about = plan.net_live + plan.net_live / 64 + 16;
    vals[i] = sweep_vals_bytes(std::min(about, plan.slot_cap(16u >> i)), 1 << i);
  }
  for (;;) {
    double best = 1e300;
    int bi = -1;
    for (int i = 3; i >= 0; --i) {
      if (vals[i] > share1) continue;
      for (uint32_t t = 32; t <= 1024; t += 32) {
        const double c = sweep_shape_cost(plan.net, 1 << i, t, vals[i], smem_per_sm, words);
        if (c < best * 0.99) {
          best = c;
          bi = i;
          threads = (int)t;
        }
      }
    }
    if (bi < 0 && !exact[0]) bi = 0;  // the estimate may be too high: ask the schedule
    if (bi < 0) return false;
    M = 1 << bi;
    if (exact[bi]) break;
    const Schedule& sc = sched_at(M);
    exact[bi] = true;
    vals[bi] = sched_fits(sc, M, share1) ? sweep_vals_bytes(sc.max_live, M) : share1 + 1;
  }
  return true;
}

}  // namespace fsimb

bool fsimb_handle::default_shape(int& M, int& threads) {
  return default_sweep_shape(
      plan, [&](int m) -> const Schedule& { return cached_schedule(m); },
      (uint32_t)std::min<uint64_t>(pats.W, kTileWords), smem_optin, smem_per_sm, M, threads);
}

GoodView fsimb_handle::good_view(uint32_t W) const {
  return GoodView{d_gates.as<uint4>(), d_level_off.as<uint32_t>(), d_pwords.as<uint64_t>(),
                  d_good.as<uint64_t>(), (uint32_t)nl.n_pi, nl.N, nl.n_levels, W};
}

void fsimb_handle::tune_shape(cudaStream_t s) {
  const uint32_t N = plan.N;
  const uint32_t n_sweeps = (uint32_t)plan.sweeps.size();
  for (auto& e : tune_ev)
    if (!e) CK(cudaEventCreate(&e));
  launch_good(good_view(tile_words(pats.W, 0)), nl.level_off.data(), n_sms, s);  // tile 0
  // every stride-th sweep: at most 1 in 16 and about 4,096 of them, so a
  // candidate's run stays short on large circuits
  const uint32_t stride =
      std::max<uint32_t>(1, std::max<uint32_t>(std::min<uint32_t>(16, n_sweeps / 2048), n_sweeps / 4096));
  std::vector<uint32_t> list;
  for (uint32_t i = 0; i < n_sweeps; i += stride) list.push_back(i);
  upload(d_tune_list, list, s);
  float best_ms = 1e30f;
  int bM = 0, bT = 0;
  // The default shape is the incumbent: a candidate replaces it only when
  // faster by more than 2% on the sample (the sample favours no shape, but
  // its time carries a few percent of noise).
  int dM = 0, dT = 0;
  if (!default_shape(dM, dT)) {
    tuned_M = tuned_T = 0;
    tuned_words = kTileWords;  // of no tile
    tuned_gen = plan_gen;
    return;
  }
  float default_ms = -1;
  std::vector<SweepShape> cands{{dM, dT}};
  for (const SweepShape& c :
       likely_shapes(plan, (uint32_t)std::min<uint64_t>(pats.W, kTileWords), smem_optin, smem_per_sm, 10))
    if (!(c.M == dM && c.threads == dT)) cands.push_back(c);
  const size_t share1 = sweep_smem_share(smem_optin, smem_per_sm, 1);
  for (const SweepShape& cd : cands) {
    const int M = cd.M, T = cd.threads;
    if (!sched_fits(cached_schedule(M), M, share1)) continue;
    const Schedule& sc = use_schedule(M, T, s);
    const size_t smem = std::max<size_t>(16, sweep_vals_bytes(sc.max_live, M));
    CK(sweep_set_smem(M, sc.direct, share1));
    int got = 0;
    CK(sweep_occupancy(M, sc.direct, T, smem, &got));
    if (got < 1) continue;
    SweepArgs sa{};
    sa.blob = d_recs.as<uint4>();
    sa.lvl = d_lvl.as<uint4>();
    sa.level = d_level.as<uint32_t>();
    sa.li = d_li.as<uint32_t>();
    sa.fi_off = d_fi_off.as<uint32_t>();
    sa.fi_idx = d_fi_idx.as<uint32_t>();
    sa.type = d_type.as<uint8_t>();
    sa.inj = d_inj.as<InjRec>();
    sa.list = d_tune_list.as<uint32_t>();
    sa.n_list = (uint32_t)list.size();
    sa.n_tiles = 1;
    sa.n_sweeps = n_sweeps;
    sa.n_words = tile_words(pats.W, 0);
    sa.max_gate_level = plan.max_gate_level;
    sa.N = N;
    sa.good = d_good.as<uint64_t>();
    sa.out = d_out.as<uint64_t>();
    sa.queue = d_queue.as<int>();
    sa.stream_recs = sc.stream_recs;
    sa.fix0 = sc.fix0;
    sa.inj_slot = sc.max_live - 1;
    sa.split = sc.split;
    const int nb = (int)std::min<uint64_t>((uint64_t)n_sms * got, (uint64_t)sa.n_list * ((sa.n_words + M - 1) / M));
    // an untimed run of the first candidate warms the GPU up; then the
    // fastest of two timed runs counts
    float ms = 1e30f;
    for (int rep = (&cd == &cands[0]) ? -1 : 0; rep < 2; ++rep) {
      CK(cudaMemsetAsync(d_queue.p, 0, sizeof(int), s));
      CK(cudaEventRecord(tune_ev[0], s));
      CK(launch_sweep(M, sc.direct, T, nb, smem, sa, s));
      CK(cudaEventRecord(tune_ev[1], s));
      CK(cudaEventSynchronize(tune_ev[1]));
      float x = 0;
      CK(cudaEventElapsedTime(&x, tune_ev[0], tune_ev[1]));
      if (rep >= 0) ms = std::min(ms, x);
    }
    if (default_ms < 0 && M == dM && T == dT) {
      default_ms = ms;
      best_ms = ms;
      bM = M;
      bT = T;
    } else if (ms < (default_ms > 0 && bM == dM && bT == dT ? 0.98f : 1.0f) * best_ms) {
      best_ms = ms;
      bM = M;
      bT = T;
    }
  }
  tuned_M = bM;
  tuned_T = bT;
  tuned_words = tile_words(pats.W, 0);
  tuned_gen = plan_gen;
}

void fsimb_handle::run(const fsimb_opts* opts) {
  if (device < 0) throw CudaError{"host-only handle: no GPU to run on"};
  if (!has_ckt || !has_faults || !has_pats) throw StateError{"load circuit, faults and patterns first"};
  fsimb_opts o{};
  if (opts) {
    // callers built against the layout before n_detect pass a shorter struct
    const size_t min_size = offsetof(fsimb_opts, n_detect);
    if (opts->struct_size != 0 && opts->struct_size < min_size) throw ArgError{"fsimb_opts.struct_size too small"};
    std::memcpy(&o, opts, opts->struct_size ? std::min<size_t>(opts->struct_size, sizeof o) : sizeof o);
  }
  if (o.words_per_item && o.words_per_item != 1 && o.words_per_item != 2 && o.words_per_item != 4 &&
      o.words_per_item != 8)
    throw ArgError{"words_per_item must be 0, 1, 2, 4 or 8"};
  if (o.block_threads && (o.block_threads < 32 || o.block_threads > 1024 || o.block_threads % 32))
    throw ArgError{"block_threads must be 0 or a multiple of 32 in 32..1024"};
  if (o.ctas_per_sm > 8) throw ArgError{"ctas_per_sm must be 0..8"};
  if (o.sweep_variant > 2) throw ArgError{"sweep_variant must be 0, 1 or 2"};
  if (o.sweep_variant == 2 && o.words_per_item > 2)
    throw ArgError{"the global-memory sweep takes 1 or 2 words per item"};
  const uint32_t n_detect = std::max<uint32_t>(o.n_detect, 1);
  CK(cudaSetDevice(device));
  cudaStream_t s = o.stream ? (cudaStream_t)o.stream : stream;
  has_results = false;

  if (!plan_valid) {
    build_plan(nl, faults, plan);
    plan_valid = true;
    plan_uploaded = false;
    sched_M = 0;
  }
  const uint32_t N = plan.N;
  const uint64_t F = faults.size();
  const uint64_t W = pats.W;
  const uint64_t tiles = (W + kTileWords - 1) / kTileWords;
  const uint64_t W_pad = tiles * kTileWords;
  const uint32_t n_sweeps = (uint32_t)plan.sweeps.size();
  const uint32_t n_roots = (uint32_t)plan.roots.size();
  const uint32_t n_exact = (uint32_t)plan.exact_fault.size();
  if (W_pad > (1ull << 31) || tiles * (uint64_t)N * kTileWords > (1ull << 40))
    throw LimitError{"pattern block too large"};

  cudaEvent_t e0 = ev(0), e1 = ev(1), e2 = ev(2), e3 = ev(3);
  CK(cudaEventRecord(e0, s));
  if (!plan_uploaded) {
    upload(d_type, nl.type, s);
    upload(d_fi_off, nl.fi_off, s);
    upload(d_fi_idx, nl.fi_idx, s);
    upload(d_level, plan.net.lev_up, s);
    upload(d_gates, plan.net.gates, s);
    upload(d_level_off, plan.level_off, s);
    upload(d_roots, plan.roots, s);
    upload(d_members, plan.members, s);
    upload(d_traced, plan.traced, s);
    upload(d_traced_slot, plan.traced_slot, s);
    upload(d_inj, plan.sweeps, s);
    upload(d_exact, plan.exact_fault, s);
    eflag_uploaded = false;
    plan_uploaded = true;
  }
  if (!pats_uploaded) {
    upload(d_pwords, pats.words, s);
    pats_uploaded = true;
  }
  CK(cudaEventRecord(upload_ev, s));
  uint64_t launches = 1;  // results init
  d_good.ensure(tiles * N * kTileWords * 8);
  const size_t share1 = sweep_smem_share(smem_optin, smem_per_sm, 1);
  // The documented limit counts every gate's live value (the schedules fold
  // some of them away): levels beyond it keep to the global-memory sweep,
  // and explicit shapes beyond it stay refused.
  auto gates_fit = [&](int m, size_t bytes) {
    return plan.max_live <= kMaxSlots && sweep_vals_bytes(plan.max_live, m) <= bytes;
  };
  // Tiles of one launch: in count mode as many as kTileScratch bytes hold the
  // sweep outputs and sensitivities of (and fewer than 2^31 sweep items), so
  // that a run of few tiles has one sweep launch and one tracing launch and
  // their last CTAs run dry once; drop mode compacts after every tile.
  // 6,586 gates, 5 tiles: 2.36 + 0.14 -> 2.23 + 0.04 ms; 2,000 gates, 2 tiles: 0.132 +
  // 0.044 -> 0.113 + 0.023 ms.  Their room is asked for last, and a device that
  // does not have it runs one tile at a time.
  constexpr uint64_t kTileScratch = 512ull << 20;
  const uint32_t n_slots = (uint32_t)(plan.members.size() + plan.roots.size());
  const uint64_t tile_bytes = ((uint64_t)n_sweeps + n_slots + 1) * kTileWords * 8;
  uint64_t group = 1;
  if (!o.drop && o.sweep_variant != 2 && gates_fit(1, share1) && one_tile_gen != plan_gen) {
    const uint64_t by_items = (1ull << 31) / ((uint64_t)std::max(n_sweeps, 1u) * kTileWords);
    group = std::max<uint64_t>(1, std::min(tiles, std::min(kTileScratch / tile_bytes, by_items)));
  }
  auto scratch = [&](uint64_t n) {
    d_sens.ensure(n * std::max<uint32_t>(n_slots, 1) * kTileWords * 8);
    d_out.ensure(n * std::max<uint32_t>(n_sweeps, 1) * kTileWords * 8);
  };
  d_count.ensure(std::max<uint64_t>(F, 1) * 8);
  d_first.ensure(std::max<uint64_t>(F, 1) * 8);
  d_lastflag.ensure(std::max<uint64_t>(F, 1));
  d_queue.ensure((tiles + 1) * sizeof(int));
  d_records.ensure(F * sizeof(fsimb_fault_result) + 16);
  if (o.drop) {
    d_root_list[0].ensure(std::max<uint32_t>(n_roots, 1) * 4);
    d_root_list[1].ensure(std::max<uint32_t>(n_roots, 1) * 4);
    d_sweep_list.ensure(std::max<uint32_t>(n_sweeps, 1) * 4);
    d_exact_list[0].ensure(std::max<uint32_t>(n_exact, 1) * 4);
    d_exact_list[1].ensure(std::max<uint32_t>(n_exact, 1) * 4);
    d_nout.ensure(16);
  }

  // Sweep shape: explicit options, the autotuned shape of this plan, or the
  // default.  Circuits whose live values do not fit in shared memory take
  // the global-memory sweep.
  double tune_ms_now = 0;
  int M = 0, threads = 0;
  bool wide = o.sweep_variant == 2;
  size_t smem = 0;
  const Schedule* sched = nullptr;
  auto no_room = [&](uint32_t live, int m, size_t bytes, int ctas) {
    return LimitError{"a sweep needs " + std::to_string(live) + " live values; shared memory holds " +
                      std::to_string(bytes / (8 * m)) + " at " + std::to_string(m) + " word(s) per item and " +
                      std::to_string(ctas) + " CTA(s) per SM"};
  };
  if (!wide && n_sweeps && !gates_fit(1, share1)) {
    if (o.sweep_variant == 1) throw no_room(plan.max_live, 1, share1, 1);
    wide = true;
  }
  const bool explicit_shape = o.words_per_item || o.block_threads || o.ctas_per_sm;
  if (!wide && n_sweeps) {
    if (explicit_shape) {
      const int ctas = o.ctas_per_sm ? (int)o.ctas_per_sm : 1;
      const size_t budget = sweep_smem_share(smem_optin, smem_per_sm, ctas);
      M = o.words_per_item ? (int)o.words_per_item : 8;
      for (;; M /= 2) {
        if (gates_fit(M, budget) && sched_fits(cached_schedule(M), M, budget)) break;
        if (o.words_per_item || M == 1)
          throw no_room(std::max(plan.max_live, cached_schedule(M).max_live), M, budget, ctas);
      }
      threads = o.block_threads ? (int)o.block_threads : (int)pick_sweep_threads(cached_schedule(M));
    } else if (o.tune && tiles) {
      if (!tuned_holds()) {
        const auto t0 = std::chrono::steady_clock::now();
        scratch(1);
        tune_shape(s);
        tune_ms_now =
            std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
      }
      M = tuned_M;
      threads = tuned_T;
    } else if (!default_shape(M, threads)) {
      M = 0;
    }
    if (!M) {  // no schedule fits: the global-memory sweep
      if (o.sweep_variant == 1) throw no_room(cached_schedule(1).max_live, 1, share1, 1);
      wide = true;
    }
  }
  int blocks = 0, occ_got = 0;
  if (wide) {
    group = 1;
    M = o.words_per_item == 1 || (!o.words_per_item && W == 1) ? 1 : 2;
    // An item's levels are walked by its CTA alone, so few items take larger
    // CTAs: as long as their threads fit on the SMs.  240 items of 50,000-gate
    // levels: 0.76 -> 0.22 ms; 37,858 sweeps keep 256 threads.
    const uint64_t tile_items = (uint64_t)n_sweeps * ((std::min<uint64_t>(W, kTileWords) + M - 1) / M);
    for (threads = 1024; threads > 256 && tile_items * threads > 2048ull * n_sms; threads /= 2) {}
    if (!eflag_uploaded && n_sweeps) {
      std::vector<uint8_t> fl(N, 0);
      for (uint32_t e = plan.n_pi; e < N; ++e)
        fl[e] = (uint8_t)((plan.net.live[e] && nl.type[e] != G_PO) ? 1 : 0) | (uint8_t)(plan.po_drv[e] ? 2 : 0);
      upload(d_eflag, fl, s);
      eflag_uploaded = true;
    }
    CK(sweep_wide_occupancy(M, threads, &occ_got));
    const uint64_t per_block = (uint64_t)N * M * 8;
    const uint64_t cap = std::max<uint64_t>((uint64_t)n_sms, (4ull << 30) / std::max<uint64_t>(per_block, 1));
    blocks = (int)std::max<uint64_t>(
        1, std::min({(uint64_t)n_sms * std::max(occ_got, 1), cap, std::max<uint64_t>(tile_items, 1)}));
    if (n_sweeps) d_gvals.ensure((size_t)blocks * per_block);
  } else if (n_sweeps) {
    sched = &use_schedule(M, threads, s);
    smem = std::max<size_t>(16, sweep_vals_bytes(sched->max_live, M));
  }
  try {
    scratch(group);
  } catch (const CudaError&) {
    if (group == 1) throw;
    one_tile_gen = plan_gen;
    group = 1;
    d_sens.release();
    d_out.release();
    scratch(1);
  }
  // control words: the error word, then a work counter per tile
  int* err_word = d_queue.as<int>();
  int* queue = err_word + 1;
  launch_init_results(d_count.as<unsigned long long>(), d_first.as<unsigned long long>(),
                      d_lastflag.as<uint8_t>(), (uint32_t)F, err_word, (uint32_t)tiles + 1, s);
  CK(cudaEventRecord(e1, s));

  // 2. good machine
  launches += launch_good(good_view((uint32_t)W), nl.level_off.data(), n_sms, s);
  CK(cudaGetLastError());
  good_tiles = tiles;
  good_P = pats.P;
  CK(cudaEventRecord(e2, s));

  if (!wide && n_sweeps) {
    CK(sweep_set_smem(M, sched->direct, share1));
    CK(sweep_occupancy(M, sched->direct, threads, smem, &occ_got));
    if (occ_got < 1) throw LimitError{"sweep kernel does not fit on an SM with this shape"};
    blocks = n_sms * occ_got;
  }

  // 3. tiles
  uint32_t n_sw = n_sweeps, n_rt = n_roots, n_ex = n_exact;
  const uint32_t* sw_list = nullptr;
  const uint32_t* rt_list = nullptr;
  const uint32_t* ex_list = nullptr;
  int cur = 0;
  uint64_t items = 0, dense = 0, alg_bytes = 0;
  float ms_sweep = 0, ms_ffr = 0;
  const uint32_t gates_end = plan.level_off[std::min(plan.max_gate_level + 1, plan.n_levels)];
  std::vector<uint32_t> host_sw;  // only for the dense-work counter in drop mode
  uint64_t n_groups = 0;
  for (uint64_t t = 0; t < tiles; t += group, ++n_groups) {
    const uint32_t n_tiles = (uint32_t)std::min(group, tiles - t);
    const uint64_t* good_t = d_good.as<uint64_t>() + t * (uint64_t)N * kTileWords;
    cudaEvent_t a0 = ev(5 + 3 * n_groups), a1 = ev(6 + 3 * n_groups), a2 = ev(7 + 3 * n_groups);
    CK(cudaEventRecord(a0, s));
    if (n_sw) {
      const uint32_t n_words = tile_words(W, t + n_tiles - 1);
      const uint64_t subtiles = (uint64_t)(n_tiles - 1) * (kTileWords / M) + (n_words + M - 1) / M;
      const int nb = (int)std::min<uint64_t>((uint64_t)blocks, n_sw * subtiles);
      if (wide) {
        SweepWideArgs wa{};
        wa.level = d_level.as<uint32_t>();
        wa.level_off = d_level_off.as<uint32_t>();
        wa.fi_off = d_fi_off.as<uint32_t>();
        wa.fi_idx = d_fi_idx.as<uint32_t>();
        wa.type = d_type.as<uint8_t>();
        wa.eflag = d_eflag.as<uint8_t>();
        wa.inj = d_inj.as<InjRec>();
        wa.list = sw_list;
        wa.n_list = n_sw;
        wa.n_words = n_words;
        wa.max_gate_level = plan.max_gate_level;
        wa.N = N;
        wa.good = good_t;
        wa.out = d_out.as<uint64_t>();
        wa.queue = queue + t;
        wa.gvals = d_gvals.as<uint64_t>();
        CK(launch_sweep_wide(M, threads, nb, wa, s));
      } else {
        SweepArgs sa{};
        sa.blob = d_recs.as<uint4>();
        sa.lvl = d_lvl.as<uint4>();
        sa.level = d_level.as<uint32_t>();
        sa.li = d_li.as<uint32_t>();
        sa.fi_off = d_fi_off.as<uint32_t>();
        sa.fi_idx = d_fi_idx.as<uint32_t>();
        sa.type = d_type.as<uint8_t>();
        sa.inj = d_inj.as<InjRec>();
        sa.list = sw_list;
        sa.n_list = n_sw;
        sa.n_tiles = n_tiles;
        sa.n_sweeps = n_sweeps;
        sa.n_words = n_words;
        sa.max_gate_level = plan.max_gate_level;
        sa.N = N;
        sa.good = good_t;
        sa.out = d_out.as<uint64_t>();
        sa.queue = queue + t;
        sa.stream_recs = sched->stream_recs;
        sa.fix0 = sched->fix0;
        sa.inj_slot = sched->max_live - 1;
        sa.split = sched->split;
        sa.err = err_word;
        sa.wait_ns = kWaitTestNs;
        sa.wait_test = (o.wait_test && t == 0) ? 1u : 0u;
        CK(launch_sweep(M, sched->direct, threads, nb, smem, sa, s));
      }
      ++launches;
      items += (uint64_t)n_sw * subtiles;
      if (!sw_list) {
        dense += plan.dense_sweep_gates * subtiles * M;
        alg_bytes += plan.dense_sweep_bytes * subtiles * M;
      } else {
        host_sw.resize(n_sw);
        CK(cudaMemcpyAsync(host_sw.data(), sw_list, n_sw * 4, cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        for (uint32_t si : host_sw) {
          uint32_t L0 = nl.level[plan.sweeps[si].stored] + 1;
          if (L0 <= plan.max_gate_level) {
            dense += (uint64_t)(plan.eval_prefix[gates_end] - plan.eval_prefix[plan.level_off[L0]]) * subtiles * M;
            alg_bytes += (plan.nfp_prefix[gates_end] - plan.nfp_prefix[plan.level_off[L0]]) * subtiles * M;
          }
        }
      }
    }
    CK(cudaEventRecord(a1, s));
    FfrArgs fa{};
    fa.roots = d_roots.as<RootRec>();
    fa.list = rt_list;
    fa.n_list = n_rt;
    fa.members = d_members.as<MemberRec>();
    fa.traced = d_traced.as<TracedRec>();
    fa.traced_slot = d_traced_slot.as<uint32_t>();
    fa.N = N;
    fa.n_sweeps = n_sweeps;
    fa.n_slots = n_slots;
    fa.n_tiles = n_tiles;
    fa.fi_off = d_fi_off.as<uint32_t>();
    fa.fi_idx = d_fi_idx.as<uint32_t>();
    fa.type = d_type.as<uint8_t>();
    fa.good = good_t;
    fa.obs = d_out.as<uint64_t>();
    fa.sens = d_sens.as<uint64_t>();
    fa.tile = (uint32_t)t;
    fa.W = (uint32_t)W;
    fa.P = pats.P;
    fa.drop = o.drop ? 1 : 0;
    fa.n_detect = n_detect;
    fa.count = d_count.as<unsigned long long>();
    fa.first = d_first.as<unsigned long long>();
    fa.lastflag = d_lastflag.as<uint8_t>();
    launch_ffr(fa, s);
    launches += n_rt ? 1 : 0;
    ExactArgs xa{};
    xa.exact_fault = d_exact.as<uint32_t>();
    xa.list = ex_list;
    xa.n_exact = n_ex;
    xa.first_sweep = plan.n_stem_sweeps;
    xa.out = d_out.as<uint64_t>();
    xa.n_sweeps = n_sweeps;
    xa.n_tiles = n_tiles;
    xa.tile = (uint32_t)t;
    xa.W = (uint32_t)W;
    xa.P = pats.P;
    xa.drop = o.drop ? 1 : 0;
    xa.n_detect = n_detect;
    xa.count = fa.count;
    xa.first = fa.first;
    xa.lastflag = fa.lastflag;
    launch_exact(xa, s);
    launches += n_ex ? 1 : 0;
    CK(cudaGetLastError());
    CK(cudaEventRecord(a2, s));
    if (o.drop && t + 1 < tiles) {
      CK(cudaMemsetAsync(d_nout.p, 0, 16, s));
      DropArgs da{};
      da.roots = d_roots.as<RootRec>();
      da.in_list = rt_list;
      da.n_in = n_rt;
      da.n_in_pad = (n_rt + 31) / 32 * 32;
      da.traced = d_traced.as<TracedRec>();
      da.exact_fault = d_exact.as<uint32_t>();
      da.exact_in = ex_list;
      da.n_exact_in = n_ex;
      da.first_exact_sweep = plan.n_stem_sweeps;
      da.count = d_count.as<unsigned long long>();
      da.n_detect = n_detect;
      da.out_roots = d_root_list[cur].as<uint32_t>();
      da.out_sweeps = d_sweep_list.as<uint32_t>();
      da.out_exact = d_exact_list[cur].as<uint32_t>();
      da.n_out = d_nout.as<uint32_t>();
      launch_drop(da, s);
      ++launches;
      CK(cudaGetLastError());
      uint32_t nout[4] = {0, 0, 0, 0};
      CK(cudaMemcpyAsync(nout, d_nout.p, 16, cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      n_rt = nout[0];
      n_sw = nout[1];
      n_ex = nout[2];
      rt_list = d_root_list[cur].as<uint32_t>();
      sw_list = d_sweep_list.as<uint32_t>();
      ex_list = d_exact_list[cur].as<uint32_t>();
      cur ^= 1;
      if (n_rt == 0 && n_ex == 0) {
        CK(cudaEventSynchronize(a2));
        float x = 0;
        CK(cudaEventElapsedTime(&x, a0, a1));
        ms_sweep += x;
        CK(cudaEventElapsedTime(&x, a1, a2));
        ms_ffr += x;
        break;
      }
    }
    if (o.drop) {
      CK(cudaEventSynchronize(a2));
      float x = 0;
      CK(cudaEventElapsedTime(&x, a0, a1));
      ms_sweep += x;
      CK(cudaEventElapsedTime(&x, a1, a2));
      ms_ffr += x;
    }
  }
  CK(cudaEventRecord(e3, s));

  // 4. results
  const uint64_t last_rd = W ? W - 1 : 0;
  launch_results(ResultArgs{d_count.as<unsigned long long>(), d_first.as<unsigned long long>(),
                            d_lastflag.as<uint8_t>(), err_word, d_records.as<ulonglong2>(), last_rd, (uint32_t)F,
                            W ? 1u : 0u},
                 s);
  ++launches;
  CK(cudaGetLastError());
  const size_t record_bytes = F * sizeof(fsimb_fault_result);
  const double last_ms = stats.ms_compute;  // of the run before
  cudaEvent_t e4 = ev(4);
  // The records come back to pageable memory first, and to page-locked memory
  // once locking is cheap against the run (in count mode it runs beside the
  // kernels) or the pageable copies have cost as much.  Locking takes 1.1 to 4 ms
  // and 0.3 to 3 ms per MB, a pageable copy 10 us more at 45 KB, 17 us at 130 KB, 0.1 ms
  // at 1.3 MB, 0.3 to 0.6 ms at 4 MB and 0.8 ms at 24 MB.  Locked on its second run, a
  // handle of 400 gates and 64 patterns took 2.5 ms for it, against 0.15 ms.
  const double record_mb = (double)record_bytes * 1e-6, lock_us = 1500 + 500 * record_mb;
  bool pinned = h_records.n >= record_bytes + 16;
  if (!pinned && host_records.size() > F &&
      (last_ms * 1e3 > lock_us * (o.drop ? 10 : 2) || paged_us > lock_us)) {
    pinned = h_records.try_ensure(record_bytes + 16);
    paged_us = 0;
  }
  if (pinned) {
    std::vector<fsimb_fault_result>().swap(host_records);
  } else {
    host_records.resize(F + 1);
    paged_us += 12 + 80 * record_mb;
  }
  char* dst = pinned ? h_records.as<char>() : reinterpret_cast<char*>(host_records.data());
  CK(cudaMemcpyAsync(dst, d_records.p, record_bytes + 16, cudaMemcpyDeviceToHost, s));
  CK(cudaEventRecord(e4, s));
  CK(cudaStreamSynchronize(s));
  uint64_t kerr = 0;
  std::memcpy(&kerr, dst + record_bytes, sizeof kerr);
  if (kerr) throw CudaError{"a sweep kernel's wait test reached its time limit; results discarded"};
  if (!o.drop) {
    for (uint64_t g = 0; g < n_groups; ++g) {
      float x = 0;
      CK(cudaEventElapsedTime(&x, ev(5 + 3 * g), ev(6 + 3 * g)));
      ms_sweep += x;
      CK(cudaEventElapsedTime(&x, ev(6 + 3 * g), ev(7 + 3 * g)));
      ms_ffr += x;
    }
  }
  static_assert(sizeof(fsimb_fault_result) == 32, "k_results writes two 16-byte halves");
  records = reinterpret_cast<const fsimb_fault_result*>(dst);
  n_records = F;
  has_results = true;

  float x = 0;
  stats = fsimb_stats{};
  CK(cudaEventElapsedTime(&x, e0, e4));
  stats.ms_total = x;
  CK(cudaEventElapsedTime(&x, e0, e1));
  stats.ms_h2d = x;
  CK(cudaEventElapsedTime(&x, e1, e2));
  stats.ms_good = x;
  stats.ms_sweep = ms_sweep;
  stats.ms_ffr = ms_ffr;
  CK(cudaEventElapsedTime(&x, e3, e4));
  stats.ms_d2h = x;
  stats.n_tiles = tiles;
  stats.n_stem_sweeps = plan.n_stem_sweeps;
  stats.n_exact_sweeps = n_exact;
  stats.n_traced_faults = plan.traced.size();
  stats.n_roots = n_roots;
  stats.sweep_items = items;
  stats.dense_gate_words = dense;
  stats.sweep_alg_bytes = alg_bytes;
  stats.kernel_launches = launches;
  CK(cudaEventElapsedTime(&x, e1, e3));
  stats.ms_compute = x;
  stats.good_gate_words = (uint64_t)(N - plan.n_pi) * W_pad;
  stats.max_live = sched ? sched->max_live : 0;
  stats.bank_conflict_groups = sched ? sched->conflict_groups : 0;
  stats.bank_access_groups = sched ? sched->access_groups : 0;
  stats.sweep_variant = wide ? 2 : 1;
  stats.hbm_bytes_per_tile = (uint64_t)N * kTileWords * 8 + (uint64_t)n_sweeps * (kTileWords * 8 + sizeof(InjRec)) +
                             (sched ? sched->bytes() : wide ? (uint64_t)N * 10 + nl.fi_idx.size() * 4 : 0);
  stats.ms_tune = tune_ms_now;
  stats.ctas_per_sm = (uint32_t)occ_got;
  stats.words_per_item = (uint32_t)M;
  stats.block_threads = (uint32_t)threads;
  stats.blocks = (uint32_t)blocks;
  stats.smem_bytes = (uint32_t)smem;
  stats.device_bytes = device_bytes();
}

extern "C" {

int fsimb_create(int device, fsimb_handle** out) {
  if (!out) return FSIMB_ERR_ARG;
  *out = nullptr;
  fsimb_handle* h = nullptr;
  try {
    h = new fsimb_handle();
    if (device >= 0) {
      int n = 0;
      cudaError_t e = cudaGetDeviceCount(&n);
      if (e != cudaSuccess || device >= n) {
        g_create_error = std::string("no usable CUDA device ") + std::to_string(device) + ": " +
                         (e != cudaSuccess ? cudaGetErrorString(e) : "index out of range");
        cudaGetLastError();
        delete h;
        return FSIMB_ERR_CUDA;
      }
      int major = 0;
      CK(cudaSetDevice(device));
      CK(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
      if (major < 10) throw CudaError{"device is not sm_100 (Blackwell)"};
      int sms = 0, optin = 0;
      CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
      CK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
      int per_sm = 0;
      CK(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device));
      h->device = device;
      h->n_sms = sms;
      h->smem_optin = (size_t)optin;
      h->smem_per_sm = (size_t)per_sm;
      CK(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
      CK(cudaEventCreateWithFlags(&h->upload_ev, cudaEventDisableTiming));
    }
  } catch (const CudaError& e) {
    g_create_error = e.msg;
    delete h;
    return FSIMB_ERR_CUDA;
  } catch (const std::bad_alloc&) {
    g_create_error = "host allocation failed";
    delete h;
    return FSIMB_ERR_NOMEM;
  }
  *out = h;
  return FSIMB_OK;
}

int fsimb_destroy(fsimb_handle* h) {
  if (!h) return FSIMB_ERR_ARG;
  delete h;
  return FSIMB_OK;
}

const char* fsimb_last_error(const fsimb_handle* h) {
  return h ? h->err.c_str() : g_create_error.c_str();
}

int fsimb_load_files(fsimb_handle* h, const char* ckt, const char* flst, const char* ptn) {
  API_BEGIN(h)
  if (!ckt || !flst || !ptn) throw ArgError{"null path"};
  std::string a = read_file(ckt), b = read_file(flst), c = read_file(ptn);
  h->load_ckt(a.data(), a.size());
  h->load_flst(b.data(), b.size());
  h->load_ptn(c.data(), c.size());
  API_END(h)
}

int fsimb_load_buffers(fsimb_handle* h, const char* ckt, size_t ckt_len, const char* flst,
                       size_t flst_len, const char* ptn, size_t ptn_len) {
  API_BEGIN(h)
  if (!ckt || !flst || !ptn) throw ArgError{"null buffer"};
  h->load_ckt(ckt, ckt_len);
  h->load_flst(flst, flst_len);
  h->load_ptn(ptn, ptn_len);
  API_END(h)
}

int fsimb_load_circuit(fsimb_handle* h, const char* ckt, size_t ckt_len) {
  API_BEGIN(h)
  if (!ckt) throw ArgError{"null buffer"};
  h->load_ckt(ckt, ckt_len);
  API_END(h)
}

int fsimb_set_faults(fsimb_handle* h, const uint32_t* site, const uint8_t* pin,
                     const uint8_t* value, uint64_t n) {
  API_BEGIN(h)
  if (!h->has_ckt) throw StateError{"load a circuit first"};
  if (n && (!site || !value)) throw ArgError{"null fault arrays"};
  std::vector<Fault> fs(n);
  for (uint64_t i = 0; i < n; ++i) {
    if (site[i] >= h->nl.N) throw ArgError{"fault site out of range at " + std::to_string(i)};
    uint8_t p = pin ? pin[i] : 0;
    if (p > h->nl.fanin_count(site[i])) throw ArgError{"fault pin out of range at " + std::to_string(i)};
    fs[i] = Fault{site[i], p, (uint8_t)(value[i] ? 1 : 0)};
  }
  h->faults = std::move(fs);
  h->has_faults = true;
  h->gen = h->plan_gen = next_generation();
  h->plan_valid = false;
  h->plan_uploaded = false;
  h->has_results = false;
  API_END(h)
}

int fsimb_set_fault_text(fsimb_handle* h, const char* flst, size_t flst_len) {
  API_BEGIN(h)
  if (!flst) throw ArgError{"null buffer"};
  h->load_flst(flst, flst_len);
  API_END(h)
}

int fsimb_set_patterns(fsimb_handle* h, const uint64_t* words, uint64_t num_patterns) {
  API_BEGIN(h)
  if (!h->has_ckt) throw StateError{"load a circuit first"};
  const uint64_t W = (num_patterns + 63) / 64;
  if (W && !words) throw ArgError{"null pattern words"};
  if (W * h->nl.n_pi > (1ull << 36)) throw LimitError{"pattern block too large"};
  if (h->pats.words.capacity() >= W * h->nl.n_pi) {  // into the room the last patterns had
    h->pats.words.assign(words, words + W * h->nl.n_pi);
    h->pats.P = num_patterns;
    h->pats.W = W;
  } else {
    Patterns p;
    p.P = num_patterns;
    p.W = W;
    p.words.assign(words, words + W * h->nl.n_pi);
    h->pats = std::move(p);
  }
  h->has_pats = true;
  h->gen = next_generation();
  h->has_results = false;
  h->good_tiles = 0;
  h->pats_uploaded = false;
  API_END(h)
}

int fsimb_run(fsimb_handle* h, const fsimb_opts* opts) {
  API_BEGIN(h)
  h->run(opts);
  API_END(h)
}

int fsimb_results(const fsimb_handle* hc, fsimb_fault_result* out, uint64_t n) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!h->has_results) throw StateError{"no results: call fsimb_run first"};
  if (n != h->n_records || (n && !out)) throw ArgError{"result buffer size must equal the fault count"};
  if (n) std::memcpy(out, h->records, n * sizeof(fsimb_fault_result));
  API_END(h)
}

int fsimb_found_fault_to_pattern(const fsimb_handle* hc, uint64_t* out, uint64_t n) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!h->has_results) throw StateError{"no results: call fsimb_run first"};
  if (n != 2 * h->n_records || (n && !out)) throw ArgError{"buffer size must be 2 * faults"};
  for (size_t f = 0; f < h->n_records; ++f) {
    out[2 * f] = h->records[f].ref_last_round_flag;
    out[2 * f + 1] = h->records[f].ref_last_rd;
  }
  API_END(h)
}

int fsimb_good_values(const fsimb_handle* hc, uint64_t round, uint64_t* out, uint64_t n) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!h->good_tiles || h->good_P != h->pats.P) throw StateError{"no good values: call fsimb_run first"};
  if (round >= h->pats.W) throw ArgError{"round out of range"};
  if (n != h->nl.N || !out) throw ArgError{"buffer size must equal the element count"};
  CK(cudaSetDevice(h->device));
  const uint64_t tile = round / kTileWords, lane = round % kTileWords;
  const uint32_t bits = h->pats.bits(round);
  // into the run's scratch where it is large enough (a full device may have
  // no room for more)
  DevBuf& b = h->d_sens.n >= n * 8 ? h->d_sens : h->d_out.n >= n * 8 ? h->d_out : h->d_round;
  b.ensure(n * 8);
  launch_round(h->d_good.as<uint64_t>() + (tile * h->nl.N) * kTileWords + lane, h->nl.N,
               bits >= 64 ? ~0ull : ((1ull << bits) - 1), b.as<uint64_t>(), h->stream);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(out, b.p, n * 8, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  API_END(h)
}

int fsimb_get_info(const fsimb_handle* hc, fsimb_info* out) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!out) throw ArgError{"null output"};
  if (!h->has_ckt) throw StateError{"no circuit loaded"};
  *out = fsimb_info{};
  out->num_pis = h->nl.n_pi;
  out->num_pos = h->nl.n_po;
  out->num_gates = h->nl.n_gates;
  out->num_wires = h->nl.n_wires;
  out->num_elements = h->nl.N;
  out->num_levels = h->nl.ref_per_level.empty() ? h->nl.n_levels : h->nl.ref_per_level.size();
  out->num_faults = h->has_faults ? h->faults.size() : 0;
  out->num_patterns = h->has_pats ? h->pats.P : 0;
  out->num_rounds = h->has_pats ? h->pats.W : 0;
  API_END(h)
}

int fsimb_set_loader(fsimb_handle* h, int mode, int threads) {
  API_BEGIN(h)
  if (mode < FSIMB_LOAD_AUTO || mode > FSIMB_LOAD_DEVICE) throw ArgError{"loader mode must be 0, 1 or 2"};
  if (threads < 0 || threads > 1024) throw ArgError{"loader threads must be 0..1024"};
  h->load_mode = mode;
  h->load_threads = threads;
  API_END(h)
}

int fsimb_get_load_info(const fsimb_handle* hc, fsimb_load_info* out) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!out) throw ArgError{"null output"};
  if (!h->has_ckt) throw StateError{"no circuit loaded"};
  const LoadInfo& li = h->load_info;
  *out = fsimb_load_info{};
  out->on_device = li.on_device;
  out->handed_back = li.handed_back;
  out->threads = (uint32_t)li.threads;
  out->waves = li.waves;
  out->ms_total = li.ms_total;
  out->ms_tokenize = li.ms_tokenize;
  out->ms_device = li.ms_device;
  API_END(h)
}

int fsimb_get_stats(const fsimb_handle* hc, fsimb_stats* out) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!out) throw ArgError{"null output"};
  *out = h->stats;
  API_END(h)
}

int fsimb_topo_map(const fsimb_handle* hc, uint64_t* out, uint64_t n) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!h->has_ckt) throw StateError{"no circuit loaded"};
  if (n != h->nl.N || !out) throw ArgError{"buffer size must equal the element count"};
  std::copy(h->nl.tpg.begin(), h->nl.tpg.end(), out);
  API_END(h)
}

int fsimb_levels(const fsimb_handle* hc, uint64_t* out, uint64_t n) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!h->has_ckt) throw StateError{"no circuit loaded"};
  if (n != h->nl.N || !out) throw ArgError{"buffer size must equal the element count"};
  const auto& level = h->nl.ref_level.empty() ? h->nl.level : h->nl.ref_level;
  for (uint64_t i = 0; i < n; ++i) out[i] = level[i];
  API_END(h)
}

int fsimb_gates_per_level(const fsimb_handle* hc, uint64_t* out, uint64_t n) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!h->has_ckt) throw StateError{"no circuit loaded"};
  const auto& per = h->nl.ref_per_level.empty() ? h->nl.per_level : h->nl.ref_per_level;
  if (n != per.size() || !out) throw ArgError{"buffer size must equal the level count"};
  std::copy(per.begin(), per.end(), out);
  API_END(h)
}

int fsimb_types(const fsimb_handle* hc, uint8_t* out, uint64_t n) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!h->has_ckt) throw StateError{"no circuit loaded"};
  if (n != h->nl.N || !out) throw ArgError{"buffer size must equal the element count"};
  std::copy(h->nl.type.begin(), h->nl.type.end(), out);
  API_END(h)
}

int fsimb_faults(const fsimb_handle* hc, uint32_t* site, uint8_t* pin, uint8_t* value, uint64_t n) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!h->has_faults) throw StateError{"no faults loaded"};
  if (n != h->faults.size()) throw ArgError{"buffer size must equal the fault count"};
  for (uint64_t i = 0; i < n; ++i) {
    if (site) site[i] = h->faults[i].site;
    if (pin) pin[i] = h->faults[i].pin;
    if (value) value[i] = h->faults[i].value;
  }
  API_END(h)
}

int fsimb_fault_costs(fsimb_handle* h, uint64_t* group, uint64_t* cost, uint64_t n) {
  API_BEGIN(h)
  if (!h->has_ckt || !h->has_faults) throw StateError{"load a circuit and faults first"};
  if (n != h->faults.size()) throw ArgError{"buffer size must equal the fault count"};
  if (!h->plan_valid) {
    build_plan(h->nl, h->faults, h->plan);
    h->plan_valid = true;
    h->plan_uploaded = false;
    h->sched_M = 0;
  }
  const Plan& P = h->plan;
  const Netlist& nl = h->nl;
  const uint32_t gates_end = nl.level_off[std::min(P.max_gate_level + 1, nl.n_levels)];
  auto sweep_gates = [&](uint32_t elem) -> uint64_t {
    const uint32_t L0 = nl.level[elem] + 1;
    return L0 <= P.max_gate_level ? gates_end - nl.level_off[L0] : 0;
  };
  // traced faults: one group per FFR root (its sweep, when it has one, plus
  // the tracing of its members); exact faults: one group each
  for (const RootRec& rr : P.roots) {
    const bool swept = nl.type[rr.root] != G_PO && !P.po_drv[rr.root] && P.gate_fo[rr.root];
    const uint64_t c = 1 + (swept ? sweep_gates(rr.root) : 0) + (rr.mem_end - rr.mem_begin);
    for (uint32_t i = rr.flt_begin; i < rr.flt_end; ++i) {
      const uint32_t f = P.traced[i].fault;
      if (group) group[f] = rr.root;
      if (cost) cost[f] = c;
    }
  }
  for (uint32_t j = 0; j < P.exact_fault.size(); ++j) {
    const uint32_t f = P.exact_fault[j];
    if (group) group[f] = (uint64_t)nl.N + j;
    if (cost) cost[f] = 1 + sweep_gates(P.sweeps[P.n_stem_sweeps + j].elem);
  }
  API_END(h)
}

int fsimb_patterns(const fsimb_handle* hc, uint64_t* out, uint64_t n) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!h->has_pats) throw StateError{"no patterns loaded"};
  if (n != h->pats.words.size() || (n && !out)) throw ArgError{"buffer size must equal rounds * PIs"};
  std::copy(h->pats.words.begin(), h->pats.words.end(), out);
  API_END(h)
}

static int emit_text(const std::string& s, char** text, size_t* len) {
  char* p = (char*)std::malloc(s.size() + 1);
  if (!p) return FSIMB_ERR_NOMEM;
  std::memcpy(p, s.data(), s.size());
  p[s.size()] = 0;
  *text = p;
  if (len) *len = s.size();
  return FSIMB_OK;
}

static const char* type_name(uint8_t t) {
  static const char* names[] = {"INV", "AND", "OR", "XOR", "NAND", "NOR", "XNOR", "MUX", "CLKBUF", "PI", "PO"};
  return t <= G_PO ? names[t] : "UNKNOWN";
}

int fsimb_dot(const fsimb_handle* hc, char** text, size_t* len) {
  fsimb_handle* h = const_cast<fsimb_handle*>(hc);
  API_BEGIN(h)
  if (!text) throw ArgError{"null output"};
  if (!h->has_ckt) throw StateError{"no circuit loaded"};
  const Netlist& nl = h->nl;
  const uint64_t g0 = nl.n_pi, p0 = nl.n_pi + nl.n_gates;
  // Node names: PI_i, Gate_j_TYPE (j = index among gates), PO_k.
  auto src_name = [&](uint32_t e) {
    if (nl.type[e] == G_PI) return "PI_" + std::to_string(e);
    return "Gate_" + std::to_string(e - g0) + "_" + type_name(nl.type[e]);
  };
  std::string out = "digraph G {\n\tsubgraph cluster_0 {\n\t\tcolor=black;\n"
                    "\t\tnode [style=filled,color=lightgrey];\n";
  for (uint64_t e = g0; e < nl.N; ++e) {
    const std::string dst = e < p0 ? "Gate_" + std::to_string(e - g0) + "_" + type_name(nl.type[e]) + ";"
                                   : "PO_" + std::to_string(e - p0) + ";";
    for (uint32_t k = nl.fi_off[e]; k < nl.fi_off[e + 1]; ++k)
      out += "\t\t" + src_name(nl.fi_idx[k]) + " -> " + dst + "\n";
  }
  out += "\t}\n\n";
  for (uint64_t i = 0; i < nl.n_pi; ++i) out += "\tPI_" + std::to_string(i) + "  [shape=Msquare];\n";
  for (uint64_t i = 0; i < nl.n_po; ++i) out += "\tPO_" + std::to_string(i) + "  [shape=Msquare];\n";
  out += "}\n\n";
  char* p = (char*)std::malloc(out.size() + 1);
  if (!p) throw std::bad_alloc();
  std::memcpy(p, out.data(), out.size() + 1);
  *text = p;
  if (len) *len = out.size();
  API_END(h)
}

int fsimb_gen_circuit(const fsimb_gen_config* cfg, char** text, size_t* len) {
  if (!cfg || !text) return FSIMB_ERR_ARG;
  try {
    GenConfig g;
    g.seed = cfg->seed;
    g.n_gates = cfg->n_gates;
    g.n_pi = cfg->n_pi;
    g.n_po = cfg->n_po;
    g.n_levels = cfg->n_levels;
    if (cfg->window) g.window = cfg->window;
    g.p_fanin3 = cfg->p_fanin3;
    if (cfg->type_mask) g.type_mask = cfg->type_mask;
    g.hub_frac = cfg->hub_frac;
    if (cfg->hub_fo_min) g.hub_fo_min = cfg->hub_fo_min;
    if (cfg->hub_fo_max) g.hub_fo_max = cfg->hub_fo_max;
    if (cfg->fo_min) g.fo_min = cfg->fo_min;
    if (cfg->fo_max) g.fo_max = cfg->fo_max;
    g.p_unused = cfg->p_unused;
    g.shuffle_ids = cfg->shuffle_ids;
    if (g.n_pi == 0 || g.n_levels == 0) {
      g_create_error = "generator needs at least one PI and one level";
      return FSIMB_ERR_ARG;
    }
    if (g.hub_fo_max < g.hub_fo_min || g.fo_max < g.fo_min) {
      g_create_error = "generator fanout range is empty";
      return FSIMB_ERR_ARG;
    }
    return emit_text(generate_ckt(g), text, len);
  } catch (const std::bad_alloc&) {
    return FSIMB_ERR_NOMEM;
  }
}

int fsimb_gen_faults(const char* ckt, size_t ckt_len, int kind, char** text, size_t* len) {
  if (!ckt || !text || kind < 0 || kind > 2) return FSIMB_ERR_ARG;
  try {
    Netlist nl;
    parse_ckt(ckt, ckt_len, nl);
    std::vector<Fault> fs;
    build_fault_list(nl, (FaultListKind)kind, fs);
    return emit_text(write_flst(nl, fs, kind != 0), text, len);
  } catch (const ParseError& e) {
    g_create_error = e.msg;
    return FSIMB_ERR_PARSE;
  } catch (const std::bad_alloc&) {
    return FSIMB_ERR_NOMEM;
  }
}

int fsimb_gen_patterns(uint64_t seed, uint64_t n_patterns, uint64_t n_pi, double biased_pi_frac,
                       double p_one_biased, char** text, size_t* len) {
  if (!text || n_pi == 0) return FSIMB_ERR_ARG;
  try {
    PatternConfig pc;
    pc.seed = seed;
    pc.n_patterns = n_patterns;
    pc.biased_pi_frac = biased_pi_frac;
    pc.p_one_biased = p_one_biased;
    Patterns p;
    generate_patterns(pc, n_pi, p);
    return emit_text(write_ptn(p, n_pi), text, len);
  } catch (const std::bad_alloc&) {
    return FSIMB_ERR_NOMEM;
  }
}

void fsimb_free_text(char* text) { std::free(text); }

}  // extern "C"

// ------------------------------------------------------------ no-allocation
// Good-machine PO words for up to one tile of pattern words, for callers that
// must not allocate device memory on the call (for example code running under
// a fixed device-memory budget handed out up front, or a serving loop that may
// not take the implicit device synchronisation of cudaMalloc/cudaFree).  The
// element values, which the regular path keeps in a buffer sized per circuit,
// live here in one file-scope device array of fixed size, shared by every call
// on a device.
namespace {

constexpr uint32_t kNoAllocMaxElements = 32768;  // 32,768 elements x 32 words x 8 B = 8 MiB
static __device__ __align__(256) uint64_t g_noalloc_values[(size_t)kNoAllocMaxElements * kTileWords];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
uint64_t* g_noalloc_ptr[kNoAllocMaxDevices] = {};

__global__ void k_good_level_static(const uint8_t* type, const uint32_t* fi_off,
                                    const uint32_t* fi_idx, const uint64_t* pwords,
                                    uint32_t n_words, uint32_t n_pi, uint32_t po_begin,
                                    uint32_t n_po, uint32_t lo, uint32_t hi, uint64_t* vals,
                                    uint64_t* po_out) {
  const uint32_t n = (hi - lo) * kTileWords;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += gridDim.x * blockDim.x) {
    const uint32_t lane = idx % kTileWords;
    const uint32_t e = lo + idx / kTileWords;
    const uint8_t t = type[e];
    uint64_t v;
    if (t == G_PI) {
      v = lane < n_words ? pwords[(uint64_t)lane * n_pi + e] : 0ull;
    } else {
      const uint32_t f0 = fi_off[e];
      uint32_t nf = fi_off[e + 1] - f0;
      if (t == G_INV || t == G_CLKBUF || t == G_PO) nf = 1;
      uint64_t in[4] = {0, 0, 0, 0};
      for (uint32_t k = 0; k < nf && k < 4; ++k) in[k] = vals[(uint64_t)fi_idx[f0 + k] * kTileWords + lane];
      uint64_t r = in[0];
      switch (t) {
        case G_INV: r = ~r; break;
        case G_AND: case G_NAND:
          for (uint32_t k = 1; k < nf; ++k) r &= in[k];
          if (t == G_NAND) r = ~r;
          break;
        case G_OR: case G_NOR:
          for (uint32_t k = 1; k < nf; ++k) r |= in[k];
          if (t == G_NOR) r = ~r;
          break;
        case G_XOR: case G_XNOR:
          for (uint32_t k = 1; k < nf; ++k) r ^= in[k];
          if (t == G_XNOR) r = ~r;
          break;
        case G_MUX: r = (in[2] & in[1]) | (in[0] & (uint64_t)(in[2] == 0)); break;
        default: break;  // CLKBUF, PO: copy
      }
      v = r;
    }
    vals[(uint64_t)e * kTileWords + lane] = v;
    if (e >= po_begin && e - po_begin < n_po && lane < n_words)
      po_out[(uint64_t)lane * n_po + (e - po_begin)] = v;
  }
}

// Address of the static array on the current device, looked up once per
// device (host code cannot use the array's name as a device address).  A
// device reset ends the handles on that device and invalidates the address.
uint64_t* noalloc_scratch(int device) {
  if (device < 0 || device >= kNoAllocMaxDevices) throw ArgError{"device index out of range"};
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[device]) {
    void* p = nullptr;
    CK(cudaGetSymbolAddress(&p, g_noalloc_values));
    g_noalloc_ptr[device] = (uint64_t*)p;
  }
  return g_noalloc_ptr[device];
}

}  // namespace

extern "C" int fsimb_good_po_noalloc(fsimb_handle* h, const uint64_t* d_pattern_words,
                                     uint32_t n_words, uint64_t* d_po_words, void* stream) {
  API_BEGIN(h)
  if (h->device < 0) throw CudaError{"host-only handle: no GPU to run on"};
  if (!h->has_ckt || !h->plan_uploaded)
    throw StateError{"the circuit is not on the device yet: call fsimb_run once first"};
  if (n_words == 0 || n_words > kTileWords) throw ArgError{"n_words must be in 1..32"};
  if (!d_pattern_words || !d_po_words) throw ArgError{"null device pointer"};
  if (h->nl.N > kNoAllocMaxElements)
    throw LimitError{"circuit has " + std::to_string(h->nl.N) + " elements; the no-allocation "
                     "entry point holds at most " + std::to_string(kNoAllocMaxElements)};
  CK(cudaSetDevice(h->device));
  uint64_t* vals = noalloc_scratch(h->device);
  cudaStream_t s = stream ? (cudaStream_t)stream : h->stream;
  // the circuit arrays were uploaded by the last fsimb_run, maybe on another stream
  CK(cudaStreamWaitEvent(s, h->upload_ev, 0));
  const uint32_t po_begin = (uint32_t)(h->nl.n_pi + h->nl.n_gates);
  for (uint32_t l = 0; l < h->nl.n_levels; ++l) {
    const uint32_t lo = h->nl.level_off[l], hi = h->nl.level_off[l + 1];
    if (hi == lo) continue;
    const uint32_t n = (hi - lo) * kTileWords;
    const uint32_t blocks = std::min<uint32_t>((n + 255) / 256, 148u * 16u);
    k_good_level_static<<<blocks, 256, 0, s>>>(h->d_type.as<uint8_t>(), h->d_fi_off.as<uint32_t>(),
                                                h->d_fi_idx.as<uint32_t>(), d_pattern_words, n_words,
                                                (uint32_t)h->nl.n_pi, po_begin, (uint32_t)h->nl.n_po,
                                                lo, hi, vals, d_po_words);
  }
  CK(cudaGetLastError());
  API_END(h)
}
