// Internal declarations shared by the library's translation units: error
// types thrown inside the library and turned into status codes at the C ABI,
// device buffers, and the per-circuit handle (struct fsimb_handle of
// include/fsimb.h).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <functional>
#include <new>
#include <string>
#include <vector>

#include "../../include/fsimb.h"
#include "fsimb_kernels.cuh"
#include "fsimb_loader.h"
#include "fsimb_netlist.h"
#include "fsimb_plan.h"

namespace fsimb {

struct CudaError {
  std::string msg;
};
struct StateError {
  std::string msg;
};
struct ArgError {
  std::string msg;
};
struct IoError {
  std::string msg;
};

// The error is cleared: left as the thread's last error, the next launch
// check, of any handle, would take it for its own.
#define CK(call)                                                                            \
  do {                                                                                      \
    cudaError_t e_ = (call);                                                                \
    if (e_ != cudaSuccess) {                                                                \
      cudaGetLastError();                                                                   \
      throw ::fsimb::CudaError{std::string(#call) + ": " + cudaGetErrorString(e_)};         \
    }                                                                                       \
  } while (0)

struct DevBuf {
  void* p = nullptr;
  size_t n = 0;
  void ensure(size_t bytes) {
    if (bytes <= n && p) return;
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
    if (bytes == 0) bytes = 16;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e != cudaSuccess) {
      p = nullptr;
      cudaGetLastError();
      throw CudaError{"cudaMalloc(" + std::to_string(bytes) + " bytes): " + cudaGetErrorString(e)};
    }
    n = bytes;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  template <class T>
  T* as() const {
    return reinterpret_cast<T*>(p);
  }
};

template <class T>
inline void upload(DevBuf& b, const std::vector<T>& v, cudaStream_t s) {
  b.ensure(v.size() * sizeof(T));
  if (!v.empty()) CK(cudaMemcpyAsync(b.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
}

// Largest sweep CTA (the kernels' register caps).
constexpr uint32_t kMaxSweepThreads = 1024;

// Sweep CTA size for one thread per record of a level: the multiple of 32
// that splits the typical (90th percentile) level into equal rounds, so no
// thread idles long before the per-level barrier.
inline uint32_t pick_sweep_threads(const Schedule& sc) {
  std::vector<uint32_t> widths;
  for (size_t l = 0; l + 1 < sc.rec_off.size(); ++l)
    if (sc.rec_off[l + 1] > sc.rec_off[l]) widths.push_back(sc.rec_off[l + 1] - sc.rec_off[l]);
  uint32_t w = 64;
  if (!widths.empty()) {
    std::nth_element(widths.begin(), widths.begin() + widths.size() * 9 / 10, widths.end());
    w = std::max<uint32_t>(widths[widths.size() * 9 / 10], 1);
  }
  uint32_t best = 64;
  double best_cost = 1e30;
  for (uint32_t k = 1; k <= 64; ++k) {
    uint32_t t = (w + k - 1) / k;
    t = std::max<uint32_t>(64, (t + 31) / 32 * 32);
    if (t > kMaxSweepThreads) continue;
    const double cost = (double)k * t + 8.0 * k;  // issued slots + per-round overhead
    if (cost < best_cost) {
      best_cost = cost;
      best = t;
    }
  }
  return best;
}

// Dynamic shared memory one sweep CTA may take when `occ` CTAs share an SM
// (each CTA also holds the kernel's static __shared__ variables and the
// 1 KB the hardware reserves per CTA).
inline size_t sweep_smem_share(size_t smem_optin, size_t smem_per_sm, int occ) {
  const size_t static_smem = 512, reserved = 1024;
  const size_t budget = smem_optin > static_smem + reserved ? smem_optin - static_smem - reserved : 0;
  if (occ <= 1) return budget;
  const size_t per = smem_per_sm / (size_t)occ;
  return per > static_smem + reserved ? std::min(budget, per - static_smem - reserved) : 0;
}

// Pattern words of tile t of a block of W words.
inline uint32_t tile_words(uint64_t W, uint64_t t) {
  return (uint32_t)std::min<uint64_t>(kTileWords, W > t * kTileWords ? W - t * kTileWords : 0);
}

// Bytes of a sweep CTA's value slots: max_live slots of M words, 16-byte rounded.
inline uint32_t sweep_vals_bytes(uint32_t max_live, int M) {
  return (uint32_t)(((size_t)max_live * M * 8 + 15) / 16 * 16);
}

// Whether the schedule at M words per item has its records and its slots fit
// `bytes` of shared memory.
inline bool sched_fits(const Schedule& sc, int M, size_t bytes) {
  return sc.max_live <= max_slots(sc.G) && sweep_vals_bytes(sc.max_live, M) <= bytes;
}

// Page-locked host staging buffer.
struct PinnedBuf {
  void* p = nullptr;
  size_t n = 0;
  void ensure(size_t bytes) {
    if (bytes <= n && p) return;
    release();
    if (bytes == 0) bytes = 16;
    cudaError_t e = cudaMallocHost(&p, bytes);
    if (e != cudaSuccess) {
      p = nullptr;
      cudaGetLastError();
      throw CudaError{"cudaMallocHost(" + std::to_string(bytes) + " bytes): " + cudaGetErrorString(e)};
    }
    n = bytes;
  }
  // As ensure(); false, with nothing held, where the memory cannot be locked.
  bool try_ensure(size_t bytes) {
    try {
      ensure(bytes);
    } catch (const CudaError&) {
    }
    return p != nullptr;
  }
  void release() {
    if (p) cudaFreeHost(p);
    p = nullptr;
    n = 0;
  }
  template <class T>
  T* as() const {
    return reinterpret_cast<T*>(p);
  }
};

// Sweep launch shape: words per item and CTA size.
struct SweepShape {
  int M;
  int threads;
};

// Modelled cost of a sweep shape (cycles of an SM per tile of `words` pattern
// words and sweep) with `vals` bytes of slots; the shapes within 1.5x of the
// cheapest, cheapest first, at most `most` of them.
double sweep_shape_cost(const SweepNet& net, int M, uint32_t threads, size_t vals, size_t smem_per_sm,
                        uint32_t words);
std::vector<SweepShape> likely_shapes(const Plan& plan, uint32_t words, size_t smem_optin, size_t smem_per_sm,
                                      size_t most);

// Default sweep shape of a circuit: the cheapest for a tile of `words` pattern
// words.  sched_at(M) returns the schedule at M.  False if no schedule fits
// shared memory, not even at one word per item.
bool default_sweep_shape(const Plan& plan, const std::function<const Schedule&(int)>& sched_at,
                         uint32_t words, size_t smem_optin, size_t smem_per_sm, int& M, int& threads);

// A fresh value for fsimb_handle::gen: every change of a handle's circuit,
// faults or patterns gets a number no other state of any handle had.
uint64_t next_generation();

}  // namespace fsimb

struct fsimb_handle {
  int device = -1;
  int n_sms = 0;
  size_t smem_optin = 0, smem_per_sm = 0;
  cudaStream_t stream = nullptr;
  std::string err;
  uint64_t gen = 0;       // changes whenever circuit, faults or patterns change
  uint64_t plan_gen = 0;  // changes whenever circuit or faults change

  fsimb::Netlist nl;
  bool has_ckt = false;
  std::vector<fsimb::Fault> faults;
  bool has_faults = false;
  fsimb::Patterns pats;
  bool has_pats = false;

  fsimb::Plan plan;
  bool plan_valid = false;
  bool plan_uploaded = false;
  // Schedules built so far for this plan, per words per item (1, 2, 4, 8).
  fsimb::Schedule sched_cache[4];
  int sched_M = 0, sched_T = 0;   // the one on the device, and its CTA size (0: none)
  uint64_t sched_cache_gen[4] = {0, 0, 0, 0};
  // Autotuned sweep shape of plan_gen (fsimb_opts.tune), timed on a tile of
  // tuned_words pattern words.
  uint64_t tuned_gen = 0;
  uint32_t tuned_words = 0;
  int tuned_M = 0, tuned_T = 0;
  cudaEvent_t tune_ev[2] = {nullptr, nullptr};
  // Recorded after each fsimb_run's uploads, on the run's stream: work on
  // another stream that reads the circuit arrays waits for it.
  cudaEvent_t upload_ev = nullptr;

  fsimb::DevBuf d_type, d_fi_off, d_fi_idx, d_recs, d_level, d_level_off, d_gates, d_li;
  fsimb::DevBuf d_lvl;     // schedule: stream and live-in offsets per level
  fsimb::DevBuf d_eflag;   // wide-circuit sweep: per element, evaluated / drives a PO
  fsimb::DevBuf d_gvals;   // wide-circuit sweep: per-CTA value regions
  fsimb::DevBuf d_roots, d_members, d_traced, d_traced_slot, d_inj, d_exact;
  fsimb::DevBuf d_pwords, d_good, d_out, d_sens, d_count, d_first, d_lastflag, d_queue;
  fsimb::DevBuf d_root_list[2], d_sweep_list, d_exact_list[2], d_nout, d_tune_list;
  uint64_t one_tile_gen = 0;  // plan_gen whose group of tiles found no room on the device
  uint64_t good_tiles = 0;  // tiles held in d_good
  uint64_t good_P = 0;
  bool pats_uploaded = false;  // d_pwords holds the current patterns
  bool eflag_uploaded = false; // d_eflag holds the current plan's element flags

  // The last run's records: in host_records or h_records after fsimb_run, in
  // host_records after a batch's run.
  fsimb::DevBuf d_records, d_round;
  fsimb::PinnedBuf h_records;
  double paged_us = 0;  // what pageable record copies have cost so far
  std::vector<fsimb_fault_result> host_records;
  const fsimb_fault_result* records = nullptr;
  uint64_t n_records = 0;
  bool has_results = false;
  fsimb_stats stats{};
  std::vector<cudaEvent_t> events;

  ~fsimb_handle() {
    if (device >= 0) {
      cudaSetDevice(device);
      for (fsimb::DevBuf* b : {&d_type, &d_fi_off, &d_fi_idx, &d_recs, &d_level, &d_level_off, &d_gates,
                        &d_lvl, &d_eflag, &d_gvals, &d_li, &d_roots, &d_members, &d_traced, &d_traced_slot, &d_inj, &d_exact,
                        &d_pwords, &d_good, &d_out, &d_sens, &d_count, &d_first, &d_lastflag,
                        &d_queue, &d_root_list[0], &d_root_list[1], &d_sweep_list,
                        &d_exact_list[0], &d_exact_list[1], &d_nout, &d_tune_list, &d_records, &d_round})
        b->release();
      h_records.release();
      for (auto e : events) cudaEventDestroy(e);
      for (auto e : tune_ev)
        if (e) cudaEventDestroy(e);
      if (upload_ev) cudaEventDestroy(upload_ev);
      if (stream) cudaStreamDestroy(stream);
    }
  }

  cudaEvent_t ev(size_t i) {
    while (events.size() <= i) {
      cudaEvent_t e;
      CK(cudaEventCreate(&e));
      events.push_back(e);
    }
    return events[i];
  }

  uint64_t device_bytes() const {
    uint64_t s = 0;
    for (const fsimb::DevBuf* b : {&d_type, &d_fi_off, &d_fi_idx, &d_recs, &d_level, &d_level_off, &d_gates,
                            &d_lvl, &d_eflag, &d_gvals, &d_li, &d_roots, &d_members, &d_traced, &d_traced_slot, &d_inj, &d_exact,
                            &d_pwords, &d_good, &d_out, &d_sens, &d_count, &d_first, &d_lastflag,
                            &d_queue, &d_root_list[0], &d_root_list[1], &d_sweep_list,
                            &d_exact_list[0], &d_exact_list[1], &d_nout, &d_tune_list, &d_records, &d_round})
      s += b->n;
    return s;
  }

  void invalidate_circuit() {
    has_faults = false;
    has_pats = false;
    plan_valid = false;
    plan_uploaded = false;
    sched_M = 0;
    has_results = false;
    good_tiles = 0;
  }

  // Circuit loader (fsimb_set_loader): 0 automatic, 1 host, 2 device.
  int load_mode = 0;
  int load_threads = 0;
  fsimb::LoadInfo load_info;

  void load_ckt(const char* t, size_t n) {
    fsimb::Netlist tmp;
    const bool dev = device >= 0 && (load_mode == 2 || (load_mode == 0 && n >= fsimb::kDeviceLoadBytes));
    const auto t0 = std::chrono::steady_clock::now();
    fsimb::LoadInfo li;
    bool built = false;
    if (dev) {
      try {
        built = fsimb::parse_ckt_device(t, n, tmp, device, stream, load_threads, li);
      } catch (const fsimb::CudaError&) {
        // no room on the device (or the like): the host reader still can
        cudaStreamSynchronize(stream);
        cudaGetLastError();
        built = false;
      }
    }
    if (!built) {
      fsimb::parse_ckt(t, n, tmp);
      li = fsimb::LoadInfo{};
      li.handed_back = dev;
      li.threads = 1;
      li.ms_total = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }
    load_info = li;
    nl = std::move(tmp);
    has_ckt = true;
    gen = plan_gen = fsimb::next_generation();
    invalidate_circuit();
    faults.clear();
    pats = fsimb::Patterns();
  }
  void load_flst(const char* t, size_t n) {
    if (!has_ckt) throw fsimb::StateError{"load a circuit first"};
    std::vector<fsimb::Fault> tmp;
    fsimb::parse_flst(t, n, nl, tmp);
    faults = std::move(tmp);
    has_faults = true;
    gen = plan_gen = fsimb::next_generation();
    plan_valid = false;
    plan_uploaded = false;
    has_results = false;
  }
  void load_ptn(const char* t, size_t n) {
    if (!has_ckt) throw fsimb::StateError{"load a circuit first"};
    fsimb::Patterns tmp;
    fsimb::parse_ptn(t, n, nl, tmp);
    pats = std::move(tmp);
    has_pats = true;
    gen = fsimb::next_generation();
    has_results = false;
    good_tiles = 0;
    pats_uploaded = false;
  }

  void run(const fsimb_opts* opts);
  // The schedule at M words per item for the current plan (cached per M).
  fsimb::Schedule& cached_schedule(int M);
  // The schedule at M packed for T threads, uploaded unless it is there.
  const fsimb::Schedule& use_schedule(int M, int T, cudaStream_t s);
  // The circuit's good machine on the device for the first W pattern words.
  fsimb::GoodView good_view(uint32_t W) const;
  // default_sweep_shape for this circuit and the plain sweep kernel.
  bool default_shape(int& M, int& threads);
  // Whether the tuned shape holds for the current patterns: it was timed on
  // this plan, and on no fewer words a tile, up to the next power of two (the
  // words an item may take).  By the cost model a shape of one word takes 2.3
  // (50,000 gates) to 3.1 (2,000 gates) times the best shape's time on a full
  // tile.  For fewer words it is kept, so a plan is tuned six times at most.
  bool tuned_holds() const {
    uint32_t p = 1;  // tuned_words up to a power of two
    while (p < tuned_words) p *= 2;
    return tuned_gen == plan_gen && fsimb::tile_words(pats.W, 0) <= p;
  }
  // Times candidate shapes on a strided sample of tile 0's sweeps and keeps
  // the fastest in tuned_M / tuned_T (0: none fits shared memory).  Needs the
  // plan and the patterns on the device.
  void tune_shape(cudaStream_t s);
};

// Wraps a C ABI body: exceptions become status codes and (h)->err.
#define API_BEGIN(h)                                    \
  if (!(h)) return FSIMB_ERR_ARG;                       \
  try {
#define API_END(h)                                      \
  }                                                     \
  catch (const fsimb::ParseError& e) {                  \
    (h)->err = e.msg;                                   \
    return FSIMB_ERR_PARSE;                             \
  }                                                     \
  catch (const fsimb::CudaError& e) {                   \
    (h)->err = e.msg;                                   \
    return FSIMB_ERR_CUDA;                              \
  }                                                     \
  catch (const fsimb::LimitError& e) {                  \
    (h)->err = e.msg;                                   \
    return FSIMB_ERR_LIMIT;                             \
  }                                                     \
  catch (const fsimb::StateError& e) {                  \
    (h)->err = e.msg;                                   \
    return FSIMB_ERR_STATE;                             \
  }                                                     \
  catch (const fsimb::ArgError& e) {                    \
    (h)->err = e.msg;                                   \
    return FSIMB_ERR_ARG;                               \
  }                                                     \
  catch (const fsimb::IoError& e) {                     \
    (h)->err = e.msg;                                   \
    return FSIMB_ERR_IO;                                \
  }                                                     \
  catch (const std::bad_alloc&) {                       \
    (h)->err = "host allocation failed";                \
    return FSIMB_ERR_NOMEM;                             \
  }                                                     \
  catch (const std::exception& e) {                     \
    (h)->err = e.what();                                \
    return FSIMB_ERR_ARG;                               \
  }                                                     \
  (h)->err.clear();                                     \
  return FSIMB_OK;
