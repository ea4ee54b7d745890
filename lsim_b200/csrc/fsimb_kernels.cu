// B200 (sm_100a) kernels of the stuck-at fault simulator.
//
//   k_good         good machine: a CTA takes a few words through all levels.
//   k_good_level   the same, one launch per level, for very wide levels.
//   k_sweep<M>     persistent: each CTA pulls (sweep, M-word subtile) items from
//                  a device work counter and re-simulates the levels above the
//                  injection point with all live values in shared memory
//                  (slots, a bank-conflict-free order and a stream of gate
//                  records per CTA size laid out on the host).  Writes the OR
//                  over POs of (faulty ^ good) per word.
//   k_sweep_wide<M> the same sweep for circuits whose live values do not
//                  fit in shared memory: values in a per-CTA region of global
//                  memory indexed by element.
//   k_ffr          one warp per FFR root, lanes = the 32 words of a tile:
//                  backward critical-path tracing inside the FFR and the
//                  per-fault detection word, count and first pattern.
//   k_exact        the same epilogue for faults simulated by an exact sweep.
//   k_drop         fault dropping: warp-aggregated stream compaction of the
//                  roots / sweeps that still carry faults below the N-detect
//                  limit.
//
// Word semantics follow fsim/simulation.cpp: gates act on whole 64-bit words
// (fsim/simulation.cpp:979-1124), the last round keeps its high bits until
// the PO comparison masks them (fsim/simulation.cpp:94-102, 174-178), and a
// detecting bit b of round rd with `bits` valid bits is pattern
// rd*64 + bits-1-b.
#include "fsimb_kernels.cuh"

#include <algorithm>
#include <type_traits>

namespace fsimb {

namespace {

// Gate families: AND/OR/NAND/NOR/INV/CLKBUF/PO are io ^ AND(in ^ ii);
// XOR/XNOR are io ^ XOR(in).  Bit t of each mask is the property of type t.
constexpr uint32_t kIiMask = (1u << G_OR) | (1u << G_NOR);
constexpr uint32_t kIoMask = (1u << G_INV) | (1u << G_OR) | (1u << G_NAND) | (1u << G_XNOR);
constexpr uint32_t kXfMask = (1u << G_XOR) | (1u << G_XNOR);

__device__ __forceinline__ uint64_t bmask(uint32_t bit) { return 0ull - (uint64_t)bit; }

// Evaluates one word.  in[k] for k >= nf is ignored.
__device__ __forceinline__ uint64_t eval_word(uint32_t t, uint32_t nf, uint64_t a, uint64_t b,
                                              uint64_t c, uint64_t d) {
  if (t == G_MUX) {
    // (s & b) | (a & !s) with a logical not (fsim/simulation.cpp:1056)
    return (c & b) | (a & (uint64_t)(c == 0));
  }
  const uint64_t ii = bmask((kIiMask >> t) & 1u);
  const uint64_t io = bmask((kIoMask >> t) & 1u);
  const bool xf = (kXfMask >> t) & 1u;
  const uint64_t fill_ao = ~ii;
  if (nf < 2) b = xf ? 0ull : fill_ao;
  if (nf < 3) c = xf ? 0ull : fill_ao;
  if (nf < 4) d = xf ? 0ull : fill_ao;
  const uint64_t ao = (a ^ ii) & (b ^ ii) & (c ^ ii) & (d ^ ii);
  const uint64_t xo = a ^ b ^ c ^ d;
  return (xf ? xo : ao) ^ io;
}

__device__ __forceinline__ uint32_t round_bits(uint64_t P, uint32_t W, uint32_t w) {
  if (w >= W) return 0;
  return (P / (64ull * (w + 1))) ? 64u : (uint32_t)(P % 64);
}

__device__ __forceinline__ uint64_t bits_mask(uint32_t bits) {
  return bits >= 64 ? ~0ull : ((1ull << bits) - 1ull);
}

// (a ^ i) & b, and x & y or x ^ y by the mask k: one LOP3 each.
__device__ __forceinline__ uint32_t and_inv(uint32_t a, uint32_t i, uint32_t b) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0x28;" : "=r"(r) : "r"(a), "r"(i), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t and_or_xor(uint32_t x, uint32_t y, uint32_t k) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0x68;" : "=r"(r) : "r"(x), "r"(y), "r"(k));
  return r;
}

// ---------------------------------------------------------------- good
// V consecutive words (1 or 2) of a gate.
template <int V>
struct GoodWords {
  uint64_t v[4][V];
};
__device__ __forceinline__ uint32_t gate_type(const uint4& r) {
  return r.x >> 31 | r.y >> 31 << 1 | r.z >> 31 << 2 | r.w >> 31 << 3;
}
template <int V>
__device__ __forceinline__ GoodWords<V> good_inputs(const uint4& r, const uint64_t* g) {
  GoodWords<V> x;
  const uint32_t in[4] = {r.x & kNoInput, r.y & kNoInput, r.z & kNoInput, r.w & kNoInput};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint64_t* p = g + (uint64_t)in[k] * 32;
    const bool has = in[k] != kNoInput;
    if constexpr (V == 2) {
      const ulonglong2 q = has ? *reinterpret_cast<const ulonglong2*>(p) : make_ulonglong2(0, 0);
      x.v[k][0] = q.x;
      x.v[k][1] = q.y;
    } else {
      x.v[k][0] = has ? *p : 0ull;
    }
  }
  return x;
}
// AND and XOR families by masks, as 32-bit halves: a missing input is zeros,
// inverted in an AND; MUX by its own rule.
template <int V>
__device__ __forceinline__ void good_store(const uint4& r, const GoodWords<V>& x, uint64_t* p) {
  const uint32_t t = gate_type(r);
  uint64_t o[V];
  if (t == G_MUX) {
#pragma unroll
    for (int j = 0; j < V; ++j) o[j] = eval_word(t, 3, x.v[0][j], x.v[1][j], x.v[2][j], 0ull);
  } else {
    const uint32_t ii = 0u - ((kIiMask >> t) & 1u), io = 0u - ((kIoMask >> t) & 1u), kx = 0u - ((kXfMask >> t) & 1u);
    const uint32_t i1 = (r.y & kNoInput) == kNoInput ? ~kx : ii, i2 = (r.z & kNoInput) == kNoInput ? ~kx : ii,
                   i3 = (r.w & kNoInput) == kNoInput ? ~kx : ii;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      uint32_t h[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        auto half = [&](int k) { return (uint32_t)(x.v[k][j] >> (32 * q)); };
        uint32_t y = and_or_xor(half(0) ^ ii, half(1) ^ i1, kx);
        y = and_or_xor(y, half(2) ^ i2, kx);
        h[q] = and_or_xor(y, half(3) ^ i3, kx) ^ io;
      }
      o[j] = (uint64_t)h[0] | (uint64_t)h[1] << 32;
    }
  }
  if constexpr (V == 2)
    *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(o[0], o[1]);
  else
    *p = o[0];
}

// All levels of the words [w0, w0 + P) by one CTA: words are independent, so
// a level needs a barrier, not a launch.  A thread takes two words (one at P
// = 1) of an element, so P / 2 consecutive lanes share an element; a word
// beyond the patterns that shares a thread with the last one is computed
// from its zeros.  200,000 gates, 150 levels: 1,024 words 2.18 -> 0.95 ms (P =
// 8); 6,586 gates, 157 words 270 -> 57 us; 400 gates, one word 67 -> 14 us
// (P = 1), against one launch per level.
template <int P>
__device__ __forceinline__ void good_words(const GoodView& a, uint32_t w0) {
  constexpr int V = P == 1 ? 1 : 2, L = P / V;  // words per thread, lanes per element
  const uint32_t t = threadIdx.x / L, step = blockDim.x / L, w = w0 + threadIdx.x % L * V;
  const bool on = w < a.W;
  uint64_t* g = a.good + ((uint64_t)(w >> 5) * a.N) * 32 + (w & 31u);
  if (on)
    for (uint32_t e = t; e < a.n_pi; e += step)
#pragma unroll
      for (int j = 0; j < V; ++j) g[(uint64_t)e * 32 + j] = w + j < a.W ? a.pwords[(uint64_t)(w + j) * a.n_pi + e] : 0ull;
  __syncthreads();
  // Steps of U elements a thread: the next step's gate records (and the next
  // level's bound) are loaded before this step's words are waited for, so a
  // level costs the words' latency and a barrier.
  constexpr int U = 2;
  const uint4 none = make_uint4(kNoInput, kNoInput, kNoInput, kNoInput);
  auto bound = [&](uint32_t level) { return a.level_off[min(level, a.n_levels - 1) + 1]; };
  uint32_t l = 1, hi = bound(1), e = a.level_off[1] + t, hi1 = bound(2), hi2 = bound(3);
  uint4 q[U];
#pragma unroll
  for (int u = 0; u < U; ++u) q[u] = e + u * step < hi ? a.gates[e + u * step] : none;
  while (l < a.n_levels) {
    // the step after this one: (level, element) and its bound
    const bool last = e - t + U * step >= hi;  // the same for every thread of the CTA
    const uint32_t ne = last ? hi + t : e + U * step, nh = last ? hi1 : hi;
    if (last) {
      hi1 = hi2;
      hi2 = bound(l + 3);
    }
    uint4 nq[U];
#pragma unroll
    for (int u = 0; u < U; ++u) nq[u] = ne + u * step < nh ? a.gates[ne + u * step] : none;
    if (on && e < hi) {
      GoodWords<V> x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = good_inputs<V>(q[u], g);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (e + u * step < hi) good_store<V>(q[u], x[u], g + (uint64_t)(e + u * step) * 32);
    }
    if (last) {
      __syncthreads();
      ++l;
    }
    hi = nh;
    e = ne;
#pragma unroll
    for (int u = 0; u < U; ++u) q[u] = nq[u];
  }
}

template <int P>
__global__ void __launch_bounds__(1024) k_good(GoodView a) { good_words<P>(a, blockIdx.x * P); }

// One level of all words, for circuits whose levels are too wide for the
// words' CTAs to cover (launch_good): one thread per (element, word).
__global__ void k_good_level(GoodView a, uint32_t lo, uint32_t hi) {
  const uint64_t n = (uint64_t)(hi - lo) * a.W;
  for (uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
       idx += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t w = (uint32_t)(idx % a.W);
    const uint32_t e = lo + (uint32_t)(idx / a.W);
    uint64_t* g = a.good + ((uint64_t)(w >> 5) * a.N) * 32 + (w & 31u);
    if (e < a.n_pi) {
      g[(uint64_t)e * 32] = a.pwords[(uint64_t)w * a.n_pi + e];
    } else {
      const uint4 q = a.gates[e];
      good_store<1>(q, good_inputs<1>(q, g), g + (uint64_t)e * 32);
    }
  }
}

// ---------------------------------------------------------------- bounded wait
// (the wait test's only: the sweeps' barriers are the CTA's own)
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for the barrier's phase `parity` for at most limit_ns nanoseconds of
// the global timer (and at most 2^26 polls); false if it gave up, so the
// caller reports an error instead of hanging.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
  if (mbar_try(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  for (uint32_t it = 0; it < (1u << 26); ++it) {
    if (mbar_try(bar, parity)) return true;
    if (global_ns() - t0 > limit_ns) return false;
  }
  return false;
}

// Index of the last prefix entry <= x (prefix[0] = 0, n entries).
__device__ __forceinline__ uint32_t find_prefix(const unsigned long long* prefix, uint32_t n,
                                                unsigned long long x) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (prefix[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}

// ---------------------------------------------------------------- sweep
// Per-circuit pointers a sweep item reads (one circuit, one tile).
struct SweepView {
  const uint4* blob;       // record stream for this CTA size (fsimb_plan.h)
  const uint4* lvl;        // per level: its first record in the stream, its range in li
  const uint32_t* level;   // element -> level, or kFolded | consumer
  const uint32_t* li;      // (element, slot) pairs
  const uint32_t* fi_off;
  const uint32_t* fi_idx;
  const uint8_t* type;
  const uint64_t* good;    // tile [N][32]
  uint32_t max_gate_level;
  uint32_t stream_recs;
  uint32_t fix0;           // 16-byte offset of the fix entries in blob
  uint32_t inj_slot;       // the injection slot (the last one)
  uint32_t split;          // levels are ordered by kind
};

// Element x's word w of the tile with its input `pin` (any input that reads
// `from` when pin < 0) at v; the other inputs hold their good values.
template <class V>
__device__ __forceinline__ uint64_t eval_with(const V& a, uint32_t x, int pin, uint32_t from, uint64_t v,
                                              uint32_t w) {
  const uint8_t t = a.type[x];
  const uint32_t f0 = a.fi_off[x];
  uint32_t nf = a.fi_off[x + 1] - f0;
  if (t == G_INV || t == G_CLKBUF || t == G_PO) nf = 1;
  uint64_t in[4] = {0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if ((uint32_t)k < nf) {
      const uint32_t f = a.fi_idx[f0 + k];
      in[k] = k == pin || (pin < 0 && f == from) ? v : a.good[(uint64_t)f * 32 + w];
    }
  }
  return eval_word(t, nf, in[0], in[1], in[2], in[3]);
}

// Word w of the injection's stored element with the fault: the faulty word
// of inj.elem, taken up through the gates it is folded into (each has one
// consumer, whose other inputs are good).
template <class V>
__device__ __forceinline__ uint64_t inj_value(const V& a, const InjRec& inj, uint32_t w) {
  uint32_t x = inj.elem;
  if (!(inj.mode & kInjStuck)) return ~a.good[(uint64_t)x * 32 + w];
  const uint64_t sv = (inj.mode & kInjValue) ? ~0ull : 0ull;
  const uint32_t pin = inj.mode >> kInjPinShift;
  uint64_t v = pin ? eval_with(a, x, (int)pin - 1, 0u, sv, w) : sv;
  for (uint32_t lv = a.level[x]; lv & kFolded; lv = a.level[x]) {
    const uint32_t c = lv & ~kFolded;
    v = eval_with(a, c, -1, x, v, w);
    x = c;
  }
  return v;
}

// Chunk of a slot: 16 bytes, two words (one 8-byte word at M = 1), as 32-bit
// registers so that inversion masks are one register each.
template <int M>
struct Chunk {
  static constexpr int R = M == 1 ? 2 : 4;
  uint32_t r[R];
};
template <int M>
__device__ __forceinline__ Chunk<M> lds(uint32_t addr) {
  Chunk<M> c;
  if constexpr (M == 1)
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(c.r[0]), "=r"(c.r[1]) : "r"(addr));
  else
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(c.r[0]), "=r"(c.r[1]), "=r"(c.r[2]), "=r"(c.r[3])
                 : "r"(addr));
  return c;
}
// The same for a literal that may be absent (has == 0: zeros), without a
// branch: neighbouring records differ in their literal counts.
template <int M>
__device__ __forceinline__ Chunk<M> lds_if(uint32_t addr, uint32_t has) {
  Chunk<M> c;
  if constexpr (M == 1) {
    c.r[0] = c.r[1] = 0u;
    asm volatile("{ .reg .pred p; setp.ne.u32 p, %3, 0; @p ld.shared.v2.u32 {%0, %1}, [%2]; }"
                 : "+r"(c.r[0]), "+r"(c.r[1])
                 : "r"(addr), "r"(has));
  } else {
    c.r[0] = c.r[1] = c.r[2] = c.r[3] = 0u;
    asm volatile("{ .reg .pred p; setp.ne.u32 p, %5, 0; @p ld.shared.v4.u32 {%0, %1, %2, %3}, [%4]; }"
                 : "+r"(c.r[0]), "+r"(c.r[1]), "+r"(c.r[2]), "+r"(c.r[3])
                 : "r"(addr), "r"(has));
  }
  return c;
}
template <int M>
__device__ __forceinline__ void sts(uint32_t addr, const Chunk<M>& c) {
  if constexpr (M == 1)
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(c.r[0]), "r"(c.r[1]) : "memory");
  else
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(c.r[0]), "r"(c.r[1]), "r"(c.r[2]),
                 "r"(c.r[3])
                 : "memory");
}
// A record (fsimb_plan.h RecKind): two words, four at one word per item.
template <int M>
using RecWords = typename std::conditional<M == 1, uint4, uint2>::type;

// Byte offset of slot k of a record, to be masked by kOffMask: one shift.
// Chunk c of a lane's order is the slot's chunk (first ^ c), its offset
// (offset & mask) ^ (rot ^ 16c) with rot 16 bytes times the lane's first
// chunk: one LOP3; the slots' base address is left to the load.
template <int M>
struct SlotBits {
  static constexpr int kShift = M == 1 ? 3 : M == 2 ? 4 : M == 4 ? 5 : 6;  // 8 * M bytes a slot
  static constexpr uint32_t kOffMask = kRecSlot << kShift;
};
template <int M>
__device__ __forceinline__ uint32_t slot_off(const RecWords<M>& q, int k) {
  const uint32_t w = k < 2 ? q.x : q.y;
  if constexpr (M == 1) {
    const uint32_t h = k < 2 ? q.z : q.w;
    const int sh = 14 * (k & 1);
    return ((w >> sh & kRecSlot) | (h >> sh & kRecSlot) << 14) * 8u;
  } else {
    return (k & 1) ? w >> (14 - SlotBits<M>::kShift) : w << SlotBits<M>::kShift;
  }
}
template <int M>
__device__ __forceinline__ uint32_t chunk_at(uint32_t off, uint32_t rot, uint32_t c) {
  if constexpr (M == 1) return off;
  return (off & SlotBits<M>::kOffMask) ^ (rot ^ 16u * c);
}

// A cluster record on all M words.  vb: shared address of the slots.  Two
// chunks are in flight at a time.  KIND kRecNop: any AND or XOR, by masks.
template <int M, int KIND>
__device__ __forceinline__ void cluster_eval(uint32_t vb, uint32_t rot, const RecWords<M> q) {
  constexpr int C = (M >= 2) ? M / 2 : 1;
  constexpr int U = C >= 2 ? 2 : 1;
  constexpr int R = Chunk<M>::R;
  constexpr bool kAny = KIND == kRecNop;
  constexpr bool kThree = KIND == kRecAnd3 || KIND == kRecXor3;
  const uint32_t o0 = slot_off<M>(q, 0), o1 = slot_off<M>(q, 1), o2 = slot_off<M>(q, 2), oo = slot_off<M>(q, 3);
  const uint32_t i0 = (uint32_t)((int32_t)q.x >> 31), i1 = (uint32_t)((int32_t)(q.x << 1) >> 31);
  const uint32_t i2 = (uint32_t)((int32_t)(q.x << 2) >> 31), io = (uint32_t)((int32_t)(q.x << 3) >> 31);
  const uint32_t kind = (q.y >> kRecKindShift) & 7u;
  const uint32_t kx = kind >= kRecXor2 ? ~0u : 0u;
  static_assert(kRecAnd3 % 2 == 0 && kRecXor3 % 2 == 0 && kRecAnd2 % 2 == 1 && kRecXor2 % 2 == 1, "third literal");
#pragma unroll
  for (int c = 0; c < C; c += U) {
    Chunk<M> a[U], b[U], d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      a[u] = lds<M>(vb + chunk_at<M>(o0, rot, c + u));
      b[u] = lds<M>(vb + chunk_at<M>(o1, rot, c + u));
      if constexpr (kThree) d[u] = lds<M>(vb + chunk_at<M>(o2, rot, c + u));
      if constexpr (kAny) d[u] = lds_if<M>(vb + chunk_at<M>(o2, rot, c + u), ~kind & 1u);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        uint32_t x = a[u].r[r];
        if constexpr (kAny) {
          x = and_or_xor(and_or_xor(x ^ i0, b[u].r[r] ^ i1, kx), d[u].r[r] ^ i2, kx) ^ io;
        } else if constexpr (KIND == kRecXor2) {
          x = x ^ b[u].r[r] ^ io;
        } else if constexpr (KIND == kRecXor3) {
          x = x ^ b[u].r[r] ^ d[u].r[r];
          x ^= io;
        } else {
          x = and_inv(b[u].r[r], i1, x ^ i0);
          if constexpr (kThree) x = and_inv(d[u].r[r], i2, x);
          x ^= io;
        }
        a[u].r[r] = x;
      }
      sts<M>(vb + chunk_at<M>(oo, rot, c + u), a[u]);
    }
  }
}

// (s & b) | (a & !s) with a logical not of the whole 64-bit select word
// (fsim/simulation.cpp:1056).
template <int M>
__device__ __forceinline__ void mux_eval(uint32_t vb, uint32_t rot, const RecWords<M> q) {
  constexpr int C = (M >= 2) ? M / 2 : 1;
  const uint32_t o0 = slot_off<M>(q, 0), o1 = slot_off<M>(q, 1), o2 = slot_off<M>(q, 2), oo = slot_off<M>(q, 3);
#pragma unroll
  for (int c = 0; c < C; ++c) {
    Chunk<M> a = lds<M>(vb + chunk_at<M>(o0, rot, c));
    const Chunk<M> b = lds<M>(vb + chunk_at<M>(o1, rot, c)), s = lds<M>(vb + chunk_at<M>(o2, rot, c));
#pragma unroll
    for (int r = 0; r < Chunk<M>::R; r += 2) {
      const uint32_t not_s = (s.r[r] | s.r[r + 1]) == 0u;
      a.r[r] = (s.r[r] & b.r[r]) | (a.r[r] & not_s);
      a.r[r + 1] = s.r[r + 1] & b.r[r + 1];
    }
    sts<M>(vb + chunk_at<M>(oo, rot, c), a);
  }
}

// A wide record: its description d, runtime type.
template <int M>
__device__ __forceinline__ void wide_eval(uint32_t vb, const uint4* d) {
  constexpr int C = (M >= 2) ? M / 2 : 1;
  constexpr int VC = (M >= 2) ? 2 : 1;
  const uint4 f = d[0], g = d[1];
  const uint32_t t = g.y & 15u, nf = (g.y >> 4) & 15u;
#pragma unroll 1
  for (int c = 0; c < C; ++c) {
    const uint32_t vc = vb + 16u * c;
    Chunk<M> x = lds<M>(vc + 8u * M * f.x);
    const Chunk<M> i1 = lds_if<M>(vc + 8u * M * f.y, nf > 1), i2 = lds_if<M>(vc + 8u * M * f.z, nf > 2),
                   i3 = lds_if<M>(vc + 8u * M * f.w, nf > 3);
#pragma unroll
    for (int v = 0; v < VC; ++v) {
      auto word = [&](const Chunk<M>& k) { return (uint64_t)k.r[2 * v] | (uint64_t)k.r[2 * v + 1] << 32; };
      const uint64_t r = eval_word(t, nf, word(x), word(i1), word(i2), word(i3));
      x.r[2 * v] = (uint32_t)r;
      x.r[2 * v + 1] = (uint32_t)(r >> 32);
    }
    sts<M>(vc + 8u * M * g.x, x);
  }
}

// A direct PO record: the driver's words from its inputs, by masks as in
// good_store, against its good words.  A thread's chunk order is the
// clusters' (the lanes of a phase read different banks), so the lanes'
// words do not line up: each sets the bits that the CTA's words do not
// have yet, which after a few records is nearly none.  Bound by the inputs'
// shared-memory reads and the good words' latency: 20,000 drivers after six levels of
// 500 gates, 2,048 patterns, all stems 3.4 ms; every lane on the same chunk with
// po_eval's reduction 5.6 (four lanes of a phase on a bank); slots and PO records
// 11.0, at one word an item.
template <int M>
__device__ __forceinline__ void direct_eval(uint32_t vb, uint32_t rot, const uint4* d, const uint64_t* good_w0,
                                            uint32_t* acc) {
  constexpr int C = (M >= 2) ? M / 2 : 1;
  constexpr int R = Chunk<M>::R;
  const uint4 f = d[0], g = d[1];
  const uint32_t t = g.y & 15u, nf = (g.y >> 4) & 15u;
  const uint32_t ii = 0u - ((kIiMask >> t) & 1u), io = 0u - ((kIoMask >> t) & 1u), kx = 0u - ((kXfMask >> t) & 1u);
  const uint32_t i1 = nf > 1 ? ii : ~kx, i2 = nf > 2 ? ii : ~kx, i3 = nf > 3 ? ii : ~kx;
  const uint64_t* good_row = good_w0 + (uint64_t)g.x * 32;
#pragma unroll 1
  for (int c = 0; c < C; ++c) {
    const uint32_t o = M == 1 ? 0u : rot ^ 16u * c, vc = vb + o;  // o: the chunk's bytes in its slot
    Chunk<M> w;
    if constexpr (M == 1) {
      const uint2 q = *reinterpret_cast<const uint2*>(good_row);
      w.r[0] = q.x, w.r[1] = q.y;
    } else {
      const uint4 q = *reinterpret_cast<const uint4*>(good_row + o / 8);
      w.r[0] = q.x, w.r[1] = q.y, w.r[2] = q.z, w.r[3] = q.w;
    }
    const Chunk<M> x0 = lds<M>(vc + 8u * M * f.x), x1 = lds_if<M>(vc + 8u * M * f.y, nf > 1),
                   x2 = lds_if<M>(vc + 8u * M * f.z, nf > 2), x3 = lds_if<M>(vc + 8u * M * f.w, nf > 3);
    uint32_t any = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      uint32_t x;
      if (t == G_MUX) {
        const uint32_t not_s = (x2.r[r & ~1] | x2.r[r | 1]) == 0u;
        x = (x2.r[r] & x1.r[r]) | (r & 1 ? 0u : x0.r[r] & not_s);
      } else {
        x = and_or_xor(and_or_xor(x0.r[r] ^ ii, x1.r[r] ^ i1, kx), x2.r[r] ^ i2, kx);
        x = and_or_xor(x, x3.r[r] ^ i3, kx) ^ io;
      }
      w.r[r] ^= x;
      any |= w.r[r];
    }
    if (any) {
      volatile uint32_t* at = acc + o / 4;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (w.r[r] & ~at[r]) atomicOr(acc + o / 4 + r, w.r[r]);
    }
  }
}

// A PO record: the driver's difference from its good words, to the CTA's
// words in shared memory by one atomic per warp and 32-bit half (registers
// for them would cost every other record).
template <int M>
__device__ __forceinline__ void po_eval(uint32_t vb, const RecWords<M> q, const uint64_t* good_w0, uint32_t* acc) {
  constexpr int C = (M >= 2) ? M / 2 : 1;
  const unsigned lanes = __activemask();
  const bool leader = (threadIdx.x & 31u) == (uint32_t)(__ffs(lanes) - 1);
  const uint32_t o = slot_off<M>(q, 3);
  const uint64_t* good_row = good_w0 + (uint64_t)q.x * 32;
#pragma unroll
  for (int c = 0; c < C; ++c) {  // every lane the same chunk: the lanes' words line up
    Chunk<M> x = lds<M>(vb + chunk_at<M>(o, 0u, c)), g;
    if constexpr (M == 1) {
      const uint2 w = *reinterpret_cast<const uint2*>(good_row);
      g.r[0] = w.x, g.r[1] = w.y;
    } else {
      const uint4 w = *reinterpret_cast<const uint4*>(good_row + 2 * c);
      g.r[0] = w.x, g.r[1] = w.y, g.r[2] = w.z, g.r[3] = w.w;
    }
#pragma unroll
    for (int r = 0; r < Chunk<M>::R; ++r) {
      const uint32_t diff = __reduce_or_sync(lanes, x.r[r] ^ g.r[r]);
      if (leader && diff) atomicOr(acc + 4 * c + r, diff);
    }
  }
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

template <int M, bool D>
__device__ __forceinline__ void record_eval(uint32_t vb, uint32_t rot, bool split, const RecWords<M> q,
                                            const uint4* blob, const uint64_t* good_w0, uint32_t* acc) {
  const uint32_t kind = (q.y >> kRecKindShift) & 7u;
  if (kind >= kRecMux) {
    if (kind == kRecMux)
      mux_eval<M>(vb, rot, q);
    else if (D && kind == kRecPo && (q.x & kPoDirect))
      direct_eval<M>(vb, rot, blob + (q.x & ~kPoDirect), good_w0, acc);
    else if (kind == kRecPo)
      po_eval<M>(vb, q, good_w0, acc);
    else
      wide_eval<M>(vb, blob + q.x);
  } else if (kind == kRecNop) {  // padding
  } else if (!split) {
    cluster_eval<M, kRecNop>(vb, rot, q);
  } else if (kind == kRecAnd3) {  // records are in kind order, so a warp mostly takes one path
    cluster_eval<M, kRecAnd3>(vb, rot, q);
  } else if (kind == kRecAnd2) {
    cluster_eval<M, kRecAnd2>(vb, rot, q);
  } else if (kind == kRecXor3) {
    cluster_eval<M, kRecXor3>(vb, rot, q);
  } else {
    cluster_eval<M, kRecXor2>(vb, rot, q);
  }
}

// A CTA of one warp needs no barrier between levels, only the warp's order.
__device__ __forceinline__ void cta_sync() {
  if (blockDim.x == 32)
    __syncwarp();
  else
    __syncthreads();
}

// M words per item, one thread per record holding all M words.  Slots are
// M*8 bytes; a thread reads a slot as C = M/2 16-byte chunks (one 8-byte word
// for M = 1).  The host orders each level in groups of G = 16/M consecutive
// positions whose slots have distinct residues mod G (for every literal and
// the output), and packs them so that within a phase of 8 lanes (16 for M =
// 1) lane l takes position (l % C) * G + l / C; with chunk (l % C) ^ i at step
// i the 8 chunks a phase touches lie in 8 different bank quads: the loads
// and stores of a sweep are free of bank conflicts wherever the host found
// such groups.
//
// A thread reads its records straight from global memory (L1 / L2), kAhead
// rounds ahead: the stream is padded per level to rounds of one record per
// thread, so the next address is one addition away and a level's end is a
// bit of its last round's records.
//
// One item: the levels above the injection element for M words starting at
// word w0 of the tile; writes the OR of PO differences to out_row[w0..w0+M).
template <int M, bool D>
__device__ __forceinline__ void sweep_item(uint64_t* vals, unsigned long long* acc, const SweepView& v,
                                           const InjRec inj, uint32_t w0, uint64_t* out_row) {
  constexpr int C = (M >= 2) ? M / 2 : 1;   // chunks per slot
  constexpr int PH = (M == 1) ? 16 : 8;     // lanes per shared-memory phase
  const int tid = threadIdx.x, nth = blockDim.x;
  const int pl = tid & (PH - 1);
  const uint32_t vb = smem_u32(vals), rot = 16u * ((uint32_t)pl % C);
  const uint32_t x = inj.stored;
  const uint4 lv = v.lvl[inj.level];
  if (tid < M) {
    acc[tid] = 0ull;
    if (inj.mode & kInjReachesPo) acc[tid] = inj_value(v, inj, w0 + tid) ^ v.good[(uint64_t)x * 32 + w0 + tid];
  }
  const uint32_t first = inj.level <= v.max_gate_level ? lv.x : v.stream_recs;
  if (first < v.stream_recs) {
    const RecWords<M>* rp = reinterpret_cast<const RecWords<M>*>(v.blob) + first + tid;
    // Three rounds at M = 4, the shape of large circuits: 100,000 gates 11.84 ->
    // 11.75 ms, 200,000 gates 341.5 -> 336.4; four 11.67 and 335.3, but 30,000
    // gates 2.90 -> 2.95.  At M = 8 three cost 6 % (6,586 gates) to 23 % (small).
    constexpr int kAhead = M == 4 ? 3 : 2;
    static_assert(kAhead <= (int)kPrefetch, "the stream's padding");
    RecWords<M> q[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j, rp += nth) q[j] = *rp;
    // Values live at the start level come from the good machine (copied
    // asynchronously, four list entries in flight per thread), except the
    // injection element itself.
    const uint32_t i1 = lv.z;
    const uint2* li = reinterpret_cast<const uint2*>(v.li);
    for (uint32_t i = lv.y + tid; i < i1; i += 4 * nth) {
      uint2 es[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) es[j] = (i + j * nth < i1) ? li[i + j * nth] : make_uint2(0xFFFFFFFFu, 0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (es[j].x == 0xFFFFFFFFu) continue;
        uint64_t* dst = vals + (size_t)es[j].y * M;
        if (es[j].x == x) {
#pragma unroll 1
          for (int m = 0; m < M; ++m) dst[m] = inj_value(v, inj, w0 + m);
        } else {
          const uint64_t* src = v.good + (uint64_t)es[j].x * 32 + w0;
          if constexpr (M == 1) {
            cp_async8(dst, src);
          } else {
#pragma unroll
            for (int q = 0; q < M / 2; ++q) cp_async16(dst + 2 * q, src + 2 * q);
          }
        }
      }
    }
    // A flip of an alias goes to the injection slot, which the fix entries
    // of its list read after their levels.
    const uint4* fx = nullptr;
    uint32_t fix_at = 0xFFFFFFFFu;
    if (inj.fix) {
      fx = v.blob + v.fix0 + 2 * (size_t)(inj.fix - 1);
      fix_at = fx[1].x;
      if (tid < M)
        vals[(size_t)v.inj_slot * M + tid] =
            inj_value(v, inj, w0 + tid) ^ ((inj.mode & kInjAliasInv) ? ~0ull : 0ull);
    }
    cp_async_wait_all();
    cta_sync();
    const uint64_t* good_w0 = v.good + w0;
    uint32_t* acc32 = reinterpret_cast<uint32_t*>(acc);
    auto round = [&](const RecWords<M> q, uint32_t at) {
      record_eval<M, D>(vb, rot, v.split, q, v.blob, good_w0, acc32);
      if (q.y & kRecEnd) {
        cta_sync();
        if (at == fix_at) {
          const uint32_t n = fx[1].y;
          for (uint32_t i = tid; i < n; i += nth)
            record_eval<M, D>(vb, rot, v.split, *reinterpret_cast<const RecWords<M>*>(fx + 2 * i), v.blob, good_w0,
                           acc32);
          fx += 2 * n;
          fix_at = fx[1].x;
          cta_sync();
        }
      }
    };
    // kAhead rounds a turn, so that a record's registers are loaded again
    // only after its evaluation and nothing waits for a load early.
    for (uint32_t at = first;;) {
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        round(q[j], at);
        q[j] = *rp;
        rp += nth;
        at += nth;
        if (at >= v.stream_recs) goto done;
      }
    }
  done:;
  }
  cta_sync();
  if (tid < M) out_row[w0 + tid] = acc[tid];
}

// Test hook of the error word: a wait on a barrier that nothing completes runs
// out and the launch reports it.  Nothing else in a sweep waits on an mbarrier.
__device__ __forceinline__ void sweep_wait_test(uint64_t* bar, uint64_t wait_ns, int* err) {
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    if (!mbar_wait(bar, 0, wait_ns)) atomicExch(err, 1);
  }
}

// Register caps: 1,024 threads an SM at up to 4 words per item.  D: the stream
// has direct PO records (their code beside the others costs every sweep 1 to
// 3 %: 50,000 gates 53.5 -> 55.1 ms).
template <int M, bool D>
__global__ void __maxnreg__(64) k_sweep(SweepArgs a) {
  extern __shared__ __align__(128) uint64_t vals[];  // [max_live][M]
  __shared__ unsigned long long acc[M];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t s_item;
  if (a.wait_test && blockIdx.x == 0) {
    sweep_wait_test(&bar, a.wait_ns, a.err);
    return;
  }
  // Items are (tile, sweep, subtile), tile-major.  Only subtiles that hold
  // pattern words: the last tile of a block is rarely full (16 words of 32
  // for 1,000 patterns), and the tracing masks the others.
  constexpr uint32_t subtiles = kTileWords / M;
  const uint32_t last_sub = (a.n_words + M - 1) / M;
  const uint32_t per_tile = a.n_list * subtiles;
  const uint32_t n_items = (a.n_tiles - 1) * per_tile + a.n_list * last_sub;
  // The next item's number is asked for while the current one runs.
  uint32_t next = blockIdx.x;
  for (;;) {
    if (threadIdx.x == 0) {
      s_item = next;
      next = gridDim.x + (uint32_t)atomicAdd(a.queue, 1);
    }
    cta_sync();
    const uint32_t item = s_item;
    if (item >= n_items) return;
    const uint32_t tile = min(item / per_tile, a.n_tiles - 1);
    const uint32_t rem = item - tile * per_tile;
    const uint32_t sub = tile == a.n_tiles - 1 ? last_sub : subtiles;
    const uint32_t li = rem / sub;
    const uint32_t w0 = (rem % sub) * M;
    const uint32_t si = a.list ? a.list[li] : li;
    const SweepView v{a.blob, a.lvl, a.level, a.li, a.fi_off, a.fi_idx, a.type,
                      a.good + (uint64_t)tile * a.N * 32,
                      a.max_gate_level, a.stream_recs, a.fix0, a.inj_slot, a.split};
    sweep_item<M, D>(vals, acc, v, a.inj[si], w0, a.out + ((uint64_t)tile * a.n_sweeps + si) * 32);
  }
}

// Batch form: the circuits of one launch, each with its own work counter.
// Every CTA walks the circuits in order and takes (tile, sweep, subtile)
// items of each until its counter runs out, so items are consumed in
// circuit order as from one queue.  The loop index is uniform and the
// circuit fields come from the kernel parameters: the compiler keeps the
// pointers in uniform registers, as for k_sweep.
template <int M, bool D>
__global__ void __maxnreg__(64) k_sweep_batch(const __grid_constant__ BatchSweepParams p) {
  extern __shared__ __align__(128) uint64_t vals[];
  __shared__ unsigned long long acc[M];
  __shared__ uint32_t s_item;
  constexpr uint32_t subtiles = kTileWords / M;
  for (uint32_t ci = 0; ci < p.n_circ; ++ci) {
    const SweepCirc& c = p.c[ci];
    const uint32_t per_tile = c.n_sweeps * subtiles;
    // The next item's number is asked for while the current one runs.
    unsigned long long next = threadIdx.x == 0 ? atomicAdd(p.queue + ci, 1ull) : 0ull;
    for (;;) {
      if (threadIdx.x == 0) {
        s_item = next < c.n_items ? (uint32_t)next : 0xFFFFFFFFu;
        if (next < c.n_items) next = atomicAdd(p.queue + ci, 1ull);
      }
      cta_sync();
      const uint32_t item = s_item;
      if (item == 0xFFFFFFFFu) {
        cta_sync();  // s_item is written for the next circuit only after all have read it
        break;
      }
      // The last tile has items only for the subtiles that hold pattern words.
      const uint32_t tile = min(item / per_tile, c.tiles - 1);
      const uint32_t rem = item - tile * per_tile;
      const uint32_t sub = tile == c.tiles - 1 ? c.last_sub : subtiles;
      const uint32_t si = rem / sub;
      const uint32_t w0 = (rem % sub) * M;
      const SweepView v{c.blob, c.lvl, c.level, c.li, c.fi_off, c.fi_idx, c.type,
                        c.good + (uint64_t)tile * c.N * 32, c.max_gate_level, c.stream_recs, c.fix0, c.inj_slot, c.split};
      sweep_item<M, D>(vals, acc, v, c.inj[si], w0, c.out + ((uint64_t)tile * c.n_sweeps + si) * 32);
    }
  }
}

// ---------------------------------------------------------------- wide circuits
// Sweep for circuits whose live values do not fit in shared memory: every
// CTA keeps the values of its item in its own region of global memory,
// indexed by element (gvals + block * N * M), which L2 mostly holds.  A
// fanin below the start level other than the injection element reads the
// good machine directly, so an item starts without copying live values.
// Threads take (element, word) pairs of a level; one barrier per level.
template <int M>
__global__ void __launch_bounds__(1024) k_sweep_wide(SweepWideArgs a) {
  __shared__ unsigned long long acc[M];
  __shared__ uint32_t s_item;
  uint64_t* gv = a.gvals + (size_t)blockIdx.x * a.N * M;
  const uint32_t tid = threadIdx.x, nth = blockDim.x;
  const uint32_t m = tid % M, step = nth / M;
  const uint32_t subtiles = (a.n_words + M - 1) / M;  // those that hold pattern words
  const uint32_t n_items = a.n_list * subtiles;
  for (;;) {
    if (tid == 0) s_item = atomicAdd(a.queue, 1);
    __syncthreads();
    const uint32_t item = s_item;
    __syncthreads();
    if (item >= n_items) return;
    const uint32_t li = item / subtiles;
    const uint32_t w0 = (item % subtiles) * M;
    const uint32_t si = a.list ? a.list[li] : li;
    const InjRec inj = a.inj[si];
    const uint32_t x = inj.stored;
    const uint32_t L0 = a.level[x] + 1;
    const uint32_t lo0 = L0 <= a.max_gate_level ? a.level_off[L0] : 0;
    if (tid < M) {
      const uint64_t fv = inj_value(a, inj, w0 + tid);
      gv[(size_t)x * M + tid] = fv;
      acc[tid] = (inj.mode & kInjReachesPo) ? fv ^ a.good[(uint64_t)x * 32 + w0 + tid] : 0ull;
    }
    __syncthreads();
    uint64_t pacc = 0;
    const uint32_t w = w0 + m;
    for (uint32_t L = L0; L <= a.max_gate_level; ++L) {
      const uint32_t lo = a.level_off[L], hi = a.level_off[L + 1];
      for (uint32_t e = lo + tid / M; e < hi; e += step) {
        const uint8_t fl = a.eflag[e];
        if (!(fl & 1u)) continue;
        const uint8_t t = a.type[e];
        const uint32_t f0 = a.fi_off[e];
        uint32_t nf = a.fi_off[e + 1] - f0;
        if (t == G_INV || t == G_CLKBUF || t == G_PO) nf = 1;
        uint64_t in[4] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if ((uint32_t)q < nf) {
            const uint32_t f = a.fi_idx[f0 + q];
            in[q] = (f < lo0 && f != x) ? a.good[(uint64_t)f * 32 + w] : gv[(size_t)f * M + m];
          }
        }
        const uint64_t r = eval_word(t, nf, in[0], in[1], in[2], in[3]);
        gv[(size_t)e * M + m] = r;
        if (fl & 2u) pacc |= r ^ a.good[(uint64_t)e * 32 + w];
      }
      __syncthreads();
    }
    if (pacc) atomicOr(&acc[m], (unsigned long long)pacc);
    __syncthreads();
    if (tid < M) a.out[(uint64_t)si * 32 + w0 + tid] = acc[tid];
  }
}

// ---------------------------------------------------------------- FFR tracing
// Bits where flipping input `pin` of element p flips p's output, for bitwise
// gate types (MUX never reaches this path).
template <class V>
__device__ __forceinline__ uint64_t local_sens(const V& a, uint32_t p, uint32_t pin, uint32_t lane) {
  const uint8_t t = a.type[p];
  if (t == G_XOR || t == G_XNOR) return ~0ull;
  if (t == G_INV || t == G_CLKBUF || t == G_PO) return pin == 0 ? ~0ull : 0ull;
  if (t == G_MUX || t == G_PI) return 0ull;
  const bool orf = (t == G_OR || t == G_NOR);
  const uint32_t f0 = a.fi_off[p], f1 = a.fi_off[p + 1];
  uint64_t s = ~0ull;
  for (uint32_t k = f0; k < f1; ++k) {
    if (k - f0 == pin) continue;
    const uint64_t g = a.good[(uint64_t)a.fi_idx[k] * 32 + lane];
    s &= orf ? ~g : g;
  }
  return s;
}

__device__ __forceinline__ void record(unsigned long long* count, unsigned long long* first,
                                       uint8_t* lastflag, uint32_t f, uint64_t D, uint32_t w,
                                       uint32_t bits, uint32_t W, uint32_t lane) {
  const unsigned ball = __ballot_sync(0xFFFFFFFFu, D != 0ull);
  const unsigned cnt = __reduce_add_sync(0xFFFFFFFFu, (unsigned)__popcll(D));
  if (ball) {
    const int fl = __ffs(ball) - 1;
    if ((int)lane == fl) {
      // lowest pattern index in the lowest detecting word: highest set bit
      const unsigned long long idx =
          (unsigned long long)w * 64ull + bits - 64ull + (unsigned long long)__clzll((long long)D);
      atomicMin(&first[f], idx);
      atomicAdd(&count[f], (unsigned long long)cnt);
    }
  }
  if (w == W - 1) lastflag[f] = D != 0ull;
}

// What tracing reads of one circuit's tile.
struct FfrView {
  const MemberRec* members;
  const TracedRec* traced;
  const uint32_t* traced_slot;
  const uint32_t* fi_off;
  const uint32_t* fi_idx;
  const uint8_t* type;
  const uint64_t* good;      // tile [N][32]
  const uint64_t* obs;       // tile [n_sweeps][32]
  uint64_t* sens;            // tile [n_slots][32]: slot i = members[i], then the roots
  unsigned long long* count;
  unsigned long long* first;
  uint8_t* lastflag;
  uint64_t P;
  uint32_t W, tile;
  uint32_t drop_at;          // skip faults whose count reached this (0: none)
};

// One FFR on one tile by one warp, lanes = words.
__device__ __forceinline__ void ffr_root(const FfrView& a, const RootRec& rr, uint32_t lane) {
  const uint32_t w = a.tile * 32 + lane;
  const uint32_t bits = round_bits(a.P, a.W, w);
  uint64_t obs = rr.obs == kObsOne ? ~0ull : rr.obs == kObsZero ? 0ull : a.obs[(uint64_t)rr.obs * 32 + lane];
  obs &= bits_mask(bits);
  a.sens[(uint64_t)rr.slot * 32 + lane] = ~0ull;
  for (uint32_t i = rr.mem_begin; i < rr.mem_end; ++i) {
    const MemberRec m = a.members[i];
    a.sens[(uint64_t)i * 32 + lane] = a.sens[(uint64_t)m.p_slot * 32 + lane] & local_sens(a, m.p, m.pin, lane);
  }
  for (uint32_t i = rr.flt_begin; i < rr.flt_end; ++i) {
    const TracedRec tr = a.traced[i];
    if (a.drop_at && a.count[tr.fault] >= a.drop_at) continue;  // dropped after an earlier tile
    uint64_t s = a.sens[(uint64_t)a.traced_slot[i] * 32 + lane], gv;
    if (tr.pin == 0) {
      gv = a.good[(uint64_t)tr.elem * 32 + lane];
    } else {
      s &= local_sens(a, tr.elem, tr.pin - 1, lane);
      gv = a.good[(uint64_t)a.fi_idx[a.fi_off[tr.elem] + tr.pin - 1] * 32 + lane];
    }
    const uint64_t D = s & (gv ^ (tr.value ? ~0ull : 0ull)) & obs;
    record(a.count, a.first, a.lastflag, tr.fault, D, w, bits, a.W, lane);
  }
}

// One warp per (tile, root).
__global__ void __launch_bounds__(256) k_ffr(FfrArgs a) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t unit = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (unit >= (uint64_t)a.n_list * a.n_tiles) return;
  const uint32_t t = (uint32_t)(unit / a.n_list), i = (uint32_t)(unit % a.n_list);
  const FfrView v{a.members, a.traced, a.traced_slot, a.fi_off, a.fi_idx, a.type,
                  a.good + (uint64_t)t * a.N * 32, a.obs + (uint64_t)t * a.n_sweeps * 32,
                  a.sens + (uint64_t)t * a.n_slots * 32, a.count, a.first, a.lastflag, a.P, a.W, a.tile + t,
                  a.drop ? a.n_detect : 0u};
  ffr_root(v, a.roots[a.list ? a.list[i] : i], lane);
}

// One warp per (tile, exact fault).
__global__ void __launch_bounds__(256) k_exact(ExactArgs a) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t unit = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (unit >= (uint64_t)a.n_exact * a.n_tiles) return;
  const uint32_t t = (uint32_t)(unit / a.n_exact), i = (uint32_t)(unit % a.n_exact);
  const uint32_t j = a.list ? a.list[i] : i;
  const uint32_t f = a.exact_fault[j];
  if (a.drop && a.count[f] >= a.n_detect) return;  // dropped after an earlier tile
  const uint32_t w = (a.tile + t) * 32 + lane;
  const uint32_t bits = round_bits(a.P, a.W, w);
  const uint64_t D = a.out[((uint64_t)t * a.n_sweeps + a.first_sweep + j) * 32 + lane] & bits_mask(bits);
  record(a.count, a.first, a.lastflag, f, D, w, bits, a.W, lane);
}

// ---------------------------------------------------------------- batches
// One CTA per (circuit, kGoodBatchWords words) of the batch.
__global__ void __launch_bounds__(256) k_good_batch(BatchUnits u) {
  const uint32_t ci = find_prefix(u.unit_prefix, u.n_circ, blockIdx.x);
  const BatchCirc& c = u.circs[ci];
  const GoodView v{c.gates, c.level_off, c.pwords, c.good, c.n_pi, c.N, c.n_levels,
                   min(c.W, c.tiles * kTileWords)};
  good_words<kGoodBatchWords>(v, (uint32_t)(blockIdx.x - u.unit_prefix[ci]) * kGoodBatchWords);
}

// One warp per (circuit, tile, root).
__global__ void __launch_bounds__(256) k_ffr_batch(BatchUnits u, unsigned long long n_units) {
  const uint32_t lane = threadIdx.x & 31u;
  const unsigned long long unit = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (unit >= n_units) return;
  const uint32_t ci = find_prefix(u.unit_prefix, u.n_circ, unit);
  const BatchCirc& c = u.circs[ci];
  const unsigned long long local = unit - u.unit_prefix[ci];
  const uint32_t tile = (uint32_t)(local / c.n_roots);
  const FfrView v{c.members, c.traced, c.traced_slot, c.fi_off, c.fi_idx, c.type,
                  c.good + (uint64_t)tile * c.N * 32, c.out + (uint64_t)tile * c.n_sweeps * 32,
                  c.sens + (uint64_t)tile * c.n_slots * 32, c.count, c.first, c.lastflag, c.P, c.W, tile, 0u};
  ffr_root(v, c.roots[(uint32_t)(local % c.n_roots)], lane);
}

// One warp per (circuit, tile, exact fault).
__global__ void __launch_bounds__(256) k_exact_batch(BatchUnits u, unsigned long long n_units) {
  const uint32_t lane = threadIdx.x & 31u;
  const unsigned long long unit = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (unit >= n_units) return;
  const uint32_t ci = find_prefix(u.unit_prefix, u.n_circ, unit);
  const BatchCirc& c = u.circs[ci];
  const unsigned long long local = unit - u.unit_prefix[ci];
  const uint32_t tile = (uint32_t)(local / c.n_exact);
  const uint32_t j = (uint32_t)(local % c.n_exact);
  const uint32_t w = tile * 32 + lane;
  const uint32_t bits = round_bits(c.P, c.W, w);
  const uint64_t D = c.out[((uint64_t)tile * c.n_sweeps + c.n_stem_sweeps + j) * 32 + lane] & bits_mask(bits);
  record(c.count, c.first, c.lastflag, c.exact_fault[j], D, w, bits, c.W, lane);
}

// Counters of a run before its first tile; n_zero control words.
__global__ void k_init_results(unsigned long long* count, unsigned long long* first, uint8_t* lastflag, uint32_t F,
                               int* zero, uint32_t n_zero) {
  const uint32_t stride = gridDim.x * blockDim.x, i0 = blockIdx.x * blockDim.x + threadIdx.x;
  for (uint32_t i = i0; i < F; i += stride) {
    count[i] = 0ull;
    first[i] = ~0ull;
    lastflag[i] = 0;
  }
  for (uint32_t i = i0; i < n_zero; i += stride) zero[i] = 0;
}

// The caller's result records (32 bytes: flags, first pattern, count, last
// round) in one array with the error word behind it: one copy to
// page-locked memory instead of four to pageable memory and a host loop over
// the faults (400 gates: 51 -> 17 us after the last kernel; 738,943
// faults: 0.82 + 4.6 -> 0.43 ms).
__global__ void k_results(ResultArgs a) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < a.F) {
    const unsigned long long n = a.count[i], f = a.first[i];
    const unsigned long long flags = (n ? 1ull : 0ull) | (a.any_rounds && a.lastflag[i] ? 256ull : 0ull);
    a.out[2 * (size_t)i] = make_ulonglong2(flags, f);  // ~0: none, as -1
    a.out[2 * (size_t)i + 1] = make_ulonglong2(n, a.last_rd);
  } else if (i == a.F) {
    a.out[2 * (size_t)a.F] = make_ulonglong2((unsigned long long)*a.err, 0ull);
  }
}

// One round's good words of all elements, masked to its valid bits, in one
// array (the tile's rows are 256 bytes apart).
__global__ void k_round(const uint64_t* good, uint32_t N, uint64_t mask, uint64_t* out) {
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < N; e += gridDim.x * blockDim.x)
    out[e] = good[(uint64_t)e * 32] & mask;
}

// Keeps the roots that still carry an undetected traced fault and emits the
// sweep each of them needs; keeps undetected exact faults and their sweeps.
// Warp-aggregated appends: one atomic per warp and output list.
__global__ void k_drop(DropArgs a) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31u;
  const unsigned lt = (1u << lane) - 1u;
  const bool root_part = i < a.n_in_pad;  // uniform per warp (n_in_pad % 32 == 0)
  bool keep = false, sweep = false;
  uint32_t id = 0, sw = 0;
  if (root_part) {
    if (i < a.n_in) {
      id = a.in_list ? a.in_list[i] : i;
      const RootRec rr = a.roots[id];
      for (uint32_t k = rr.flt_begin; k < rr.flt_end && !keep; ++k)
        keep = a.count[a.traced[k].fault] < a.n_detect;
      sweep = keep && rr.obs != kObsOne && rr.obs != kObsZero;
      sw = rr.obs;
    }
  } else {
    const uint32_t j = i - a.n_in_pad;
    if (j < a.n_exact_in) {
      id = a.exact_in ? a.exact_in[j] : j;
      keep = a.count[a.exact_fault[id]] < a.n_detect;
      sweep = keep;
      sw = a.first_exact_sweep + id;
    }
  }
  const unsigned bk = __ballot_sync(0xFFFFFFFFu, keep);
  const unsigned bs = __ballot_sync(0xFFFFFFFFu, sweep);
  uint32_t base_k = 0, base_s = 0;
  if (lane == 0) {
    if (bk) base_k = atomicAdd(&a.n_out[root_part ? 0 : 2], (uint32_t)__popc(bk));
    if (bs) base_s = atomicAdd(&a.n_out[1], (uint32_t)__popc(bs));
  }
  base_k = __shfl_sync(0xFFFFFFFFu, base_k, 0);
  base_s = __shfl_sync(0xFFFFFFFFu, base_s, 0);
  if (keep) (root_part ? a.out_roots : a.out_exact)[base_k + __popc(bk & lt)] = id;
  if (sweep) a.out_sweeps[base_s + __popc(bs & lt)] = sw;
}

}  // namespace

void launch_good_batch(const BatchUnits& u, unsigned long long n_units, cudaStream_t s) {
  if (!n_units) return;
  k_good_batch<<<(unsigned)n_units, 256, 0, s>>>(u);
}

void launch_ffr_batch(const BatchUnits& u, unsigned long long n_units, cudaStream_t s) {
  if (!n_units) return;
  k_ffr_batch<<<(unsigned)((n_units * 32 + 255) / 256), 256, 0, s>>>(u, n_units);
}

void launch_exact_batch(const BatchUnits& u, unsigned long long n_units, cudaStream_t s) {
  if (!n_units) return;
  k_exact_batch<<<(unsigned)((n_units * 32 + 255) / 256), 256, 0, s>>>(u, n_units);
}

void launch_init_results_batch(unsigned long long* count, unsigned long long* first, uint8_t* lastflag,
                               uint64_t F, cudaStream_t s) {
  if (!F) return;
  const uint64_t blocks = std::min<uint64_t>((F + 255) / 256, 4096);
  k_init_results<<<(unsigned)blocks, 256, 0, s>>>(count, first, lastflag, (uint32_t)std::min<uint64_t>(F, 0xFFFFFFFFull),
                                                  nullptr, 0);
}

// The sweep kernels at M words per item, without and with direct records.
using SweepFn = void (*)(SweepArgs);
using SweepBatchFn = void (*)(BatchSweepParams);
static SweepFn sweep_fn(int M, bool direct) {
  switch (M) {
    case 1: return direct ? k_sweep<1, true> : k_sweep<1, false>;
    case 2: return direct ? k_sweep<2, true> : k_sweep<2, false>;
    case 4: return direct ? k_sweep<4, true> : k_sweep<4, false>;
    case 8: return direct ? k_sweep<8, true> : k_sweep<8, false>;
  }
  return nullptr;
}
static SweepBatchFn sweep_batch_fn(int M, bool direct) {
  switch (M) {
    case 1: return direct ? k_sweep_batch<1, true> : k_sweep_batch<1, false>;
    case 2: return direct ? k_sweep_batch<2, true> : k_sweep_batch<2, false>;
    case 4: return direct ? k_sweep_batch<4, true> : k_sweep_batch<4, false>;
    case 8: return direct ? k_sweep_batch<8, true> : k_sweep_batch<8, false>;
  }
  return nullptr;
}
template <class Fn>
static cudaError_t set_smem(Fn fn, size_t smem) {
  return fn ? cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : cudaErrorInvalidValue;
}
template <class Fn>
static cudaError_t occupancy(Fn fn, int threads, size_t smem, int* blocks_per_sm) {
  return fn ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, threads, smem) : cudaErrorInvalidValue;
}
template <class Fn, class Args>
static cudaError_t launch_fn(Fn fn, int threads, int blocks, size_t smem, const Args& a, cudaStream_t s) {
  if (!fn) return cudaErrorInvalidValue;
  fn<<<blocks, threads, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t sweep_batch_set_smem(int M, bool direct, size_t smem) { return set_smem(sweep_batch_fn(M, direct), smem); }
cudaError_t sweep_batch_occupancy(int M, bool direct, int threads, size_t smem, int* blocks_per_sm) {
  return occupancy(sweep_batch_fn(M, direct), threads, smem, blocks_per_sm);
}
cudaError_t launch_sweep_batch(int M, bool direct, int threads, int blocks, size_t smem, const BatchSweepParams& p,
                               cudaStream_t s) {
  return launch_fn(sweep_batch_fn(M, direct), threads, blocks, smem, p, s);
}
cudaError_t sweep_set_smem(int M, bool direct, size_t smem) { return set_smem(sweep_fn(M, direct), smem); }
cudaError_t sweep_occupancy(int M, bool direct, int threads, size_t smem, int* blocks_per_sm) {
  return occupancy(sweep_fn(M, direct), threads, smem, blocks_per_sm);
}
cudaError_t launch_sweep(int M, bool direct, int threads, int blocks, size_t smem, const SweepArgs& a, cudaStream_t s) {
  return launch_fn(sweep_fn(M, direct), threads, blocks, smem, a, s);
}

uint32_t launch_good(const GoodView& a, const uint32_t* level_off, int n_sms, cudaStream_t s) {
  if (!a.W || !a.N) return 0;
  // Words per CTA: as few as leave at most one CTA an SM.
  uint32_t p = 1;
  while (p < 8 && (a.W + p - 1) / p > (uint32_t)n_sms) p *= 2;
  // Time by levels, us: a barrier, latency and the elements' share for the
  // words' CTAs against a launch and all words' share of the chip.  Measured
  // us a level: 32 words at 1,333 gates 3.2 against 4.5, at 5,000 11.6 against
  // 5.2, at 50,000 105 against 15; 1,024 words at 1,333 gates 6.2 against 13,
  // at 50,000 197 against 279.
  const uint32_t waves = ((a.W + p - 1) / p + (uint32_t)n_sms - 1) / (uint32_t)n_sms;
  const double per_elem = (p == 8 ? 3.9e-3 : p == 4 ? 2.6e-3 : 2.1e-3) * waves;
  double by_words = 0, by_levels = 0;
  for (uint32_t l = 1; l < a.n_levels; ++l) {
    const double n = level_off[l + 1] - level_off[l];
    by_words += 1 + n * per_elem;
    by_levels += 4.5 + n * a.W * 5.4e-6;
  }
  if (by_words > by_levels) {
    uint32_t launches = 0;
    for (uint32_t l = 0; l < a.n_levels; ++l) {
      const uint64_t n = (uint64_t)(level_off[l + 1] - level_off[l]) * a.W;
      if (!n) continue;
      const uint64_t blocks = std::min<uint64_t>((n + 255) / 256, 64ull * n_sms);
      k_good_level<<<(unsigned)blocks, 256, 0, s>>>(a, level_off[l], level_off[l + 1]);
      ++launches;
    }
    return launches;
  }
  // A thread per element of a typical level and pair of words: more would
  // only run the loop's overhead.
  const uint64_t lanes = (uint64_t)(a.N - a.n_pi) / std::max<uint32_t>(a.n_levels - 1, 1) * 5 / 4 * std::max(p / 2, 1u);
  const unsigned threads = (unsigned)std::min<uint64_t>(1024, std::max<uint64_t>(64, (lanes + 31) / 32 * 32));
  const unsigned blocks = (a.W + p - 1) / p;
  switch (p) {
    case 1: k_good<1><<<blocks, threads, 0, s>>>(a); break;
    case 2: k_good<2><<<blocks, threads, 0, s>>>(a); break;
    case 4: k_good<4><<<blocks, threads, 0, s>>>(a); break;
    default: k_good<8><<<blocks, threads, 0, s>>>(a); break;
  }
  return 1;
}

cudaError_t launch_sweep_wide(int M, int threads, int blocks, const SweepWideArgs& a, cudaStream_t s) {
  switch (M) {
    case 1: k_sweep_wide<1><<<blocks, threads, 0, s>>>(a); break;
    case 2: k_sweep_wide<2><<<blocks, threads, 0, s>>>(a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t sweep_wide_occupancy(int M, int threads, int* blocks_per_sm) {
  switch (M) {
    case 1: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_sweep_wide<1>, threads, 0);
    case 2: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_sweep_wide<2>, threads, 0);
  }
  return cudaErrorInvalidValue;
}

void launch_ffr(const FfrArgs& a, cudaStream_t s) {
  if (a.n_list == 0) return;
  const int threads = 256;
  const uint64_t blocks = ((uint64_t)a.n_list * a.n_tiles * 32 + threads - 1) / threads;
  k_ffr<<<(unsigned)blocks, threads, 0, s>>>(a);
}

void launch_exact(const ExactArgs& a, cudaStream_t s) {
  if (a.n_exact == 0) return;
  const int threads = 256;
  const uint64_t blocks = ((uint64_t)a.n_exact * a.n_tiles * 32 + threads - 1) / threads;
  k_exact<<<(unsigned)blocks, threads, 0, s>>>(a);
}

void launch_init_results(unsigned long long* count, unsigned long long* first, uint8_t* lastflag,
                         uint32_t F, int* zero, uint32_t n_zero, cudaStream_t s) {
  const uint32_t n = std::max(F, n_zero);
  if (n == 0) return;
  k_init_results<<<std::min<uint32_t>((n + 255) / 256, 4096), 256, 0, s>>>(count, first, lastflag, F, zero, n_zero);
}

void launch_results(const ResultArgs& a, cudaStream_t s) {
  k_results<<<a.F / 256 + 1, 256, 0, s>>>(a);
}

void launch_round(const uint64_t* good, uint32_t N, uint64_t mask, uint64_t* out, cudaStream_t s) {
  if (N) k_round<<<std::min<uint32_t>((N + 255) / 256, 4096), 256, 0, s>>>(good, N, mask, out);
}

void launch_drop(const DropArgs& a, cudaStream_t s) {
  const uint64_t n = (uint64_t)a.n_in_pad + a.n_exact_in;
  if (n == 0) return;
  k_drop<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
}

}  // namespace fsimb
