// logprobs_batch: per row the log-softmax of one token and the top_n largest raw logits as log
// probabilities (tools/server_chat.h:417-441; zero/runz.cpp:478-484 scores perplexity with the
// same sum). One launch, one pass. Many rows: a CTA to a row. Fewer: the rows, cut into units of
// columns, are dealt out to the CTAs in equal runs of consecutive units (lp_plan): a CTA takes the end
// of one row, some whole rows and the beginning of another, so that a row is cut only where one CTA's
// share ends. Every such piece of a row is read once, straight into registers (a tile of
// four 16-byte chunks a thread, the next tile's loads in flight while one is worked on), and gives
//  - per thread a sum of exponentials relative to a reference value of the thread's own, in fp64;
//  - notes of the threads' tiles that may hold one of the top_n largest elements, which are read
//    again at the piece's end.
// After a piece's first tile no thread waits for another. The CTA that finishes a cut row last merges its
// pieces (left in the workspace) and writes the row's output.
//
// What bounds it: memory, then the special-function unit (one ex2 per logit, 16 a clock and SM:
// 59 us for 1024 x 262144, next to 83 us for its 537 MB); what the kernel takes on top are the pieces'
// ends and beginnings. 1024 x 262144 bf16: 20 alternatives 216 -> 147 us, none 134 -> 114 us; 512 x
// 151936 fp32, none: 80 -> 62 us; 8 x 151936 fp32, 20 alternatives 22 -> 15 us (a row through a
// shared-memory ring with two barriers a tile, the candidates' buffer kept by the whole CTA, -> this;
// graph replays). A masked front of a row (7 of 8 columns, 512 x 262144 bf16, 20 alternatives): -inf
// 410 -> 59 us, -1e30 432 -> 110.
#include <algorithm>
#include <type_traits>

#include "plan.h"
#include "select.cuh"
#include "stream.cuh"

namespace arcs {

constexpr int kLpThreads = 128;               // threads of a CTA
constexpr int kLpCap = 1024;                  // candidate buffer of a CTA
constexpr int kLpTrig = kLpCap - kLpThreads;    // prune once it has grown past this
// CTAs per SM the work is dealt out to. With alternatives five, which leaves the compiler enough
// registers (64 alternatives 185 -> 169 us, 256: 433 -> 287 us); without them six (111 -> 105 us).
__host__ __device__ constexpr int lp_per_sm(bool top) { return top ? 5 : 6; }
constexpr int kLpChunks = 4;                  // 16-byte chunks a thread holds of one tile
constexpr int kLpTileBytes = kLpChunks * kLpThreads * 16;
constexpr int kLpAhead = 3;                   // tiles ahead of the one worked on that are asked into the L2 cache
constexpr int kLpFew = 64;                    // up to so many alternatives one maximum per thread gives a tight threshold
// records a CTA keeps of threads and tiles whose maximum reached the threshold of the moment: one a thread of
// the first tile, then about as many as alternatives wanted (plus a seventh) each time the piece doubles.
// Each time another kLpMark have come the threshold is raised out of turn (a masked region has ended).
template <int TOP> constexpr int kLpRec = TOP == 0 ? 1 : TOP == 1 ? 1536 : 3072;
template <int TOP> constexpr uint32_t kLpMark = TOP == 0 ? 0 : (kLpRec<TOP> - kLpThreads) / 4;

struct LpPart {      // what a piece leaves for the merge
  double z;          // sum of exp(l - M) over the piece
  float M;           // the largest of its threads' references (-inf: nothing but NaN or -inf)
  int32_t cnt;       // entries in its candidate list
};

struct LogprobDev {
  const void* logits;
  int64_t row_stride;
  int32_t B, V;
  int32_t unit, row_units;         // columns per unit, units per row
  uint32_t run, longer;            // units every CTA takes, CTAs that take one more (the first ones)
  int32_t max_pieces;              // pieces a row can be cut into
  const int32_t* token;
  int32_t top_n, top_stride;
  double* logprob;
  double* lse;
  int32_t* top_id;
  double* top_logprob;
  unsigned int* ws_ctr;            // [B] pieces of the row that have finished, 0 between launches
  LpPart* ws_part;                 // [B][max_pieces]
  unsigned long long* ws_list;     // [B][max_pieces][n] composites
  int32_t* status;
};

constexpr float kL2e = 1.44269502162933349609375f;  // log2 e rounded to fp32

__device__ __forceinline__ float ex2(float x) {
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x));
  return e;
}
// a float that is neither negative, infinite nor NaN, widened by integer operations (the conversion
// instruction shares the special-function unit with the exponentials; zero comes out as 2^-127)
__device__ __forceinline__ double widen_pos(float x) {
  const uint32_t b = __float_as_uint(x);
  return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}

// the largest element of several chunks (NaN ignored), a chunk of -inf
template <typename T> struct LpElem;
template <> struct LpElem<float> {
  static constexpr uint32_t kNothing = 0xFF800000u;
  static __device__ __forceinline__ float tile_max(const uint4 (&q)[kLpChunks]) {
    float m = Elem<float>::chunk_max(q[0]);
#pragma unroll
    for (int j = 1; j < kLpChunks; ++j) m = fmaxf(m, Elem<float>::chunk_max(q[j]));
    return m;
  }
};
template <> struct LpElem<__nv_bfloat16> {
  static constexpr uint32_t kNothing = 0xFF80FF80u;
  static __device__ __forceinline__ float tile_max(const uint4 (&q)[kLpChunks]) {
    __nv_bfloat162 m[kLpChunks];
#pragma unroll
    for (int j = 0; j < kLpChunks; ++j) {
      const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&q[j]);
      m[j] = __hmax2(__hmax2(p[0], p[1]), __hmax2(p[2], p[3]));  // NaN-ignoring packed max
    }
#pragma unroll
    for (int w = kLpChunks / 2; w > 0; w >>= 1)
#pragma unroll
      for (int j = 0; j < w; ++j) m[j] = __hmax2(m[j], m[j + w]);
    return fmaxf(__low2float(m[0]), __high2float(m[0]));
  }
};

// A thread's running sum of exponentials: S * 2^c = sum of 2^(l * kL2e) over what it has seen, c
// the rounded product ref * kL2e. A term is ex2(fma(l, kL2e, -c)): one rounding, and c's own is
// made good once, when the sum is taken (scaled()). The terms of a chunk are added in fp32, the
// chunks in fp64. The reference is at least every element the thread has seen: the terms that make
// up a peaked sum are exact ones. Against fp64 sums the log of a row's sum has an rms error of
// 0.9e-8 (fp32 normal logits, 512 rows of 151936; 1.1e-8 when exponents were rounded twice).
// That holds while c's own rounding is small: up to |ref| = 2^24 it is at most 1. Beyond (logits masked
// with a large negative number, above all) c is a NaN, and S the sum of 2^((l - ref) * kL2e): a float
// so large has neighbours 1 away or more, so that l - ref is exact or leaves a term without weight.
constexpr float kLpNear = 16777216.0f;
__device__ __forceinline__ float lp_c(float ref) { return fabsf(ref) <= kLpNear ? __fmul_rn(ref, kL2e) : NAN; }
struct LpSum {
  float ref = -INFINITY, c = NAN;
  double S = 0.0;
  __device__ __forceinline__ double off() const { return c == c ? (double)ref * (double)kL2e - (double)c : 0.0; }  // exact: what the terms' exponents are short of
  __device__ __forceinline__ double scaled() const { return S == 0.0 ? 0.0 : S * exp2(-off()); }                   // sum of exp(l - ref)
  // a new, larger reference
  __device__ __forceinline__ void raise(float m) {
    const LpSum from = *this;
    ref = m;
    c = lp_c(m);
    if (S == 0.0) return;
    if (c == c && from.c == from.c) S *= exp2((double)from.c - (double)c);
    else S = from.scaled() * exp((double)from.ref - (double)m) * exp2(off());
  }
  // exp(v - ref) in fp64, without the exponential where it has no digits or is one
  __device__ __forceinline__ double term(float v) const {
    const double d = (double)v - (double)ref;
    return v != v || d < -750.0 ? 0.0 : d == 0.0 ? 1.0 : exp(d);
  }
  // one more value, in the slow way
  __device__ __forceinline__ void one(float v) {
    if (v > ref) raise(v);
    if (ref > -INFINITY) S += term(v) * exp2(off());
  }
};
// The rare steps of the main loop are calls: what they need in registers is then spilled around
// them and not in the loop itself.
__device__ __noinline__ double lp_rescale(double S, float ref, float m) {
  LpSum s;
  s.S = S;
  s.ref = ref;
  s.c = lp_c(ref);
  s.raise(m);
  return s.S;
}
// (the thread's chunks first, first + kLpThreads, ... of a piece with nchunk of them at body, read once more)
template <typename T>
__device__ __noinline__ double lp_tile_slow(double S, float ref, const char* body, int first, int nchunk) {
  LpSum s;
  s.ref = ref;
  s.c = lp_c(ref);
  double z = 0.0;
  const int end = min(nchunk, first + kLpChunks * kLpThreads);
  for (int i = first; i < end; i += kLpThreads) {
    const uint4 q = ldg128_stream(body + (size_t)i * 16);
#pragma unroll
    for (int e = 0; e < Elem<T>::kPerChunk; ++e) z += s.term(Elem<T>::get(q, e));  // (none exceeds the reference)
  }
  return S + z * exp2(s.off());
}
// The sums of a tile's chunks relative to a reference far from zero, the tile read once more (with
// alternatives the loop has no registers left for a second form of the terms).
template <typename T>
__device__ __noinline__ float4 lp_terms_far(float ref, const char* body, int first, int nchunk) {
  constexpr int E = Elem<T>::kPerChunk;
  static_assert(kLpChunks == 4, "a float a chunk");
  float z[kLpChunks];
  uint4 q[kLpChunks];
#pragma unroll
  for (int j = 0; j < kLpChunks; ++j) q[j] = ldg128_stream_if(body + (size_t)(first + j * kLpThreads) * 16, first + j * kLpThreads < nchunk, LpElem<T>::kNothing);
#pragma unroll
  for (int j = 0; j < kLpChunks; ++j) {
    float e[E];
#pragma unroll
    for (int i = 0; i < E; ++i) e[i] = ex2(__fmul_rn(__fsub_rn(Elem<T>::get(q[j], i), ref), kL2e));
#pragma unroll
    for (int w = E / 2; w > 0; w >>= 1)
#pragma unroll
      for (int i = 0; i < w; ++i) e[i] += e[i + w];
    z[j] = e[0];
  }
  return make_float4(z[0], z[1], z[2], z[3]);
}
// What the threads have published of their own maxima belongs to disjoint sets of elements, so the
// n-th largest of it is a lower bound of the n-th largest element: the threshold (a key,
// inclusive, 16-bit resolution) rises to it. One warp calls.
template <int PER>
__device__ __noinline__ void lp_raise_threshold(const uint32_t* keys, int n, uint32_t* tkey) {
  const uint32_t k = warp_kth16<PER>(keys, n);
  if ((threadIdx.x & 31) == 0) asm volatile("red.shared.max.u32 [%0], %1;" ::"r"(smem_addr(tkey)), "r"(k) : "memory");
}

// The same after the first tile, whose threads are all there: an element of a later tile has a higher
// id than the n elements found, so that it must exceed the n-th of them, not only reach it. What lies
// in a region of equal logits (masked ones, -inf among them) is then not noted again tile by tile.
template <int PER>
__device__ __noinline__ void lp_first_threshold(const uint32_t* keys, int n, uint32_t* tkey) {
  const uint32_t k = warp_kth16<PER>(keys, n);
  uint32_t m = 0xFFFFFFFFu;  // the smallest key at or above that bound: n keys are not below it
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const uint32_t x = keys[i * 32 + (threadIdx.x & 31)];
    if (x >= k) m = min(m, x);
  }
  m = __reduce_min_sync(0xFFFFFFFFu, m);
  if ((threadIdx.x & 31) == 0 && k != 0u) asm volatile("red.shared.max.u32 [%0], %1;" ::"r"(smem_addr(tkey)), "r"(m + 1u) : "memory");  // (no bound: fewer than n numbers)
}

// The n best of the tiles noted, when more of their elements reach the threshold than the buffer
// holds (masses of equal logits in the first tile). Called by all threads.
template <typename T>
__device__ __noinline__ void lp_take_noted(const SegPlan& p, const T* row, const Sel& sel, const PruneScratch& ps, const uint32_t* rec_at, int noted) {
  constexpr int E = Elem<T>::kPerChunk;
  const int tid = threadIdx.x, nchunk = p.body_bytes / 16;
  __syncthreads();
  if (tid == 0) {
    *sel.cnt = 0;
    *sel.tau = 0ull;
  }
  __syncthreads();
  for (int i0 = 0; i0 < noted * kLpChunks; i0 += kLpThreads) {  // (a chunk to a thread)
    const int i = i0 + tid;
    const uint32_t r = i < noted * kLpChunks ? rec_at[i / kLpChunks] : 0u;
    const int ci = i < noted * kLpChunks ? ((int)(r >> 8) * kLpChunks + i % kLpChunks) * kLpThreads + (int)(r & 255u) : nchunk;
    const uint4 q = ci < nchunk ? ldg128_stream(p.body + (size_t)(uint32_t)ci * 16) : make_uint4(0, 0, 0, 0);
    const unsigned long long tau = *sel.tau;
    uint32_t bits = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) bits |= (ci < nchunk && comp_of(key_of(Elem<T>::get(q, e)), p.body_first + ci * E + e) > tau ? 1u : 0u) << e;
    push_all<kLpThreads>(sel, ps, bits, [&](int e, uint32_t& ky, int32_t& id) {
      id = p.body_first + ci * E + e;
      ky = key_of(Elem<T>::get(q, e));
    });
  }
  const bool hv = tid < p.head_n, tv = tid < p.tail_n;
  push_all<kLpThreads>(sel, ps, (hv ? 1u : 0u) | (tv ? 2u : 0u), [&](int idx, uint32_t& ky, int32_t& id) {
    id = idx == 0 ? p.lo + tid : p.tail_first + tid;
    ky = key_of(Elem<T>::load(row + id));
  });
}

// The n best of a piece read once more, element by element (slow, and rare: the notes overflowed,
// with ascending data). Called by all threads.
template <typename T>
__device__ __noinline__ void lp_reread(const SegPlan& p, const T* row, const Sel& sel, const PruneScratch& ps) {
  constexpr int E = Elem<T>::kPerChunk;
  const int tid = threadIdx.x, nchunk = p.body_bytes / 16;
  __syncthreads();
  if (tid == 0) {
    *sel.cnt = 0;
    *sel.tau = 0ull;
  }
  __syncthreads();
  for (int c0 = 0; c0 < nchunk; c0 += kLpChunks * kLpThreads) {
    uint4 q[kLpChunks];
    uint32_t bits = 0;
    const uint32_t tkey = (uint32_t)(*sel.tau >> 32);
#pragma unroll
    for (int j = 0; j < kLpChunks; ++j) {
      const int ci = c0 + j * kLpThreads + tid;
      q[j] = ci < nchunk ? ldg128_stream(p.body + (size_t)ci * 16) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int e = 0; e < E; ++e) bits |= (ci < nchunk && key_of(Elem<T>::get(q[j], e)) >= tkey ? 1u : 0u) << (j * E + e);
    }
    push_all<kLpThreads>(sel, ps, bits, [&](int idx, uint32_t& ky, int32_t& id) {
      const int j = idx / E;
      uint4 c = q[0];
#pragma unroll
      for (int x = 1; x < kLpChunks; ++x)
        if (j == x) c = q[x];
      id = p.body_first + (c0 + j * kLpThreads + tid) * E + idx % E;
      ky = key_of(Elem<T>::get(c, idx % E));
    });
  }
  const bool hv = tid < p.head_n, tv = tid < p.tail_n;
  push_all<kLpThreads>(sel, ps, (hv ? 1u : 0u) | (tv ? 2u : 0u), [&](int idx, uint32_t& ky, int32_t& id) {
    id = idx == 0 ? p.lo + tid : p.tail_first + tid;
    ky = key_of(Elem<T>::load(row + id));
  });
}

// the first unit of a CTA's run, and the CTA whose run holds a unit
__host__ __device__ inline uint32_t lp_first_unit(uint32_t cta, uint32_t run, uint32_t longer) { return cta * run + (cta < longer ? cta : longer); }
__host__ __device__ inline uint32_t lp_cta_of(uint32_t u, uint32_t run, uint32_t longer) {
  const uint32_t split = longer * (run + 1);
  return u < split ? u / (run + 1) : longer + (u - split) / run;
}

// what the threads of a CTA share
template <int TOP>
struct LpShared {
  static constexpr int OWN = TOP == 2 ? kLpChunks : 1;  // maxima a thread keeps
  unsigned long long tau, m64;
  double red_s[kLpThreads / 32], lse;
  alignas(16) uint32_t keys[TOP ? OWN * kLpThreads : 4];  // what the threads publish of their maxima (read four at a time)
  float rec_max[kLpRec<TOP>];                           // threads' maxima of tiles that reached the threshold
  uint32_t rec_at[kLpRec<TOP>];                         // ... tile << 8 | thread
  uint32_t bkey[TOP ? kLpCap : 1];                      // the piece's candidates
  int32_t bid[TOP ? kLpCap : 1];
  uint32_t hist[TOP ? 512 : 1];
  uint32_t tk[TOP ? kTmpCap : 1];
  int32_t ti[TOP ? kTmpCap : 1];
  float red_m[kLpThreads / 32];
  uint32_t wkey[kLpThreads / 32];
  uint32_t nkey;                                        // the threshold of the main loop: keys from which on a tile is noted
  uint32_t tkey;                                        // the piece's last one: keys from which on an element is a candidate
  int rec, cnt, misc[8], flag, cnts[kMaxSeg];
};

// The end of a piece (columns of units s0 .. s1 of row b): its sum and candidates, the merge of the
// row's pieces, the row's output. ref, z: the thread's sum. Called by all threads; a function of its
// own, so that the main loop's registers are not spilled for it.
template <typename T, int TOP>
__device__ __noinline__ void lp_close(const LogprobDev& a, LpShared<TOP>& sh, int b, int s0, int s1, int tiles, float M, double z) {
  constexpr int E = Elem<T>::kPerChunk;
  constexpr int OWN = LpShared<TOP>::OWN;
  const int tid = threadIdx.x;
  const int n = TOP ? min(a.top_n, a.V) : 0;
  const Sel sel{sh.bkey, sh.bid, &sh.cnt, &sh.tau, n, kLpTrig, kLpCap};
  const PruneScratch ps{sh.hist, sh.tk, sh.ti, sh.misc, &sh.m64};
  const T* row = reinterpret_cast<const T*>(a.logits) + (size_t)b * a.row_stride;
  const SegPlan p = make_plan(row, s0 * a.unit, min(a.V, s1 * a.unit));
  const int nchunk = p.body_bytes / 16;
  const bool hv = tid < p.head_n, tv = tid < p.tail_n;
  const float vh = TOP && hv ? Elem<T>::load(row + p.lo + tid) : -INFINITY;
  const float vt = TOP && tv ? Elem<T>::load(row + p.tail_first + tid) : -INFINITY;
  // a warp's (reference, sum of exponentials relative to it) from its lanes' pairs, and the CTA's from
  // its warps' (left in sh.red_m / sh.red_s; called by warp 0)
  auto warp_lse = [&](float& m, double& z) {
    float M = m;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xFFFFFFFFu, M, o));
    z = m > -INFINITY ? z * exp((double)m - (double)M) : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xFFFFFFFFu, z, o);
    m = M;
  };
  auto cta_lse = [&](float& m, double& z) {
    const int w = tid & 31;
    m = w < kLpThreads / 32 ? sh.red_m[w] : -INFINITY;
    z = w < kLpThreads / 32 ? sh.red_s[w] : 0.0;
    warp_lse(m, z);
  };
  auto rank_of = [&](int i, int c) -> int {  // composites are unique: an entry's place is the number of entries above it
    const uint64_t ci = comp_of(sh.bkey[i], sh.bid[i]);
    int rank = 0;
    for (int j = 0; j < c; ++j) rank += comp_of(sh.bkey[j], sh.bid[j]) > ci;
    return rank;
  };

  // ---- the piece's sum, and its candidates: a last threshold, and the elements of the tiles noted
  // that reach it to the buffer (a little more than n as a rule); afterwards sh.bkey / sh.bid hold c
  // entries, the n best among them
  warp_lse(M, z);
  if ((tid & 31) == 0) {
    sh.red_m[tid >> 5] = M;
    sh.red_s[tid >> 5] = z;
  }
  if (tid == 0) {
    sh.cnt = sh.misc[0] = 0;
    sh.tkey = 0u;
  }
  __syncthreads();
  if (TOP && tid < 32) lp_raise_threshold<OWN * kLpThreads / 32>(sh.keys, n, &sh.tkey);
  if (TOP) __syncthreads();
  if (tid < 32) cta_lse(M, z);
  int c = 0;
  if (TOP) {
    const uint32_t tkey = sh.tkey;
    const float tf = floor_value(tkey);
    const int have = tiles > 0 ? sh.rec : 0;
    int noted = 0;
    if (have <= kLpRec<TOP>) {
      // the records that reach it, closed up (in place: a round's are all read before any is
      // written, at or before the round's first place)
      for (int i0 = 0; i0 < have; i0 += kLpThreads) {
        const int i = i0 + tid;
        const bool in = i < have && sh.rec_max[i] >= tf;
        const uint32_t at = i < have ? sh.rec_at[i] : 0u;
        __syncthreads();
        if (in) sh.rec_at[sm_atomic_add(&sh.misc[0], 1u)] = at;
      }
      __syncthreads();
      auto keep = [&](float v, int32_t id) {
        const uint32_t ky = key_of(v);
        if (!(v >= tf) || ky == 0u) return;
        const uint32_t at = sm_atomic_add(&sh.cnt, 1u);
        if (at < (uint32_t)kLpCap) {
          sh.bkey[at] = ky;
          sh.bid[at] = id;
        }
      };
      noted = sh.misc[0];
      for (int i = tid; i < noted * kLpChunks; i += kLpThreads) {  // (a chunk to a thread, from the L2 cache as a rule)
        const uint32_t r = sh.rec_at[i / kLpChunks];
        const int ci = ((int)(r >> 8) * kLpChunks + i % kLpChunks) * kLpThreads + (int)(r & 255u);
        if (ci >= nchunk) continue;
        const uint4 ch = ldg128_stream(p.body + (size_t)(uint32_t)ci * 16);
        if (!(Elem<T>::chunk_max(ch) >= tf) || sm_ld_volatile(&sh.cnt) > (uint32_t)kLpCap) continue;  // (overflowed: below)
#pragma unroll
        for (int e = 0; e < E; ++e) keep(Elem<T>::get(ch, e), p.body_first + ci * E + e);
      }
      if (hv) keep(vh, p.lo + tid);
      if (tv) keep(vt, p.tail_first + tid);
    }
    __syncthreads();
    if (have > kLpRec<TOP>) lp_reread<T>(p, row, sel, ps);
    else if (sh.cnt > kLpCap) lp_take_noted<T>(p, row, sel, ps, sh.rec_at, noted);
    if (sh.cnt > 512) {
      __syncthreads();
      sel_prune<1, kLpThreads>(sel, n, ps, tid);
      __syncthreads();
    }
    c = min(sh.cnt, kLpCap);
  }

  const uint32_t row_u = (uint32_t)b * (uint32_t)a.row_units;
  const int cta0 = (int)lp_cta_of(row_u, a.run, a.longer);
  const int pieces = (int)lp_cta_of(row_u + (uint32_t)a.row_units - 1u, a.run, a.longer) - cta0 + 1;
  const int piece = (int)blockIdx.x - cta0;
  if (pieces > 1) {
    // ---- leave the piece's results; the CTA that finishes the row last merges them
    const size_t slot = (size_t)b * a.max_pieces + piece;
    for (int i = tid; i < c; i += kLpThreads) {
      const int rank = rank_of(i, c);
      if (rank < n) a.ws_list[slot * n + rank] = comp_of(sh.bkey[i], sh.bid[i]);
    }
    if (tid == 0) {
      LpPart pt;
      pt.z = z;
      pt.M = M;
      pt.cnt = min(c, n);
      a.ws_part[slot] = pt;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      sh.flag = atomicAdd(&a.ws_ctr[b], 1u) == (unsigned)pieces - 1u;
      if (sh.flag) a.ws_ctr[b] = 0u;  // left at zero for the next launch
    }
    __syncthreads();
    if (!sh.flag) return;  // (every warp is past its reads of the shared arrays, but for sh.flag: written again behind two barriers)
    __threadfence();
    float pm = -INFINITY;
    double pz = 0.0;
    int pc = 0;
    if (tid < pieces) {
      const LpPart* src = &a.ws_part[(size_t)b * a.max_pieces + tid];
      pz = __ldcg(&src->z);
      pm = __ldcg(&src->M);
      pc = __ldcg(&src->cnt);
    }
    if (TOP) {
      // The lists are sorted. The n-th largest of their first entries (as many of each as there is
      // room for) bounds the row's n-th from below; what exceeds it goes through the buffer, all
      // lists' first entries, then all second ones, until no list has one left.
      if (tid == 0) {
        sh.cnt = 0;
        sh.tau = 0ull;
      }
      if (tid < pieces) sh.cnts[tid] = pc;
      __syncthreads();
      const unsigned long long* lists = a.ws_list + (size_t)b * a.max_pieces * n;
#pragma unroll
      for (int j = 0; j < OWN; ++j) {
        const int e = j * kLpThreads + tid, x = e / pieces, g = e - x * pieces;
        sh.keys[e] = x < sh.cnts[g] ? comp_key(__ldcg(&lists[(size_t)g * n + x])) : 0u;
      }
      __syncthreads();
      if (tid < 32) {
        const uint32_t k = warp_kth16<OWN * kLpThreads / 32>(sh.keys, n);
        if (tid == 0 && k != 0u) sh.tau = ((unsigned long long)k << 32) - 1ull;
      }
      __syncthreads();
      for (int e0 = 0; e0 < pieces * n; e0 += kLpThreads) {
        const int e = e0 + tid, x = e / pieces, g = e - x * pieces;
        const unsigned long long cm = x < sh.cnts[g] ? __ldcg(&lists[(size_t)g * n + x]) : 0ull;
        const bool have = cm > sh.tau;
        if (!__syncthreads_or(have)) break;  // (kLpThreads entries hold one of every list at least)
        push_all<kLpThreads>(sel, ps, have ? 1u : 0u, [&](int, uint32_t& ky, int32_t& id) {
          ky = comp_key(cm);
          id = comp_id(cm);
        });
      }
      __syncthreads();
      if (sh.cnt > 256) sel_prune<1, kLpThreads>(sel, n, ps, tid);
      __syncthreads();
      c = min(sh.cnt, kLpCap);
    }
    static_assert(kMaxSeg <= 64 && kMaxSeg <= kLpThreads, "the pieces' sums lie with two warps");
    if (tid < 64) {
      warp_lse(pm, pz);
      if ((tid & 31) == 0) {
        sh.red_m[tid >> 5] = pm;
        sh.red_s[tid >> 5] = pz;
      }
    } else if (tid < 64 + kLpThreads / 32 - 2) {
      sh.red_m[tid - 62] = -INFINITY;
    }
    __syncthreads();
    if (tid < 32) cta_lse(M, z);
  }

  // ---- the row's output
  if (tid == 0) {
    const double lse = (double)M + log(z);  // tools/server_chat.h:422
    sh.lse = lse;
    if (a.lse) a.lse[b] = lse;
    if (a.logprob) {
      const int32_t tok = a.token ? a.token[b] : -1;
      if (tok >= a.V) raise_status(a.status, ARCS_ERR_ARG);
      a.logprob[b] = (tok >= 0 && tok < a.V) ? (double)Elem<T>::load(row + tok) - lse : (double)NAN;  // :427
    }
  }
  if (TOP) {
    __syncthreads();
    const double lse = sh.lse;
    for (int i = tid; i < c; i += kLpThreads) {
      const int rank = rank_of(i, c);
      if (rank < n) {
        a.top_id[(size_t)b * a.top_stride + rank] = sh.bid[i];
        a.top_logprob[(size_t)b * a.top_stride + rank] = (double)value_of(sh.bkey[i]) - lse;
      }
    }
  }
}

// TOP: 0 no alternatives, 1 up to kLpFew (a threshold from one maximum a thread), 2 any number (four
// maxima a thread)
template <typename T, int TOP>
__global__ void __launch_bounds__(kLpThreads, lp_per_sm(TOP != 0)) logprob_kernel(const __grid_constant__ LogprobDev a) {
  constexpr int E = Elem<T>::kPerChunk;
  constexpr int OWN = LpShared<TOP>::OWN;
  static_assert(OWN * kLpThreads < 1024, "the search counts to 1023");
  static_assert(kLpChunks * E <= 32, "a thread's elements of one tile are tracked in a 32-bit mask");
  __shared__ __align__(16) LpShared<TOP> sh;

  const int tid = threadIdx.x;
  const int n = TOP ? min(a.top_n, a.V) : 0;
  uint32_t u = lp_first_unit(blockIdx.x, a.run, a.longer);
  const uint32_t u_end = lp_first_unit(blockIdx.x + 1, a.run, a.longer);

  while (u < u_end) {
    // ---- the next piece
    const int b = (int)(u / (uint32_t)a.row_units), s0 = (int)(u - (uint32_t)b * (uint32_t)a.row_units);
    const int s1 = (int)min((uint32_t)a.row_units, (uint32_t)s0 + (u_end - u));
    u += (uint32_t)(s1 - s0);
    const T* row = reinterpret_cast<const T*>(a.logits) + (size_t)b * a.row_stride;
    const SegPlan p = make_plan(row, s0 * a.unit, min(a.V, s1 * a.unit));
    const int nchunk = p.body_bytes / 16;
    const char* mine = p.body + (size_t)tid * 16;
    auto fetch = [&](uint4 (&q)[kLpChunks], int t) {
      const char* from = mine + (size_t)t * kLpTileBytes;
      if ((t + 1) * (kLpChunks * kLpThreads) <= nchunk) {
#pragma unroll
        for (int j = 0; j < kLpChunks; ++j) q[j] = ldg128_stream(from + j * kLpThreads * 16);
      } else {
        const int c0 = t * kLpChunks * kLpThreads + tid;
#pragma unroll
        for (int j = 0; j < kLpChunks; ++j) q[j] = ldg128_stream_if(from + j * kLpThreads * 16, c0 + j * kLpThreads < nchunk, LpElem<T>::kNothing);
      }
    };
    if (tid == 0 && p.body_bytes > 0) prefetch_l2(p.body, min(kLpAhead * kLpTileBytes, p.body_bytes));
    uint4 qa[kLpChunks], qb[kLpChunks];  // the tile being worked on and the next, in turn
    fetch(qa, 0);
    const bool hv = tid < p.head_n, tv = tid < p.tail_n;  // the few elements outside the 16-byte aligned body
    const float vh = hv ? Elem<T>::load(row + p.lo + tid) : -INFINITY;
    const float vt = tv ? Elem<T>::load(row + p.tail_first + tid) : -INFINITY;

    LpSum sum;
    float own[OWN];  // the largest values this thread itself has seen
#pragma unroll
    for (int i = 0; i < OWN; ++i) own[i] = -INFINITY;
    auto publish = [&]() {
#pragma unroll
      for (int i = 0; i < OWN; ++i) sh.keys[i * kLpThreads + tid] = own[i] > -INFINITY ? key_of(own[i]) : 0u;
    };
    if (tid == 0) {
      sh.rec = kLpThreads;  // (the first tile's records have places of their own)
      sh.nkey = 0u;
    }

    const int tiles = (nchunk + kLpChunks * kLpThreads - 1) / (kLpChunks * kLpThreads);
    uint32_t mark = kLpThreads + kLpMark<TOP>;  // the number of notes at which the warp does so out of turn
    auto tile = [&](auto odd, int t, const uint4 (&q)[kLpChunks], uint4 (&nq)[kLpChunks]) {
      constexpr bool kOdd = decltype(odd)::value;  // (t is odd: what only even or only odd tiles do is left out of the other's code)
      if (t + 1 < tiles) fetch(nq, t + 1);
      if (tid == 0 && t + kLpAhead < tiles) prefetch_l2(p.body + (size_t)(t + kLpAhead) * kLpTileBytes, min(kLpTileBytes, p.body_bytes - (t + kLpAhead) * kLpTileBytes));
      const float tm = LpElem<T>::tile_max(q);
      if (TOP == 2) {
#pragma unroll
        for (int j = 0; j < OWN; ++j) own[j] = fmaxf(own[j], Elem<T>::chunk_max(q[j]));
      } else if (TOP == 1) {
        own[0] = fmaxf(own[0], tm);
      }
      if (!kOdd && t == 0) {
        // The CTA's largest element so far is every thread's first reference: a thread then meets a
        // larger one, and pays for the rescaling of its sum, some 32 times a row and not at every
        // maximum of its own.
        const uint32_t wk = __reduce_max_sync(0xFFFFFFFFu, tm > -INFINITY ? key_of(tm) : 0u);
        if ((tid & 31) == 0) sh.wkey[tid >> 5] = wk;
        if (TOP) {
          // (numbers only, -inf among them where every chunk is one of the row's)
          const bool whole = nchunk >= kLpChunks * kLpThreads;
#pragma unroll
          for (int i = 0; i < OWN; ++i) {
            const float m = OWN == 1 ? tm : Elem<T>::chunk_max(q[i]);
            sh.keys[i * kLpThreads + tid] = m > -INFINITY || (whole && m == m) ? key_of(m) : 0u;
          }
          sh.rec_max[tid] = tm;
          sh.rec_at[tid] = tid;
        }
        __syncthreads();
        uint32_t mk = sh.wkey[0];
#pragma unroll
        for (int w = 1; w < kLpThreads / 32; ++w) mk = max(mk, sh.wkey[w]);
        if (mk != 0u) {
          sum.ref = value_of(mk);
          sum.c = lp_c(sum.ref);
        }
        if (TOP && tid < 32) lp_first_threshold<OWN * kLpThreads / 32>(sh.keys, n, &sh.nkey);
      } else if (tm > sum.ref) {
        if (sum.S != 0.0) sum.S = lp_rescale(sum.S, sum.ref, tm);
        sum.ref = tm;
        sum.c = lp_c(tm);
      }
      // ---- the sum of exponentials
      {
        float z[kLpChunks];
        auto terms = [&](auto exponent) {
#pragma unroll
          for (int j = 0; j < kLpChunks; ++j) {
            float e[E];
#pragma unroll
            for (int i = 0; i < E; ++i) e[i] = ex2(exponent(Elem<T>::get(q[j], i)));
#pragma unroll
            for (int w = E / 2; w > 0; w >>= 1)
#pragma unroll
              for (int i = 0; i < w; ++i) e[i] += e[i + w];
            z[j] = e[0];
          }
        };
        if (sum.c == sum.c) terms([&](float v) { return fmaf(v, kL2e, -sum.c); });
        else if (TOP == 0) terms([&](float v) { return __fmul_rn(__fsub_rn(v, sum.ref), kL2e); });
        else if (sum.ref > -INFINITY) {
          const float4 far = lp_terms_far<T>(sum.ref, p.body, t * kLpChunks * kLpThreads + tid, nchunk);
          z[0] = far.x;
          z[1] = far.y;
          z[2] = far.z;
          z[3] = far.w;
        } else z[0] = z[1] = z[2] = z[3] = INFINITY;
        if ((z[0] + z[1]) + (z[2] + z[3]) < 1e30f) {
          sum.S += (widen_pos(z[0]) + widen_pos(z[1])) + (widen_pos(z[2]) + widen_pos(z[3]));
        } else if (sum.ref > -INFINITY) {  // (nothing but -inf so far: nothing to add)
          sum.S = lp_tile_slow<T>(sum.S, sum.ref, p.body, t * kLpChunks * kLpThreads + tid, nchunk);  // (a NaN or an infinity)
        }
      }
      // ---- a tile that may hold one of the n best is noted, to be looked into at the piece's end
      if (TOP && (kOdd || t > 0)) {
        if (tm >= floor_value(sm_ld_volatile(&sh.nkey))) {
          const uint32_t at = sm_atomic_add(&sh.rec, 1u);
          if (at < (uint32_t)kLpRec<TOP>) {
            sh.rec_max[at] = tm;
            sh.rec_at[at] = (uint32_t)t << 8 | (uint32_t)tid;
          }
        }
      }
      // ---- after tiles 1, 3, 7, 15, ..., and where notes come thick (a look every four tiles: one every two
      // costs 2 % of the kernel), the threads publish their maxima. (No barrier: what another warp has not
      // published yet only leaves the threshold lower. The warps take turns at raising it, but each does
      // that finds many notes.)
      if (TOP && kOdd && (t == 1 || (t & 2) != 0)) {
        const uint32_t rec = __shfl_sync(0xFFFFFFFFu, sm_ld_volatile(&sh.rec), 0);
        const bool many = rec >= mark && rec < (uint32_t)kLpRec<TOP>;
        if ((t & (t + 1)) == 0 || many) {
          publish();
          __syncwarp();
          if (many || (tid >> 5) == (__ffs(t + 1) & (kLpThreads / 32 - 1))) lp_raise_threshold<OWN * kLpThreads / 32>(sh.keys, n, &sh.nkey);
          if (many) mark = rec + kLpMark<TOP>;
        }
      }
    };
    if (u < u_end && tid == 0) {  // (the next row's first tile is asked for in time)
      const uintptr_t next = (reinterpret_cast<uintptr_t>(row + a.row_stride) + 15) & ~(uintptr_t)15;
      const int bytes = (int)min((int64_t)kLpTileBytes, (int64_t)a.V * (int)sizeof(T) - 16) & ~15;
      if (bytes > 0) prefetch_l2(reinterpret_cast<const void*>(next), bytes);
    }
    for (int t = 0; t < tiles; t += 2) {
      tile(std::false_type(), t, qa, qb);
      if (t + 1 < tiles) tile(std::true_type(), t + 1, qb, qa);
    }
    if (hv) sum.one(vh);
    if (tv) sum.one(vt);
    if (TOP) {
      own[0] = fmaxf(own[0], fmaxf(vh, vt));
      publish();
    }
    lp_close<T, TOP>(a, sh, b, s0, s1, tiles, sum.ref, sum.scaled());
    __syncthreads();  // (the next piece takes the shared arrays over)
  }
}

}  // namespace arcs

using namespace arcs;

// Rows enough for the GPU, or short ones, are not cut: a row to a CTA, nothing handed over and no
// workspace used, so that such calls may overlap as they like. (Cutting them too, and dealing the
// pieces out evenly, was measured: none wanted, 512 x 151936 fp32 53 us against 59, 1024 x 262144
// bf16 99 against 113; 20 alternatives 75 / 74 and 139 / 140, 600 x 50000 bf16 39 / 27.)
constexpr int32_t kLpManyRows = 3 * kSmCount, kLpShortRow = 8192;
static bool lp_whole(int32_t B, int32_t V) { return B >= kLpManyRows || V <= kLpShortRow; }
// How B rows of V columns are dealt out: whole, or cut into units of `unit` columns (a multiple of
// 2048, at most kMaxSeg to a row) that are given in equal runs to the CTAs, which all fit the GPU at
// once: a row is cut only where one CTA's share ends. A row's units lie with at most max_pieces CTAs.
// Where that would be less than kLpOwnPiece columns a CTA, no CTA gets the end of one row and the
// beginning of the next, which would cost it a second piece's fixed time (7 us with alternatives: 56 x
// 30000 fp32, 5 alternatives, 20 us when runs straddle rows, 15 when not): a unit to a CTA. Up to twice
// as many columns, too, where that leaves an eighth of the CTAs without a unit at most.
constexpr int32_t kLpOwnPiece = 8192;
struct LpPlan {
  int32_t unit, row_units, max_pieces;
  uint32_t run, longer;
  unsigned grid;
};
static LpPlan lp_plan(int32_t B, int32_t V, int32_t top_n) {
  LpPlan p;
  if (lp_whole(B, V)) {
    p.unit = V;
    p.row_units = p.max_pieces = 1;
    p.run = 1;
    p.longer = 0;
    p.grid = (unsigned)B;
    return p;
  }
  const int32_t ctas = kSmCount * lp_per_sm(top_n > 0);
  const int64_t share = (int64_t)B * V / ctas;
  const bool own = share < kLpOwnPiece || (share < 2 * kLpOwnPiece && ctas / B * B * 8 >= ctas * 7);
  const int32_t most = own ? std::min(kMaxSeg, std::max(1, ctas / B)) : kMaxSeg;
  p.unit = std::max(top_n > 0 ? 4096 : 2048, ((V - 1) / most + 2048) / 2048 * 2048);  // (a list costs more to merge than a sum)
  p.row_units = (V + p.unit - 1) / p.unit;
  const uint32_t total = (uint32_t)B * (uint32_t)p.row_units;
  p.grid = std::min<uint32_t>(total, (uint32_t)ctas);
  p.run = total / p.grid;
  p.longer = total % p.grid;
  p.max_pieces = (int32_t)std::min<uint32_t>(p.row_units, ((uint32_t)p.row_units - 1 + p.run - 1) / p.run + 1);
  return p;
}

extern "C" size_t arcs_logprobs_workspace_bytes(int32_t B, int32_t V, int32_t top_n) {
  if (B <= 0 || V <= 0 || top_n < 0) return 0;
  if (lp_whole(B, V)) return 16;  // (not used)
  const LpPlan p = lp_plan(B, V, top_n);
  return 256 + (((size_t)B * 4 + 255) & ~(size_t)255) + (size_t)B * p.max_pieces * (sizeof(LpPart) + (size_t)top_n * 8);
}

extern "C" int arcs_logprobs_batch(const arcs_logprob_args* g, void* stream) {
  if (int inj = fault_injected()) return inj;
  if (!g || !g->logits || g->B <= 0 || g->V <= 0 || g->row_stride < g->V || (g->dtype != ARCS_F32 && g->dtype != ARCS_BF16))
    return set_error(ARCS_ERR_ARG, "logprobs_batch: bad argument");
  if (g->top_n < 0 || g->top_n > ARCS_KCAP) return set_error(ARCS_ERR_TOPK, "logprobs_batch: top_n must be 0 .. ARCS_KCAP");
  if (g->top_n > 0 && (!g->top_id || !g->top_logprob || g->top_stride < g->top_n))
    return set_error(ARCS_ERR_ARG, "logprobs_batch: top_n given without top_id / top_logprob of at least top_n entries per row");
  if (g->token && !g->logprob) return set_error(ARCS_ERR_ARG, "logprobs_batch: token given without logprob");
  LogprobDev a;
  a.logits = g->logits;
  a.row_stride = g->row_stride;
  a.B = g->B;
  a.V = g->V;
  const LpPlan plan = lp_plan(g->B, g->V, g->top_n);
  a.unit = plan.unit;
  a.row_units = plan.row_units;
  a.run = plan.run;
  a.longer = plan.longer;
  a.max_pieces = plan.max_pieces;
  a.token = g->token;
  a.top_n = g->top_n;
  a.top_stride = g->top_stride;
  a.logprob = g->logprob;
  a.lse = g->lse;
  a.top_id = g->top_id;
  a.top_logprob = g->top_logprob;
  a.status = g->status;
  a.ws_ctr = nullptr;
  a.ws_part = nullptr;
  a.ws_list = nullptr;
  if (!lp_whole(g->B, g->V)) {
    if (!g->workspace || g->workspace_bytes < arcs_logprobs_workspace_bytes(g->B, g->V, g->top_n))
      return set_error(ARCS_ERR_WORKSPACE, "logprobs_batch: workspace too small");
    if ((reinterpret_cast<uintptr_t>(g->workspace) & 15u) != 0) return set_error(ARCS_ERR_WORKSPACE, "logprobs_batch: workspace must be 16-byte aligned");
    char* ws = static_cast<char*>(g->workspace);
    a.ws_ctr = reinterpret_cast<unsigned int*>(ws);
    ws += ((size_t)g->B * 4 + 255) & ~(size_t)255;
    a.ws_part = reinterpret_cast<LpPart*>(ws);
    ws += (size_t)g->B * a.max_pieces * sizeof(LpPart);
    a.ws_list = reinterpret_cast<unsigned long long*>(ws);
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
#define ARCS_LAUNCH(T)                                                                            \
  do {                                                                                            \
    if (g->top_n == 0) logprob_kernel<T, 0><<<plan.grid, kLpThreads, 0, st>>>(a);                   \
    else if (g->top_n <= kLpFew) logprob_kernel<T, 1><<<plan.grid, kLpThreads, 0, st>>>(a);         \
    else logprob_kernel<T, 2><<<plan.grid, kLpThreads, 0, st>>>(a);                                 \
  } while (0)
  if (g->dtype == ARCS_F32) ARCS_LAUNCH(float);
  else ARCS_LAUNCH(__nv_bfloat16);
#undef ARCS_LAUNCH
  return check_launch("logprobs_batch");
}
