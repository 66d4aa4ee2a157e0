// resident_kernel: a row held whole in the shared memory of a few SMs, from its logits to its token.
//
// While the rows of a call fit on the chip, a cluster of CTAs takes each: every CTA fetches one slice
// of the row with bulk copies (TMA) and keeps it, so that nothing has to be handed from one kernel
// to another, and no threshold has to be found before the data have passed:
//  1. while the slice is on its way, the CTA enters the history's ids that fall into it in a hash
//     table, which counts them, and looks the biases' columns up there;
//  2. each such column is adjusted with the exact fp32 arithmetic of Sampler::adjusted
//     (tools/sampler.h:147-176) and kept in the table; a NaN takes its place in the slice;
//  3. the k-th largest of the threads' own maxima bounds the slice's k-th element from below; what
//     reaches it, and the adjusted columns that do, are the slice's candidates (a few more than k);
//  4. the cluster's first CTA reads the others' candidates out of their shared memory, ranks them
//     and follows tools/sampler.h:54-77.
// What bounds it: latency, spread over all steps. 1 x 151936 fp32, history 64 (8 CTAs of 76 KB), in us
// from the CTA's start: lists 0.7, slice there 2.0, maxima 2.9, threshold 4.0, candidates 5.8, cluster
// barrier 7.7, fetched and cut 9.6, ranked 10.6, token 12.9; a call 31 -> 15 us. 8 x 262144 fp32
// 45 -> 22 us, 64 x 151936 bf16 (two CTAs of 152 KB a row) about 38 -> 23 us.
#pragma once
#include "sample_finish_warp.cuh"

namespace arcs {

constexpr int kResThreads = 256;
constexpr int kResParts = 8;      // bulk copies (and barriers) a slice arrives by
constexpr int kResCap = 1024;     // candidates of a slice; a longer list is cut to the k best
constexpr int kResOwn = 4;        // maxima a thread keeps
constexpr int kResMaxList = 2048; // longest history + bias lists taken

struct ResShared {
  unsigned long long tau, m64, floor;       // floor: composites at or below it are not among the slice's (the row's) k best
  uint64_t bars[kResParts];
  double spr[ARCS_KCAP + 1], cum[ARCS_KCAP];
  alignas(16) uint32_t keys[kResOwn * kResThreads];  // the threads' maxima; later the prune's counters
  alignas(16) unsigned long long comp[kResCap];      // composites to rank
  uint32_t key[kResCap];                    // the slice's candidates (read by the cluster's first CTA)
  int32_t id[kResCap];
  uint32_t mkey[kResCap];                   // the row's
  int32_t mid[kResCap];
  uint32_t tk[kTmpCap];
  int32_t ti[kTmpCap];
  float sv[ARCS_KCAP];
  int32_t sid[ARCS_KCAP];
  int cnt, mcnt, misc[8], failed, off[17];
  uint32_t scal[16];                        // the elements before and after the aligned body, as float bits
};

// Slots of the table of a slice's history columns: at most four fifths of them are taken.
__host__ __device__ inline int res_slots(int max_hist) {
  if (max_hist <= 0) return 0;
  int slots = 2;
  while (4 * slots < 5 * max_hist) slots <<= 1;
  return slots;
}
// the table (column, what is known of it and then its adjusted key), the row's bias list (id, value, the same)
__host__ __device__ inline size_t res_list_bytes(int max_hist, int max_bias) { return (size_t)res_slots(max_hist) * 8 + (size_t)max_bias * 12; }

// the place of a column in the table (linear probing; -1: not there), entered first if `enter`
__device__ __forceinline__ int res_find(int32_t* h_col, int slots, int32_t c, bool enter) {
  if (slots == 0) return -1;
  uint32_t at = ((uint32_t)c * 2654435761u >> 12) & (uint32_t)(slots - 1);
  for (int n = 0; n < slots; ++n) {
    const int32_t was = enter ? (int32_t)sm_atomic_cas(&h_col[at], 0xFFFFFFFFu, (uint32_t)c) : h_col[at];
    if (was == c) return (int)at;
    if (was == -1) return enter ? (int)at : -1;
    at = (at + 1) & (uint32_t)(slots - 1);
  }
  return -1;  // (not reached when entering: the table has more places than the history has entries)
}

template <typename T>
__global__ void __launch_bounds__(kResThreads, 2) resident_kernel(const __grid_constant__ SampleDev a, int ctas, int slice) {
  extern __shared__ __align__(128) char res_smem[];
  ResShared& s = *reinterpret_cast<ResShared*>(res_smem);
  constexpr int E = Elem<T>::kPerChunk;
  constexpr int NT = kResThreads;
  const int all_slots = res_slots(a.max_hist);
  int32_t* const h_col = reinterpret_cast<int32_t*>(res_smem + ((sizeof(ResShared) + 15) & ~(size_t)15));
  uint32_t* const h_info = reinterpret_cast<uint32_t*>(h_col + all_slots);
  int32_t* const b_id = reinterpret_cast<int32_t*>(h_info + all_slots);
  float* const b_val = reinterpret_cast<float*>(b_id + a.max_bias);
  uint32_t* const b_info = reinterpret_cast<uint32_t*>(b_val + a.max_bias);
  char* const data = res_smem + (((size_t)(reinterpret_cast<char*>(b_info + a.max_bias) - res_smem) + 127) & ~(size_t)127);

  const int tid = threadIdx.x, lane = tid & 31;
  const int rank = (int)blockIdx.x % ctas, b = (int)blockIdx.x / ctas;
  const T* row = reinterpret_cast<const T*>(a.logits) + (size_t)b * a.row_stride;
  const int32_t lo = min(a.V, rank * slice), hi = min(a.V, lo + slice);
  const SegPlan p = make_plan(row, lo, hi);
  const int nchunk = p.body_bytes / 16;
  constexpr int kRound = kResOwn * NT;  // chunks the threads look at together: chunk c is thread c % NT's, its maximum number c / NT % kResOwn
  const int part = ((nchunk + kResParts - 1) / kResParts + kRound - 1) / kRound * kRound;  // chunks a copy brings
  if (tid == 0) {
    for (int i = 0; i < kResParts; ++i) mbar_init(&s.bars[i], 1);
    mbar_init_fence();
    for (int i = 0; i < kResParts; ++i) {
      const int n = min(part, nchunk - i * part);
      if (n <= 0) break;
      mbar_expect_tx(&s.bars[i], (uint32_t)n * 16u);
      bulk_load(data + (size_t)i * part * 16, p.body + (size_t)i * part * 16, (uint32_t)n * 16u, &s.bars[i]);
    }
    s.cnt = s.failed = 0;
  }
  const RowCfg r = row_cfg<false>(a, b);
  if (rank == 0 && tid == 0) {
    if (r.k_bad) raise_status(a.status, ARCS_ERR_TOPK);
    if (!r.lists_ok) raise_status(a.status, ARCS_ERR_LIST);
  }
  // the elements outside the aligned body
  const int sc_n = p.head_n + p.tail_n;
  const int32_t sc_col = tid < p.head_n ? lo + tid : p.tail_first + tid - p.head_n;
  if (tid < sc_n) s.scal[tid] = __float_as_uint(Elem<T>::load(row + sc_col));
  // ---- the listed columns of the slice
  const bool lists = r.touched_on;
  const int L_all = lists && r.pen_on ? r.H : 0, NB = lists ? r.NB : 0;
  const int slots = res_slots(L_all);  // (what this row's history takes of the table)
  for (int i = tid; i < slots; i += NT) {
    h_col[i] = -1;
    h_info[i] = 0u;
  }
  __syncthreads();
  if (lists) {
    const int32_t Vg = a.v_global > 0 ? a.v_global : a.V;
    const int32_t w0 = window_start(r);
    // A column of the table counts its occurrences in the history and holds whether one lies in the
    // repeat window (bit 31). A warp enters a column it holds several times once.
    constexpr int kAhead = 4;  // entries a thread fetches at once
    for (int i0 = 0; i0 < L_all; i0 += kAhead * NT) {
      int32_t t[kAhead];
#pragma unroll
      for (int x = 0; x < kAhead; ++x) t[x] = i0 + x * NT + tid < L_all ? __ldg(&a.hist_ids[r.h0 + i0 + x * NT + tid]) : -1;
#pragma unroll
      for (int x = 0; x < kAhead; ++x) {
        const int32_t c = t[x] >= 0 && t[x] < Vg ? t[x] - a.id_base : -1;
        const bool in = c >= lo && c < hi;
        const unsigned any = __ballot_sync(0xFFFFFFFFu, in);
        if (!in) continue;
        const unsigned same = __match_any_sync(any, c);
        if (lane != __ffs(same) - 1) continue;
        const int at = res_find(h_col, slots, c, true);
        const int last = i0 + x * NT + (tid & ~31) + 31 - __clz(same);
        sm_red_add(&h_info[at], (uint32_t)__popc(same));
        if (last >= w0) sm_red_or(&h_info[at], 1u << 31);
      }
      __syncwarp();
    }
    for (int i = tid; i < NB; i += NT) {
      b_id[i] = __ldg(&a.bias_ids[r.q0 + i]);
      b_val[i] = __ldg(&a.bias_vals[r.q0 + i]);
    }
    __syncthreads();
  }
  bool ok = true;
  auto wait_part = [&](int i) {
    if (i * part < nchunk) ok = ok && mbar_wait_warp(&s.bars[i], 0u);
  };
  if (lists) {
    // What applies to a column, while the slice is on its way. It is taken by its first bias entry (bit 30
    // set there), or, without one, by its place in the table (bit 30 not set).
    constexpr uint32_t kBias = 1u << 30;
    for (int i = tid; i < NB; i += NT) {
      const int32_t c = b_id[i] - a.id_base;
      bool first = b_id[i] >= 0 && c >= lo && c < hi;
      for (int j = 0; j < i && first; ++j) first = b_id[j] != b_id[i];
      uint32_t o = 0u;
      if (first) {
        o = kBias;
        const int at = res_find(h_col, slots, c, false);
        if (at >= 0) {
          o |= h_info[at];
          h_info[at] = o;
        }
      }
      b_info[i] = o;
    }
    __syncthreads();
    for (int i = 0; i < kResParts; ++i) wait_part(i);
    // one column adjusted (tools/sampler.h:154-174): the raw logit from the slice, a NaN into its place
    for (int i = tid; i < NB + slots; i += NT) {
      const uint32_t o = i < NB ? b_info[i] : h_info[i - NB];
      const int32_t c = i < NB ? b_id[i] - a.id_base : h_col[i - NB];
      uint32_t* const key = i < NB ? &b_info[i] : &h_info[i - NB];
      if (i < NB ? !(o & kBias) : c < 0 || (o & kBias)) {
        *key = 0u;  // (no column of its own: as a NaN, never a candidate)
        continue;
      }
      float v;
      if (c >= p.body_first && c < p.tail_first) {
        T* at = reinterpret_cast<T*>(data) + (c - p.body_first);
        v = Elem<T>::from_smem(reinterpret_cast<const char*>(at));
        if (sizeof(T) == 4) *reinterpret_cast<uint32_t*>(at) = 0x7FFFFFFFu;
        else *reinterpret_cast<unsigned short*>(at) = 0x7FFFu;
      } else {
        uint32_t* at = &s.scal[c < p.body_first ? c - lo : p.head_n + c - p.tail_first];
        v = __uint_as_float(*at);
        *at = 0x7FFFFFFFu;
      }
      bool ban = false;
      for (int j = i; j < NB; ++j) {  // :154-155 in list order, duplicates add again
        if (b_id[j] != c + a.id_base) continue;
        if (b_val[j] > -100.0f) v = __fadd_rn(v, b_val[j]);
        else ban = true;
      }
      const uint32_t cnt = o & (kBias - 1u);
      if (cnt > 0) v = penalise(r, v, cnt, (o >> 31) != 0u);
      if (ban) v = ARCS_BANNED;                                                                        // :174
      *key = key_of(v);
    }
    __syncthreads();
  }

  // ---- the slice's threshold
  float own[kResOwn];
#pragma unroll
  for (int j = 0; j < kResOwn; ++j) own[j] = -INFINITY;
  for (int i = 0; i < kResParts; ++i) {
    wait_part(i);
    const int end = min(nchunk, (i + 1) * part);
    for (int c0 = i * part + tid; c0 < end; c0 += kRound) {
#pragma unroll
      for (int j = 0; j < kResOwn; ++j)
        if (c0 + j * NT < end) own[j] = fmaxf(own[j], Elem<T>::chunk_max(lds128(data + (size_t)(c0 + j * NT) * 16)));
    }
  }
  const float sc = tid < sc_n ? __uint_as_float(s.scal[tid]) : NAN;
  if (!ok) {
    // a copy did not land in time: all that were issued get one more bounded wait, so that none is
    // still on its way when the CTA gives its shared memory up
    for (int i = 0; i < kResParts; ++i)
      if (i * part < nchunk) mbar_wait_warp(&s.bars[i], 0u);
    s.failed = 1;
  }
  const int kB = r.kB;
  const bool few = kB <= 64;  // one maximum a thread gives a tight threshold
  {
    float m = fmaxf(own[0], sc);
#pragma unroll
    for (int j = 1; j < kResOwn; ++j) m = fmaxf(m, own[j]);
    if (few) {
      s.keys[tid] = m > -INFINITY ? key_of(m) : 0u;
    } else {
#pragma unroll
      for (int j = 0; j < kResOwn; ++j) s.keys[j * NT + tid] = own[j] > -INFINITY ? key_of(own[j]) : 0u;
      if (tid == NT - 1) s.keys[kResOwn * NT - 1] = 0u;  // (the search counts to 1023)
    }
  }
  __syncthreads();
  if (tid < 32) {
    const uint32_t k = few ? warp_kth16<NT / 32>(s.keys, kB) : warp_kth16<kResOwn * NT / 32>(s.keys, kB);
    if (tid == 0) s.floor = k ? ((unsigned long long)k << 32) - 1ull : 0ull;
  }
  __syncthreads();
  // ---- its candidates
  const int n_list = lists ? NB + slots : 0;  // places that may hold an adjusted column
  auto listed_key = [&](int i) { return i < NB ? b_info[i] : h_info[i - NB]; };
  auto listed_id = [&](int i) { return i < NB ? b_id[i] : h_col[i - NB] + a.id_base; };
  const unsigned long long flo = s.floor;
  {
    const uint32_t tkey = (uint32_t)((flo + 1ull) >> 32);
    const float tf = floor_value(flo ? tkey : 0u);
    auto keep = [&](uint32_t ky, int32_t id) {
      if (ky == 0u || comp_of(ky, id) <= flo) return;
      const uint32_t at = sm_atomic_add(&s.cnt, 1u);
      if (at < (uint32_t)kResCap) {
        s.key[at] = ky;
        s.id[at] = id;
      }
    };
    // the chunks behind a maximum that reaches it, looked through by the whole warp
#pragma unroll
    for (int j = 0; j < kResOwn; ++j) {
      unsigned hot = __ballot_sync(0xFFFFFFFFu, own[j] >= tf && !s.failed);
      while (hot != 0u) {
        const int src = (tid & ~31) + __ffs(hot) - 1;
        hot &= hot - 1u;
        for (int c = j * NT + src + lane * kRound; c < nchunk; c += 32 * kRound) {
          const uint4 q = lds128(data + (size_t)c * 16);
          uint32_t bits = 0;
#pragma unroll
          for (int e = 0; e < E; ++e) bits |= (Elem<T>::get(q, e) >= tf ? 1u : 0u) << e;
          while (bits != 0u) {
            const int e = __ffs(bits) - 1;
            bits &= bits - 1u;
            keep(key_of(elem_of_words<T>(q.x, q.y, q.z, q.w, e)), p.body_first + c * E + e + a.id_base);
          }
        }
      }
    }
    if (sc >= tf) keep(key_of(sc), sc_col + a.id_base);
    for (int i = tid; i < n_list; i += NT) keep(listed_key(i), listed_id(i));
  }
  __syncthreads();
  if (s.cnt > kResCap) {
    // too many (masses of equal logits, a handful of elements a thread): the k best, exactly, by pushes and prunes
    __syncthreads();  // (every thread has read the count that brings it here, before it is set to zero)
    if (tid == 0) {
      s.cnt = 0;
      s.tau = 0ull;
    }
    __syncthreads();
    const Sel sel{s.key, s.id, &s.cnt, &s.tau, kB, kResCap - NT, kResCap};
    const PruneScratch ps{s.keys, s.tk, s.ti, s.misc, &s.m64};
    for (int c0 = 0; c0 < nchunk; c0 += NT) {
      const int c = c0 + tid;
      const uint4 q = c < nchunk ? lds128(data + (size_t)c * 16) : make_uint4(0, 0, 0, 0);
      uint32_t bits = 0;
#pragma unroll
      for (int e = 0; e < E; ++e) bits |= (c < nchunk && comp_of(key_of(Elem<T>::get(q, e)), p.body_first + c * E + e + a.id_base) > s.tau ? 1u : 0u) << e;
      push_all<NT>(sel, ps, bits, [&](int e, uint32_t& ky, int32_t& id) {
        ky = key_of(elem_of_words<T>(q.x, q.y, q.z, q.w, e));
        id = p.body_first + c * E + e + a.id_base;
      });
    }
    push_all<NT>(sel, ps, tid < sc_n ? 1u : 0u, [&](int, uint32_t& ky, int32_t& id) {
      ky = key_of(sc);
      id = sc_col + a.id_base;
    });
    for (int i0 = 0; i0 < n_list; i0 += NT) {
      const int i = i0 + tid;
      push_all<NT>(sel, ps, i < n_list ? 1u : 0u, [&](int, uint32_t& ky, int32_t& id) {
        ky = listed_key(i);
        id = listed_id(i);
      });
    }
    __syncthreads();
  }

  // ---- the row: the first CTA takes the others' candidates
  cluster_arrive();
  cluster_wait();
  if (rank != 0) {
    cluster_arrive();
    cluster_wait();  // (its shared memory is read until then)
    return;
  }
  const Sel sel{s.mkey, s.mid, &s.mcnt, &s.tau, kB, kResCap - NT, kResCap};
  const PruneScratch ps{s.keys, s.tk, s.ti, s.misc, &s.m64};
  if (tid < 32) {
    const int n = lane < ctas ? min((int)cluster_ld(&s.cnt, lane), kResCap) : 0;
    unsigned long long f = lane < ctas ? cluster_ld64(&s.floor, lane) : 0ull;
    const bool bad = lane < ctas && cluster_ld(&s.failed, lane) != 0u;
    int inc = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xFFFFFFFFu, inc, d);
      if (lane >= d) inc += t;
    }
    f = warp_max_u64(f);  // (that slice alone holds k elements above it)
    if (lane < 16) s.off[lane + 1] = inc;
    const bool any_bad = __any_sync(0xFFFFFFFFu, bad);
    if (lane == 0) {
      s.off[0] = 0;
      s.tau = f;
      s.mcnt = 0;
      s.misc[4] = any_bad;
    }
  } else {
    for (int i = tid - 32; i < 256; i += NT - 32) s.keys[i] = 0u;
  }
  __syncthreads();
  const int total = s.off[ctas];
  if (total <= 4 * NT) {
    // As a rule: fetched in one go, and a tighter threshold read off their counts by the upper 16 bits
    // of their keys, before they are kept.
    uint32_t k0[4];
    int32_t i0[4];
    const uint32_t base = (uint32_t)(s.tau >> 48);
    const unsigned long long tau0 = s.tau;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int e = x * NT + tid;
      k0[x] = 0u;
      i0[x] = 0;
      if (e < total) {
        int g = 0;
        for (int y = 1; y < ctas; ++y) g += e >= s.off[y];
        k0[x] = cluster_ld(&s.key[e - s.off[g]], g);
        i0[x] = (int32_t)cluster_ld(&s.id[e - s.off[g]], g);
      }
    }
#pragma unroll
    for (int x = 0; x < 4; ++x)
      if (k0[x] != 0u && comp_of(k0[x], i0[x]) > tau0) sm_red_add(&s.keys[min((k0[x] >> 16) - base, 255u)], 1u);
    __syncthreads();
    if (tid < 32) {
      int d, kr;
      bool ex;
      find_bin(s.keys, kB, d, kr, ex);
      if (d > 0 && lane == 0) s.tau = max(tau0, ((unsigned long long)((base + (uint32_t)d) << 16) << 32) - 1ull);
    }
    __syncthreads();
    bool hot = false;
    const unsigned long long tau1 = s.tau;
#pragma unroll
    for (int x = 0; x < 4; ++x)
      if (x * NT < total) sel_offer(sel, k0[x] != 0u && comp_of(k0[x], i0[x]) > tau1, k0[x], i0[x], hot);
  } else {
    for (int e0 = 0; e0 < total; e0 += NT) {
      const int e = e0 + tid;
      int g = 0;
      for (int x = 1; x < ctas; ++x) g += e >= s.off[x];
      const bool have = e < total;
      push_all<NT>(sel, ps, have ? 1u : 0u, [&](int, uint32_t& ky, int32_t& id) {
        ky = cluster_ld(&s.key[e - s.off[g]], g);
        id = (int32_t)cluster_ld(&s.id[e - s.off[g]], g);
      });
    }
  }
  __syncthreads();
  cluster_arrive();
  if (s.misc[4]) {
    if (tid == 0) {
      raise_status(a.status, ARCS_ERR_TIMEOUT);
      a.token[b] = -1;
    }
    cluster_wait();
    return;
  }
  if (s.mcnt > 512) {
    sel_prune<1, NT>(sel, kB, ps, tid);
    __syncthreads();
  }
  // candidates best first: ranked by counting (composites are unique)
  const int m = min(s.mcnt, kResCap);
  const int nB = min(m, kB);
  for (int i = tid; i < m + 4; i += NT)
    if (i < kResCap) s.comp[i] = i < m ? comp_of(s.mkey[i], s.mid[i]) : 0ull;
  __syncthreads();
  for (int i = tid; i < m; i += NT) {
    const unsigned long long mine = s.comp[i];
    int above = 0;
#pragma unroll 4
    for (int j = 0; j < m; j += 2) {
      const ulonglong2 c = *reinterpret_cast<const ulonglong2*>(&s.comp[j]);
      above += (c.x > mine) + (c.y > mine);
    }
    if (above < nB) {
      s.sv[above] = value_of(comp_key(mine));
      s.sid[above] = comp_id(mine);
    }
  }
  __syncthreads();
  if (tid < 32) {
    bool bans = false;  // Sampler::bans_: any bias entry <= -100, in range or not (tools/sampler.h:34)
    for (int i = lane; i < r.NB && r.lists_ok; i += 32) bans = bans || __ldg(&a.bias_vals[r.q0 + i]) <= -100.0f;
    choose_token(a, b, r, __any_sync(0xFFFFFFFFu, bans), nB, s.sv, s.sid, s.spr, s.cum);
  }
  cluster_wait();
}

}  // namespace arcs
