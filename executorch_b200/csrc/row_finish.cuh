// Second kernel of the fast sampling path: one block per row turns what row_sweep.cuh left into the
// exact softmax sum and, for a nucleus (or top-k set) that fits the block's lists, into the token.
// Included by fast_path.cu inside its unnamed namespace (uses its helpers).
//
//   1. the row's unit records: which units are "events" (the running sum may leave its binade
//      there, or the row starts there), which lanes need another look
//   2. side by side: the exact terms of the event units; of every reported lane the 16 logits
//      again, its unsure terms exactly (their increments replace the approximate ones) and its
//      candidates exactly (listed). An exact half-way term makes its unit's increment depend on the
//      parity of the running significand: such a unit gets a two-parity summary.
//   3. one warp joins the runs of units between events and the events' terms, in order
//      (exact_math.cuh). Every assumption of the sweep is checked here -- a run must be entered in
//      its binade and must not leave it -- so the sum is the reference's or the row is
//      "undecided" and goes to sample_rows_kernel untouched
//   4. the rest of sample_topp / sample_topk on the candidate list (small_tail)
//
// What bounds it: latency. A row is some thousand terms' work in a chain of a dozen block-wide
// steps, so all rows of a batch run side by side, two blocks of 512 threads per SM.

constexpr int kFinThreads = kThreads;   // the tail's helpers are written for kThreads threads
constexpr int kFinEvents = 22;          // event units of a row (2 KB of shared memory each)
constexpr int kFinTables = 4;           // binades in which an event's terms are summarised
constexpr int kFinTies = 96;            // exact half-way terms
constexpr int kFinGroups = 6144;        // lanes that need another look
constexpr int kFinCand = 3072;          // candidates
constexpr int kFinFirst = 256;          // lanes whose candidates are listed at once
constexpr int kFinListLanes = 1536;     // up to this many lanes list their candidates one by one
constexpr int kFinBins = 4096;          // beyond that they are counted in bins (row_nucleus.cuh)
constexpr int kFinBinShift = 8;         // positions inside a bin
constexpr int kLongZones = 120;         // bins whose entries are added one by one
constexpr int kLongList = 1536;         // entries in those
constexpr int kNearPart = 376;          // nuclei of up to 16 times as many (a warp's part) are listed by index
constexpr int kNear = kNearPart * kWarps;
constexpr int kSampleHalfLanes = 6144;  // of longer rows a sample of this size says where the nucleus ends
constexpr int kLongTies = 24;           // half-way terms
constexpr int kLongBinade = 108;        // the lowest binade that a bin is rounded for
constexpr int kFinQueue = 64;           // a warp's queue of terms to evaluate

// How an event will probably go: the sum enters it in binade k, the lanes in front of lane l (32: all)
// add up to `front`, the 16 terms of lane l carry it into binade k2, and the lanes behind l add
// `behind` there. A half-way term on either side changes the increments by *_d when the significand
// in front of it (*_at increments in) is odd.
struct __align__(16) EventPlan {
  int k, l, front, upto;  // upto: with lane l's own increments in binade k
  int k2, behind;
  int front_at, front_d, behind_at, behind_d;
  int ok, pad;
};

// The tail's share: candidates by probability.
constexpr int kTailBins = 1024;      // value bins: exponent and 5 mantissa bits, from the floor up
constexpr int kTailBinShift = 18;
struct FinishTail {
  unsigned cnt[kTailBins], ofs[kTailBins];  // per bin: entries, and the sum of their 13 mantissa bits below the bin's
  unsigned first[kTailBins];                // entries in larger bins
  unsigned long long ck[kFinCand];          // (probability, inverted index), grouped by bin
  alignas(16) float p[kFinCand + 32];       // sorted
  int idx[kFinCand];
};

// Its share when the candidates are counted in bins (the counts are in FinishShared::hist).
struct __align__(16) FinishLongFront {
  uint8_t code[kFinBins];  // 128 + zone, or 1 + binade - kLongBinade
  alignas(4) uint16_t count[kFinBins];
  int zone_bin[kLongZones], zone_start[kLongZones], zone_n[kLongZones], zone_fill[kLongZones];
  int zone_k[kLongZones];         // the binade of the bins in front of a zone
  uint32_t zone_q[kLongZones];    // increments of all bins in front of it (modulo 2^32)
  float zone_in[kLongZones];      // the running sum in front of it
  int4 zone[kLongZones + 1];                        // in order: start, entries, zone_k, zone_q
  alignas(16) unsigned long long entry[kLongList];  // (probability, inverted index), grouped by zone
  alignas(16) float sorted[kLongList + 4];          // the probabilities in order
  uint16_t order[kLongList];                        // of `sorted`
  uint8_t zone_of[kLongList];
  int queue_fill[kWarps];
  int n_tie, tie[kLongTies];
  int n_near[kWarps];
};
struct FinishLong : FinishLongFront {
  char unused[kFinEvents * kUnit * sizeof(float) - sizeof(FinishLongFront)];
  uint16_t group_kept[kFinGroups];  // (the group list stays)
  union {
    struct {
      uint32_t queue[kWarps][kFinQueue];
      int members[kSwMaxUnits];
    };
    uint32_t near[kWarps][kNearPart + 64];
  };
};

// One row's constants for the passes of row_nucleus.cuh.
struct LongRow {
  const void* row;
  int shift, vocab, n_units;
  float inv_t, mx, raw_max, c1;
  // which half-lanes: of every lane, or of the group list
  int all, n_half;
  int step;  // every how many-th
  // the bins (BinMap)
  float scale;
  uint32_t limit;
  float x_lo, x_hi;  // a range of logits
  // the exact sum; terms are 2^(x c1 - r_row), times s_lo and s_hi in binade kLongBinade
  float sum, r_row, s_lo, s_hi;
};

struct __align__(16) FinishShared {
  static constexpr bool kExt = false;
  static constexpr bool kHasLut = false;
  uint64_t exp_tab[kExpTableSize];
  LongRow lr;
  float redf[kWarps];
  int redi[kWarps], redf_i[kWarps];
  SeqSummary wsum[3][kWarps];  // seqsum_tile
  int first[2];
  float s_bcast;
  int hit_found, hit_idx;
  float hit_val;
  int wcnt[kWarps];
  float wmass[kWarps];
  int tail_bin, tail_cnt, tail_last, tail_pos;
  float tail_cum, tail_mass;
  int misc_i[1];
  int level_cnt[kLevels];
  int n_task, n_task2, n_cand, n_tie, bad;
  float sum, coin, start_sum, mass;
  int ev_unit[kFinEvents + 1];
  float ev_sum[kFinEvents];  // what each event adds to the sum
  int4 run[kFinEvents + 1];  // between events: increments (entered even, odd), binade (0: only zeros)
  union alignas(16) {
    struct {
      float pool[kFinEvents][kUnit];       // exact terms of the event units, swizzled (pool_chunk)
      uint16_t group[kFinGroups];          // unit * 32 + lane; those with unsure terms first
      EventPlan plan[kFinEvents];
      float ev_tot[kFinEvents];                      // sums of the events' terms, roughly
      alignas(16) int tab_k[kFinEvents][kFinTables];             // the binades
      alignas(16) unsigned tab_tie[kFinEvents][kFinTables];      // lanes with an exact half-way term in that binade
      int tab_inc[kFinEvents][kFinTables][32];       // inclusive sums of the lanes' increments
      signed char tab_d[kFinEvents][kFinTables][32]; // change of a lane's increment when entered odd
      uint32_t tie[kFinTies];                        // padded position | kTieUp
      uint32_t info[kSwMaxUnits];
      int a0[kSwMaxUnits];                           // increments of the units, entered with an even significand
      signed char a1d[kSwMaxUnits];                  // the same for an odd one, minus a0
      uint32_t queue[kWarps][kFinQueue];   // terms to evaluate exactly: padded position | kQ...
    };
    FinishTail t;
    FinishLong l;
  } u;
  union {
    Entry cand[kFinCand];
    uint32_t hist[kFinBins];
  };
};
static_assert(sizeof(FinishLongFront) < kFinEvents * kUnit * sizeof(float), "the group list stays where it is");
static_assert(sizeof(FinishShared) <= 115712, "two blocks per SM");
constexpr uint32_t kTieUp = 1u << 31;
constexpr uint32_t kQCand = 1u << 31, kQUnsure = 1u << 30, kQPos = (1u << 30) - 1u;

// Slot of the 16-byte chunk `c` (terms 4 c ...) of an event's terms: rotated so that the 16
// consecutive terms of neighbouring lanes fall into distinct banks.
__device__ __forceinline__ int pool_chunk(int c) { return c ^ ((c >> 3) & 7); }

// A lane's 16 logits of the unit at padded position p0 (unit_pos order); -inf outside the row.
template <typename T>
__device__ __forceinline__ void load8_padded(const T* row, int shift, int vocab, int p, float (&x)[8]) {
  const int i0 = p - shift;
  if (i0 >= 0 && i0 + 8 <= vocab) {
    const uint4* src = reinterpret_cast<const uint4*>(row + i0);
    if constexpr (sizeof(T) == 4) {
      const uint4 a = __ldg(src), b = __ldg(src + 1);
      x[0] = __uint_as_float(a.x); x[1] = __uint_as_float(a.y); x[2] = __uint_as_float(a.z); x[3] = __uint_as_float(a.w);
      x[4] = __uint_as_float(b.x); x[5] = __uint_as_float(b.y); x[6] = __uint_as_float(b.z); x[7] = __uint_as_float(b.w);
    } else {
      const uint4 a = __ldg(src);
      const T* t = reinterpret_cast<const T*>(&a);
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = to_f32(t[j]);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = (i0 + j >= 0 && i0 + j < vocab) ? to_f32(row[i0 + j]) : -INFINITY;
  }
}
template <typename T>
__device__ __forceinline__ void load_unit_lane(const T* row, int shift, int vocab, int p0, float (&x)[16]) {
  const int lane = threadIdx.x & 31;
  const int i0 = p0 - shift;
  if (i0 >= 0 && i0 + kUnit <= vocab) {  // the usual case; every load in flight at once
    constexpr int kV = sizeof(T) / 2;
    uint4 raw[2 * kV];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int v = 0; v < kV; ++v)
        raw[q * kV + v] = __ldg(reinterpret_cast<const uint4*>(row + i0 + unit_pos(lane, q)) + v);
    const T* t = reinterpret_cast<const T*>(raw);
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = to_f32(t[j]);
  } else {
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = i0 + unit_pos(lane, q) + j;
        x[q * 8 + j] = (i >= 0 && i < vocab) ? to_f32(row[i]) : -INFINITY;
      }
  }
}

struct FinishArgs {
  SweepArgs s;
  unsigned long long* rng_states;
  int64_t* out_ids;
  PeerOut peers;
  int* retry_rows;
  int* retry_count;
  int* retry_count_next;  // cleared for the next call, or null
};

// Ordered composition of the lanes' summaries; the result is in every lane.
__device__ __forceinline__ SeqSummary warp_compose(SeqSummary s) {
  const int lane = threadIdx.x & 31;
  if (!__any_sync(0xffffffffu, s.a0 != s.a1)) {
    const unsigned t = __reduce_add_sync(0xffffffffu, (unsigned)s.a0);  // 32 * kSeqSat = 2^31
    s.a0 = s.a1 = t < (unsigned)kSeqSat ? (int)t : kSeqSat;
    return s;
  }
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    SeqSummary o;
    o.a0 = __shfl_up_sync(0xffffffffu, s.a0, d);
    o.a1 = __shfl_up_sync(0xffffffffu, s.a1, d);
    if (lane >= d) s = seq_compose(o, s);
  }
  s.a0 = __shfl_sync(0xffffffffu, s.a0, 31);
  s.a1 = __shfl_sync(0xffffffffu, s.a1, 31);
  return s;
}

// Exclusive block-wide prefix sum of a non-negative count. One barrier; the slots are free again
// after the next one.
__device__ __forceinline__ int finish_scan(int* slots, int v, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += o;
  }
  if (lane == 31) slots[warp] = inc;
  __syncthreads();
  const int w = lane < kWarps ? slots[lane] : 0;
  *total = __reduce_add_sync(0xffffffffu, w);
  return __reduce_add_sync(0xffffffffu, lane < warp ? w : 0) + inc - v;
}

// The exact terms of one event unit into the pool, and its summaries in the binades that the
// sweep's estimate leaves open (by one warp).
template <typename T, typename Term>
__device__ __forceinline__ void finish_event(FinishShared& sm, const T* row, int shift, int vocab, int e, Term exact_term) {
  const int lane = threadIdx.x & 31;
  const int u = sm.ev_unit[e];
  float4* pool4 = reinterpret_cast<float4*>(sm.u.pool[e]);
  {
    float x[16];
    load_unit_lane(row, shift, vocab, u * kUnit, x);
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = exact_term(x[j]);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int c = q * 64 + lane * 2;
      pool4[pool_chunk(c)] = make_float4(x[q * 8], x[q * 8 + 1], x[q * 8 + 2], x[q * 8 + 3]);
      pool4[pool_chunk(c + 1)] = make_float4(x[q * 8 + 4], x[q * 8 + 5], x[q * 8 + 6], x[q * 8 + 7]);
    }
  }
  __syncwarp();
  if (e == 0) {
    // the row's first terms that are not zero: nothing is in front of them, so the sum can be formed
    // at once (it leaves a binade every few terms: plain additions, by every lane alike)
    float s = 0.0f;
#pragma unroll 8
    for (int c = 0; c < kUnit / 4; ++c) {
      const float4 f = pool4[pool_chunk(c)];
      s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, f.x), f.y), f.z), f.w);
    }
    if (lane == 0) sm.start_sum = s;
    return;
  }
  float v[16];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 f = pool4[pool_chunk(lane * 4 + q)];
    v[4 * q] = f.x;
    v[4 * q + 1] = f.y;
    v[4 * q + 2] = f.z;
    v[4 * q + 3] = f.w;
  }
  float tot = 0.0f;
#pragma unroll
  for (int j = 0; j < 16; ++j) tot += v[j];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, d);
  if (lane == 0) sm.u.ev_tot[e] = tot;
  const uint32_t info = sm.u.info[u];
  const int klo = unit_binade(info), span = (int)unit_span(info);
  const int nt = span == (int)kUnitSpanOpen ? 0 : (span < kFinTables - 1 ? span + 1 : kFinTables);
  for (int t = 0; t < kFinTables; ++t) {
    // the lowest two and the highest two of the open binades
    const int k = t < nt ? (t < 2 ? klo + t : klo + span - (nt - 1 - t)) : 0;
    if (lane == 0) sm.u.tab_k[e][t] = k;
    if (k == 0) continue;
    // increments as in chunk_increment_fast: exact unless a term is 2^23 units or more, and then
    // the sum leaves the binade anyway
    const float inv_u = seq_inv_u(k);
    float acc0 = 0.0f, acc1 = 0.0f, md = 0.0f;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float tt = __fmaf_rn(v[j], inv_u, 8388608.0f);
      const float q = __fsub_rn(tt, 8388608.0f);
      md = fmaxf(md, fabsf(__fmaf_rn(v[j], inv_u, -q)));
      if (j & 1) acc1 = __fadd_rn(acc1, q); else acc0 = __fadd_rn(acc0, q);
    }
    int inc = (int)fminf(__fadd_rn(acc0, acc1), 33554432.0f);
    const unsigned ties = __ballot_sync(0xffffffffu, !(md < 0.5f));
    if (ties != 0u) {
      // exact half-way terms: two-parity summaries of the lanes that hold them
      int d = 0;
      if (!(md < 0.5f)) {
        SeqSummary two;
        seq_identity(&two);
#pragma unroll
        for (int j = 0; j < 16; ++j) seq_push_scaled(&two, v[j], inv_u);
        inc = two.a0;
        d = two.a1 - two.a0;
      }
      sm.u.tab_d[e][t][lane] = (signed char)d;
    }
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += o;
    }
    sm.u.tab_inc[e][t][lane] = inc;
    if (lane == 0) sm.u.tab_tie[e][t] = ties;
  }
}

// Adds the terms of event e to the exact running sum s (one warp, warp-uniform s): lanes are applied
// by their summaries up to the first whose terms carry the sum out of its binade; those 16
// terms are added for real, and so on.
__device__ __forceinline__ float finish_apply_event(FinishShared& sm, int e, float s) {
  const int lane = threadIdx.x & 31;
  const float4* pool4 = reinterpret_cast<const float4*>(sm.u.pool[e]);
  int f = 0;  // lanes in front of f are in s
  while (f < 32) {
    const int k = seq_kb(s), n = seq_n(s);
    const unsigned has = __ballot_sync(0xffffffffu, lane < kFinTables && sm.u.tab_k[e][lane & (kFinTables - 1)] == k);
    if (has == 0u) break;
    const int t = __ffs(has) - 1;
    const int inc = sm.u.tab_inc[e][t][lane];
    unsigned ties = sm.u.tab_tie[e][t];
    const int base = f > 0 ? __shfl_sync(0xffffffffu, inc, f - 1) : 0;
    int end = n + (inc - base);  // the significand behind this lane (lanes from f on)
    for (ties = ties >> f << f; ties != 0u; ties &= ties - 1u) {
      const int l = __ffs(ties) - 1;
      const int in = l > f ? __shfl_sync(0xffffffffu, end, l - 1) : n;
      if ((in & 1) && lane >= l) end += sm.u.tab_d[e][t][l];
    }
    const unsigned out = __ballot_sync(0xffffffffu, lane >= f && end >= kSeqLimit);
    const int l = out != 0u ? __ffs(out) - 1 : 32;
    if (l < 32) {
      float4 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = pool4[pool_chunk(l * 4 + q)];
      const int before = __shfl_sync(0xffffffffu, end, l > 0 ? l - 1 : 0);
      s = seq_value(k, l > f ? before : n);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, v[q].x), v[q].y), v[q].z), v[q].w);
      f = l + 1;
    } else {
      return seq_value(k, __shfl_sync(0xffffffffu, end, 31));
    }
  }
  if (f < 32) {
    // no summary for this binade: the general way for the other lanes
    float v[kChunk];
#pragma unroll
    for (int q = 0; q < kChunk / 4; ++q) {
      const float4 x = pool4[pool_chunk(lane * 4 + q)];
      v[4 * q] = lane >= f ? x.x : 0.0f;
      v[4 * q + 1] = lane >= f ? x.y : 0.0f;
      v[4 * q + 2] = lane >= f ? x.z : 0.0f;
      v[4 * q + 3] = lane >= f ? x.w : 0.0f;
    }
    int hp;
    float hs;
    seqsum_warp<false>(v, s, 0.0f, 0, 0, &hp, &hs);
  }
  return s;
}

// The rest of sample_topp / sample_topk on the row's candidates (all of them in sm.cand, unordered):
// value bins over the probabilities, from the largest bin down to the first that surely holds the
// nucleus (or the k largest); those entries grouped by bin and ranked inside their bin, i.e.
// sorted by (probability descending, index ascending); then the reference's cumulative sum
// (sampler.cpp:146-156; the top-k sum of :105-108) and draw (:162-169), whose sums are the same
// numbers in the same order. Returns false, with nothing decided, when the list does not hold the
// nucleus; *mass is then the mass it does hold. `complete`: the list holds every entry that passes
// the crop.
__device__ __forceinline__ bool finish_tail(FinishShared& sm, float e_floor, float sum, float cutoff, float topp, int topk,
                                            bool use_topk, bool complete, float coin, int* token, float* mass) {
  FinishTail& t = sm.u.t;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = sm.n_cand;
  for (int b = tid; b < kTailBins; b += kFinThreads) t.cnt[b] = t.ofs[b] = 0u;
  if (tid == 0) {
    sm.tail_bin = -1;
    sm.tail_pos = 0x7fffffff;
  }
  __syncthreads();
  const int base = (int)(f32_bits(__fdiv_rn(e_floor, sum)) >> kTailBinShift);  // bin of the smallest probability
  for (int i = tid; i < n; i += kFinThreads) {
    const uint32_t pb = f32_bits(__fdiv_rn(bits_f32(sm.cand[i].key), sum));
    sm.cand[i].key = pb;
    int b = (int)(pb >> kTailBinShift) - base;
    b = b < kTailBins ? b : kTailBins - 1;
    if (use_topk || bits_f32(pb) >= cutoff) {  // the crop (sampler.cpp:136-143)
      atomicAdd(&t.cnt[b], 1u);
      atomicAdd(&t.ofs[b], (pb >> 5) & 0x1FFFu);
    }
  }
  __syncthreads();
  // thread t: bins 1023 - 2 t and 1022 - 2 t; counts and masses (rounded down) of the larger bins
  const int b0 = kTailBins - 1 - 2 * tid, b1 = b0 - 1;
  const int c0 = (int)t.cnt[b0], c1 = (int)t.cnt[b1];
  auto bin_mass = [&](int b, int c) {
    const uint32_t edge = (uint32_t)(b + base) << kTailBinShift;
    return (float)c * bits_f32(edge) + (float)t.ofs[b] * (bits_f32(edge & 0x7F800000u) * (32.0f / 8388608.0f));
  };
  const float m0 = c0 > 0 ? bin_mass(b0, c0) : 0.0f, m1 = c1 > 0 ? bin_mass(b1, c1) : 0.0f;
  int ci = c0 + c1;
  float mi = m0 + m1;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int oc = __shfl_up_sync(0xffffffffu, ci, d);
    const float om = __shfl_up_sync(0xffffffffu, mi, d);
    if (lane >= d) {
      ci += oc;
      mi += om;
    }
  }
  if (lane == 31) {
    sm.wcnt[warp] = ci;
    sm.wmass[warp] = mi;
  }
  __syncthreads();
  int pre_c = 0, all_c = 0;
  float pre_m = 0.0f, all_m = 0.0f;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const int c = sm.wcnt[w];
    const float m = sm.wmass[w];
    if (w < warp) {
      pre_c += c;
      pre_m += m;
    }
    all_c += c;
    all_m += m;
  }
  ci += pre_c;
  mi += pre_m;
  t.first[b0] = (unsigned)(ci - c0 - c1);
  t.first[b1] = (unsigned)(ci - c1);
  // the margin covers the rounding of the reference's own running sum
  auto enough = [&](int c, float m) {
    return use_topk ? c >= topk : m >= topp * 1.002f + 0.001f + (float)c * 4.8e-7f;
  };
  const int found = __reduce_max_sync(0xffffffffu, enough(ci - c1, mi - m1) ? b0 : (enough(ci, mi) ? b1 : -1));
  if (lane == 0 && found >= 0) atomicMax(&sm.tail_bin, found);
  __syncthreads();
  *mass = all_m;
  const bool whole = sm.tail_bin < 0;  // everything listed is needed
  if (whole && !complete) return false;
  const int bin_lo = whole ? 0 : sm.tail_bin;
  const int n_b = whole ? all_c : (int)(t.first[bin_lo] + t.cnt[bin_lo]);
  if (n_b <= 0) return false;
  __syncthreads();
  for (int b = tid; b < kTailBins; b += kFinThreads) t.ofs[b] = t.first[b];  // fill pointers
  __syncthreads();
  for (int i = tid; i < n; i += kFinThreads) {
    const Entry en = sm.cand[i];
    int b = (int)(en.key >> kTailBinShift) - base;
    b = b < kTailBins ? b : kTailBins - 1;
    if (b >= bin_lo && (use_topk || bits_f32(en.key) >= cutoff)) {
      t.ck[atomicAdd(&t.ofs[b], 1u)] = ((unsigned long long)en.key << 32) | (uint32_t)(0x7FFFFFFF - en.idx);
    }
  }
  __syncthreads();
  for (int i = tid; i < n_b; i += kFinThreads) {
    const unsigned long long mine = t.ck[i];
    int b = (int)((uint32_t)(mine >> 32) >> kTailBinShift) - base;
    b = b < kTailBins ? b : kTailBins - 1;
    const int lo = (int)t.first[b], hi = lo + (int)t.cnt[b];
    int rank = lo;
    for (int j = lo; j < hi; ++j) rank += t.ck[j] > mine ? 1 : 0;
    t.p[rank] = bits_f32((uint32_t)(mine >> 32));
    t.idx[rank] = (int)(0x7FFFFFFFu - (uint32_t)(mine & 0xFFFFFFFFull));
  }
  // what is added: everything sorted, or the k largest; zeros behind it change no sum
  const int lim = use_topk && topk < n_b ? topk : n_b;
  __syncthreads();
  if (tid < 32 && lim + tid < kFinCand + 32) t.p[lim + tid] = 0.0f;
  __syncthreads();
  float* prefix = reinterpret_cast<float*>(t.ck);  // the partial sums (the keys are not needed any more)
  if (lim <= kRankSortMax) {
    // one thread adds 16 at a time, the next 16 already on their way
    if (tid == 0) {
      const float4* p4 = reinterpret_cast<const float4*>(t.p);
      float4* pre4 = reinterpret_cast<float4*>(prefix);
      float acc = 0.0f;
      int last = -1;
      float4 q[4], nq[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) q[k] = p4[k];
      for (int i = 0; i < lim; i += 16) {
#pragma unroll
        for (int k = 0; k < 4; ++k) nq[k] = p4[(i >> 2) + 4 + k];  // at most 16 entries behind the padding's start
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float4 o;
          o.x = acc = __fadd_rn(acc, q[k].x);
          o.y = acc = __fadd_rn(acc, q[k].y);
          o.z = acc = __fadd_rn(acc, q[k].z);
          o.w = acc = __fadd_rn(acc, q[k].w);
          pre4[(i >> 2) + k] = o;
          q[k] = nq[k];
        }
        if (!use_topk && acc > topp) {  // the partial sums only grow: the first one above topp is among these
          last = i;
          break;
        }
      }
      sm.tail_last = last;
    }
    __syncthreads();
    int last = sm.tail_last;
    if (last >= 0) {
      if (tid < 32) {
        const unsigned above = __ballot_sync(0xffffffffu, lane < 16 && prefix[last + lane] > topp);
        if (lane == 0) sm.tail_last = last + __ffs(above) - 1;
      }
      __syncthreads();
      last = sm.tail_last;
    } else if (use_topk || (whole && complete)) {
      // top-k keeps its k entries; top-p keeps everything when the sum never exceeds topp
      // (the "in case of rounding errors" branch, sampler.cpp:152)
      last = lim - 1;
    } else {
      return false;
    }
    const float rr = __fmul_rn(coin, prefix[last]);  // sampler.cpp:162
    const bool above = tid <= last && prefix[tid] > rr;
    const unsigned bal = __ballot_sync(0xffffffffu, above);
    if (bal != 0u && lane == 0) atomicMin(&sm.tail_pos, (tid & ~31) + __ffs(bal) - 1);
    __syncthreads();
    const int fa = sm.tail_pos;
    *token = t.idx[fa <= last ? fa : last];
    return true;
  }
  // a longer list: by tiles of the whole block
  int rp = 0;
  auto search = [&](float thr, int limit, int* pos, float* cum) {
    float s = 0.0f;
    for (int tb = 0; tb < limit; tb += kTile) {
      float v[kChunk];
#pragma unroll
      for (int j = 0; j < kChunk; ++j) {
        const int k = tb + tid * kChunk + j;
        v[j] = k < limit ? t.p[k] : 0.0f;
      }
      if (seqsum_tile<true>(sm, v, s, rp, thr, tb, limit, pos, cum)) return true;
    }
    *cum = s;
    return false;
  };
  int last = lim - 1;
  float cum;
  if (use_topk) {
    search(INFINITY, lim, &last, &cum);
    last = lim - 1;
  } else if (!search(topp, lim, &last, &cum)) {
    if (!(whole && complete)) return false;
    last = lim - 1;
  }
  int pos = last;
  float at;
  if (!search(__fmul_rn(coin, cum), last + 1, &pos, &at)) pos = last;
  *token = t.idx[pos];
  return true;
}

// Adds the terms of event e to the exact running sum s, looking for the first position at which it
// exceeds thr (seqsum_warp). p0: position of the event's first term in the row.
__device__ __forceinline__ bool finish_search_event(FinishShared& sm, int e, float& s, float thr, int p0, int vocab, int* hit) {
  const int lane = threadIdx.x & 31;
  const float4* pool4 = reinterpret_cast<const float4*>(sm.u.pool[e]);
  float v[kChunk];
#pragma unroll
  for (int q = 0; q < kChunk / 4; ++q) {
    const float4 x = pool4[pool_chunk(lane * 4 + q)];
    v[4 * q] = x.x;
    v[4 * q + 1] = x.y;
    v[4 * q + 2] = x.z;
    v[4 * q + 3] = x.w;
  }
  float at;
  return seqsum_warp<true>(v, s, thr, p0, vocab, hit, &at);
}

#include "row_nucleus.cuh"

// Lane e: the plan of event e, from the sum in front of it as the runs and events in front of it
// estimate it (good to a few hundred units of the last place; a lane's increments are thousands).
__device__ __forceinline__ void plan_event(FinishShared& sm, int e, float in) {
  EventPlan p = {};
  const int k = seq_kb(in), n = seq_n(in);
  const int4 tk = *reinterpret_cast<const int4*>(sm.u.tab_k[e]);
  auto table = [&](int b) { return tk.x == b ? 0 : (tk.y == b ? 1 : (tk.z == b ? 2 : (tk.w == b ? 3 : -1))); };
  const int t = table(k);
  if (t >= 0) {
    const int* inc = sm.u.tab_inc[e][t];
    int l = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (n + inc[l + step - 1] < kSeqLimit) l += step;
    if (l == 31 && n + inc[31] < kSeqLimit) l = 32;
    p.k = k;
    p.l = l;
    p.front = l > 0 ? inc[l - 1] : 0;
    p.ok = 1;
    auto half_way = [&](unsigned ties, const int* a, int tt, int base, int* at, int* d) {
      if (__popc(ties) > 1) p.ok = 0;
      if (ties != 0u) {
        const int q = __ffs(ties) - 1;
        *at = (q > 0 ? a[q - 1] : 0) - base;
        *d = sm.u.tab_d[e][tt][q];
      }
    };
    half_way(sm.u.tab_tie[e][t] & (l < 32 ? (1u << l) - 1u : 0xFFFFFFFFu), inc, t, 0, &p.front_at, &p.front_d);
    if (l < 32) {
      p.upto = inc[l];
      const long long after = (long long)n + inc[l];  // in units of binade k
      p.k2 = k + (31 - __clz((int)(after >> 23)));
      const int t2 = table(p.k2);
      if (t2 < 0 || p.k2 == k) {
        p.ok = 0;
      } else {
        const int* inc2 = sm.u.tab_inc[e][t2];
        p.behind = inc2[31] - inc2[l];
        if ((after >> (p.k2 - k)) + p.behind >= kSeqLimit - 64) p.ok = 0;  // probably leaves that binade, too
        half_way(sm.u.tab_tie[e][t2] & (l < 31 ? 0xFFFFFFFFu << (l + 1) : 0u), inc2, t2, inc2[l], &p.behind_at,
                 &p.behind_d);
      }
    }
  }
  sm.u.plan[e] = p;
}

// The exact sequential sum of the row from its runs and events, by one warp; with kMulti up to the
// first position at which it exceeds thr, looked for in the events from unit hit_unit on (*hit >= 0
// when there is one). False when an assumption of the sweep does not hold.
//
// It is one chain of dependent steps over some ten events, so each step is made short: where an event
// leaves its binade is worked out beforehand from estimates, a lane per event, and what remains in
// the chain is to check that, an integer addition, 16 float additions, and another integer addition
// (130 cycles; the general form with its votes and shuffles takes 1200). An event that goes
// differently takes the general form.
template <bool kMulti>
__device__ __forceinline__ bool finish_replay(FinishShared& sm, int n_ev, float thr, int hit_unit, int shift, int vocab,
                                           float* sum, int* hit) {
  const int lane = threadIdx.x & 31;
  {
    const int4 r4 = lane <= n_ev ? sm.run[lane] : make_int4(0, 0, 0, 0);
    const float run = r4.z > 0 ? (float)r4.x * bits_f32((uint32_t)(r4.z > 23 ? r4.z - 23 : 0) << 23) : 0.0f;
    const float tot = lane < n_ev ? (lane == 0 ? sm.start_sum : sm.u.ev_tot[lane]) : 0.0f;
    float in = run + tot;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const float o = __shfl_up_sync(0xffffffffu, in, d);
      if (lane >= d) in += o;
    }
    const float before = __shfl_up_sync(0xffffffffu, in, 1);
    if (lane > 0 && lane < n_ev) plan_event(sm, lane, before + run);
  }
  __syncwarp();
  float s = 0.0f;
#pragma unroll 1
  for (int e = 0; e <= n_ev; ++e) {
    const int4 r4 = sm.run[e];
    int k = seq_kb(s), n = seq_n(s);
    if (r4.z != 0) {
      n += (n & 1) ? r4.y : r4.x;  // at most 2^24 + 2^26
      if (r4.z != k || n >= kSeqLimit) return false;
      s = seq_value(k, n);
      if (kMulti && !(s <= thr)) return false;
    }
    if (e == n_ev) break;
    const float before = s;
    if (kMulti && sm.ev_unit[e] >= hit_unit) {
      if (finish_search_event(sm, e, s, thr, sm.ev_unit[e] * kUnit - shift, vocab, hit)) break;
    } else if (e == 0) {
      s = sm.start_sum;
    } else {
      const EventPlan p = sm.u.plan[e];
      const float4* pool4 = reinterpret_cast<const float4*>(sm.u.pool[e]);
      float4 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = pool4[pool_chunk((p.l & 31) * 4 + q)];
      int in = n + p.front;
      if ((n + p.front_at) & 1) in += p.front_d;
      bool good = p.ok != 0 && p.k == k && in < kSeqLimit;
      float r = seq_value(k, in);
      if (p.l < 32) {
        good = good && n + p.upto >= kSeqLimit + 2;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          r = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(r, v[q].x), v[q].y), v[q].z), v[q].w);
        const int n2 = seq_n(r);
        int out = n2 + p.behind;
        if ((n2 + p.behind_at) & 1) out += p.behind_d;
        good = good && seq_kb(r) == p.k2 && out < kSeqLimit;
        r = seq_value(p.k2, out);
      }
      s = good ? r : finish_apply_event(sm, e, s);
      if (kMulti && !(s <= thr)) return false;  // the estimate says so
    }
    if (!(s < 3.0e38f)) return false;
    if (kMulti && lane == 0) sm.ev_sum[e] = s - before;
  }
  *sum = s;
  return true;
}

// kMulti: some row may be sampled without a crop (the second pass, which costs registers).
template <typename T, bool kMulti>
__global__ void __launch_bounds__(kFinThreads, 2) row_finish_kernel(const FinishArgs fa, ExpTable table) {
  extern __shared__ __align__(16) unsigned char finish_smem[];
  FinishShared& sm = *reinterpret_cast<FinishShared*>(finish_smem);
  const SweepArgs& a = fa.s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t i = blockIdx.x, r = a.row0 + i;
  const T* row = static_cast<const T*>(a.logits) + r * a.row_stride;
  const int shift = row_shift(row), vocab = a.vocab;
  const int n_units = (shift + vocab + kUnit - 1) / kUnit;
  grid_launch_dependents();  // the pass over the rows handed on may take its place
  if (tid < kExpTableSize) sm.exp_tab[tid] = table.t[tid];
  sm.u.a1d[tid] = 0;
  if (tid == 0) sm.mass = 0.0f;
  if (tid == 0) sm.n_task = sm.n_task2 = sm.n_cand = sm.n_tie = sm.bad = 0;
  grid_dependency_wait();  // the sweep's records are complete and visible from here on

  // ---- 1. the unit records (the row's head and RNG state meanwhile). Past the L1 cache: a block that
  // became resident early may share its SM with readers of older contents.
  uint4 rec = make_uint4(0u, 0u, kUnitZero, 0u), lv4 = make_uint4(~0u, ~0u, ~0u, ~0u);
  if (tid < n_units) {
    const uint4* src = reinterpret_cast<const uint4*>(a.units + i * (int64_t)a.units_pitch + tid);
    rec = __ldcg(src);
    lv4 = __ldcg(src + 1);
  }
  const uint32_t level[4] = {lv4.x, lv4.y, lv4.z, lv4.w};
  const float4 head4 = __ldcg(reinterpret_cast<const float4*>(a.heads + r));
  unsigned long long rng = 0ull;
  if (tid == 0) {
    if (fa.rng_states != nullptr) rng = fa.rng_states[r];
    if (blockIdx.x == 0 && fa.retry_count_next != nullptr) *fa.retry_count_next = 0;
  }
  const RowMode mode = row_mode(a, r);
  const bool use_topk = mode.topk > 0;
  const bool use_topp = !use_topk && mode.topp > 0.0f && mode.topp < 1.0f;
  const bool use_list = use_topk || use_topp;
  const float inv_t = mode.inv_t;
  const float mx = head4.x, raw_max = head4.y;
  const int head_state = __float_as_int(head4.w);
  int token = 0;
  // a greedy row among sampled ones: its argmax lies in a lane on level 0
  if (mode.greedy) {
    sm.misc_i[0] = 0x7fffffff;
    __syncthreads();
    int best = 0x7fffffff;
    for (unsigned m = tid < n_units ? lanes_up_to(level, 0) : 0u; m != 0u; m &= m - 1u) {
      const int l = __ffs(m) - 1;
      for (int q = 0; q < 2; ++q) {
        const int p = tid * kUnit + unit_pos(l, q);
        float x[8];
        load8_padded(row, shift, vocab, p, x);
#pragma unroll
        for (int j = 7; j >= 0; --j)
          if (x[j] == raw_max && p + j >= shift && p + j - shift < best) best = p + j - shift;
      }
    }
    best = __reduce_min_sync(0xffffffffu, best);
    if (lane == 0) atomicMin(&sm.misc_i[0], best);
    __syncthreads();
    // strict '>' in index order (sampler.cpp:44-56): a NaN in element 0 is never replaced, and of
    // equal maxima (all -inf included) the first stays
    const float first = to_f32(row[0]);
    best = sm.misc_i[0];
    store_token(fa.out_ids, fa.peers, r, (first != first || best >= vocab || raw_max == -INFINITY) ? 0 : best);
    return;
  }
  const float c1 = __fmul_rn(inv_t, kLog2eHi);
  if (use_list && tid == 0) {
    LongRow& lr = sm.lr;
    lr.row = row;
    lr.shift = shift;
    lr.vocab = vocab;
    lr.n_units = n_units;
    lr.inv_t = inv_t;
    lr.mx = mx;
    lr.raw_max = raw_max;
    lr.c1 = c1;
    lr.step = 1;
  }
  const RowScale rs = row_scale(mx);
  // The terms of the sum being formed: e (first pass), or e / sum (multinomial, second pass: the
  // running cdf of sampler.cpp:58-70, up to the unit in which it passes the coin)
  float sum = 1.0f, inv_sum = 1.0f, thr = INFINITY;
  bool probs = false;
  int hit_unit = 0x7fffffff;  // first unit in which the running sum may pass thr
  auto exact_term = [&](float x) {
    const float e = expf_ref(__fsub_rn(__fmul_rn(x, inv_t), mx), sm.exp_tab);
    return kMulti && probs ? __fdiv_rn(e, sum) : e;
  };
  auto scales = [&](uint32_t info, float* lo, float* hi) {
    unit_scales(rs, mx, unit_ref(info), unit_binade(info), lo, hi);
    if (kMulti && probs) {  // three more roundings
      *lo *= inv_sum * (1.0f - 4e-7f);
      *hi *= inv_sum * (1.0f + 4e-7f);
    }
  };

  bool decided = head_state >= 0 && fabsf(mx) < 10000.0f;  // block-uniform throughout
  int known = kRowUnknown;

  bool listing = use_list;
  bool counted = false, all_lanes = false;  // candidates are counted in bins; those of every lane
  int n_more = 0;        // lanes that are looked at for candidates in a second round
  float e_floor = INFINITY, list_floor = INFINITY;
  const float cutoff = __fdiv_rn(__fsub_rn(1.0f, mode.topp), (float)(vocab - 1));
  const float temperature = 1.0f / inv_t;
  for (;;) {
    const bool zero = (rec.z & kUnitZero) != 0u;
    const bool event = !zero && (unit_span(rec.z) != 0u || (kMulti && tid >= hit_unit));
    sm.u.info[tid] = rec.z;
    sm.u.a0[tid] = (zero || event) ? 0 : (int)rec.x;
    const unsigned unsure_mask = (zero || event) ? 0u : rec.y;
    int n_groups, n_unsure, n_ev;
    int top_level = -1;
    {
      if (use_list) {
        // lanes on every level, and from them the level down to which candidates are listed first: for
        // top-k the first with at least k lanes (every such lane holds an entry that large, so the k
        // largest are among what is listed); for top-p as many levels as kFinFirst lanes cover
        if (tid < kLevels) sm.level_cnt[tid] = 0;
        __syncthreads();
        int mine = 0;
#pragma unroll
        for (int t = 0; t < kLevels - 1; ++t) {
          const int c = __reduce_add_sync(0xffffffffu, tid < n_units ? __popc(lanes_up_to(level, t)) : 0);
          if (lane == t) mine = c;
        }
        if (lane < kLevels - 1 && mine > 0) atomicAdd(&sm.level_cnt[lane], mine);
        __syncthreads();
        const int upto = lane < kLevels - 1 ? sm.level_cnt[lane] : 0x7fffffff;
        const unsigned b = __ballot_sync(0xffffffffu, use_topk ? upto >= mode.topk : upto > kFinFirst);
        top_level = use_topk ? __ffs(b) - 1 : __ffs(b) - 2;  // bit kLevels - 1 is set in any case
        if (top_level > kLevels - 2) top_level = kLevels - 2;
        e_floor = top_level >= 0 ? level_floor(top_level) : 2.0f;
        if (use_topp) e_floor = fmaxf(e_floor, cutoff * 0.999999f);  // the sum is at least 1
      }
      // lanes with unsure terms first, then lanes with candidates only
      unsigned cmask = listing && top_level >= 0 && tid < n_units ? lanes_up_to(level, top_level) & ~unsure_mask : 0u;
      int tot_u, tot_c;
      const int pre_u = finish_scan(sm.redi, (__popc(unsure_mask) << 10) | (event ? 1 : 0), &tot_u);
      const int pre_c = finish_scan(sm.redf_i, __popc(cmask), &tot_c);
      n_unsure = tot_u >> 10;  // at most 512 events (10 bits) and 16384 lanes
      n_ev = tot_u & 1023;
      if (n_unsure + tot_c > kFinGroups) {
        // candidates all over the row: none is listed here
        listing = false;
        e_floor = INFINITY;
        cmask = 0u;
        tot_c = 0;
      }
      n_groups = n_unsure + tot_c;
      if (n_groups > kFinGroups || n_ev > kFinEvents) {
        decided = false;
      } else {
        if (event) sm.ev_unit[pre_u & 1023] = tid;
        int slot = pre_u >> 10;
        for (unsigned m = unsure_mask; m != 0u; m &= m - 1u) sm.u.group[slot++] = (uint16_t)(tid * 32 + __ffs(m) - 1);
        slot = n_unsure + pre_c;
        for (unsigned m = cmask; m != 0u; m &= m - 1u) sm.u.group[slot++] = (uint16_t)(tid * 32 + __ffs(m) - 1);
      }
      if (tid == 0) sm.ev_unit[n_ev < kFinEvents ? n_ev : kFinEvents] = n_units;
    }
    __syncthreads();

    if (decided) {
      // Half-lanes [32 * task, ...) of the group list, one per thread: which of their logits are
      // candidates (terms in [lo, hi)) or, for the first n_u groups, unsure; then those terms exactly,
      // packed, one per lane. By one warp.
      auto look = [&](int task, int n_g, int n_u, float lo, float hi) {
        const float x_low = candidate_logit_bound(__logf(lo), mx, temperature);
        const int h = task * 32 + lane;
        float x[8];
        unsigned um = 0u, cm = 0u;
        int p = 0;
        if (h < 2 * n_g) {
          const int g = sm.u.group[h >> 1];
          const int u = g >> 5;
          p = u * kUnit + unit_pos(g & 31, h & 1);
          load8_padded(row, shift, vocab, p, x);
#pragma unroll
          for (int j = 0; j < 8; ++j) cm |= x[j] >= x_low ? 1u << j : 0u;
          if ((h >> 1) < n_u) {
            const uint32_t info = sm.u.info[u];
            const float r_unit = (float)unit_ref(info);
            float s_lo, s_hi;
            scales(info, &s_lo, &s_hi);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float tau = ex2_approx(__fmaf_rn(x[j], c1, -r_unit));
              if (__float_as_uint(__fmaf_rn(tau, s_lo, kRoundMagic)) != __float_as_uint(__fmaf_rn(tau, s_hi, kRoundMagic)))
                um |= 1u << j;
            }
          }
        }
        uint32_t* queue = sm.u.queue[warp];
        unsigned am = um | cm;
        float mass = 0.0f;
        for (;;) {
          int n_q = __popc(am), inc = n_q;
#pragma unroll
          for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += o;
          }
          const int tot = __shfl_sync(0xffffffffu, inc, 31);
          if (tot == 0) break;
          int slot = inc - n_q;
          while (am != 0u && slot < kFinQueue) {
            const int j = __ffs(am) - 1;
            queue[slot++] = (uint32_t)(p + j) | ((cm >> j & 1u) ? kQCand : 0u) | ((um >> j & 1u) ? kQUnsure : 0u);
            am &= am - 1u;
          }
          __syncwarp();
          const int n_e = tot < kFinQueue ? tot : kFinQueue;
          for (int e = lane; e < n_e; e += 32) {
            const uint32_t el = queue[e];
            const int pe = (int)(el & kQPos), u = pe / kUnit;
            const float xs = to_f32(row[pe - shift]);
            const float v = exact_term(xs);
            if ((el & kQCand) && v >= lo && v < hi) {
              const int c = atomicAdd(&sm.n_cand, 1);
              mass += v;
              if (c < kFinCand) {
                Entry en;
                en.key = f32_bits(v);
                en.idx = pe - shift;
                sm.cand[c] = en;
              }
            }
            if (el & kQUnsure) {
              const uint32_t info = sm.u.info[u];
              float s_lo, s_hi;
              scales(info, &s_lo, &s_hi);
              const float tau = ex2_approx(__fmaf_rn(xs, c1, -(float)unit_ref(info)));
              const int approx = (int)(__float_as_uint(__fmaf_rn(tau, s_lo, kRoundMagic)) - kRoundMagicBits);
              const float t = fminf(__fmul_rn(v, seq_inv_u(unit_binade(info))), 67108864.0f);
              const float m = rintf(t);
              if (fabsf(t - m) == 0.5f) {
                const int c = atomicAdd(&sm.n_tie, 1);
                if (c < kFinTies) sm.u.tie[c] = (uint32_t)pe | (m > t ? kTieUp : 0u);
              }
              const int d = (int)m - approx;
              if (d != 0) atomicAdd(&sm.u.a0[u], d);
            }
          }
          __syncwarp();
        }
        if (hi > 2.0f) {  // the first pass: the mass listed
#pragma unroll
          for (int d = 16; d > 0; d >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, d);
          if (lane == 0 && mass > 0.0f) atomicAdd(&sm.mass, mass);
        }
      };
      auto next_task = [&](int* counter) {
        int task = 0;
        if (lane == 0) task = atomicAdd(counter, 1);
        return __shfl_sync(0xffffffffu, task, 0);
      };
      // ---- 2. events, a warp each, and the reported lanes; whichever warp is free takes the next task
      const int n_tasks = n_ev + (2 * n_groups + 31) / 32;
      for (;;) {
        const int task = next_task(&sm.n_task);
        if (task >= n_tasks) break;
        if (task < n_ev)
          finish_event(sm, row, shift, vocab, task, exact_term);
        else
          look(task - n_ev, n_groups, n_unsure, listing ? e_floor : INFINITY, INFINITY);
      }
      __syncthreads();
      const int n_tie = sm.n_tie;
      // Top-p whose nucleus is not in the list yet: the level (and the part of it) down to which the
      // lanes' largest terms make up for what is missing, a little more to be safe. Those lanes are looked
      // at while one warp forms the sum.
      n_more = 0;
      float e_more = e_floor;
      if (use_topp && listing && !(e_floor <= cutoff * head4.z * 0.98f)) {
        const int upto = lane < kLevels - 1 ? sm.level_cnt[lane] : 0;
        const int below = __shfl_up_sync(0xffffffffu, upto, 1);
        const float goal = (mode.topp * 1.002f + 0.003f) * head4.z;
        const float w = 0.72f * bits_f32((uint32_t)(127 - lane) << 23);  // mean term of a lane on level `lane`
        const float own = lane > top_level && lane < kLevels - 1 ? (float)(upto - (lane > 0 ? below : 0)) * w : 0.0f;
        float m = own;
#pragma unroll
        for (int d = 1; d < kLevels; d <<= 1) {
          const float o = __shfl_up_sync(0xffffffffu, m, d);
          if (lane >= d) m += o;
        }
        const float missing = goal - sm.mass;
        if (missing > 0.0f) {  // block-uniform
          const unsigned b = __ballot_sync(0xffffffffu, lane < kLevels - 1 && m >= missing * 1.1f);
          if (b == 0u) {
            listing = false;  // not even all levels
          } else {
            const int t = __ffs(b) - 1;
            const float in = __shfl_sync(0xffffffffu, m - own, t), of = __shfl_sync(0xffffffffu, own, t);
            const float part = fminf((missing * 1.1f - in) / of + 0.1f, 1.0f);
            e_more = fmaxf(level_floor(t) * exp2f(1.0f - part), cutoff * 0.999999f);
            const unsigned gmask = tid < n_units ? lanes_up_to(level, t) : 0u;
            int slot = finish_scan(sm.redi, __popc(gmask), &n_more);
            if (n_more > kFinGroups) {
              listing = false;
              n_more = 0;
            } else {
              for (unsigned g = gmask; g != 0u; g &= g - 1u) sm.u.group[slot++] = (uint16_t)(tid * 32 + __ffs(g) - 1);
              if (n_more > kFinListLanes) counted = true;
            }
          }
        }
      }
      if (use_topp && !listing) {
        // a nucleus all over the row: whatever passes the crop
        counted = all_lanes = true;
        e_more = cutoff * head4.z * 0.98f;
      }
      if (counted) {
        if (tid == 0) {
          set_bins(sm.lr, candidate_logit_bound(__logf(e_more), mx, temperature));
          sm.lr.all = all_lanes ? 1 : 0;
          sm.lr.n_half = all_lanes ? n_units * (kUnit / 8) : 2 * n_more;
          sm.lr.step = (sm.lr.n_half + kSampleHalfLanes - 1) / kSampleHalfLanes;
        }
        for (int q = tid; q < kFinBins; q += kFinThreads) sm.hist[q] = 0u;
      }
      if (n_tie > kFinTies) decided = false;
      if (decided) {
        // ---- exact half-way terms, a warp each. Such a term makes the significand even: it is rounded
        // up or down by the parity in front of it, i.e. by the parity of the increments since the
        // half-way term in front of it in the unit (which left the significand even), or since the
        // unit's start (then the result depends on the parity at which the unit is entered).
        for (int e = warp; e < n_tie; e += kWarps) {
          const uint32_t tie = sm.u.tie[e];
          const int p = (int)(tie & ~kTieUp), u = p / kUnit;
          int prev = u * kUnit - 1;
          for (int q = lane; q < n_tie; q += 32) {
            const int o = (int)(sm.u.tie[q] & ~kTieUp);
            if (o < p && o > prev) prev = o;
          }
          prev = __reduce_max_sync(0xffffffffu, prev);
          const uint32_t info = sm.u.info[u];
          const int r_unit = unit_ref(info);
          float s_lo, s_hi, x[16];
          scales(info, &s_lo, &s_hi);
          load_unit_lane(row, shift, vocab, u * kUnit, x);
          unsigned par = 0u, um = 0u;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int pj = u * kUnit + unit_pos(lane, j >> 3) + (j & 7);
            const float tau = ex2_approx(__fmaf_rn(x[j], c1, -(float)r_unit));
            const unsigned lo = __float_as_uint(__fmaf_rn(tau, s_lo, kRoundMagic));
            const unsigned hi = __float_as_uint(__fmaf_rn(tau, s_hi, kRoundMagic));
            if (pj > prev && pj < p) {
              par ^= lo;
              um |= lo != hi ? 1u << j : 0u;
            }
          }
          for (; um != 0u; um &= um - 1u) {  // the unsure ones exactly
            const int j = __ffs(um) - 1;
            const float xs = to_f32(row[u * kUnit + unit_pos(lane, j >> 3) + (j & 7) - shift]);
            const float tau = ex2_approx(__fmaf_rn(xs, c1, -(float)r_unit));
            const float t = fminf(__fmul_rn(exact_term(xs), seq_inv_u(unit_binade(info))), 67108864.0f);
            par ^= __float_as_uint(__fmaf_rn(tau, s_lo, kRoundMagic)) ^ (unsigned)(int)rintf(t);
          }
          par = __popc(__ballot_sync(0xffffffffu, (par & 1u) != 0u)) & 1u;
          if (lane == 0) {
            // a0 counts the term rounded to the even one of its two neighbours m; kTieUp: that is the
            // upper one
            const int up = (tie & kTieUp) ? 1 : 0;
            const int c_even = par ? (up ? -1 : 1) : 0, c_odd = par ? 0 : (up ? -1 : 1);
            if (c_even != 0) atomicAdd(&sm.u.a0[u], c_even);
            if (prev < u * kUnit) sm.u.a1d[u] = (signed char)(c_odd - c_even);
          }
        }
        __syncthreads();
        // ---- 3. the runs of ordinary units in front of each event and behind the last
        for (int e = warp; e <= n_ev; e += kWarps) {
          const int u0 = e > 0 ? sm.ev_unit[e - 1] + 1 : 0, u1 = sm.ev_unit[e];
          SeqSummary tot;
          seq_identity(&tot);
          int kmin = 255, kmax = 0;
          for (int ub = u0; ub < u1; ub += 32) {
            const int u = ub + lane;
            SeqSummary s;
            seq_identity(&s);
            if (u < u1) {
              const uint32_t info = sm.u.info[u];
              if ((info & kUnitZero) == 0u) {
                const int k = unit_binade(info);
                kmin = k < kmin ? k : kmin;
                kmax = k > kmax ? k : kmax;
                const uint32_t v = (uint32_t)sm.u.a0[u];
                s.a0 = v < (uint32_t)kSeqSat ? (int)v : kSeqSat;
                s.a1 = s.a0 + sm.u.a1d[u];
              }
            }
            tot = seq_compose(tot, warp_compose(s));
          }
          kmin = __reduce_min_sync(0xffffffffu, kmin);
          kmax = __reduce_max_sync(0xffffffffu, kmax);
          if (lane == 0) {
            sm.run[e] = make_int4(tot.a0, tot.a1, kmax == 0 ? 0 : (kmin == kmax ? kmin : -1), 0);
          }
        }
        __syncthreads();
        // ---- the exact sequential sum, by one warp
        if (warp == 0) {
          int hit = -1;
          float s = 0.0f;
          bool ok = finish_replay<kMulti>(sm, n_ev, thr, hit_unit, shift, vocab, &s, &hit);
          // a cdf that passes the coin nowhere in the units that were looked at, but has units behind them
          if (probs && hit < 0 && sm.tail_last < n_units - 1) ok = false;
          if (lane == 0) {
            if (!probs) {
              sm.sum = s;
              sm.coin = next_coin(&rng);
            }
            sm.bad = ok ? 0 : 1;
            sm.tail_pos = hit;  // (-1 but for the multinomial hit)
          }
        } else if (counted) {
          bin_count<T>(sm, warp - 1, kWarps - 1);
        } else if (n_more > 0) {
          for (;;) {
            const int task = next_task(&sm.n_task2);
            if (32 * task >= 2 * n_more) break;
            look(task, n_more, 0, e_more, e_floor);
          }
        }
        __syncthreads();
        list_floor = e_floor;
        e_floor = e_more;
        if (sm.bad) decided = false;
      }
    }
    if (!kMulti || !decided || use_list || probs) break;
    // ---- multinomial: the exact sum is known. Estimates of the cdf behind every unit from the units'
    // shares of the sum, the binades they leave open, and the units in which the cdf may pass the
    // coin; then the increments of the units in front of those, as in the sweep, for e / sum.
    probs = true;
    sum = sm.sum;
    inv_sum = __frcp_rn(sum);
    thr = sm.coin;
    float* share = reinterpret_cast<float*>(sm.cand);  // (no candidates in this mode)
    uint32_t* masks = reinterpret_cast<uint32_t*>(sm.cand) + kSwMaxUnits;
    {
      const uint32_t v = (uint32_t)sm.u.a0[tid];
      share[tid] = (zero || event) ? 0.0f : (float)v * bits_f32((uint32_t)(unit_binade(rec.z) - 23) << 23);
      __syncthreads();
      if (tid < n_ev) share[sm.ev_unit[tid]] = sm.ev_sum[tid];
      if (tid == 0) sm.tail_pos = sm.tail_last = n_units - 1;
      __syncthreads();
      const float own = share[tid];
      float inc = own;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const float o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += o;
      }
      if (lane == 31) sm.wmass[warp] = inc;
      __syncthreads();
      float front = 0.0f;
      for (int w = 0; w < warp; ++w) front += sm.wmass[w];
      const float q_in = (front + inc - own) * inv_sum, q_out = (front + inc) * inv_sum;
      const float margin = sweep_margin((tid + 1) * kUnit);
      int klo = seq_kb(q_in * (1.0f - margin));
      const int khi = seq_kb(q_out * (1.0f + margin));
      uint32_t span = (uint32_t)(khi > klo ? khi - klo : 0);
      if (span > 62u) span = 62u;
      if (q_in <= 0.0f || klo < 27) span = kUnitSpanOpen;
      if (klo < 27) klo = 27;
      if (tid < n_units && q_out * (1.0f + margin) > thr) atomicMin(&sm.tail_pos, tid);
      if (tid < n_units && q_out * (1.0f - margin) > thr) atomicMin(&sm.tail_last, tid);
      __syncthreads();
      hit_unit = sm.tail_pos;
      const int last_unit = sm.tail_last;
      // units behind the last one count as zero: nothing is added there
      rec.z = (uint32_t)klo | (span << kUnitSpanShift) | (zero || tid > last_unit ? kUnitZero : 0u) | (rec.z & 0xFFFF0000u);
      sm.u.info[tid] = rec.z;
      sm.u.a1d[tid] = 0;
      if (tid == 0) sm.n_task = sm.n_task2 = sm.n_tie = 0;
    }
    __syncthreads();
    const int n_sweep = hit_unit < n_units ? hit_unit : n_units;
    for (int u = warp; u < n_sweep; u += kWarps) {
      const uint32_t info = sm.u.info[u];
      if (unit_span(info) != 0u || (info & kUnitZero) != 0u) continue;
      float s_lo, s_hi, x[16];
      load_unit_lane(row, shift, vocab, u * kUnit, x);
      scales(info, &s_lo, &s_hi);
      const float nr = -(float)unit_ref(info);
      uint32_t acc = 0u, acc_hi = 0u;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float tau = ex2_approx(__fmaf_rn(x[j], c1, nr));
        acc += __float_as_uint(__fmaf_rn(tau, s_lo, kRoundMagic));
        acc_hi += __float_as_uint(__fmaf_rn(tau, s_hi, kRoundMagic));
      }
      const unsigned unsure = __ballot_sync(0xffffffffu, acc != acc_hi);
      const unsigned inc = __reduce_add_sync(0xffffffffu, acc);
      if (lane == 0) {
        sm.u.a0[u] = (int)(inc - 512u * kRoundMagicBits);
        masks[u] = unsure;
      }
    }
    __syncthreads();
    rec.x = (uint32_t)sm.u.a0[tid];
    rec.y = masks[tid];
    __syncthreads();
  }
  if (probs) known = kRowSum;
  if (decided) {
    // ---- 4. the sum is exact: finish on the candidate list, or hand the row on with its sum
    const float coin = sm.coin;
    known = kRowSum;
    sum = sm.sum;
    decided = probs;
    if (probs) token = sm.tail_pos >= 0 ? sm.tail_pos : vocab - 1;
    const int n_a = sm.n_cand;
    if (!probs && use_list) {
      if (!counted && listing && n_a <= kFinCand) {
        const bool complete = use_topp && e_floor <= cutoff * sum * 0.999999f;
        float mass;
        decided = finish_tail(sm, e_floor, sum, cutoff, mode.topp, mode.topk, use_topk, complete, coin, &token, &mass);
      }
      if (!decided) {
        __syncthreads();
        if (!counted && tid == 0) sm.lr.all = 1;
        token = finish_long<T>(sm, counted, n_more, e_floor, list_floor, sm.mass, sum, cutoff, mode.topp, mode.topk,
                            use_topk, coin);
        decided = token >= 0;
      }
      if (!decided) known = kRowLong;
    }
  }
  if (decided) {
    store_token(fa.out_ids, fa.peers, r, token);
    if (tid == 0) fa.rng_states[r] = rng;  // advanced by next_coin
  } else if (tid == 0) {
    RowHead h;
    h.mx = mx;
    h.raw_max = raw_max;
    h.sum = known != kRowUnknown ? sm.sum : 0.0f;
    h.state = known;
    a.heads[r] = h;
    fa.retry_rows[atomicAdd(fa.retry_count, 1)] = (int)r;
  }
}
