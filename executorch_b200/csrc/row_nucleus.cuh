// The end of sample_topp for nuclei that are too long for a list of their entries, and of
// sample_topk when the sweep's levels do not reach down to the k-th entry. Included by
// row_finish.cuh, whose shared state it uses.
//
// The reference sorts the candidates and adds their probabilities one by one (sampler.cpp:146-169).
// Sorting tens of thousands of entries is not needed for that: while the running sum stays inside
// a binade every term adds round(p / ulp) to its integer significand, whatever the order. So
//
//   1. the logits are counted in narrow bins of equal width, largest logits first; the counts and the
//      mean positions inside the bins give the running sum at every bin's edge to a few parts in 10^5
//   2. bins in which it may enter another binade, pass topp or pass the coin are "zones" (some two
//      dozen): their entries are listed, ranked and added one by one. Of every other bin the
//      increments are added up, in any order; they come from an approximate term rounded twice, a
//      little too low and a little too high, and from the exact term where the two differ
//   3. one warp joins both, checking that each stretch between zones is entered and left in the
//      binade that it was rounded for. So a wrong estimate can only end in "undecided".
//
// An exact half-way term makes its bin's sum depend on the parity of the significand in front of it
// (a row has a few: one in 2^(24 - n) terms that add about 2^n is one). Such a bin becomes a zone,
// whose entries take a third look at the row.
//
// What bounds it: instructions and shared-memory atomics, about 8, 18 and 7 per logit in the passes
// over the row (which comes from the L2 cache).

struct BinMap {
  float raw_max, scale;
  uint32_t limit;
  // bits >= limit: below the lowest bin (also -inf)
  __device__ __forceinline__ uint32_t bits(float x) const {
    return __float_as_uint(__fmaf_rn(__fsub_rn(raw_max, x), scale, 8388610.0f));
  }
  // a logit above every one in bin b or below it
  __device__ __forceinline__ float upper(int b) const {
    const float d = __fdividef((float)(b << kFinBinShift) - 4.0f, scale);
    return raw_max - d + 1.0e-6f * (fabsf(raw_max) + fabsf(d));
  }
  // a logit below every one whose bits are below `bits`
  __device__ __forceinline__ float lower(uint32_t bits) const {
    const float d = __fdividef((float)(bits - 0x4B000000u), scale);
    return raw_max - d - 1.0e-6f * (fabsf(raw_max) + d);
  }
  static __device__ __forceinline__ int bin(uint32_t bits) { return (int)((bits >> kFinBinShift) & (uint32_t)(kFinBins - 1)); }
};
constexpr uint32_t kBinBits = 0x4B000000u;  // bits of 2^23

__device__ __forceinline__ void set_bins(LongRow& lr, float x_low) {
  lr.scale = __fdividef((float)((kFinBins - 2) << kFinBinShift), fmaxf(lr.raw_max - x_low, 1.0e-20f));
  lr.limit = kBinBits + (uint32_t)(kFinBins << kFinBinShift);
}

// Eight logits as they lie in memory.
template <typename T>
struct Raw8 {
  uint4 v[sizeof(T) / 2];
  __device__ __forceinline__ float operator[](int j) const { return to_f32(reinterpret_cast<const T*>(v)[j]); }
};

// (LongRow, the constants of the passes, lies in shared memory: the passes are functions of their own, so
// that none of their loops shares its registers with the rest of the kernel.)
__device__ __forceinline__ BinMap row_bins(const LongRow& lr) {
  BinMap m;
  m.raw_max = lr.raw_max;
  m.scale = lr.scale;
  m.limit = lr.limit;
  return m;
}

// Padded position of half-lane h (8 logits): of the group list, or of the whole row.
__device__ __forceinline__ int half_lane_pos(const FinishShared& sm, bool all, int h) {
  if (all) return h * 8;
  const int g = sm.u.group[h >> 1];
  return (g >> 5) * kUnit + unit_pos(g & 31, h & 1);
}

// Calls f(logits, padded position, limit) for the half-lanes of the group list or the row, a warp's
// 32 at a time (of which every lr.step-th are taken); limit is that of the bins, or 0 where a lane has nothing. Warps first, first + 1, ...
// of `warps` take part; first 0 also takes the row's ragged ends. 64 bytes per thread are on their way at
// any time: with one block on an SM that is 32 KB, what hides the L2 cache's latency; no load stands
// behind a condition (one outside the row reads some other place of it).
template <typename T, bool kAll, typename F>
__device__ __forceinline__ void each_full_half_lane(const FinishShared& sm, int first, int warps, F f) {
  constexpr int kAhead = 8 / sizeof(T);
  const int lane = threadIdx.x & 31, stride = warps * 32 * sm.lr.step;
  const T* row = static_cast<const T*>(sm.lr.row);
  const int shift = sm.lr.shift, n_half = sm.lr.n_half, last = sm.lr.vocab - 8;
  const uint32_t limit = sm.lr.limit;
  const int some = (8 - shift) & 7;  // an aligned place in the row
  Raw8<T> w[kAhead];
  auto place = [&](int h) { return h < n_half ? half_lane_pos(sm, kAll, h) - shift : -1; };
  auto load = [&](int i0, Raw8<T>& to) {
    const uint4* src = reinterpret_cast<const uint4*>(row + ((unsigned)i0 <= (unsigned)last ? i0 : some));
#pragma unroll
    for (int q = 0; q < (int)(sizeof(T) / 2); ++q) to.v[q] = __ldg(src + q);
  };
  int h = first * 32 * sm.lr.step + lane;
#pragma unroll
  for (int u = 0; u < kAhead; ++u) load(place(h + u * stride), w[u]);
#pragma unroll 1
  for (int h0 = h - lane; h0 < n_half; h0 += kAhead * stride) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const Raw8<T> x = w[u];
      load(place(h + kAhead * stride), w[u]);
      const int i0 = place(h);
      f(x, i0 + shift, (unsigned)i0 <= (unsigned)last ? limit : 0u);
      h += stride;
    }
  }
}
// The chunks in which the row starts (lane 0) and ends (lane 1), where they are not whole; true: there is
// one for this lane.
template <typename T>
__device__ __forceinline__ bool ragged_ends(const LongRow& lr, int* pos, Raw8<T>& x) {
  const int lane = threadIdx.x & 31, vocab = lr.vocab, last = vocab - 8;
  const int p = lane == 0 ? 0 : (lr.shift + vocab - 1) & ~7, i0 = p - lr.shift;
  const bool ragged = lane < 2 && !((unsigned)i0 <= (unsigned)last && last >= 8) && !(lane == 1 && p == 0);
  T* t = reinterpret_cast<T*>(x.v);
#pragma unroll
  for (int j = 0; j < 8; ++j)
    t[j] = ragged && i0 + j >= 0 && i0 + j < vocab ? static_cast<const T*>(lr.row)[i0 + j] : static_cast<T>(-INFINITY);
  *pos = p;
  return ragged;
}
template <typename T, typename F>
__device__ __forceinline__ void each_half_lane(const FinishShared& sm, int first, int warps, F f) {
  if (sm.lr.vocab >= 16) {
    if (sm.lr.all != 0)
      each_full_half_lane<T, true>(sm, first, warps, f);
    else
      each_full_half_lane<T, false>(sm, first, warps, f);
  }
  if (first == 0) {
    int p;
    Raw8<T> x;
    const bool ragged = ragged_ends<T>(sm.lr, &p, x);
    f(x, p, ragged ? sm.lr.limit : 0u);
  }
}

// Which of eight logits lie in [lo, hi]: logit j is bit j of 32-bit logits; of 16-bit ones, compared two
// at a time, logits 2 k and 2 k + 1 are bits k and 16 + k. Without an upper bound (kUpper) one
// instruction per logit.
template <typename T>
struct RangeFilter;
template <>
struct RangeFilter<float> {
  float lo, hi;
  __device__ __forceinline__ RangeFilter(float l, float h) : lo(l), hi(h) {}
  template <bool kUpper>
  __device__ __forceinline__ uint32_t mask(const Raw8<float>& w, int) const {
    uint32_t m = 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) m |= w[j] >= lo && (!kUpper || w[j] <= hi) ? 1u << j : 0u;
    return m;
  }
  static __device__ __forceinline__ int logit(int bit) { return bit; }
};
template <typename T2>
struct RangeFilter16 {
  T2 lo, hi;
  template <bool kUpper>
  __device__ __forceinline__ uint32_t mask(const uint4 (&v)[1], int up) const {
    const uint32_t w[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
    uint32_t m = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const T2 x = *reinterpret_cast<const T2*>(&w[k]);
      uint32_t in = __hge2_mask(x, lo);
      if (kUpper) in &= __hle2_mask(x, hi);
      m |= in & (0x00010001u << (k + up));
    }
    return m;
  }
  static __device__ __forceinline__ int logit(int bit) { return ((bit & 15) << 1) | (bit >> 4); }
};
template <>
struct RangeFilter<__nv_bfloat16> : RangeFilter16<__nv_bfloat162> {
  __device__ __forceinline__ RangeFilter(float l, float h) {
    lo = __bfloat162bfloat162(__float2bfloat16_rd(fmaxf(l, -3.0e38f)));
    hi = __bfloat162bfloat162(__float2bfloat16_ru(fminf(h, 3.0e38f)));
  }
  template <bool kUpper>
  __device__ __forceinline__ uint32_t mask(const Raw8<__nv_bfloat16>& w, int up) const {
    return RangeFilter16<__nv_bfloat162>::template mask<kUpper>(w.v, up);
  }
};
template <>
struct RangeFilter<__half> : RangeFilter16<__half2> {
  __device__ __forceinline__ RangeFilter(float l, float h) {
    lo = __half2half2(__float2half_rd(fmaxf(l, -65504.0f)));
    hi = __half2half2(__float2half_ru(fminf(h, 65504.0f)));
  }
  template <bool kUpper>
  __device__ __forceinline__ uint32_t mask(const Raw8<__half>& w, int up) const {
    return RangeFilter16<__half2>::template mask<kUpper>(w.v, up);
  }
};

// Calls f(mask, position of chunk 0, of chunk 1) for the logits in [lo, hi] (some just outside may be
// among them), 16-bit logits 16 at a time (bits 4 .. 7 and 20 .. 23 are chunk 1's), 32-bit ones 8.
template <typename T, bool kUpper, bool kAll, typename F>
__device__ __forceinline__ void each_full_in_range(const FinishShared& sm, int first, int warps, float lo, float hi, F f) {
  constexpr int kChunks = sizeof(T) == 2 ? 2 : 1;
  const int lane = threadIdx.x & 31, stride = warps * 32;
  const T* row = static_cast<const T*>(sm.lr.row);
  const int shift = sm.lr.shift, n_half = sm.lr.n_half, last = sm.lr.vocab - 8;
  const int some = (8 - shift) & 7;
  const RangeFilter<T> filter(lo, hi);
  Raw8<T> w[2][kChunks];
  auto place = [&](int h) { return h < n_half ? half_lane_pos(sm, kAll, h) - shift : -1; };
  auto load = [&](int h, Raw8<T> (&to)[kChunks]) {
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
      const int i0 = place(h + c * stride);
      const uint4* src = reinterpret_cast<const uint4*>(row + ((unsigned)i0 <= (unsigned)last ? i0 : some));
#pragma unroll
      for (int q = 0; q < (int)(sizeof(T) / 2); ++q) to[c].v[q] = __ldg(src + q);
    }
  };
  int h = first * 32 + lane;
  load(h, w[0]);
  load(h + kChunks * stride, w[1]);
#pragma unroll 1
  for (int h0 = first * 32; h0 < n_half; h0 += 2 * kChunks * stride) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      uint32_t m = 0u;
      int p[2] = {0, 0};
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        const int i0 = place(h + c * stride);
        const uint32_t in = filter.template mask<kUpper>(w[u][c], 4 * c);
        m |= (unsigned)i0 <= (unsigned)last ? in : 0u;
        p[c] = i0 + shift;
      }
      load(h + 2 * kChunks * stride, w[u]);
      f(m, p[0], p[1]);
      h += kChunks * stride;
    }
  }
}
template <typename T, bool kUpper, typename F>
__device__ __forceinline__ void each_in_range(const FinishShared& sm, int first, int warps, float lo, float hi, F f) {
  if (sm.lr.vocab >= 16) {
    if (sm.lr.all != 0)
      each_full_in_range<T, kUpper, true>(sm, first, warps, lo, hi, f);
    else
      each_full_in_range<T, kUpper, false>(sm, first, warps, lo, hi, f);
  }
  if (first == 0) {
    int p;
    Raw8<T> x;
    const bool ragged = ragged_ends<T>(sm.lr, &p, x);
    const uint32_t m = RangeFilter<T>(lo, hi).template mask<kUpper>(x, 0);
    f(ragged ? m : 0u, p, 0);
  }
}

// 1. Counts: per bin the number of logits (upper 12 bits) and the sum of their positions inside it.
// More than 4095 in a bin spoil the estimates, no more than that.
template <typename T>
__device__ __noinline__ void bin_count(FinishShared& sm, int first, int warps) {
  const BinMap bins = row_bins(sm.lr);
  each_half_lane<T>(sm, first, warps, [&](const Raw8<T>& w, int, uint32_t limit) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t b = bins.bits(w[j]);
      if (b < limit) atomicAdd(&sm.hist[BinMap::bin(b)], (1u << 20) | (b & ((1u << kFinBinShift) - 1u)));
    }
  });
}

constexpr int kBinsPerThread = kFinBins / kFinThreads;

// 2. What the counts say: the zones, and the binade that every other bin is rounded for. `coin`
// and topp: where the walks end. Returns the number of zones; -1: the mass in the bins does not reach
// topp; -2: too much for the lists.
__device__ __noinline__ int long_plan(FinishShared& sm, float topp, float coin, int* listed) {
  // The margin around the estimated sum: it covers the estimates' own error and what the roundings of
  // the running sum add up to where thousands of equal terms are rounded alike.
  constexpr float kLow = 1.0f - 3.0e-4f, kHigh = 1.0f + 3.0e-4f;
  FinishLong& L = sm.u.l;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = tid * kBinsPerThread;
  const float step = -__fdividef(sm.lr.c1, sm.lr.scale), scale = ex2_approx(-2.0f * step) * __frcp_rn(sm.lr.sum);
  auto bin_mass = [&](int b, uint32_t w) {
    const float n = (float)(w >> 20);
    const float t = (float)(b << kFinBinShift) + __fdividef((float)(w & 0xFFFFFu), n);
    return w >> 20 ? n * ex2_approx(t * step) * scale : 0.0f;
  };
  float own = 0.0f;
#pragma unroll
  for (int q = 0; q < kBinsPerThread; ++q) own += bin_mass(b0 + q, sm.hist[b0 + q]);
  float inc = own;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const float o = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += o;
  }
  if (lane == 31) sm.wmass[warp] = inc;
  if (tid == 0) {
    sm.tail_bin = -1;
    sm.s_bcast = 0.0f;
    sm.tail_cnt = 0;
  }
  for (int q = tid; q < kLongList; q += kFinThreads) {
    L.sorted[q] = 0.0f;
    L.zone_of[q] = 255;
  }
  __syncthreads();
  float front = 0.0f, all = 0.0f;
#pragma unroll
  for (int q = 0; q < kWarps; ++q) {
    const float x = sm.wmass[q];
    if (q < warp) front += x;
    all += x;
  }
  if (!(all * kLow > topp)) return -1;  // block-uniform
  front += inc - own;
  if (front <= topp && front + own > topp * kLow)  // the largest term near topp (of this thread's bins)
    atomicMax(reinterpret_cast<int*>(&sm.s_bcast), (int)f32_bits(ex2_approx((float)(b0 << kFinBinShift) * step) * scale));
  __syncthreads();
  const float r_lo = coin * topp, r_hi = coin * (topp + sm.s_bcast);
  uint32_t mask = 0u;
  int elems = 0, inside = 0, last = -1;
  float m = front;
#pragma unroll
  for (int q = 0; q < kBinsPerThread; ++q) {
    const uint32_t w = sm.hist[b0 + q];
    const float lo = m * kLow;
    m += bin_mass(b0 + q, w);
    const float hi = m * kHigh;
    const int k = seq_kb(lo);
    // (bins that seem empty, too: every bin above the limit has the binade of the bins in front of it)
    L.code[b0 + q] = (uint8_t)(k < kLongBinade ? 1 : k - kLongBinade + 1);
    L.count[b0 + q] = (uint16_t)(w >> 20);
    sm.hist[b0 + q] = 0u;
    if (!(lo > topp)) {
      last = b0 + q;
      inside += (int)(w >> 20);
      if (w != 0u && (k != seq_kb(hi) || k < kLongBinade || hi > topp || (lo <= r_hi && hi >= r_lo))) {
        mask |= 1u << q;
        elems += (int)((w >> 20) + 3u) & ~3;
      }
    }
  }
  int n_zones;
  int z = finish_scan(sm.redi, __popc(mask), &n_zones);
  int at = finish_scan(sm.redf_i, elems, listed);
  last = __reduce_max_sync(0xffffffffu, last);
  inside = __reduce_add_sync(0xffffffffu, inside);
  if (lane == 0) {
    atomicMax(&sm.tail_bin, last);
    atomicAdd(&sm.tail_cnt, inside);
  }
  if (n_zones > kLongZones - kLongTies || *listed > kLongList) return -2;  // block-uniform
  for (; mask != 0u; mask &= mask - 1u, ++z) {
    const int b = b0 + __ffs(mask) - 1, n = L.count[b];
    L.zone_k[z] = (int)L.code[b] - 1 + kLongBinade;
    L.code[b] = (uint8_t)(128 + z);
    L.zone_bin[z] = b;
    L.zone_start[z] = at;
    L.zone_n[z] = n;
    L.zone_fill[z] = 0;
    at += (n + 3) & ~3;
  }
  __syncthreads();
  if (tid == 0) sm.lr.limit = kBinBits + (uint32_t)((sm.tail_bin + 1) << kFinBinShift);
  __syncthreads();
  return n_zones;
}


// Entry i exactly: into its zone's list, or its increment into its bin. kMode 2 (top-k): into sm.cand.
template <int kMode, typename T>
__device__ __forceinline__ void long_exact(FinishShared& sm, const BinMap& bins, uint32_t i) {
  FinishLong& L = sm.u.l;
  const float x = to_f32(static_cast<const T*>(sm.lr.row)[i]);
  const float v = expf_ref(__fsub_rn(__fmul_rn(x, sm.lr.inv_t), sm.lr.mx), sm.exp_tab);
  if (kMode == 2) {
    const int c = atomicAdd(&sm.n_cand, 1);
    if (c < kFinCand) {
      Entry en;
      en.key = f32_bits(v);
      en.idx = (int)i;
      sm.cand[c] = en;
    }
    return;
  }
  const float p = __fdiv_rn(v, sm.lr.sum);
  const int bin = BinMap::bin(bins.bits(x));
  const int code = L.code[bin];
  if (code >= 128) {
    const int z = code - 128, k = atomicAdd(&L.zone_fill[z], 1);
    if (k < L.zone_n[z]) {
      const int s = L.zone_start[z] + k;
      L.entry[s] = ((unsigned long long)f32_bits(p) << 32) | (uint32_t)(0x7FFFFFFF - (int)i);
      L.zone_of[s] = (uint8_t)z;
    }
  } else {
    const float t = fminf(__fmul_rn(p, seq_inv_u(code - 1 + kLongBinade)), 67108864.0f);
    const float m = rintf(t);
    if (fabsf(t - m) == 0.5f) {
      // once per bin: the upper bit of its count tells (of 16-bit logits hundreds are equal)
      const uint32_t bit = 0x8000u << (16 * (bin & 1));
      if (!(atomicOr(reinterpret_cast<uint32_t*>(L.count) + (bin >> 1), bit) & bit)) {
        const int f = atomicAdd(&L.n_tie, 1);
        if (f < kLongTies) L.tie[f] = bin;
      }
    }
    atomicAdd(&sm.hist[bin], (uint32_t)(int)m);
  }
}

// The increment of a term whose two roundings agree; false when they do not, or when its bin is a zone.
struct TermScale {
  float c1, r_row, s_lo, s_hi;
};
__device__ __forceinline__ TermScale term_scale(const LongRow& lr) {
  TermScale t;
  t.c1 = lr.c1;
  t.r_row = lr.r_row;
  t.s_lo = lr.s_lo;
  t.s_hi = lr.s_hi;
  return t;
}
__device__ __forceinline__ bool long_increment(const TermScale& t, float x, uint32_t code, uint32_t* inc) {
  const float tau = ex2_approx(__fmaf_rn(x, t.c1, -t.r_row));
  const uint32_t down = (code - 1u) << 23;  // one binade further up is half the scale
  const uint32_t a = __float_as_uint(__fmaf_rn(tau, bits_f32(f32_bits(t.s_lo) - down), kRoundMagic));
  const uint32_t c = __float_as_uint(__fmaf_rn(tau, bits_f32(f32_bits(t.s_hi) - down), kRoundMagic));
  *inc = a - kRoundMagicBits;
  return code < 128u && a == c;
}

// 3. The second pass over the row, when a good part of it lies above the limit: the zones' entries into
// the list (as (probability, inverted index)), the increments of all others into their bins.
template <typename T>
__device__ __noinline__ void long_pass(FinishShared& sm) {
  FinishLong& L = sm.u.l;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const BinMap bins = row_bins(sm.lr);
  const TermScale scale = term_scale(sm.lr);
  uint32_t* queue = L.queue[warp];
  int* fill = &L.queue_fill[warp];
  auto evaluate = [&](int n) {
    for (int e = lane; e < n; e += 32) long_exact<0, T>(sm, bins, queue[e]);
  };
  if (lane == 0) *fill = 0;
  __syncwarp();
  each_half_lane<T>(sm, warp, kWarps, [&](const Raw8<T>& w, int pos, uint32_t limit) {
    uint32_t am = 0u;  // entries that are evaluated exactly
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float x = w[j];
      const uint32_t b = bins.bits(x);
      if (b < limit) {
        const int bin = BinMap::bin(b);
        uint32_t inc;
        if (long_increment(scale, x, L.code[bin], &inc))
          atomicAdd(&sm.hist[bin], inc);
        else
          am |= 1u << j;
      }
    }
    while (__any_sync(0xffffffffu, am != 0u)) {
      if (am != 0u) {
        int s = atomicAdd(fill, __popc(am));
        for (; am != 0u && s < kFinQueue; am &= am - 1u) queue[s++] = (uint32_t)(pos + __ffs(am) - 1 - sm.lr.shift);
      }
      __syncwarp();
      const int n = *fill;
      if (n < kFinQueue / 2) break;  // (nothing is left over then)
      evaluate(n < kFinQueue ? n : kFinQueue);
      __syncwarp();
      if (lane == 0) *fill = 0;
      __syncwarp();
    }
  });
  evaluate(*fill);
}

// Where only some of the logits lie above the limit, a pass costs as much for those that do not, as of 32
// that a warp looks at together a few lie above nearly always. So the indices of those that do are
// collected first, a list per warp, and their scattered logits taken 32 at a time.
//
// Entries part[0, n): kMode 0 as in long_pass; 1: the entries of the zones from first_zone on; 2 (top-k):
// everything into sm.cand; 3: counts, as bin_count. The `nq` entries that wait for
// their exact evaluation are behind the list; returns how many are left.
template <int kMode, typename T>
__device__ __noinline__ int near_entries(FinishShared& sm, int first_zone, const uint32_t* part, int n, uint32_t* queue, int nq) {
  const BinMap bins = row_bins(sm.lr);
  const TermScale scale = term_scale(sm.lr);
  FinishLong& L = sm.u.l;
  const int lane = threadIdx.x & 31;
  const T* row = static_cast<const T*>(sm.lr.row);
  constexpr int kLoads = 4;
#pragma unroll 1
  for (int e0 = 0; e0 < n; e0 += kLoads * 32) {
    uint32_t i[kLoads];
    T raw[kLoads];
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const int e = e0 + q * 32 + lane;
      i[q] = part[e < n ? e : 0];
      raw[q] = row[i[q]];
    }
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const float x = to_f32(raw[q]);
      const uint32_t b = bins.bits(x);
      bool rest = false;
      if (e0 + q * 32 + lane < n && b < bins.limit) {
        const int bin = BinMap::bin(b);
        if (kMode == 3) {
          atomicAdd(&sm.hist[bin], (1u << 20) | (b & ((1u << kFinBinShift) - 1u)));
        } else if (kMode == 2) {
          rest = true;
        } else if (kMode == 1) {
          rest = L.code[bin] >= 128 + first_zone;
        } else {
          uint32_t inc;
          rest = !long_increment(scale, x, L.code[bin], &inc);
          if (!rest) atomicAdd(&sm.hist[bin], inc);
        }
      }
      if (kMode == 3) continue;
      const unsigned any = __ballot_sync(0xffffffffu, rest);
      if (any == 0u) continue;
      if (rest) queue[nq + __popc(any & ((1u << lane) - 1u))] = i[q];
      nq += __popc(any);
      if (nq >= 32) {
        __syncwarp();
        long_exact<kMode, T>(sm, bins, queue[lane]);
        const uint32_t left = queue[32 + lane];
        __syncwarp();
        nq -= 32;
        if (lane < nq) queue[lane] = left;
        __syncwarp();
      }
    }
  }
  return nq;
}
// The lists: everything above the limit, and true when it fits. kStream: it does not have to; what a
// warp has collected is taken (near_entries) whenever its list is nearly full.
template <int kMode, bool kStream, typename T>
__device__ __noinline__ bool near_pass(FinishShared& sm, bool list, int first_zone) {
  FinishLong& L = sm.u.l;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const BinMap bins = row_bins(sm.lr);
  const int shift = sm.lr.shift;
  // everything above the limit (near_entries compares exactly), or the zones' range
  const float lo = kMode == 1 ? sm.lr.x_lo : bins.lower(bins.limit), hi = sm.lr.x_hi;
  uint32_t *part = L.near[warp], *queue = part + kNearPart;
  int n = 0, nq = 0;
  if (list) {
    each_in_range<T, kMode == 1>(sm, warp, kWarps, lo, hi, [&](uint32_t m, int p0, int p1) {
      for (;;) {
        const unsigned any = __ballot_sync(0xffffffffu, m != 0u);
        if (any == 0u) break;
        if (m != 0u) {
          const int s = n + __popc(any & ((1u << lane) - 1u)), j = RangeFilter<T>::logit(__ffs(m) - 1);
          if (kStream || s < kNearPart) part[s] = (uint32_t)((j >= 8 ? p1 - 8 : p0) + j - shift);
          m &= m - 1u;
        }
        n += __popc(any);
        if (kStream && n > kNearPart - 32) {
          __syncwarp();
          nq = near_entries<kMode, T>(sm, first_zone, part, n, queue, nq);
          __syncwarp();
          n = 0;
        }
      }
    });
    if (!kStream) {
      if (lane == 0) L.n_near[warp] = n;
      return __syncthreads_and(n <= kNearPart) != 0;
    }
  } else {
    n = L.n_near[warp];
  }
  __syncwarp();
  nq = near_entries<kMode, T>(sm, first_zone, part, n, queue, nq);
  __syncwarp();
  if (lane < nq) long_exact<kMode, T>(sm, bins, queue[lane]);
  __syncthreads();
  return true;
}
// The pass that fits: over the lists, or the row, whose nucleus is dense or not.
template <int kMode, typename T>
__device__ __forceinline__ void any_pass(FinishShared& sm, bool near, bool dense, int first_zone) {
  if (near) {
    near_pass<kMode, false, T>(sm, false, first_zone);
  } else if (kMode == 0 && dense) {
    long_pass<T>(sm);
    __syncthreads();
  } else {
    near_pass<kMode, true, T>(sm, true, first_zone);
  }
}

// What a sample (bin_count of every lr.step-th half-lane) says about the nucleus: the bin in which it
// ends, with three standard deviations to spare, and (*n) how many entries it may have. Terms of at
// least `floor` are known: their mass is `mass`.
__device__ __noinline__ int long_floor(FinishShared& sm, float topp, float floor, float mass, float log_floor, int* n) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = tid * kBinsPerThread, step = sm.lr.step;
  const float slope = -__fdividef(sm.lr.c1, sm.lr.scale), scale = ex2_approx(-2.0f * slope);
  // bins that lie below the floor, roughly
  const float x_floor = floor < 2.0f ? (log_floor + sm.lr.mx) / sm.lr.inv_t : sm.lr.raw_max;
  const int b_known = floor < 2.0f ? BinMap::bin(row_bins(sm.lr).bits(fminf(x_floor, sm.lr.raw_max))) : -1;
  float m = 0.0f;
  int c = 0;
  auto add = [&](int q) {
    const uint32_t w = sm.hist[b0 + q];
    c += (int)(w >> 20);
    if (b0 + q > b_known && w >> 20)
      m += (float)(w >> 20) * scale *
           ex2_approx(((float)((b0 + q) << kFinBinShift) + __fdividef((float)(w & 0xFFFFFu), (float)(w >> 20))) * slope);
  };
#pragma unroll
  for (int q = 0; q < kBinsPerThread; ++q) add(q);
  int ci = c;
  float mi = m;
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
  if (tid == 0) {
    sm.tail_bin = kFinBins;
    sm.tail_cnt = 0x7fffffff;
  }
  __syncthreads();
  c = ci - c;
  m = mi - m;
  for (int w = 0; w < warp; ++w) {
    c += sm.wcnt[w];
    m += sm.wmass[w];
  }
  const float missing = topp * 1.001f * sm.lr.sum - mass;
  int found = kFinBins;
  for (int q = 0; q < kBinsPerThread; ++q) {
    add(q);
    if (m * (float)step * (1.0f - 3.0f * rsqrtf((float)(c + 1))) > missing) {
      found = b0 + q;
      break;
    }
  }
  const int best = __reduce_min_sync(0xffffffffu, found);
  if (lane == 0) atomicMin(&sm.tail_bin, best);
  __syncthreads();
  if (found == sm.tail_bin && found < kFinBins) sm.tail_cnt = c;
  __syncthreads();
  *n = sm.tail_cnt < 0x1000000 ? sm.tail_cnt * step : 0x7fffffff;
  return sm.tail_bin;
}

// Adds the sorted entries [a, a + n) to s, until it exceeds thr: then the entry, else -1. (Every
// lane of a warp does the same; the zeros behind a zone's entries change no sum.)
__device__ __forceinline__ int zone_walk(const FinishLong& L, int a, int n, float thr, float& s) {
  const int b = a + n;
  const float4* p4 = reinterpret_cast<const float4*>(L.sorted);
  float4 next = p4[a >> 2];
  for (int j = a; j < b; j += 4) {
    const float4 p = next;
    next = p4[(j >> 2) + 1];  // (the array is longer than the list)
    const float s0 = __fadd_rn(s, p.x), s1 = __fadd_rn(s0, p.y), s2 = __fadd_rn(s1, p.z), s3 = __fadd_rn(s2, p.w);
    if (s3 > thr) {
      const int k = s0 > thr ? 0 : (s1 > thr ? 1 : (s2 > thr ? 2 : 3));
      s = k == 0 ? s0 : (k == 1 ? s1 : (k == 2 ? s2 : s3));
      return j + k;
    }
    s = s3;
  }
  return -1;
}

// The entry's token when others of its probability may lie outside its bin: all of them, in index
// order (the order of equal probabilities), by one more pass over the row.
template <typename T>
__device__ __noinline__ int long_pick(FinishShared& sm, int bin, int rank, float x_hit, float p_hit, float dx) {
  const T* row = static_cast<const T*>(sm.lr.row);
  const int n_units = sm.lr.n_units;
  const BinMap bins = row_bins(sm.lr);
  FinishLong& L = sm.u.l;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    sm.tail_cnt = 0;
    sm.tail_pos = -1;
  }
  __syncthreads();
  auto probability = [&](float x) {
    return __fdiv_rn(expf_ref(__fsub_rn(__fmul_rn(x, sm.lr.inv_t), sm.lr.mx), sm.exp_tab), sm.lr.sum);
  };
  // bit j: logit j of the lane's 16 belongs to the group
  auto group_mask = [&](int u, int* above) {
    float x[16];
    load_unit_lane(row, sm.lr.shift, sm.lr.vocab, u * kUnit, x);
    unsigned in = 0u;
    *above = 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      if (fabsf(x[j] - x_hit) <= dx && probability(x[j]) == p_hit) {
        in |= 1u << j;
        *above += BinMap::bin(bins.bits(x[j])) < bin ? 1 : 0;
      }
    }
    return in;
  };
  for (int u = warp; u < n_units; u += kWarps) {
    int above;
    const int n = __reduce_add_sync(0xffffffffu, __popc(group_mask(u, &above)));
    above = __reduce_add_sync(0xffffffffu, above);
    if (lane == 0) {
      L.members[u] = n;
      if (above > 0) atomicAdd(&sm.tail_cnt, above);
    }
  }
  __syncthreads();
  rank += sm.tail_cnt;
  int tot;
  const int mine = tid < n_units ? L.members[tid] : 0;
  const int pre = finish_scan(sm.redf_i, mine, &tot);
  if (rank >= pre && rank < pre + mine) {
    sm.tail_bin = tid;
    sm.tail_last = rank - pre;
    sm.tail_pos = 0;
  }
  __syncthreads();
  if (sm.tail_pos < 0) return -1;
  if (warp == 0) {
    int above, left = sm.tail_last, found = -1;
    const int u = sm.tail_bin;
    const unsigned in16 = group_mask(u, &above);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      unsigned in = in16 >> (8 * q) & 0xFFu;
      const int n = __popc(in);
      int inc = n;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += o;
      }
      if (left >= inc - n && left < inc) {
        for (int k = left - (inc - n); k > 0; --k) in &= in - 1u;
        found = u * kUnit + unit_pos(lane, q) + __ffs(in) - 1 - sm.lr.shift;
      }
      left -= __shfl_sync(0xffffffffu, inc, 31);
    }
    found = __reduce_max_sync(0xffffffffu, found);
    if (lane == 0) sm.tail_pos = found;
  }
  __syncthreads();
  return sm.tail_pos;
}

// All of it. `counted`: bin_count has been over the lanes of the group list (sm.lr.all = 0, down to
// e_floor) or over the row (down to the crop); the block has been synchronised since. Returns the
// token, or -1 with nothing decided when an estimate did not hold.
template <typename T>
__device__ __noinline__ int finish_long(FinishShared& sm, bool counted, int n_groups, float e_floor, float list_floor, float list_mass,
                                        float sum, float cutoff, float topp, int topk, bool use_topk, float coin) {
  FinishLong& L = sm.u.l;
  LongRow& lr = sm.lr;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    const float inv_sum = __frcp_rn(sum);
    lr.sum = sum;
    lr.r_row = rintf(__fmul_rn(lr.raw_max, lr.c1));
    float s_lo, s_hi;
    unit_scales(row_scale(lr.mx), lr.mx, (int)lr.r_row, kLongBinade, &s_lo, &s_hi);
    lr.s_lo = s_lo * (inv_sum * (1.0f - 4e-7f));
    lr.s_hi = s_hi * (inv_sum * (1.0f + 4e-7f));
  }
  __syncthreads();
  bool refined = false, near = false;
  if (counted && lr.step > 1) {
    int n;
    const int b = long_floor(sm, topp, list_floor, list_mass, __logf(list_floor), &n);
    __syncthreads();
    const float x_low = lr.raw_max - __fdividef((float)((b + 1) << kFinBinShift), lr.scale);
    const bool fits = b < kFinBins && n < kNear - kNear / 16;
    if (tid == 0) {
      lr.step = 1;
      if (b < kFinBins) set_bins(lr, x_low);
    }
    __syncthreads();
    near = fits && near_pass<3, false, T>(sm, true, 0);
    refined = b < kFinBins;
    counted = false;
  }
  for (int attempt = 0; attempt < 5; ++attempt) {
    if (!counted) {
      __syncthreads();
      for (int q = tid; q < kFinBins; q += kFinThreads) sm.hist[q] = 0u;
      if (tid == 0) {
        if (lr.all != 0 && !refined) {
          // top-k: down to where every term is smaller than the smallest normal float
          const float lo = use_topk ? 1.2e-38f : cutoff * sum * 0.999f;
          set_bins(lr, candidate_logit_bound(__logf(lo), lr.mx, 1.0f / lr.inv_t));
        }
        lr.n_half = lr.all != 0 ? lr.n_units * (kUnit / 8) : 2 * n_groups;
      }
      __syncthreads();
      if (near) {
        near_pass<3, false, T>(sm, false, 0);
      } else {
        bin_count<T>(sm, warp, kWarps);
        __syncthreads();
      }
    }
    counted = false;
    if (tid == 0) sm.n_cand = L.n_tie = 0;
    if (use_topk) {
      // the first bin at whose lower edge k logits are counted, and one more (equal probabilities)
      int own = 0, tot;
      for (int q = 0; q < kBinsPerThread; ++q) own += (int)(sm.hist[tid * kBinsPerThread + q] >> 20);
      int n = finish_scan(sm.redi, own, &tot);
      if (tot < topk) return -1;
      if (n < topk && n + own >= topk) {
        int q = 0;
        for (; n < topk; ++q) n += (int)(sm.hist[tid * kBinsPerThread + q] >> 20);
        sm.tail_bin = tid * kBinsPerThread + q;
      }
      __syncthreads();
      if (tid == 0) {
        sm.tail_cnt = 0x7f7fffff;
        lr.limit = kBinBits + (uint32_t)((sm.tail_bin + 1) << kFinBinShift);
      }
      __syncthreads();
      near_pass<2, true, T>(sm, true, 0);
      const int n_c = sm.n_cand;
      if (n_c > kFinCand) return -1;
      for (int q = tid; q < n_c; q += kFinThreads) atomicMin(&sm.tail_cnt, (int)sm.cand[q].key);
      __syncthreads();
      const float low = bits_f32((uint32_t)sm.tail_cnt);
      float mass;
      int token;
      if (!(low > 0.0f)) return -1;
      return finish_tail(sm, low, sum, cutoff, topp, topk, true, false, coin, &token, &mass) ? token : -1;
    }
    int listed = 0;
    int zones = long_plan(sm, topp, coin, &listed);
    const bool all = lr.all != 0;
    __syncthreads();
    if (zones == -1 && (!all || refined)) {
      if (tid == 0) lr.all = 1;
      refined = near = false;
      continue;
    }
    if (zones == -2 && !refined && !near) {
      // bins as wide as this are too full: again, over the nucleus alone
      refined = true;
      if (tid == 0) set_bins(lr, lr.raw_max - __fdividef((float)((sm.tail_bin + 2) << kFinBinShift), lr.scale));
      continue;
    }
    if (zones < 0) return -1;
    const int n_in = sm.tail_cnt;
    if (!near && n_in < kNear - kNear / 16) near = near_pass<3, false, T>(sm, true, 0);
    const bool dense = n_in > 2 * lr.n_half;  // more than one in four
    any_pass<0, T>(sm, near, dense, 0);
    const int n_tie = L.n_tie;
    if (n_tie > 0) {
      if (n_tie > kLongTies) return -1;
      __syncthreads();
      if (tid == 0) {
        int z = zones, at = listed;
        for (int e = 0; e < n_tie; ++e) {
          const int b = L.tie[e], n = L.count[b] & 0xFFF;
          L.zone_k[z] = (int)L.code[b] - 1 + kLongBinade;
          L.code[b] = (uint8_t)(128 + z);
          L.zone_bin[z] = b;
          L.zone_start[z] = at;
          L.zone_n[z] = n;
          L.zone_fill[z] = 0;
          sm.hist[b] = 0u;
          at += (n + 3) & ~3;
          ++z;
        }
        sm.tail_cnt = z;
        sm.tail_last = at;
        int b_lo = 0, b_hi = kFinBins;
        for (int q = zones; q < z; ++q) {
          b_lo = max(b_lo, L.zone_bin[q]);
          b_hi = min(b_hi, L.zone_bin[q]);
        }
        const BinMap bins = row_bins(lr);
        lr.x_lo = bins.lower(kBinBits + (uint32_t)((b_lo + 1) << kFinBinShift));
        lr.x_hi = bins.upper(b_hi);
      }
      __syncthreads();
      const int old = zones;
      zones = sm.tail_cnt;
      listed = sm.tail_last;
      if (listed > kLongList) return -1;
      any_pass<1, T>(sm, near, dense, old);
    }
    // the increments in front of every zone, the zones in order, and their entries in order
    {
      int own = 0, tot;
#pragma unroll
      for (int q = 0; q < kBinsPerThread; ++q) own += (int)sm.hist[tid * kBinsPerThread + q];
      uint32_t before = (uint32_t)finish_scan(sm.redi, own, &tot);
#pragma unroll
      for (int q = 0; q < kBinsPerThread; ++q) {
        const int code = L.code[tid * kBinsPerThread + q];
        if (code >= 128) L.zone_q[code - 128] = before;
        before += sm.hist[tid * kBinsPerThread + q];
      }
    }
    __syncthreads();
    if (tid < zones) {
      const int mine = L.zone_bin[tid];
      int rank = 0;
      for (int q = 0; q < zones; ++q) rank += L.zone_bin[q] < mine ? 1 : 0;
      const bool full = L.zone_fill[tid] == L.zone_n[tid];
      L.zone[rank] = make_int4(L.zone_start[tid], full ? L.zone_n[tid] : -1, L.zone_k[tid], (int)L.zone_q[tid]);
    }
    for (int s = tid; s < listed; s += kFinThreads) {
      const int z = L.zone_of[s];
      if (z == 255) continue;
      const unsigned long long mine = L.entry[s];
      const int a = L.zone_start[z], n = L.zone_n[z];
      int rank = 0;
      if (L.zone_fill[z] == n)
        for (int j = a; j < a + n; ++j) rank += L.entry[j] > mine ? 1 : 0;
      L.sorted[a + rank] = bits_f32((uint32_t)(mine >> 32));
      L.order[a + rank] = (uint16_t)s;
    }
    if (tid == 0) sm.tail_pos = -1;
    __syncthreads();
    if (warp == 0) {
      float s = 0.0f, cum = 0.0f;
      uint32_t q_prev = 0u;
      int hit = -1, z_hit = -1;
      bool ok = true;
      int4 next = L.zone[0];
      for (int k = 0; k < zones; ++k) {
        const int4 z = next;
        next = L.zone[k + 1];
        const unsigned t = (uint32_t)z.w - q_prev;
        q_prev = (uint32_t)z.w;
        if (t != 0u) {
          ok = seq_kb(s) == z.z && t < (unsigned)(kSeqLimit - seq_n(s));
          if (ok) s = seq_value(z.z, seq_n(s) + (int)t);
          ok = ok && s <= topp;
        }
        ok = ok && z.y >= 0;
        if (lane == 0) L.zone_in[k] = s;
        if (!ok) break;
        hit = zone_walk(L, z.x, z.y, topp, s);
        if (hit >= 0) {
          z_hit = k;
          cum = s;
          break;
        }
      }
      ok = ok && hit >= 0;
      __syncwarp();
      if (ok) {
        // sampler.cpp:162-169: the first entry at which the same sum exceeds coin * cum
        const float r = __fmul_rn(coin, cum);
        if (r < cum) {
          int k = 0;
          for (int q = lane; q <= z_hit; q += 32)
            if (L.zone_in[q] <= r) k = q;
          z_hit = __reduce_max_sync(0xffffffffu, k);
          s = L.zone_in[z_hit];
          sm.misc_i[0] = hit;
          hit = zone_walk(L, L.zone[z_hit].x, L.zone[z_hit].y, r, s);
          ok = hit >= 0;
        } else {
          sm.misc_i[0] = hit;
        }
      }
      if (lane == 0 && ok) {
        sm.tail_pos = hit;
        sm.tail_last = L.zone[z_hit].x;
      }
    }
    __syncthreads();
    const int hit = sm.tail_pos;
    if (hit < 0) return -1;
    // the crop (sampler.cpp:136-143), and the floor down to which the lanes are complete
    const float p_end = L.sorted[sm.misc_i[0]];
    const bool low = !all && p_end * sum < e_floor * 1.000001f;
    if (p_end < cutoff) return -1;
    if (low) {
      __syncthreads();
      if (tid == 0) lr.all = 1;
      refined = near = false;
      continue;
    }
    const int a = sm.tail_last;
    const float p_hit = L.sorted[hit];
    const int idx = 0x7FFFFFFF - (int)(uint32_t)(L.entry[L.order[hit]] & 0xFFFFFFFFull);
    const float x_hit = to_f32(static_cast<const T*>(lr.row)[idx]);
    const BinMap bins = row_bins(lr);
    // equal probabilities come from logits this close
    const float y = __fmul_rn(x_hit, lr.inv_t);
    const float dx = (1.0e-6f + 2.5e-7f * (fabsf(y) + fabsf(lr.mx))) / lr.inv_t;
    const int bin = BinMap::bin(bins.bits(x_hit));
    int picked = idx;
    if (BinMap::bin(bins.bits(x_hit - dx)) != bin || BinMap::bin(bins.bits(fminf(x_hit + dx, lr.raw_max))) != bin) {
      int rank = 0;
      for (int j = hit - 1; j >= a && L.sorted[j] == p_hit; --j) ++rank;
      __syncthreads();
      picked = long_pick<T>(sm, bin, rank, x_hit, p_hit, dx);
      if (picked < 0) return -1;
    }
    return picked;
  }
  return -1;
}
