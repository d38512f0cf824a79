// First of the two kernels of the fast sampling path: one streaming sweep over the logits.
// Included by fast_path.cu inside its unnamed namespace (uses its helpers).
//
// The reference adds the softmax denominator in index order in float (sampler.cpp:198-203), and
// its tokens depend on every rounding of that sum. While the running sum stays in one binade
// (ulp u), an addition is an integer increment of the significand, round_half_even(e / u), and
// integer increments can be added in any order. So the row is cut into units of 512 logits and
// this kernel delivers, per unit, the sum of the increments in the binade in which the running
// sum will be when the unit is reached -- plus bit masks of the few lanes whose 16 logits need
// another look (row_finish.cuh does that, and joins the units to the exact sum).
//
//   A. per unit: largest logit, and the terms 2^(x / T * log2 e - R) with the hardware's
//      approximate exponential, R an integer near the unit's largest exponent; their sum is the
//      unit's share of the estimate. The terms stay in registers.
//   -- one exchange through distributed shared memory: row maximum, estimated prefix sums --
//   B. the terms scaled to units of the last place, t = e / u, and rounded to integers twice,
//      once with t a little low and once a little high (by eps, the bound on the error of the
//      approximate term). A lane whose two sums agree has the increments of the exact terms; a
//      lane whose sums differ is reported as unsure.
//
// What bounds it: 8 KB of HBM reads per 4096 bf16 logits against 4096 exponentials on the
// special-function pipe (16 per clock and SM) and about 10 issue slots per logit; with one
// exponential per logit the HBM side is the longer one. Hence a cluster of blocks per row
// with every logit's term in a register (a second read of the logits would mean a second
// exponential), packed float pairs (one issue slot for two logits), and the next row's slice
// copied in by one bulk asynchronous copy per block while this row is worked on.
//
// Rows of any alignment: positions are counted from the 16-byte boundary at or in front of the
// row's first logit, and what lies in front of or behind the row reads as -inf (e = 0, which
// changes no sum).

constexpr int kSwThreads = 256;
constexpr int kSwWarps = kSwThreads / 32;
constexpr int kUnit = 512;            // logits per unit: 16 per lane
constexpr int kSwMaxUnits = 512;      // per row
constexpr int kSwMaxCluster = 16;
constexpr int kSwStages = 2;
constexpr float kRoundMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds |t| < 2^22 to an integer
constexpr uint32_t kRoundMagicBits = 0x4B400000u;
constexpr float kLog2eHi = 0x1.715476p+0f;  // log2(e) as the sum of two floats
constexpr float kLog2eLo = 0x1.4ae0cp-26f;

// What the sweep leaves per unit.
struct __align__(16) UnitRec {
  uint32_t inc;     // sum of the increments (mod 2^32) in binade klo
  uint32_t unsure;  // lanes whose increments are not certain
  uint32_t info;    // klo | span << 8 | kUnitZero, and R in the upper half
  uint32_t pad;
  uint32_t level[4];  // bit b of every lane's level: how far its largest term lies below the row's
};
// A lane's level: its largest term is 2^-y with level <= y < level + 1;
// kLevels - 1 for everything further down. The finishing kernel lists candidates from the lanes up
// to a level, which it picks when it has seen how many lanes there are on every level.
constexpr int kLevels = 16;
// lanes of a unit with a level of at most t
__device__ __forceinline__ uint32_t lanes_up_to(const uint32_t (&level)[4], int t) {
  uint32_t lt = 0u, eq = 0xFFFFFFFFu;
#pragma unroll
  for (int b = 3; b >= 0; --b) {
    const uint32_t tb = (t >> b & 1) ? 0xFFFFFFFFu : 0u;
    lt |= eq & ~level[b] & tb;
    eq &= ~(level[b] ^ tb);
  }
  return lt | eq;
}
// Every term of at least this size lies in a lane up to level t (the levels are good to a few units of
// the last place of y).
__device__ __forceinline__ float level_floor(int t) { return bits_f32((uint32_t)(126 - t) << 23) * 1.0005f; }
constexpr int kUnitSpanShift = 8;         // binades that the unit may carry the sum through; 0: none
constexpr uint32_t kUnitSpanMask = 63u;
constexpr uint32_t kUnitSpanOpen = 63u;   // not known (the row's start; sums beyond the usual range)
constexpr uint32_t kUnitZero = 1u << 14;  // every term is zero
__device__ __forceinline__ int unit_binade(uint32_t info) { return (int)(info & 255u); }
__device__ __forceinline__ uint32_t unit_span(uint32_t info) { return (info >> kUnitSpanShift) & kUnitSpanMask; }
__device__ __forceinline__ int unit_ref(uint32_t info) { return (int)(int16_t)(info >> 16); }

// Lane l of a unit holds the logits at 8 l .. 8 l + 7 and 256 + 8 l .. 256 + 8 l + 7 of the unit.
__device__ __forceinline__ int unit_pos(int lane, int q) { return q * 256 + lane * 8; }

// What a row of the sweep is sampled with.
struct RowMode {
  float inv_t, topp;
  int topk;  // 0: off
  bool greedy;
};

struct SweepArgs {
  const void* logits;
  int64_t row0, rows;      // rows [row0, row0 + rows) of the batch
  int64_t row_stride;
  int vocab;
  int units_per_block;
  int units_pitch;         // UnitRec per row
  float inv_t, topp;
  int topk;
  RowSettings ext;         // per-row settings, or null pointers
  UnitRec* units;
  RowHead* heads;
};

__device__ __forceinline__ RowMode row_mode(const SweepArgs& a, int64_t r) {
  RowMode m;
  m.inv_t = a.inv_t;
  m.topp = a.topp;
  m.topk = a.topk;
  if (a.ext.temperature != nullptr) {
    const float t = a.ext.temperature[r];
    m.inv_t = t > 0.0f ? 1.0f / t : 0.0f;  // as Sampler::set_temperature: negative counts as 0
  }
  if (a.ext.topp != nullptr) m.topp = a.ext.topp[r];
  if (a.ext.topk != nullptr) m.topk = a.ext.topk[r];
  if (m.topk < 0 || m.topk >= a.vocab) m.topk = 0;
  m.greedy = m.inv_t == 0.0f;
  if (m.greedy) m.inv_t = 1.0f;
  return m;
}

// A logit below every logit whose term reaches the floor (t: the temperature, log_floor: the floor's
// logarithm, both to a few units of the last place).
__device__ __forceinline__ float candidate_logit_bound(float log_floor, float mx, float t) {
  const float x = (log_floor + mx) * t;
  return x - 1e-5f * (fabsf(x) + fabsf(mx * t)) - 1e-4f * t;
}

// The row's scale: 2^(I + F) = e^mx with I an integer; pow = 2^-F (to about 2^-22).
struct RowScale {
  int i;
  float pow;
};
__device__ __forceinline__ RowScale row_scale(float mx) {
  RowScale s;
  const float p = __fmul_rn(mx, kLog2eHi);
  const float lo = __fmaf_rn(mx, kLog2eLo, __fmaf_rn(mx, kLog2eHi, -p));
  const float i = rintf(p);
  s.i = (int)i;
  s.pow = ex2_approx(-(__fsub_rn(p, i) + lo));
  return s;
}

// Bound on the relative error of the approximate t of a unit in binade k, for every term with
// t >= 1/4 (smaller ones round to 0 whatever their error), in units of 2^-24: the reference's own
// roundings of x / T (|y|) and of y - mx (|z|), the rounding of the factor log2(e) / T (|y|) and of
// the exponent (|z|), ex2.approx twice (4 each), the rounding of the exact term (1), of the scale
// (3), and one for second-order terms.
__device__ __forceinline__ float term_eps(float mx, int k) {
  const float z = (float)(154 - k) * 0.6931472f;
  const float y = fmaxf(fabsf(mx), fabsf(mx - z));
  return (2.0f * y + 2.0f * z + 13.0f) * 5.9604645e-8f;
}

// Scale factors that take a term 2^(a - R) to t (1 - eps) and t (1 + eps) in binade k.
__device__ __forceinline__ void unit_scales(const RowScale& rs, float mx, int r_unit, int k, float* lo, float* hi) {
  const int ex = r_unit - rs.i + 150 - k;
  const float eps = term_eps(mx, k);
  // rs.pow is in (0.7, 1.5); far below the usual range every t is far below 1/2
  const float s = ex > -120 ? bits_f32(f32_bits(rs.pow) + ((uint32_t)(ex < 120 ? ex : 120) << 23)) : 0.0f;
  *lo = s * (1.0f - eps);
  *hi = s * (1.0f + eps);
}

// Relative margin around the estimated running sum inside which the sequentially rounded one is assumed
// to lie after `terms` terms: an eighth of the rigorous terms * 2^-24 (measured: below a twentieth on
// rows whose many small terms are too small to move the sum), and the estimate's own error. A row
// that breaks the assumption is noticed when the units are joined.
__device__ __forceinline__ float sweep_margin(int terms) { return (float)terms * 7.4505806e-9f + 2.0e-5f; }

// ---- packed pairs of floats
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float* a, float* b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(*a), "=f"(*b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// The 16 logits of one lane of a unit: packed maximum and float values.
template <typename T>
struct UnitLoad;
template <>
struct UnitLoad<__nv_bfloat16> {
  static __device__ __forceinline__ uint4 neg_inf() { return make_uint4(0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u); }
  static constexpr int kVecs = 2;
  static __device__ __forceinline__ float lane_max(const uint4 (&raw)[2]) {
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(raw);
    __nv_bfloat162 m = p[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) m = __hmax2(m, p[i]);
    return fmaxf(__bfloat162float(m.x), __bfloat162float(m.y));
  }
  static __device__ __forceinline__ f32x2 pair(const uint4 (&raw)[2], int i) {
    const uint32_t w = reinterpret_cast<const uint32_t*>(raw)[i];
    return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
  }
};
template <>
struct UnitLoad<__half> {
  static __device__ __forceinline__ uint4 neg_inf() { return make_uint4(0xFC00FC00u, 0xFC00FC00u, 0xFC00FC00u, 0xFC00FC00u); }
  static constexpr int kVecs = 2;
  static __device__ __forceinline__ float lane_max(const uint4 (&raw)[2]) {
    const __half2* p = reinterpret_cast<const __half2*>(raw);
    __half2 m = p[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) m = __hmax2(m, p[i]);
    return fmaxf(__half2float(m.x), __half2float(m.y));
  }
  static __device__ __forceinline__ f32x2 pair(const uint4 (&raw)[2], int i) {
    const float2 f = __half22float2(reinterpret_cast<const __half2*>(raw)[i]);
    return pack2(f.x, f.y);
  }
};
template <>
struct UnitLoad<float> {
  static __device__ __forceinline__ uint4 neg_inf() { return make_uint4(0xFF800000u, 0xFF800000u, 0xFF800000u, 0xFF800000u); }
  static constexpr int kVecs = 4;
  static __device__ __forceinline__ float lane_max(const uint4 (&raw)[4]) {
    const float* p = reinterpret_cast<const float*>(raw);
    float m = p[0];
#pragma unroll
    for (int i = 1; i < 16; ++i) m = fmaxf(m, p[i]);
    return m;
  }
  static __device__ __forceinline__ f32x2 pair(const uint4 (&raw)[4], int i) {
    const float* p = reinterpret_cast<const float*>(raw);
    return pack2(p[2 * i], p[2 * i + 1]);
  }
};

template <typename T>
__device__ __forceinline__ T neg_inf_value() {
  if constexpr (std::is_same<T, float>::value) return -INFINITY;
  else if constexpr (std::is_same<T, __half>::value) return __ushort_as_half((unsigned short)0xFC00u);
  else return __ushort_as_bfloat16((unsigned short)0xFF80u);
}

// Elements between the 16-byte boundary at or in front of a row's first logit and that logit.
template <typename T>
__device__ __forceinline__ int row_shift(const T* row) {
  return (int)((reinterpret_cast<uintptr_t>(row) & 15u) / sizeof(T));
}

// What a block tells the others about its slice of a row: largest logit, sum of the terms
// relative to 2^r, r.
struct __align__(16) SweepExchange {
  float m, est;
  int r, pad;
};

// What the compute warps need to know about a unit in phase B.
struct __align__(16) UnitPlan {
  float s_lo, s_hi;  // unit_scales
  uint32_t info;     // UnitRec::info
  float level0;      // log2 of the row's largest term
};

struct __align__(16) SweepShared {
  unsigned long long full[kSwStages];  // a stage holds its slice
  unsigned long long told[2];          // the other blocks' SweepExchange have arrived
  SweepExchange xchg[2][kSwMaxCluster];  // written by the peers through distributed shared memory
  float unit_m[32], unit_est[32];
  int unit_r[32];
  float c1[kSwStages];                 // log2(e) / T of the row in a stage
  UnitPlan plan[32];
};

template <typename T, int kUnitsPerWarp>
struct SweepLayout {
  static constexpr int kUnits = kSwWarps * kUnitsPerWarp;              // of a block
  static constexpr size_t kStage = (size_t)kUnits * kUnit * sizeof(T);  // a slice of a row
  static constexpr size_t kBytes = kSwStages * kStage + sizeof(SweepShared);
  // registers: 16 per unit for the terms, 40 or so for the rest
  static constexpr int kBlocksPerSm = kUnitsPerWarp <= 2 ? 3 : 2;
};

// Warp 0 has the slices copied in, exchanges the block's maximum and estimate with the other blocks
// and works out every unit's plan, one unit per lane, while the other warps wait (and the other
// block of the SM computes).
//
// Hand-overs inside a block: the other warps arrive at barrier 1 when their units' records are written
// (and the stage is read) and wait at barrier 2 for the plan. Between blocks: one 16-byte
// asynchronous store per pair of blocks and row, counted by the receiver's mbarrier. A block can
// be at most one row ahead of another (it needs everyone's word on row i before it sends its own
// on row i + 1), so two sets of slots suffice.
template <typename T, int kUnitsPerWarp>
__global__ void __launch_bounds__(kSwThreads, SweepLayout<T, kUnitsPerWarp>::kBlocksPerSm) row_sweep_kernel(const SweepArgs a) {
  using L = UnitLoad<T>;
  constexpr size_t kStage = SweepLayout<T, kUnitsPerWarp>::kStage;
  constexpr int kPerVec = 16 / sizeof(T);
  extern __shared__ __align__(128) unsigned char sweep_smem[];
  SweepShared& sm = *reinterpret_cast<SweepShared*>(sweep_smem + kSwStages * kStage);
  cg::cluster_group cluster = cg::this_cluster();
  const int csize = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_cl = (int)(gridDim.x / csize);
  const int first = (int)(blockIdx.x / csize);
  const int rows = (int)a.rows;
  const T* logits = static_cast<const T*>(a.logits) + a.row0 * a.row_stride;
  const int upb = a.units_per_block;
  const int pos0 = rank * upb * kUnit;  // padded position of this block's slice

  grid_launch_dependents();  // the finishing kernel may take its place; it waits for this grid
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < kSwStages; ++s)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&sm.full[s])), "r"(1u));
#pragma unroll
    for (int s = 0; s < 2; ++s)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&sm.told[s])), "r"(1u));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  cluster_arrive();  // every block of the cluster runs, and its barriers are set up, before it is written to
  cluster_wait();
  grid_dependency_wait();  // the logits (and the previous call's use of the scratch) are settled

  // Slice of row i into a stage: whole 16-byte units by one bulk copy, the ragged ends of the row
  // and the padding up to a whole unit by the lanes (-inf). Warp 0.
  auto start_slice = [&](int i, int stage) {
    T* buf = reinterpret_cast<T*>(sweep_smem + stage * kStage);
    const T* row = logits + (int64_t)i * a.row_stride;
    const int shift = row_shift(row);
    const int end = shift + a.vocab;  // padded positions [shift, end) are logits
    const int whole0 = shift > 0 ? kPerVec : 0, whole1 = end / kPerVec * kPerVec;
    int slice_end = pos0 + upb * kUnit;
    const int units_end = (end + kUnit - 1) / kUnit * kUnit;
    if (slice_end > units_end) slice_end = units_end;
    int c0 = whole0 > pos0 ? whole0 : pos0, c1 = whole1 < slice_end ? whole1 : slice_end;
    if (c1 < c0) c1 = c0 = slice_end;  // nothing for the bulk copy
    for (int p = pos0 + lane; p < c0; p += 32)
      buf[p - pos0] = p >= shift && p < end ? row[p - shift] : neg_inf_value<T>();
    for (int p = c1 + lane; p < slice_end; p += 32) buf[p - pos0] = p < end ? row[p - shift] : neg_inf_value<T>();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
      sm.c1[stage] = __fmul_rn(row_mode(a, a.row0 + i).inv_t, kLog2eHi);
      const uint32_t bar = smem_addr(&sm.full[stage]);
      if (c1 > c0) {
        const uint32_t bytes = (uint32_t)(c1 - c0) * (uint32_t)sizeof(T);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_addr(buf + (c0 - pos0))),
            "l"(row + (c0 - shift)), "r"(bytes), "r"(bar)
            : "memory");
      } else {
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
      }
    }
  };
  if (warp == 0) {
    for (int s = 0; s < kSwStages; ++s)
      if (first + s * n_cl < rows) start_slice(first + s * n_cl, s);
  }
  __syncthreads();  // the ragged ends are written

  int stage = 0, par = 0;
  uint32_t phase = 0u, told_phase = 0u;
  for (int i = first; i < rows; i += n_cl) {
    const int row_units = (row_shift(logits + (int64_t)i * a.row_stride) + a.vocab + kUnit - 1) / kUnit;
    int n_units = row_units - rank * upb;  // of this block
    n_units = n_units < 0 ? 0 : (n_units < upb ? n_units : upb);
    wait_bulk_copy(&sm.full[stage], phase);
    const float c1 = sm.c1[stage];
    const f32x2 c1p = pack2(c1, c1);
    const unsigned char* buf = sweep_smem + stage * kStage;

    // ---- A: this warp's units, j * kSwWarps + warp of the block. No branches: the units' chains of
    // latencies (load, maximum, exponentials, sum) run side by side. A unit that the row does not
    // have reads as -inf.
    f32x2 tau[kUnitsPerWarp][8];
    float lmax[kUnitsPerWarp], umax[kUnitsPerWarp];
    {
      uint4 raw[kUnitsPerWarp][L::kVecs];
#pragma unroll
      for (int j = 0; j < kUnitsPerWarp; ++j) {
        const int lu = j * kSwWarps + warp;
        const uint4* src = reinterpret_cast<const uint4*>(buf + (size_t)lu * kUnit * sizeof(T));
#pragma unroll
        for (int v = 0; v < L::kVecs; ++v) {
          // 16-bit: one vector per half of the unit; fp32: two
          constexpr int kSplit = L::kVecs / 2;
          raw[j][v] = L::neg_inf();
          if (lu < n_units) raw[j][v] = src[(v / kSplit) * 32 * kSplit + lane * kSplit + (v % kSplit)];
        }
        lmax[j] = L::lane_max(raw[j]);
      }
#pragma unroll
      for (int j = 0; j < kUnitsPerWarp; ++j) umax[j] = warp_max_f32(lmax[j]);
      float rf[kUnitsPerWarp];
      unsigned fx[kUnitsPerWarp];
#pragma unroll
      for (int j = 0; j < kUnitsPerWarp; ++j) {
        rf[j] = rintf(fmaxf(__fmul_rn(umax[j], c1), -30000.0f));
        const f32x2 nr = pack2(-rf[j], -rf[j]);
        f32x2 s2 = 0ull;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          float x, y;
          unpack2(fma2(L::pair(raw[j], p), c1p, nr), &x, &y);
          tau[j][p] = pack2(ex2_approx(x), ex2_approx(y));
          s2 = add2(s2, tau[j][p]);
        }
        float sa, sb;
        unpack2(s2, &sa, &sb);
        // the warp's sum in fixed point: at most 32 * 16 * 2^0.5 of 2^22 units
        fx[j] = __float2uint_rn((sa + sb) * 4194304.0f);
      }
#pragma unroll
      for (int j = 0; j < kUnitsPerWarp; ++j) {
        const unsigned tot = __reduce_add_sync(0xffffffffu, fx[j]);
        if (lane == 0) {
          sm.unit_m[j * kSwWarps + warp] = umax[j];
          sm.unit_est[j * kSwWarps + warp] = (float)tot * (1.0f / 4194304.0f);
          sm.unit_r[j * kSwWarps + warp] = (int)rf[j];
        }
      }
    }
    if (warp != 0) {
      asm volatile("barrier.cta.arrive 1, %0;" ::"n"(kSwThreads) : "memory");
      asm volatile("barrier.cta.sync 2, %0;" ::"n"(kSwThreads) : "memory");
    } else {
      const RowMode mode = row_mode(a, a.row0 + i);
      asm volatile("barrier.cta.sync 1, %0;" ::"n"(kSwThreads) : "memory");
      // the block's maximum and the prefix sums of its units' estimates, relative to 2^br
      float m = -INFINITY, e = 0.0f;
      int r = -30000;
      if (lane < n_units) {
        m = sm.unit_m[lane];
        e = sm.unit_est[lane];
        r = sm.unit_r[lane];
      }
      const float bm = warp_max_f32(m);
      const int br = __reduce_max_sync(0xffffffffu, r);
      e = r - br < -120 ? 0.0f : e * bits_f32((uint32_t)(r - br + 127) << 23);
      float inc = e;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const float o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += o;
      }
      const float tot = __shfl_sync(0xffffffffu, inc, 31);
      const uint32_t told = smem_addr(&sm.told[par]);
      if (lane == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(told),
                     "r"((uint32_t)(csize * sizeof(SweepExchange)))
                     : "memory");
      }
      if (lane < csize) {
        uint32_t to, bar;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(smem_addr(&sm.xchg[par][rank])), "r"(lane));
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(told), "r"(lane));
        asm volatile(
            "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to),
            "r"(f32_bits(bm)), "r"(f32_bits(tot)), "r"(br), "r"(0), "r"(bar)
            : "memory");
      }
      // what does not need the others' word
      const float margin = sweep_margin(pos0 + (lane + 1) * kUnit);
      const float m_lo = 1.0f - margin, m_hi = 1.0f + margin;
      const bool ok = wait_bulk_copy(&sm.told[par], told_phase);
      // every lane: its unit's plan
      SweepExchange x;
      x.m = -INFINITY;
      x.est = 0.0f;
      x.r = -30000;
      if (lane < csize) x = sm.xchg[par][lane];
      const float row_m = warp_max_f32(x.m);
      const int row_r = __reduce_max_sync(0xffffffffu, x.r);
      const float mx = __fmul_rn(row_m, mode.inv_t);
      const RowScale rs = row_scale(mx);
      float total = x.r - row_r >= -120 ? x.est * bits_f32((uint32_t)(x.r - row_r + 127) << 23) : 0.0f;
      float pre = (lane < rank && x.r - row_r >= -120) ? x.est * bits_f32((uint32_t)(x.r - row_r + 127) << 23) : 0.0f;
#pragma unroll
      for (int d = 1; d < kSwMaxCluster; d <<= 1) {
        pre += __shfl_xor_sync(0xffffffffu, pre, d);
        total += __shfl_xor_sync(0xffffffffu, total, d);
      }
      pre = __shfl_sync(0xffffffffu, pre, 0);
      const float my_scale = br - row_r < -120 ? 0.0f : bits_f32((uint32_t)(br - row_r + 127) << 23);
      // the binades in which the running sum may be across the unit
      const float p_in = (pre + (inc - e) * my_scale) * rs.pow;
      const float p_out = (pre + inc * my_scale) * rs.pow;
      const int k0 = row_r - rs.i;
      int klo = (int)(f32_bits(p_in * m_lo) >> 23) + k0;
      const int khi = (int)(f32_bits(p_out * m_hi) >> 23) + k0;
      uint32_t span = (uint32_t)(khi - klo < 62 ? (khi > klo ? khi - klo : 0) : 62);
      if (p_in <= 0.0f || klo < 27 || khi > 252) span = kUnitSpanOpen;
      klo = klo < 27 ? 27 : (klo > 252 ? 252 : klo);
      UnitPlan plan;
      unit_scales(rs, mx, r, klo, &plan.s_lo, &plan.s_hi);
      // every term of the unit is zero: exp underflows below -104
      const bool zero = __fsub_rn(__fmul_rn(m, mode.inv_t), mx) < -104.0f;
      plan.info = (uint32_t)klo | (span << kUnitSpanShift) | (zero ? kUnitZero : 0u) | ((uint32_t)r << 16);
      plan.level0 = mx * kLog2eHi;
      sm.plan[lane] = plan;
      asm volatile("barrier.cta.arrive 2, %0;" ::"n"(kSwThreads) : "memory");
      if (rank == 0 && lane == 0) {
        RowHead h;
        h.mx = mx;
        h.raw_max = row_m;
        h.sum = total * rs.pow * bits_f32((uint32_t)(row_r - rs.i + 127) << 23);  // the estimate
        h.state = ok ? 0 : -1;
        a.heads[a.row0 + i] = h;
      }
    }

    // ---- B
    UnitRec* out = a.units + (int64_t)i * a.units_pitch + rank * upb;
#pragma unroll
    for (int j = 0; j < kUnitsPerWarp; ++j) {
      const int lu = j * kSwWarps + warp;
      const UnitPlan plan = sm.plan[lu];
      const f32x2 lo2 = pack2(plan.s_lo, plan.s_lo), hi2 = pack2(plan.s_hi, plan.s_hi);
      const f32x2 mg = pack2(kRoundMagic, kRoundMagic);
      uint32_t acc = 0, acc_hi = 0;
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        const f32x2 q0 = fma2(tau[j][p], lo2, mg), q1 = fma2(tau[j][p], hi2, mg);
        acc += (uint32_t)q0 + (uint32_t)(q0 >> 32);
        acc_hi += (uint32_t)q1 + (uint32_t)(q1 >> 32);
      }
      const unsigned unsure = __ballot_sync(0xffffffffu, acc != acc_hi);
      const float y = fmaf(lmax[j], -c1, plan.level0);
      const int level = (int)fminf(fmaxf(y, 0.0f), (float)(kLevels - 1));
      uint32_t lv[4];
#pragma unroll
      for (int b = 0; b < 4; ++b) lv[b] = __ballot_sync(0xffffffffu, (level >> b) & 1);
      const unsigned inc = __reduce_add_sync(0xffffffffu, acc);
      if (lane == 0 && lu < n_units) {
        uint4* rec = reinterpret_cast<uint4*>(&out[lu]);
        rec[0] = make_uint4(inc - 512u * kRoundMagicBits, unsure, plan.info, 0u);
        rec[1] = make_uint4(lv[0], lv[1], lv[2], lv[3]);
      }
    }
    // the stage has been read by all: the slice of the row after the next ones
    if (warp == 0 && i + kSwStages * n_cl < rows) start_slice(i + kSwStages * n_cl, stage);
    if (++stage == kSwStages) {
      stage = 0;
      phase ^= 1u;
    }
    par ^= 1;
    if (par == 0) told_phase ^= 1u;
  }
  // nobody writes into a block that has left: a block leaves after it has heard from all the others
  // about its last row, and nothing is sent after that
}
