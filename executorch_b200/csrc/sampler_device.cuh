// Device code shared by the sampling kernels: constants, block-wide primitives, the exact
// sequential sum by block and by warp, the candidate list and the tail of a short nucleus.
#pragma once

#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <atomic>
#include <type_traits>

#include "class_math.cuh"
#include "cluster_math.cuh"
#include "exact_math.cuh"
#include "sampler_kernels.cuh"

namespace etb200 {

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kChunk = 16;                  // consecutive logits per thread per tile
constexpr int kTile = kThreads * kChunk;    // logits per tile
constexpr int kHead = 256;                  // leading terms of a sum that one thread adds sequentially
// Candidate values are binned by their float bits >> 21 (exponent + 2 mantissa bits). Bin
// kBins-1 holds 1.0; bin 0 also collects everything below the covered range (e < ~2.4e-10).
// Per bin two integers are kept: the count, and the sum of the 13 mantissa bits below the
// bin bits, which together give the bin's mass to about 2^-15 relative (always rounded
// down) without floating-point atomics.
constexpr int kBinShift = 21;
constexpr int kBins = 128;
constexpr int kBinTop = 0x3F800000 >> kBinShift;  // bin index of 1.0 before rebasing
constexpr int kBinBase = kBinTop - (kBins - 1);
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kFastSat = 1 << 25;           // per-thread clamp of chunk summaries
constexpr int kCompactSteps = 224;          // list entries compacted per segment = 448 * kThreads
constexpr float kGuessFloor = 1.0f / 8192.0f;  // first guess of a floor under the values that matter
constexpr int kListBatch = 8;               // list entries a thread loads before using any of them
constexpr int kRankSortMax = 512;           // survivor lists up to this size are rank-sorted in shared memory

// bf16 table of e by logit bit pattern: both signs, |logit| in [2^-16, 2^16). Anything else
// (zero, tiny, huge, infinite, NaN) is handled outside the table.
// Addressing is pure bit-field work so that it can run on both halves of a packed pair:
// adding kLutBias to a pattern moves the 32 covered exponents to 128..159, i.e. bits 14..12
// of the biased pattern are 100 exactly for covered values, and the slot is its low 12 bits
// (5 exponent bits, 7 mantissa bits) plus the sign as bit 12.
constexpr uint32_t kLutBias = (128u - (127u - 16u)) << 7;  // 0x0880
constexpr int kLutSize = 8192;
// A thread's kChunk staged terms are followed by 4 floats of padding: 128-bit reads of
// consecutive runs by consecutive lanes then fall into distinct banks.
constexpr int kStagePitch = kChunk + 4;

struct Entry {
  uint32_t key;  // float bits of e_i (list A) or p_i (sorted lists); positive floats order like integers
  int32_t idx;   // token index
};

// Shared state of the value-class tail (value_class_tail.cuh): a window of class counts, later
// reused for per-(tile, thread) member counts, and the block's walk record.
constexpr int kVcBins = 16384;                 // 32-bit class counters of a window (or twice as many 16-bit ones)
constexpr int kVcPer = 4;                      // classes per thread in one round of the walk
constexpr int kVcTile = kThreads * kVcPer;
constexpr int kVcSelTile = kThreads * 32;      // logits per tile of the final lookup
constexpr int kVcSelTiles = kVcBins / kThreads;
constexpr int kVcListCap = 32768;              // a 16-bit top-p row with more listed candidates takes the class tail
constexpr int kVcListProbe = 2048;             // from this many on, the count so far is extrapolated to the whole row
constexpr int kVcMinNucleus = 4096;            // ... and so does one whose list is short of this many, at least
constexpr int kVcPendCap = 8;                  // deferred tails a block collects before it runs them
constexpr int kVcCheckpoints = 6;              // window starts of one row (65536 keys / kVcBins, and one)
static_assert(kVcPer == 4, "a thread reads its four class counts as one 128-bit (or 64-bit) word");

struct VcHist {
  alignas(16) unsigned hist[kVcBins];
};
struct NoVcHist {};
struct VcControl {
  SeqSummary wsum[kWarps], wpre[kWarps], tot;
  int wcnt[kWarps], wpre_cnt[kWarps], tot_cnt;
  int hit_tid, found, kb, n, hit_b, hit_j, hit_pos;
  float cum, p;
  int ended;
  unsigned last_key;
  int loaded_hi, n_ck;
  int ck_hi[kVcCheckpoints], ck_kb[kVcCheckpoints], ck_n[kVcCheckpoints], ck_pos[kVcCheckpoints];
  int g_lo, g_hi, token;
  int tile_tot[kVcSelTiles];
  // rows whose tail is deferred until the block has left its row loop (see sample_rows_kernel)
  int n_pend;      // rows recorded in pend[]
  int class_ok;    // the current row may take the class tail
  float raw_max;   // the current row's largest logit
  struct Pending {
    long long row;
    float inv_t, mx, sum, cutoff, topp, coin, raw_max;
  } pend[kVcPendCap];
};

template <bool kLut, bool kExtended = false>
struct __align__(16) Shared {
  VcControl vcc;
  // (members read with vector loads carry their own alignas)
  static constexpr bool kHasLut = kLut;
  static constexpr bool kExt = kExtended;  // per-row settings and the fused scalar multiply
  uint64_t exp_tab[kExpTableSize];
  alignas(16) float head[kHead];  // read as float4
  SeqSummary wsum[3][kWarps];  // slots used by successive scan rounds in rotation (see seqsum_tile)
  int first[2];
  int wcnt[2][kWarps];
  float redf[kWarps];
  int redi[kWarps];
  unsigned hcnt[kBins];
  float hmass[kBins];
  float s_bcast;
  int hit_found;
  int hit_idx;
  float hit_val;
  int misc_i[4];
  float misc_f[4];
  // The table sits directly in front of the union: the value-class tail, which needs neither,
  // lays its window of class counts over both (vc_hist()).
  alignas(16) float lut[kLut ? kLutSize : 4];
  union alignas(16) {
    // terms of the row's first tile, one padded run per thread, for the one-warp start of the sum
    alignas(16) float stage[kThreads * kStagePitch];
    unsigned wbins[kWarps / 2][kBins][2];  // per warp pair and value bin: count, sum of mantissa offsets
    struct {
      unsigned short cnt[kCompactSteps][kWarps];  // survivors per (step, warp), then exclusive in step
      unsigned base[kCompactSteps];               // survivors in front of each step
    } compact;
    struct {
      unsigned long long ck[kRankSortMax];
      int rank[kRankSortMax];
    } rsort;
    struct {  // the whole tail of a row with a short nucleus, in shared memory (small_tail)
      unsigned long long ck[kRankSortMax];
      alignas(16) float p[kRankSortMax + 8];  // read four at a time, one group ahead
      int idx[kRankSortMax];
      alignas(16) float prefix[kRankSortMax + 4];
      int cnt;
      int first_above;
      int last;
      float cum;
    } small;
    struct {
      unsigned wofs[kWarps][kRadix];  // per warp and digit: count, then running output offset
      unsigned above[kRadix];
    } radix;
    typename std::conditional<kLut, NoVcHist, VcHist>::type vc;
  } u;
};

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__half v) { return __half2float(v); }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename S>
__device__ __forceinline__ float block_max(S& sm, float v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, d));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm.redf[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = sm.redf[0];
#pragma unroll
  for (int w = 1; w < kWarps; ++w) r = fmaxf(r, sm.redf[w]);
  return r;
}

// Exclusive block-wide prefix count of a per-thread count; *total gets the block sum.
template <typename S>
__device__ __forceinline__ int block_excl_count(S& sm, int cnt, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = cnt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += o;
  }
  __syncthreads();
  if (lane == 31) sm.redi[warp] = inc;
  __syncthreads();
  int pre = 0, tot = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const int c = sm.redi[w];
    if (w < warp) pre += c;
    tot += c;
  }
  *total = tot;
  return pre + inc - cnt;
}

// Summary of one thread's chunk in the binade kb of the running sum: the tie-free fast path
// first, the two-parity functions when the chunk holds an exact half-way term (or for sums
// outside the fast path's range).
__device__ __forceinline__ SeqSummary chunk_summary(const float (&v)[kChunk], int kb) {
  SeqSummary mine;
  seq_identity(&mine);
  if (kb >= 27 && kb <= 252) {
    // v / u by an exact power-of-two scaling; adding 2^23 rounds it to an integer (half to
    // even). Four interleaved accumulator pairs: short dependency chains (the partial sums
    // are integers below 2^24, hence exact, whenever the total is; otherwise the total
    // stays at or above 2^24, which is all that matters then).
    const float inv_u24 = seq_inv_u24(kb);
    float a4[4] = {0.0f, 0.0f, 0.0f, 0.0f}, t4[4] = {1.0f, 1.0f, 1.0f, 1.0f};
#pragma unroll
    for (int j = 0; j < kChunk; ++j) seq_push_fast(&a4[j & 3], &t4[j & 3], v[j], inv_u24);
    const float accf = __fadd_rn(__fadd_rn(a4[0], a4[1]), __fadd_rn(a4[2], a4[3]));
    const float tie_prod = __fmul_rn(__fmul_rn(t4[0], t4[1]), __fmul_rn(t4[2], t4[3]));
    const int acc = (int)fminf(accf, (float)kFastSat);
    mine.a0 = acc;
    mine.a1 = acc;
    if (!(tie_prod != 0.0f)) {  // zero (a tie, or an underflowed product) or NaN
      const float inv_u = seq_inv_u(kb);
      seq_identity(&mine);
#pragma unroll
      for (int j = 0; j < kChunk; ++j) seq_push_scaled(&mine, v[j], inv_u);
    }
  } else {
#pragma unroll
    for (int j = 0; j < kChunk; ++j) seq_push(&mine, v[j], kb);
  }
  if (mine.a0 > kFastSat) mine.a0 = kFastSat;
  if (mine.a1 > kFastSat) mine.a1 = kFastSat;
  return mine;
}

// ---------------------------------------------------------------------------------------
// The same exact sequential sum at warp scope: lane l holds the kChunk terms that follow
// those of lanes 0..l-1; `s` is warp-uniform. No shared memory and no block barrier, so a
// round costs one warp's instructions instead of the whole block's. Used where the running
// sum leaves its binade every few hundred terms (the start of a row). Same contract as
// seqsum_tile otherwise (pos0 = position of lane 0's first term).
// ---------------------------------------------------------------------------------------
template <bool kSearch>
__device__ __forceinline__ bool seqsum_warp(
    const float (&v)[kChunk], float& s, float thr, int pos0, int limit, int* hit_pos,
    float* hit_sum) {
  const int lane = threadIdx.x & 31;
  int consumed = 0;
  while (true) {
    const int kb = seq_kb(s);
    const int n_s = seq_n(s);
    SeqSummary mine;
    seq_identity(&mine);
    const bool active = lane >= consumed;
    if (active) mine = chunk_summary(v, kb);
    const bool two_parity = __any_sync(0xffffffffu, mine.a0 != mine.a1);
    if (!two_parity) {
      const int n_end = n_s + __reduce_add_sync(0xffffffffu, mine.a0);  // <= 2^24 + 32 * kFastSat
      bool more = n_end >= kSeqLimit;
      if (kSearch) {
        if (!more && seq_value(kb, n_end) > thr) more = true;
      }
      if (!more) {
        s = seq_value(kb, n_end);
        return false;
      }
    }
    int n_in, n_out;  // N in front of / behind this lane's chunk
    if (!two_parity) {
      int inc = mine.a0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += o;
      }
      n_in = n_s + (inc - mine.a0);
      n_out = n_s + inc;
    } else {
      SeqSummary sc = mine;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        SeqSummary o;
        o.a0 = __shfl_up_sync(0xffffffffu, sc.a0, d);
        o.a1 = __shfl_up_sync(0xffffffffu, sc.a1, d);
        if (lane >= d) sc = seq_compose(o, sc);
      }
      SeqSummary excl;
      excl.a0 = __shfl_up_sync(0xffffffffu, sc.a0, 1);
      excl.a1 = __shfl_up_sync(0xffffffffu, sc.a1, 1);
      if (lane == 0) seq_identity(&excl);
      n_in = seq_apply(n_s, excl);
      n_out = seq_apply(n_in, mine);
    }
    // the first chunk whose end value left the binade or, when searching, exceeds thr
    bool flag = active && n_out >= kSeqLimit;
    if (kSearch) {
      if (active && n_out < kSeqLimit && seq_value(kb, n_out) > thr) flag = true;
    }
    const unsigned lb = __ballot_sync(0xffffffffu, flag);
    if (lb == 0) {
      s = seq_value(kb, __shfl_sync(0xffffffffu, n_out, 31));
      return false;
    }
    const int first = __ffs(lb) - 1;
    float acc = 0.0f, hval = 0.0f;
    int found = 0, hpos = 0;
    if (lane == first) {
      // the sum in front of this chunk is exact: redo the chunk with real float additions
      acc = seq_value(kb, n_in);
#pragma unroll
      for (int j = 0; j < kChunk; ++j) {
        acc = __fadd_rn(acc, v[j]);
        if (kSearch) {
          const int pos = pos0 + lane * kChunk + j;
          if (!found && acc > thr && pos < limit) {
            found = 1;
            hpos = pos;
            hval = acc;
          }
        }
      }
    }
    s = __shfl_sync(0xffffffffu, acc, first);
    if (kSearch) {
      if (__shfl_sync(0xffffffffu, found, first)) {
        *hit_pos = __shfl_sync(0xffffffffu, hpos, first);
        *hit_sum = __shfl_sync(0xffffffffu, hval, first);
        return true;
      }
    }
    consumed = first + 1;
    if (consumed >= 32) return false;
  }
}

// ---------------------------------------------------------------------------------------
// One tile of the exact sequential float sum. Thread t holds the kChunk consecutive terms
// v[] that follow the terms of threads 0..t-1. `s` is the running sum in front of the
// tile on entry and behind it on return (block-uniform).
//
// Each round summarises every thread's chunk in the binade of s, and every warp its 32
// chunks: one integer (a warp reduction) when none of them holds an exact half-way term,
// else the two-parity summary of exact_math.cuh composed along the lanes. After ONE barrier
// every warp reads the kWarps summaries and decides, redundantly and identically, whether
// the value behind the tile is still inside the binade (and not beyond thr); then the tile
// total, a reduction or a composition of kWarps summaries, is all that is needed. Otherwise
// prefix sums down to the thread name the first chunk that leaves the binade (or holds the
// searched position); its thread redoes it with real float additions and publishes the new
// sum behind a second barrier, and the threads behind it go into the next round.
//
// Rounds rotate through three sets of shared slots (`rp`, block-uniform, carried by the
// caller across tiles), so a round needs no barrier to protect its slots from the previous
// round.
//
// With kSearch, also looks for the first term after which the running sum exceeds `thr`
// (terms at position >= limit, counted from pos0 of thread 0's first term, must be zero
// padding); on a match returns true with the position in *hit_pos and the sum reached
// there in *hit_sum (block-uniform), and `s` is then not meaningful.
// ---------------------------------------------------------------------------------------
template <bool kSearch, typename S>
__device__ __forceinline__ bool seqsum_tile(
    S& sm, const float (&v)[kChunk], float& s, int& rp, float thr, int pos0, int limit,
    int* hit_pos, float* hit_sum) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int consumed = 0;
  while (true) {
    const int kb = seq_kb(s);
    const int n_s = seq_n(s);
    SeqSummary mine;
    seq_identity(&mine);
    const bool active = tid >= consumed;
    if (active) mine = chunk_summary(v, kb);
    // Warp summary: one integer when none of the warp's chunks holds an exact half-way term
    // (a reduction), else the two-parity summary composed along the lanes (rare).
    SeqSummary lane_excl;  // two-parity summary of the lanes in front of this one (tie warps only)
    seq_identity(&lane_excl);
    SeqSummary wsum;
    const bool warp_tie = __any_sync(0xffffffffu, mine.a0 != mine.a1);
    if (!warp_tie) {
      const int wtot = __reduce_add_sync(0xffffffffu, mine.a0);  // <= 32 * kFastSat
      wsum.a0 = wsum.a1 = wtot < kFastSat ? wtot : kFastSat;
    } else {
      SeqSummary sc = mine;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        SeqSummary o;
        o.a0 = __shfl_up_sync(0xffffffffu, sc.a0, d);
        o.a1 = __shfl_up_sync(0xffffffffu, sc.a1, d);
        if (lane >= d) sc = seq_compose(o, sc);
      }
      lane_excl.a0 = __shfl_up_sync(0xffffffffu, sc.a0, 1);
      lane_excl.a1 = __shfl_up_sync(0xffffffffu, sc.a1, 1);
      if (lane == 0) seq_identity(&lane_excl);
      wsum.a0 = __shfl_sync(0xffffffffu, sc.a0, 31);
      wsum.a1 = __shfl_sync(0xffffffffu, sc.a1, 31);
    }
    if (lane == 0) sm.wsum[rp][warp] = wsum;
    __syncthreads();  // ---- barrier 1: the warp summaries are visible
    SeqSummary wt;
    seq_identity(&wt);
    if (lane < kWarps) wt = sm.wsum[rp][lane];
    const int next_rp = rp == 2 ? 0 : rp + 1;
    const bool two_parity = __any_sync(0xffffffffu, wt.a0 != wt.a1);
    int n_wend;  // N behind the warp `lane` (lanes < kWarps), for the warp-level decision
    if (!two_parity) {
      // The common round: N only grows along the tile, so if the value behind the whole tile
      // is still inside the binade (and not beyond thr), nothing in between left it: the
      // tile total is all that is needed, one reduction and no prefix sums.
      const int n_end = n_s + __reduce_add_sync(0xffffffffu, wt.a0);
      bool more = n_end >= kSeqLimit;
      if (kSearch) {
        if (!more && seq_value(kb, n_end) > thr) more = true;
      }
      if (!more) {
        s = seq_value(kb, n_end);
        rp = next_rp;
        return false;
      }
      n_wend = 0;
    } else {
      // a tie somewhere: compose the kWarps summaries; exact as long as N stays in the binade
#pragma unroll
      for (int d = 1; d < kWarps; d <<= 1) {
        SeqSummary o;
        o.a0 = __shfl_up_sync(0xffffffffu, wt.a0, d);
        o.a1 = __shfl_up_sync(0xffffffffu, wt.a1, d);
        if (lane >= d) wt = seq_compose(o, wt);
      }
      n_wend = seq_apply(n_s, wt);
      const int n_end = __shfl_sync(0xffffffffu, n_wend, kWarps - 1);
      bool more = n_end >= kSeqLimit;
      if (kSearch) {
        if (!more && seq_value(kb, n_end) > thr) more = true;
      }
      if (!more) {
        s = seq_value(kb, n_end);
        rp = next_rp;
        return false;
      }
    }
    // Some chunk leaves the binade (or holds the searched position): prefix sums per thread
    int n_in, n_out;  // N in front of / behind this thread's chunk
    if (!two_parity) {
      int inc = mine.a0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += o;
      }
      int wi = wt.a0;
#pragma unroll
      for (int d = 1; d < kWarps; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, wi, d);
        if (lane >= d) wi += o;
      }
      int pre = __shfl_sync(0xffffffffu, wi, warp > 0 ? warp - 1 : 0);
      if (warp == 0) pre = 0;
      n_wend = n_s + wi;
      n_in = n_s + pre + (inc - mine.a0);
      n_out = n_in + mine.a0;
    } else {
      // wt holds the inclusive composition over the warps; tie-free warps have not formed
      // their lanes' prefix yet
      if (!warp_tie) {
        int inc = mine.a0;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int o = __shfl_up_sync(0xffffffffu, inc, d);
          if (lane >= d) inc += o;
        }
        lane_excl.a0 = lane_excl.a1 = inc - mine.a0;
      }
      SeqSummary pre;
      pre.a0 = __shfl_sync(0xffffffffu, wt.a0, warp > 0 ? warp - 1 : 0);
      pre.a1 = __shfl_sync(0xffffffffu, wt.a1, warp > 0 ? warp - 1 : 0);
      if (warp == 0) seq_identity(&pre);
      pre = seq_compose(pre, lane_excl);
      n_in = seq_apply(n_s, pre);
      n_out = seq_apply(n_in, mine);
    }
    // Which warp holds the first chunk to redo: the first whose end value left the binade
    // (N >= 2^24) or, when searching, exceeds thr. N only grows along the tile, so this is
    // decided from the warp-end values alone, identically by every warp.
    bool wflag = lane < kWarps && n_wend >= kSeqLimit;
    if (kSearch) {
      if (lane < kWarps && n_wend < kSeqLimit && seq_value(kb, n_wend) > thr) wflag = true;
    }
    const unsigned wb = __ballot_sync(0xffffffffu, wflag);
    rp = next_rp;
    if (wb == 0) {
      // nothing left the binade: the whole tile is summarised exactly
      s = seq_value(kb, __shfl_sync(0xffffffffu, n_wend, kWarps - 1));
      return false;
    }
    const int redo_warp = __ffs(wb) - 1;
    if (warp == redo_warp) {
      bool flag = active && (n_out >= kSeqLimit);
      if (kSearch) {
        if (active && n_out < kSeqLimit && seq_value(kb, n_out) > thr) flag = true;
      }
      const unsigned lb = __ballot_sync(0xffffffffu, flag);
      const int first_lane = __ffs(lb) - 1;  // exists: this warp's end value is flagged
      if (lane == first_lane) {
        // The sum in front of this chunk is exact; redo the chunk with real float additions
        // (it leaves the binade here, or it contains the searched position).
        float acc = seq_value(kb, n_in);
        int found = 0;
#pragma unroll
        for (int j = 0; j < kChunk; ++j) {
          acc = __fadd_rn(acc, v[j]);
          if (kSearch) {
            const int pos = pos0 + tid * kChunk + j;
            if (!found && acc > thr && pos < limit) {
              found = 1;
              sm.hit_idx = pos;
              sm.hit_val = acc;
            }
          }
        }
        sm.hit_found = found;
        sm.s_bcast = acc;
        sm.first[0] = tid;
      }
    }
    __syncthreads();  // ---- barrier 2 (only in rounds that redo a chunk)
    s = sm.s_bcast;
    const int first = sm.first[0];
    const bool hit = kSearch && sm.hit_found;
    if (hit) {
      *hit_pos = sm.hit_idx;
      *hit_sum = sm.hit_val;
    }
    consumed = first + 1;
    if (hit || consumed >= kThreads) {
      __syncthreads();  // the result slots may be rewritten by the caller's next step
      return hit;
    }
    // the next round's barrier 1 orders these reads before the next writes of the slots
  }
}

// The tile behind the sequential head is where the running sum still leaves its binade every
// few hundred terms, and every such round of seqsum_tile occupies the whole block. Instead the
// tile's terms are staged in shared memory (stage_first_tile, which ends with a barrier) and
// one warp sums them 512 at a time (sum_staged_tile, block-uniform result behind a barrier)
// while the other warps wait or, between the two calls, do other work.
template <typename S>
__device__ __forceinline__ void stage_first_tile(S& sm, const float (&e)[kChunk]) {
  float4* st4 = reinterpret_cast<float4*>(sm.u.stage + threadIdx.x * kStagePitch);
#pragma unroll
  for (int q = 0; q < kChunk / 4; ++q) st4[q] = make_float4(e[4 * q], e[4 * q + 1], e[4 * q + 2], e[4 * q + 3]);
  __syncthreads();
}

template <bool kSearch, typename S>
__device__ __forceinline__ bool sum_staged_tile(
    S& sm, float& s, float thr, int vocab, int* hit_pos, float* hit_sum) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    const int span = (vocab - kHead) < kTile ? (vocab - kHead) : kTile;
    const int n_sub = (span + 32 * kChunk - 1) / (32 * kChunk);
    float sw = s, hs = 0.0f;
    int hp = 0;
    bool hit = false;
    for (int t = 0; t < n_sub && !hit; ++t) {
      float v[kChunk];
      const float4* p4 = reinterpret_cast<const float4*>(sm.u.stage + (t * 32 + lane) * kStagePitch);
#pragma unroll
      for (int q = 0; q < kChunk / 4; ++q) {
        const float4 x = p4[q];
        v[4 * q] = x.x;
        v[4 * q + 1] = x.y;
        v[4 * q + 2] = x.z;
        v[4 * q + 3] = x.w;
      }
      hit = seqsum_warp<kSearch>(v, sw, thr, kHead + t * 32 * kChunk, vocab, &hp, &hs);
    }
    if (lane == 0) {
      sm.s_bcast = sw;
      sm.hit_found = hit ? 1 : 0;
      sm.hit_idx = hp;
      sm.hit_val = hs;
    }
  }
  __syncthreads();  // the result; the staging buffer is free again
  s = sm.s_bcast;
  const bool hit = kSearch && sm.hit_found;
  if (hit) {
    *hit_pos = sm.hit_idx;
    *hit_sum = sm.hit_val;
  }
  return hit;
}

// The first terms of a sum leave a binade every few additions, which would cost one block
// round each; instead one thread adds the `count` terms staged in sm.head with real float
// additions. Same contract as seqsum_tile. Callers fill sm.head before the call and need no
// barrier in between: this function synchronises on entry and on exit.
template <bool kSearch, typename S>
__device__ __forceinline__ bool head_sum(
    S& sm, int count, float& s, float thr, int pos0, int* hit_pos, float* hit_sum) {
  __syncthreads();
  if (threadIdx.x == 0) {
    // sm.head is zero-padded to a multiple of 4, and the terms are non-negative, so the
    // partial sums only grow: test four additions at a time
    float acc = s;
    int found = 0;
    const float4* h4 = reinterpret_cast<const float4*>(sm.head);
    for (int i = 0; i < count; i += 4) {
      const float4 q = h4[i >> 2];
      const float a1 = __fadd_rn(acc, q.x);
      const float a2 = __fadd_rn(a1, q.y);
      const float a3 = __fadd_rn(a2, q.z);
      const float a4 = __fadd_rn(a3, q.w);
      if (kSearch && a4 > thr) {
        int k = 3;
        float hv = a4;
        if (a3 > thr) { k = 2; hv = a3; }
        if (a2 > thr) { k = 1; hv = a2; }
        if (a1 > thr) { k = 0; hv = a1; }
        if (i + k < count) {
          found = 1;
          sm.hit_idx = pos0 + i + k;
          sm.hit_val = hv;
        }
        acc = a4;
        break;
      }
      acc = a4;
    }
    sm.hit_found = found;
    sm.s_bcast = acc;
  }
  __syncthreads();
  s = sm.s_bcast;
  bool hit = false;
  if (kSearch && sm.hit_found) {
    *hit_pos = sm.hit_idx;
    *hit_sum = sm.hit_val;
    hit = true;
  }
  __syncthreads();  // the head buffer and the result slots may be reused after this
  return hit;
}

__device__ __forceinline__ float warp_max_f32(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// Writes the token of row r: to out_ids[r], or -- when peer buffers are given -- straight into
// every listed buffer at [offset + r] (each may live on another GPU of the node: plain
// stores over NVLink, one thread per destination). Block-uniform `token`.
__device__ __forceinline__ void store_token(
    int64_t* __restrict__ out_ids, const PeerOut& peers, int64_t r, int token) {
  if (peers.n == 0) {
    if (threadIdx.x == 0) out_ids[r] = (int64_t)token;
  } else if ((int)threadIdx.x < peers.n) {
    peers.ptr[threadIdx.x][peers.offset + r] = (int64_t)token;
  }
}

// Arrival barrier among the GPUs of a node at the end of a launch (see PeerOut). Every thread
// of every block calls it once, after its last store_token. No kernel of one GPU waits for
// another kernel of the same GPU; the wait for the other GPUs is limited to peers.wait_ns
// nanoseconds of the GPU's global timer, after which the launch records kStatusPeerTimeout in
// *status and ends (the context stays usable; the ids of the missing ranks are stale).
__device__ __forceinline__ unsigned long long global_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void peer_arrival_barrier(const PeerOut& peers, int* status) {
  if (peers.epoch == 0ull) return;  // launch-uniform
  __shared__ int is_last;
  __threadfence_system();  // this thread's id stores are ordered before the block's arrival
  __syncthreads();
  if (threadIdx.x == 0) {
    const int prev = atomicAdd(peers.blocks_done, 1);
    is_last = (prev == (int)gridDim.x - 1) ? 1 : 0;
  }
  __syncthreads();
  if (!is_last) return;  // block-uniform
  __threadfence_system();  // every block's ids before this rank's arrival marks
  if (threadIdx.x == 0) *peers.blocks_done = 0;
  if ((int)threadIdx.x < peers.n) {
    volatile unsigned long long* theirs = peers.arrive[threadIdx.x] + peers.rank;
    *theirs = peers.epoch;  // tell rank threadIdx.x that this rank's ids are in its buffer
    volatile unsigned long long* mine = peers.arrive[peers.rank] + threadIdx.x;
    const unsigned long long t0 = global_timer_ns();
    unsigned spins = 0;
    while (*mine < peers.epoch) {  // until rank threadIdx.x has told this rank
      // the timer is read every 64 polls; the poll count is a second, independent bound
      if ((++spins & 63u) == 0u && (global_timer_ns() - t0 > peers.wait_ns || spins > (1u << 30))) {
        atomicExch(status, kStatusPeerTimeout);
        break;
      }
    }
  }
  __threadfence_system();
  __syncthreads();
}

// Programmatic dependent launch: a kernel launched with the programmatic-serialization attribute
// may start while its predecessor in the stream still runs. It must wait here before it touches
// anything the predecessor writes (the wait ends when the predecessor's grid has completed and
// its writes are visible; without the attribute it returns at once). The predecessor lets its
// dependents become resident early with grid_launch_dependents().
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Bounded wait for a bulk copy. Returns false if it has not landed after about a second.
__device__ __forceinline__ bool wait_bulk_copy(unsigned long long* bar, uint32_t parity) {
  const uint32_t a = smem_addr(bar);
  for (int spin = 0; spin < (1 << 22); ++spin) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// The hardware barrier of the cluster, split so that work can sit between arrival and wait.
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// xorshift64* step and 24-bit coin of the reference (sampler.cpp:210-220).
__device__ __forceinline__ float next_coin(unsigned long long* state) {
  unsigned long long s = *state;
  s ^= s >> 12;
  s ^= s << 25;
  s ^= s >> 27;
  *state = s;
  const unsigned u = (unsigned)((s * 0x2545F4914F6CDD1Dull) >> 32);
  return (float)(u >> 8) / 16777216.0f;
}

// ---------------------------------------------------------------------------------------
// Per-row element math: e = expf(logit * inv_t - mx) (sampler.cpp:231-233 and :201), or
// e / S once the sum is known (sampler.cpp:205-207) when `probs` is set.
// ---------------------------------------------------------------------------------------
template <typename T, typename S>
struct RowMath {
  const T* row;
  int vocab;
  bool vec_ok;
  float inv_t;
  float mx;
  float sum;   // divisor when probs is set
  bool probs;
  float scale = 1.0f;  // extended entry point only: every logit is first multiplied by this, in T

  // The logit as the sampler sees it: a "multiply" logit processor folded into the load
  // (logit_processor.h:34-40 works in place on T, so the product is rounded to T).
  __device__ __forceinline__ float xform(float logit) const {
    if constexpr (S::kExt) {
      const float y = __fmul_rn(logit, scale);
      if constexpr (std::is_same<T, __nv_bfloat16>::value) return __bfloat162float(__float2bfloat16_rn(y));
      if constexpr (std::is_same<T, __half>::value) return __half2float(__float2half_rn(y));
      return y;
    } else {
      return logit;
    }
  }

  __device__ __forceinline__ float direct(float logit, const S& sm) const {
    const float e = expf_ref(__fsub_rn(__fmul_rn(xform(logit), inv_t), mx), sm.exp_tab);
    return probs ? __fdiv_rn(e, sum) : e;
  }

  // bf16 bit pattern -> table slot, or -1 when the value is outside the table
  static __device__ __forceinline__ int lut_slot(uint32_t h) {
    const uint32_t hb = h + kLutBias;
    const int slot = (int)((hb & 0x0FFFu) | ((hb >> 3) & 0x1000u));
    return (hb & 0x7000u) == 0x4000u ? slot : -1;
  }

  static __device__ __forceinline__ uint32_t lut_pattern(int slot) {
    const uint32_t hb = 0x4000u | ((uint32_t)slot & 0x0FFFu);
    return ((hb - kLutBias) & 0x7FFFu) | (((uint32_t)slot & 0x1000u) << 3);
  }

  // Fills the table for this row (bf16 only): slot -> e, or e / S when probs is set.
  __device__ __forceinline__ void build_lut(S& sm) const {
    for (int k = threadIdx.x; k < kLutSize; k += kThreads) {
      sm.lut[k] = direct(bits_f32(lut_pattern(k) << 16), sm);
    }
  }

  __device__ __forceinline__ float from_pattern(uint32_t h, const S& sm) const {
    const int slot = lut_slot(h);
    if (slot >= 0) return sm.lut[slot];
    return direct(bits_f32(h << 16), sm);
  }

  // One element (used for the sequential head and for ragged edges). 0 beyond the row.
  __device__ __forceinline__ float at(int i, const S& sm) const {
    if (i >= vocab) return 0.0f;
    if constexpr (S::kHasLut) {
      return from_pattern((uint32_t) reinterpret_cast<const unsigned short*>(row)[i], sm);
    } else {
      return direct(to_f32(row[i]), sm);
    }
  }

  // The 128-bit loads of a full, aligned chunk, separated from their use so that the next
  // tile's loads can be in flight while this tile is processed.
  static constexpr int kRawVecs = kChunk * sizeof(T) / 16;
  struct Raw {
    uint4 q[kRawVecs];
  };
  __device__ __forceinline__ bool full(int i0) const { return vec_ok && i0 + kChunk <= vocab; }
  __device__ __forceinline__ void load_raw(int i0, Raw* r) const {
#pragma unroll
    for (int q = 0; q < kRawVecs; ++q) r->q[q] = __ldg(reinterpret_cast<const uint4*>(row + i0) + q);
  }
  __device__ __forceinline__ void eval_raw(const Raw& r, const S& sm, float (&e)[kChunk]) const {
    constexpr int kPerVec = 16 / sizeof(T);
    uint32_t bad = 0u;  // bits 14..12 of a biased half that differ from 100, over the chunk
    (void)bad;
#pragma unroll
    for (int q = 0; q < kRawVecs; ++q) {
      if constexpr (S::kHasLut) {
        const uint32_t w[4] = {r.q[q].x, r.q[q].y, r.q[q].z, r.q[q].w};
        const char* lut_bytes = reinterpret_cast<const char*>(sm.lut);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // both halves at once. A carry out of the low half only happens for a low pattern
          // that is outside the table anyway, and then the whole chunk is redone below.
          const uint32_t wb = w[j] + (kLutBias | (kLutBias << 16));
          bad |= wb ^ 0x40004000u;
          const uint32_t off0 = ((wb << 2) & 0x3FFCu) | ((wb >> 1) & 0x4000u);
          const uint32_t off1 = ((wb >> 14) & 0x3FFCu) | ((wb >> 17) & 0x4000u);
          e[q * 8 + 2 * j] = *reinterpret_cast<const float*>(lut_bytes + off0);
          e[q * 8 + 2 * j + 1] = *reinterpret_cast<const float*>(lut_bytes + off1);
        }
      } else {
        const T* p = reinterpret_cast<const T*>(&r.q[q]);
#pragma unroll
        for (int j = 0; j < kPerVec; ++j) e[q * kPerVec + j] = direct(to_f32(p[j]), sm);
      }
    }
    if constexpr (S::kHasLut) {
      // every pattern is inside the table iff bits 14..12 of every biased half are 100
      if ((bad & 0x70007000u) != 0u) {
        // rare: a zero, tiny, huge or non-finite logit in this chunk; redo the chunk element by
        // element (table where possible, direct evaluation otherwise)
#pragma unroll
        for (int q = 0; q < kRawVecs; ++q) {
          const uint32_t w[4] = {r.q[q].x, r.q[q].y, r.q[q].z, r.q[q].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            e[q * 8 + 2 * j] = from_pattern(w[j] & 0xFFFFu, sm);
            e[q * 8 + 2 * j + 1] = from_pattern(w[j] >> 16, sm);
          }
        }
      }
    }
  }

  // kChunk consecutive elements starting at i0.
  __device__ __forceinline__ void chunk(int i0, const S& sm, float (&e)[kChunk]) const {
    if (vec_ok && i0 + kChunk <= vocab) {
      constexpr int kPerVec = 16 / sizeof(T);
#pragma unroll
      for (int q = 0; q < kChunk / kPerVec; ++q) {
        const uint4 raw = __ldg(reinterpret_cast<const uint4*>(row + i0) + q);
        if constexpr (S::kHasLut) {
          const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            e[q * 8 + 2 * j] = from_pattern(w[j] & 0xFFFFu, sm);
            e[q * 8 + 2 * j + 1] = from_pattern(w[j] >> 16, sm);
          }
        } else {
          const T* p = reinterpret_cast<const T*>(&raw);
#pragma unroll
          for (int j = 0; j < kPerVec; ++j) e[q * kPerVec + j] = direct(to_f32(p[j]), sm);
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < kChunk; ++j) e[j] = at(i0 + j, sm);
    }
  }
};

__device__ __forceinline__ __half2 neg_inf2(__half) {
  const __half v = __ushort_as_half((unsigned short)0xFC00);
  return __halves2half2(v, v);
}
__device__ __forceinline__ __nv_bfloat162 neg_inf2(__nv_bfloat16) {
  const __nv_bfloat16 v = __ushort_as_bfloat16((unsigned short)0xFF80);
  return __halves2bfloat162(v, v);
}

// Max over the row of logit * inv_t (softmax, sampler.cpp:191-196).
template <typename T, typename S>
__device__ __forceinline__ float row_max_scaled(
    S& sm, const RowMath<T, S>& rm, const T* __restrict__ row, int vocab, bool vec_ok, float inv_t,
    float* raw_max = nullptr) {
  const int tid = threadIdx.x;
  if (raw_max != nullptr) *raw_max = NAN;  // known only on the 16-bit path below
  if constexpr (sizeof(T) == 2) {
    if (inv_t > 0.0f) {
      // x -> fl(x * inv_t) is monotone for inv_t > 0, so the max can be taken on the raw
      // 16-bit values, two per instruction, and scaled once
      using T2 = decltype(neg_inf2(T()));
      const int nvec = vec_ok ? vocab / 8 : 0;
      T2 acc = neg_inf2(T());
      // this pass is the row's HBM read: four 128-bit loads in flight per thread
      int q = tid;
      for (; q + 3 * kThreads < nvec; q += 4 * kThreads) {
        uint4 raw[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) raw[k] = __ldg(reinterpret_cast<const uint4*>(row) + q + k * kThreads);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const T2* p = reinterpret_cast<const T2*>(&raw[k]);
          acc = __hmax2(acc, __hmax2(__hmax2(p[0], p[1]), __hmax2(p[2], p[3])));
        }
      }
      for (; q < nvec; q += kThreads) {
        const uint4 raw = __ldg(reinterpret_cast<const uint4*>(row) + q);
        const T2* p = reinterpret_cast<const T2*>(&raw);
        acc = __hmax2(acc, __hmax2(__hmax2(p[0], p[1]), __hmax2(p[2], p[3])));
      }
      float m = fmaxf(to_f32(acc.x), to_f32(acc.y));
      for (int i = nvec * 8 + tid; i < vocab; i += kThreads) m = fmaxf(m, to_f32(row[i]));
      m = block_max(sm, m);
      if (raw_max != nullptr) *raw_max = m;
      return __fmul_rn(rm.xform(m), inv_t);  // the multiply is by a positive factor: monotone too
    }
  }
  float mx = -INFINITY;
  for (int i = tid; i < vocab; i += kThreads) mx = fmaxf(mx, __fmul_rn(rm.xform(to_f32(row[i])), inv_t));
  return block_max(sm, mx);
}

// ---------------------------------------------------------------------------------------
// Stable LSD radix sort pass over a list of n entries, descending in the 8-bit digit at
// `shift`. One block; src and dst are distinct global buffers.
//
// Every warp owns a contiguous slice of the list. (1) Each warp counts the digits of its
// slice into its own 256 counters. (2) One block-wide prefix turns the counters into start
// offsets: digits in descending order, and within a digit the warps in order, which is the
// list order. (3) Each warp scatters its slice in steps of 32 entries, ranking the lanes of
// a step with a warp match and advancing its private offsets; no block barrier is needed
// inside the scatter.
// ---------------------------------------------------------------------------------------
template <typename S>
__device__ void radix_pass_desc(S& sm, const Entry* src, Entry* dst, int n, int shift) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned (*wofs)[kRadix] = sm.u.radix.wofs;
  const int per_warp = ((n + kWarps - 1) / kWarps + 31) & ~31;  // slice length, a multiple of 32
  const int lo = warp * per_warp < n ? warp * per_warp : n;
  const int hi = lo + per_warp < n ? lo + per_warp : n;
  __syncthreads();  // earlier users of the union are done
  for (int d = lane; d < kRadix; d += 32) wofs[warp][d] = 0;
  __syncwarp();
  for (int i0 = lo; i0 < hi; i0 += 32 * kListBatch) {
    uint32_t k[kListBatch];
#pragma unroll
    for (int u = 0; u < kListBatch; ++u) {  // independent loads first, so they overlap
      const int i = i0 + u * 32 + lane;
      k[u] = i < hi ? src[i].key : 0u;
    }
#pragma unroll
    for (int u = 0; u < kListBatch; ++u) {
      if (i0 + u * 32 + lane < hi) atomicAdd(&wofs[warp][(k[u] >> shift) & (kRadix - 1)], 1u);
    }
  }
  __syncthreads();
  // thread d (< 256) walks digit d over the warps; the digit totals are then prefixed in
  // descending digit order
  unsigned digit_total = 0;
  if (tid < kRadix) {
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const unsigned c = wofs[w][tid];
      wofs[w][tid] = digit_total;  // entries of this digit in earlier warps
      digit_total += c;
    }
    // suffix sums over the 256 digits: 8 warps of 32 digits each
    unsigned incl = digit_total;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned o = __shfl_down_sync(0xffffffffu, incl, d);
      if (lane + d < 32) incl += o;
    }
    sm.u.radix.above[tid] = incl - digit_total;  // larger digits inside this group of 32
    if (lane == 0) sm.redi[warp] = (int)incl;
  }
  __syncthreads();
  if (tid < kRadix) {
    unsigned above = sm.u.radix.above[tid];
    for (int w = warp + 1; w < kRadix / 32; ++w) above += (unsigned)sm.redi[w];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) wofs[w][tid] += above;
  }
  __syncthreads();
  for (int i0 = lo; i0 < hi; i0 += 32) {
    const int i = i0 + lane;
    const bool valid = i < hi;
    Entry e;
    e.key = 0;
    e.idx = 0;
    if (valid) e = src[i];
    const unsigned dg = valid ? ((e.key >> shift) & (kRadix - 1)) : 0xFFFFFFFFu;
    // rank among the lanes of this step that hold the same digit, in lane (= list) order
    const unsigned peers = __match_any_sync(0xffffffffu, dg);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    unsigned base = 0;
    if (valid) base = wofs[warp][dg];
    __syncwarp();
    if (valid) {
      dst[base + rank] = e;
      if (rank == 0) wofs[warp][dg] = base + __popc(peers);
    }
    __syncwarp();
  }
  __syncthreads();
}

// Exact cumulative sum over the key floats of a sorted list, looking for the first
// position (below `limit`) where it exceeds thr. Returns true with position and sum, else
// false with the total in *total. Short lists are summed sequentially through the head
// buffer; long ones continue with block-wide tiles.
template <typename S>
__device__ bool list_search(
    S& sm, const Entry* list, int n, int limit, float thr, int& rp, int* pos, float* sum,
    float* total) {
  const int lim = n < limit ? n : limit;
  float s = 0.0f;
  const int seq_end = lim <= 4 * kHead ? lim : kHead;
  int base = 0;
  for (; base < seq_end; base += kHead) {
    const int cnt = (seq_end - base) < kHead ? (seq_end - base) : kHead;
    __syncthreads();
    if (threadIdx.x < kHead) {
      const int i = base + threadIdx.x;
      sm.head[threadIdx.x] = (i < lim) ? bits_f32(list[i].key) : 0.0f;
    }
    if (head_sum<true>(sm, cnt, s, thr, base, pos, sum)) return true;
  }
  for (; base < lim; base += kTile) {
    float v[kChunk];
#pragma unroll
    for (int j = 0; j < kChunk; ++j) {
      const int i = base + threadIdx.x * kChunk + j;
      v[j] = (i < lim) ? bits_f32(list[i].key) : 0.0f;
    }
    if (seqsum_tile<true>(sm, v, s, rp, thr, base, lim, pos, sum)) return true;
  }
  *total = s;
  return false;
}

// ---------------------------------------------------------------------------------------
// Pieces of the top-p / top-k tail. All are block-wide and return block-uniform results.
// ---------------------------------------------------------------------------------------

// Bins the values of list A and picks the lowest value bin to keep: the largest bin b such
// that the bins >= b surely hold more than topp of the mass (top-p; the margin covers the
// rounding of the reference's own running sum) or at least topk entries (top-k). Returns
// false when even all listed entries do not suffice. *bin_out is 0 ("keep everything
// listed") in that case. *cnt_out = entries in the kept bins.
template <typename S>
__device__ bool pick_value_threshold(
    S& sm, const Entry* listA, int n_a, float sum, float topp, int topk, bool use_topk,
    int* bin_out, int* cnt_out) {
  const int tid = threadIdx.x, warp = tid >> 5;
  __syncthreads();  // earlier users of the union are done
  // per-warp integer counters, filled by one coalesced pass over the list
  for (int b = tid; b < (kWarps / 2) * kBins * 2; b += kThreads) (&sm.u.wbins[0][0][0])[b] = 0;
  __syncthreads();
  for (int i0 = 0; i0 < n_a; i0 += kListBatch * kThreads) {
    uint32_t k[kListBatch];
#pragma unroll
    for (int u = 0; u < kListBatch; ++u) {  // independent loads first, so they overlap
      const int i = i0 + u * kThreads + tid;
      k[u] = i < n_a ? listA[i].key : 0u;
    }
#pragma unroll
    for (int u = 0; u < kListBatch; ++u) {
      if (i0 + u * kThreads + tid < n_a) {
        int bin = (int)(k[u] >> kBinShift) - kBinBase;
        bin = bin < 0 ? 0 : (bin < kBins ? bin : kBins - 1);
        atomicAdd(&sm.u.wbins[warp >> 1][bin][0], 1u);
        atomicAdd(&sm.u.wbins[warp >> 1][bin][1], (k[u] >> 8) & 0x1FFFu);
      }
    }
  }
  __syncthreads();
  // Per-bin counts and the mass they hold, slightly rounded down: a value whose bits are
  // (bin << 21 | off) equals edge(bin) + off * 2^(exponent - 23), and off was accumulated with
  // its top 13 bits only. Bin 0 also holds everything below the covered range, so its mass
  // counts as 0.
  if (tid < kBins) {
    unsigned c = 0, o = 0;
#pragma unroll
    for (int w = 0; w < kWarps / 2; ++w) {
      c += sm.u.wbins[w][tid][0];
      o += sm.u.wbins[w][tid][1];
    }
    const uint32_t edge_bits = (uint32_t)(tid + kBinBase) << kBinShift;
    const float edge = bits_f32(edge_bits);
    // one unit of the 13-bit offset is 2^8 units of the last place of the bin's binade
    const float unit = bits_f32(edge_bits & 0x7F800000u) * (256.0f / 8388608.0f);
    sm.hcnt[tid] = c;
    sm.hmass[tid] = tid == 0 ? 0.0f : (float)c * edge + (float)o * unit;
  }
  __syncthreads();
  if (tid < 32) {
    float acc = 0.0f;
    unsigned cacc = 0;
    int chosen = 0, chosen_cnt = n_a;
    bool done = false;
    for (int hi = kBins - 1; hi >= 0 && !done; hi -= 32) {
      const int b = hi - tid;
      float m = (b >= 0) ? sm.hmass[b] : 0.0f;
      unsigned c = (b >= 0) ? sm.hcnt[b] : 0u;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const float om = __shfl_up_sync(0xffffffffu, m, d);
        const unsigned oc = __shfl_up_sync(0xffffffffu, c, d);
        if (tid >= d) {
          m += om;
          c += oc;
        }
      }
      const float mass_above = acc + m;
      const float cnt_above = (float)(cacc + c);
      const float need = sum * (topp * 1.002f + 0.001f + cnt_above * 4.8e-7f);
      // bin 0 is unbounded below, so it never counts as "above" anything
      const bool enough = b > 0 && (use_topk ? (cacc + c >= (unsigned)topk) : (mass_above >= need));
      const unsigned ok = __ballot_sync(0xffffffffu, enough);
      if (ok) {
        const int sel = __ffs(ok) - 1;
        chosen = hi - sel;
        chosen_cnt = (int)(cacc + __shfl_sync(0xffffffffu, c, sel));
        done = true;
      }
      acc += __shfl_sync(0xffffffffu, m, 31);
      cacc += __shfl_sync(0xffffffffu, c, 31);
    }
    if (tid == 0) {
      sm.misc_i[1] = chosen;
      sm.misc_i[2] = done ? 1 : 0;
      sm.misc_i[3] = chosen_cnt;
      sm.misc_f[1] = acc;  // mass of the bins looked at (all of them when the list was not enough)
    }
  }
  __syncthreads();
  *bin_out = sm.misc_i[1];
  *cnt_out = sm.misc_i[3];
  return sm.misc_i[2] != 0;
}

// Lists every entry of the row with e >= floor into list A, in index order. Returns the count.
template <typename T, typename S>
__device__ int gather_candidates(const RowMath<T, S>& rm, S& sm, Entry* listA, float floor) {
  const int tid = threadIdx.x;
  int n_a = 0;
  for (int base = 0; base < rm.vocab; base += kTile) {
    const int i0 = base + tid * kChunk;
    float e[kChunk];
    rm.chunk(i0, sm, e);  // 0 beyond the row, and floor > 0
    int cnt = 0;
#pragma unroll
    for (int j = 0; j < kChunk; ++j) cnt += (e[j] >= floor) ? 1 : 0;
    int tot;
    int off = n_a + block_excl_count(sm, cnt, &tot);
#pragma unroll
    for (int j = 0; j < kChunk; ++j) {
      if (e[j] >= floor) {
        Entry en;
        en.key = f32_bits(e[j]);
        en.idx = i0 + j;
        listA[off++] = en;
      }
    }
    n_a += tot;
  }
  __threadfence_block();
  __syncthreads();
  return n_a;
}

// Compacts list A into list B, in list order: entries with key >= key_lo whose probability
// e / sum passes the cutoff crop (sampler.cpp:136-143; no crop for top-k). List B holds the
// probabilities' bits. Two coalesced passes over list A per segment of kCompactSteps *
// kThreads entries: count the survivors of every (step, warp), prefix those counts, then
// write the survivors. Returns the number of survivors.
template <typename S>
__device__ int compact_candidates(
    S& sm, const Entry* listA, int n_a, Entry* listB, uint32_t key_lo, float sum, float cutoff,
    bool use_topk) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int n_b = 0;
  for (int seg0 = 0; seg0 < n_a; seg0 += kCompactSteps * kThreads) {
    const int seg_n = (n_a - seg0) < kCompactSteps * kThreads ? (n_a - seg0) : kCompactSteps * kThreads;
    const int steps = (seg_n + kThreads - 1) / kThreads;
    __syncthreads();  // earlier users of the union are done
    for (int st0 = 0; st0 < steps; st0 += kListBatch) {
      uint32_t k[kListBatch];
#pragma unroll
      for (int u = 0; u < kListBatch; ++u) {
        const int i = seg0 + (st0 + u) * kThreads + tid;
        k[u] = (st0 + u < steps && i < n_a) ? listA[i].key : 0u;
      }
#pragma unroll
      for (int u = 0; u < kListBatch; ++u) {
        if (st0 + u < steps) {  // block-uniform
          const int i = seg0 + (st0 + u) * kThreads + tid;
          const bool keep = i < n_a && k[u] >= key_lo &&
                            (use_topk || __fdiv_rn(bits_f32(k[u]), sum) >= cutoff);
          const unsigned kbal = __ballot_sync(0xffffffffu, keep);
          if (lane == 0) sm.u.compact.cnt[st0 + u][warp] = (unsigned short)__popc(kbal);
        }
      }
    }
    __syncthreads();
    // thread t owns step t: exclusive prefix inside the step, and the step total
    int step_total = 0;
    if (tid < steps) {
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const int c = sm.u.compact.cnt[tid][w];
        sm.u.compact.cnt[tid][w] = (unsigned short)step_total;
        step_total += c;
      }
    }
    int seg_total;
    const int step_base = block_excl_count(sm, step_total, &seg_total);
    if (tid < steps) sm.u.compact.base[tid] = (unsigned)(n_b + step_base);
    __syncthreads();
    for (int st0 = 0; st0 < steps; st0 += kListBatch) {
      Entry en[kListBatch];
#pragma unroll
      for (int u = 0; u < kListBatch; ++u) {
        const int i = seg0 + (st0 + u) * kThreads + tid;
        en[u].key = 0;
        en[u].idx = 0;
        if (st0 + u < steps && i < n_a) en[u] = listA[i];
      }
#pragma unroll
      for (int u = 0; u < kListBatch; ++u) {
        if (st0 + u < steps) {  // block-uniform
          const int i = seg0 + (st0 + u) * kThreads + tid;
          bool keep = false;
          if (i < n_a && en[u].key >= key_lo) {
            const float p = __fdiv_rn(bits_f32(en[u].key), sum);
            keep = use_topk || p >= cutoff;
            en[u].key = f32_bits(p);
          }
          const unsigned kbal = __ballot_sync(0xffffffffu, keep);
          if (keep) {
            listB[sm.u.compact.base[st0 + u] + sm.u.compact.cnt[st0 + u][warp] +
                  __popc(kbal & ((1u << lane) - 1u))] = en[u];
          }
        }
      }
    }
    n_b += seg_total;
  }
  __threadfence_block();
  __syncthreads();
  return n_b;
}

// Sorts list B by probability, descending; equal probabilities end up in index order. Small
// lists are rank-sorted in shared memory; larger ones take four stable LSD radix passes that
// ping-pong between list B and `spare` (after an even number of passes the result is back in
// list B).
template <typename S>
__device__ void sort_candidates(S& sm, Entry* listB, int n_b, Entry* spare) {
  const int tid = threadIdx.x;
  if (n_b <= kRankSortMax) {
    // Composite key = (probability bits, inverted index): larger means earlier in the sorted
    // order. kThreads / kRankSortMax threads share an entry, each scanning a part of the list.
    const int ent = tid & (kRankSortMax - 1), part = tid / kRankSortMax;
    Entry en;
    en.key = 0;
    en.idx = 0;
    if (tid < n_b) {
      en = listB[tid];
      sm.u.rsort.ck[tid] = ((unsigned long long)en.key << 32) | (uint32_t)(0x7FFFFFFF - en.idx);
      sm.u.rsort.rank[tid] = 0;
    }
    __syncthreads();
    if (ent < n_b) {
      const unsigned long long mine = sm.u.rsort.ck[ent];
      constexpr int kParts = kThreads / kRankSortMax;
      const int per = (n_b + kParts - 1) / kParts;
      const int j0 = part * per, j1 = (j0 + per) < n_b ? (j0 + per) : n_b;
      int rank = 0;
#pragma unroll 8
      for (int j = j0; j < j1; ++j) rank += sm.u.rsort.ck[j] > mine ? 1 : 0;
      atomicAdd(&sm.u.rsort.rank[ent], rank);
    }
    __syncthreads();
    if (tid < n_b) listB[sm.u.rsort.rank[tid]] = en;
    __threadfence_block();
  } else {
    Entry* ping = listB;
    Entry* pong = spare;
    for (int pass = 0; pass < 32 / kRadixBits; ++pass) {
      radix_pass_desc(sm, ping, pong, n_b, pass * kRadixBits);
      __threadfence_block();
      Entry* t = ping;
      ping = pong;
      pong = t;
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------------------
// The rest of sample_topp / sample_topk for a row whose survivors (list entries at or above
// the value threshold key_lo that pass the cutoff crop) number at most kRankSortMax, entirely
// in shared memory: unordered compaction (the sort key carries the index, so the list order
// does not matter), rank sort by (probability descending, index ascending), then one thread
// replays the reference's cumulative sum (sampler.cpp:146-156, or the top-k sum of
// sampler.cpp:105-108) and keeps every partial sum; the second loop of the reference
// (sampler.cpp:162-169) adds the same numbers in the same order, so its cdf values are those
// partial sums and the draw is a parallel lookup. Returns false, with nothing decided, when
// the survivors do not fit or do not suffice (the caller then takes the general path).
// `all_listed`: the list holds every entry that passes the crop and the threshold keeps all.
// ---------------------------------------------------------------------------------------
template <typename S>
__device__ bool small_tail(
    S& sm, const Entry* listA, int n_a, uint32_t key_lo, float sum, float cutoff, float topp,
    int topk, bool use_topk, bool all_listed, float coin, int* token) {
  const int tid = threadIdx.x, lane = tid & 31;
  __syncthreads();  // earlier users of the union are done
  if (tid == 0) {
    sm.u.small.cnt = 0;
    sm.u.small.first_above = 0x7fffffff;
    sm.u.small.last = -1;
    sm.u.small.cum = 0.0f;
  }
  __syncthreads();
  for (int i0 = 0; i0 < n_a; i0 += kThreads) {
    const int i = i0 + tid;
    bool keep = false;
    unsigned long long ck = 0ull;
    if (i < n_a) {
      const Entry en = listA[i];
      if (en.key >= key_lo) {
        const float p = __fdiv_rn(bits_f32(en.key), sum);
        keep = use_topk || p >= cutoff;
        ck = ((unsigned long long)f32_bits(p) << 32) | (uint32_t)(0x7FFFFFFF - en.idx);
      }
    }
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (bal != 0u) {
      int base = 0;
      if (lane == 0) base = atomicAdd(&sm.u.small.cnt, __popc(bal));
      base = __shfl_sync(0xffffffffu, base, 0);
      const int slot = base + __popc(bal & ((1u << lane) - 1u));
      if (keep && slot < kRankSortMax) sm.u.small.ck[slot] = ck;
    }
  }
  __syncthreads();
  const int n_b = sm.u.small.cnt;
  if (n_b <= 0 || n_b > kRankSortMax) return false;
  if (use_topk && n_b < topk && !all_listed) return false;
  if (tid < n_b) {
    const unsigned long long mine = sm.u.small.ck[tid];
    int rank = 0;
#pragma unroll 8
    for (int j = 0; j < n_b; ++j) rank += sm.u.small.ck[j] > mine ? 1 : 0;
    sm.u.small.p[rank] = bits_f32((uint32_t)(mine >> 32));
    sm.u.small.idx[rank] = (int)(0x7FFFFFFFu - (uint32_t)(mine & 0xFFFFFFFFull));
  }
  __syncthreads();
  // the terms beyond the ones that count read as zero (adding zero changes no partial sum)
  const int lim = use_topk ? (topk < n_b ? topk : n_b) : n_b;
  if (tid < 8) sm.u.small.p[lim + tid] = 0.0f;
  __syncthreads();
  if (tid == 0) {
    const float4* p4 = reinterpret_cast<const float4*>(sm.u.small.p);
    float4* pre4 = reinterpret_cast<float4*>(sm.u.small.prefix);
    float acc = 0.0f;
    int last = -1;
    float4 q = p4[0];
    for (int i = 0; i < lim; i += 4) {
      const float4 nq = p4[(i >> 2) + 1];  // next group, ahead of the additions
      const float a1 = __fadd_rn(acc, q.x);
      const float a2 = __fadd_rn(a1, q.y);
      const float a3 = __fadd_rn(a2, q.z);
      const float a4 = __fadd_rn(a3, q.w);
      pre4[i >> 2] = make_float4(a1, a2, a3, a4);
      if (!use_topk && a4 > topp) {  // the partial sums only grow: the first one above topp
        int k = 3;
        float hv = a4;
        if (a3 > topp) { k = 2; hv = a3; }
        if (a2 > topp) { k = 1; hv = a2; }
        if (a1 > topp) { k = 0; hv = a1; }
        last = i + k;
        acc = hv;
        break;
      }
      acc = a4;
      q = nq;
    }
    // top-k keeps its k entries; top-p keeps everything when the sum never exceeds topp
    // (the "in case of rounding errors" branch, sampler.cpp:152), which is only known to be
    // everything when all candidates were listed
    if (use_topk || (last < 0 && all_listed)) last = lim - 1;
    sm.u.small.last = last;
    sm.u.small.cum = acc;
  }
  __syncthreads();
  const int last = sm.u.small.last;
  if (last < 0) return false;
  const float r = __fmul_rn(coin, sm.u.small.cum);  // sampler.cpp:162
  {
    const bool above = tid <= last && sm.u.small.prefix[tid] > r;
    const unsigned bal = __ballot_sync(0xffffffffu, above);
    if (bal != 0u && lane == 0) atomicMin(&sm.u.small.first_above, (tid & ~31) + __ffs(bal) - 1);
  }
  __syncthreads();
  const int fa = sm.u.small.first_above;
  *token = sm.u.small.idx[fa <= last ? fa : last];
  __syncthreads();  // the union may be reused by the caller
  return true;
}

}  // namespace

// cudaFuncSetAttribute is needed once per function and device, not once per launch (the batch-1
// decode loop launches three kernels per token: the host side of a launch matters there).
struct OncePerDevice {
  std::atomic<unsigned long long> mask{0ull};
};
inline cudaError_t func_attr_once(OncePerDevice& once, const void* func, cudaFuncAttribute attr, int value) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (bit != 0ull && (once.mask.load(std::memory_order_acquire) & bit) != 0ull) return cudaSuccess;
  e = cudaFuncSetAttribute(func, attr, value);
  if (e == cudaSuccess && bit != 0ull) once.mask.fetch_or(bit, std::memory_order_release);
  return e;
}

// Launch attribute of a kernel that may become resident while its predecessor in the stream
// still runs; such a kernel calls grid_dependency_wait() before it touches anything the
// predecessor writes.
inline void programmatic_launch(cudaLaunchAttribute* attr) {
  attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr->val.programmaticStreamSerializationAllowed = 1;
}

}  // namespace etb200
