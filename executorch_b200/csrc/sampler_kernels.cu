// Token-sampling kernels for sm_100a: greedy argmax, multinomial and top-p (nucleus)
// sampling of rows x vocab logits, reproducing ExecuTorch's CPU sampler
// (extension/llm/sampler/sampler.cpp) bit for bit on the fp32 upcast of the logits.
//
// Work decomposition: one thread block per row (blocks stride over the rows of a batch).
// Logits are read in place (bf16 / fp16 / fp32, 128-bit loads when the row is 16-byte
// aligned) and never written. A sampled row makes these passes:
//
//   1. max of the temperature-scaled logits                      (HBM read of the row)
//   2. e_i = expf(x_i - max), exact sequential-order float sum S (row re-read, L2 resident);
//      top-p also appends (e_i, i) of every possible nucleus member to a per-block list.
//      For bf16 logits e_i comes from a per-row table in shared memory indexed by the
//      logit's bit pattern (a bf16 row has few distinct values), so expf runs once per
//      table entry instead of once per logit.
//   3a. multinomial: exact running cdf of e_i / S in index order until it exceeds the coin
//   3b. top-p: pick a value threshold from a histogram of the list, compact the survivors
//       with p_i = e_i / S >= cutoff, LSD-radix sort them (probability descending, stable =
//       index ascending), replay the reference's cumulative sums exactly, draw.
//
// The candidate lists of 3b live in global scratch memory owned by the caller of the launch
// functions (two buffers of vocab entries per resident block).
#include "sampler_device.cuh"

namespace etb200 {

namespace {

// Greedy choice for one row inside the sampling kernel (extended entry point): strict '>' in
// index order on the values the sampler sees, as sample_argmax (sampler.cpp:44-56) -- the
// lowest index among equal maxima, a NaN never replaces the running maximum, a NaN in
// element 0 is never replaced. Block-uniform result.
template <typename T, typename S>
__device__ int block_argmax(S& sm, const RowMath<T, S>& rm, int vocab) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float best = -INFINITY;
  int besti = 0x7fffffff;
  for (int i = tid; i < vocab; i += kThreads) {
    const float x = rm.xform(to_f32(rm.row[i]));
    if (x > best) {
      best = x;
      besti = i;
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, d);
    const int oi = __shfl_xor_sync(0xffffffffu, besti, d);
    if (ov > best || (ov == best && oi < besti)) {
      best = ov;
      besti = oi;
    }
  }
  __syncthreads();
  if (lane == 0) {
    sm.redf[warp] = best;
    sm.redi[warp] = besti;
  }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kWarps; ++w) {
      if (sm.redf[w] > best || (sm.redf[w] == best && sm.redi[w] < besti)) {
        best = sm.redf[w];
        besti = sm.redi[w];
      }
    }
    const float first = rm.xform(to_f32(rm.row[0]));
    sm.misc_i[0] = (first != first || besti == 0x7fffffff) ? 0 : besti;
  }
  __syncthreads();
  const int token = sm.misc_i[0];
  __syncthreads();
  return token;
}

#include "value_class_tail.cuh"

// ---------------------------------------------------------------------------------------
// The sampling kernel (temperature != 0): multinomial when topp is outside (0, 1), top-p
// otherwise. Follows Sampler::sample<float> (sampler.cpp:222-251).
// ---------------------------------------------------------------------------------------
template <typename T, bool kLut, bool kExt = false>
__global__ void __launch_bounds__(kThreads, 2) sample_rows_kernel(
    const T* __restrict__ logits, int64_t rows, int vocab, int64_t row_stride, float inv_t0,
    float topp0, int topk0, unsigned long long* __restrict__ rng_states,
    int64_t* __restrict__ out_ids, PeerOut peers, Entry* scratch, ExpTable table,
    int* __restrict__ status, const int* __restrict__ row_list, const int* __restrict__ row_count,
    const RowHead* __restrict__ known, RowSettings ext) {
  using S = Shared<kLut, kExt>;
  // the block's shared state exceeds the 48 KB static limit: dynamic shared memory, sized
  // sizeof(S) by the launcher
  extern __shared__ __align__(16) unsigned char smem_raw[];
  S& sm = *reinterpret_cast<S*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < kExpTableSize) sm.exp_tab[tid] = table.t[tid];
  int rp = 0;  // which set of scan-round slots the next round uses (see seqsum_tile)
  // Guessed floor under the values that matter (nucleus members / the k largest). Pass 2 lists
  // only e >= guess; if that turns out to be too high for a row, the row is regathered with
  // its exact floor and the guess is lowered for the block's later rows.
  float guess = kGuessFloor;
  __syncthreads();
  Entry* listA = scratch + (size_t)blockIdx.x * 2 * (size_t)vocab;
  Entry* listB = listA + vocab;

  // with a row list (rows that the cluster kernel left undecided) only those rows are sampled;
  // that launch may have become resident before the kernel that writes the list has ended
  if (row_list != nullptr) {
    grid_dependency_wait();
  }
  const int64_t n_todo = row_list != nullptr ? (int64_t)__ldcg(row_count) : rows;
  // Rows that finish in the value-class tail are only recorded inside the row loop; the block runs
  // those tails in batches outside it. (A call inside the loop costs every row: the state that
  // lives across it no longer fits the registers.)
  // (The bookkeeping of this lives in shared memory: the row loop has no register to spare.)
  if (tid == 0) sm.vcc.n_pend = 0;
  __syncthreads();
  int64_t it = blockIdx.x;
  for (;;) {
  for (; it < n_todo && sm.vcc.n_pend < kVcPendCap; it += gridDim.x) {
    const int64_t r = row_list != nullptr ? (int64_t)__ldcg(row_list + it) : it;
    // the row's settings: the handle's, or -- extended entry point -- its own
    // (LLMSession's SamplingConfig{temperature, top_p, top_k, seed}, llm_session.h:29-34)
    float inv_t = inv_t0, topp = topp0;
    int topk = topk0;
    if constexpr (kExt) {
      if (ext.temperature != nullptr) {
        const float t = ext.temperature[r];
        inv_t = t > 0.0f ? 1.0f / t : 0.0f;  // as Sampler::set_temperature: negative counts as 0
      }
      if (ext.topp != nullptr) topp = ext.topp[r];
      if (ext.topk != nullptr) topk = ext.topk[r];
    }
    // mode selection of Sampler::sample (sampler.cpp:239-248): top-k wins over top-p
    const bool use_topk = topk > 0 && topk < vocab;
    const bool use_topp = !use_topk && !(topp <= 0.0f || topp >= 1.0f);
    const bool use_list = use_topk || use_topp;  // modes that collect candidates during pass 2
    RowMath<T, S> rm;
    rm.row = logits + r * row_stride;
    rm.vocab = vocab;
    rm.vec_ok = (reinterpret_cast<uintptr_t>(rm.row) & 15u) == 0;
    rm.inv_t = inv_t;
    rm.sum = 1.0f;
    rm.probs = false;
    if constexpr (kExt) {
      rm.scale = ext.scale;
      if (inv_t == 0.0f) {
        // a greedy row among sampled ones (sampler.cpp:226-228): no coin, the state stays
        const int token = block_argmax(sm, rm, vocab);
        store_token(out_ids, peers, r, token);
        __syncthreads();
        continue;
      }
    }

      // ---- pass 1: max of the scaled logits
    // (or what the fast path has already found out about the row: row_finish.cuh)
    RowHead head;
    head.state = kRowUnknown;
    if (known != nullptr) {
      // past the L1 cache: this block may have become resident while row_finish_kernel was still
      // reading and writing neighbouring entries on the same SM
      const float4 h4 = __ldcg(reinterpret_cast<const float4*>(known + r));
      head.mx = h4.x;
      head.raw_max = h4.y;
      head.sum = h4.z;
      head.state = __float_as_int(h4.w);
    }
    const bool have_sum = head.state != kRowUnknown;  // block-uniform
    {
      float raw_max = head.raw_max;
      if (have_sum) {
        rm.mx = head.mx;
        __syncthreads();
      } else {
        rm.mx = row_max_scaled<T>(sm, rm, rm.row, vocab, rm.vec_ok, inv_t, &raw_max);
      }
      if constexpr (sizeof(T) == 2) {
        if (tid == 0) {
          // a 16-bit top-p row with finite logits can finish in the value-class tail
          const bool topp_row = !(topk > 0 && topk < vocab) && !(topp <= 0.0f || topp >= 1.0f);
          sm.vcc.raw_max = raw_max;
          sm.vcc.class_ok = (topp_row && fabsf(raw_max) < INFINITY && fabsf(rm.mx) < INFINITY &&
                             vocab <= kVcSelTiles * kVcSelTile) ? 1 : 0;
        }
      }
    }

    // the coin is drawn once per sampled row (sampler.cpp:237)
    if (tid == 0) {
      unsigned long long st_next = rng_states[r];
      sm.misc_f[0] = next_coin(&st_next);
      rng_states[r] = st_next;
    }
    if constexpr (kLut) {
      // the previous row's readers are behind the barriers above. Not needed by a row whose sum is
      // known and whose tail reads no terms (multinomial fills the table with probabilities).
      if (!have_sum || (use_list && head.state != kRowLong)) rm.build_lut(sm);
    }

    // ---- pass 2: e_i = expf(x_i - max) and their float sum in index order
    // (sampler.cpp:198-203). Top-p also lists every entry that can pass the cutoff crop of
    // sampler.cpp:136-143: p_i >= cutoff needs e_i >= cutoff * S and S >= 1 (the maximum
    // contributes exactly 1), so e_i >= cutoff * (1 - 1e-6) is necessary.
    const float cutoff = __fdiv_rn(__fsub_rn(1.0f, topp), (float)(vocab - 1));
    // Top-k has no crop: its exact floor is "e > 0". Both modes list only e >= max(exact
    // floor, guess) here and verify afterwards that this was enough.
    const float exact_floor0 = use_topp ? cutoff * 0.999999f : 1.4e-45f;
    const float e_floor = use_list ? fmaxf(exact_floor0, guess) : 0.0f;
    // A 16-bit top-p row whose list outgrows kVcListCap has a long nucleus: listing stops there
    // and the row is finished from its value classes instead (value_class_tail.cuh).
    bool listing = use_list;  // block-uniform
    float s = 0.0f;
    int n_a = 0;
    if (!have_sum) {
    {
      // head: the first kHead terms are added by one thread (a sum changes binade every few
      // additions at its start); their candidates are listed by all threads meanwhile
      __syncthreads();  // the table is complete
      const int cnt = vocab < kHead ? vocab : kHead;
      float e_mine = 0.0f;
      if (tid < kHead) {
        e_mine = rm.at(tid, sm);
        sm.head[tid] = e_mine;
      }
      const bool cand = use_list && tid < cnt && e_mine >= e_floor;
      const unsigned cb = __ballot_sync(0xffffffffu, cand);
      if (lane == 0) sm.wcnt[0][warp] = __popc(cb);
      __syncthreads();
      if (tid == 0) {
        float acc = 0.0f;
        const float4* h4 = reinterpret_cast<const float4*>(sm.head);
        for (int i = 0; i < cnt; i += 4) {
          const float4 q = h4[i >> 2];  // zero beyond the row
          acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, q.x), q.y), q.z), q.w);
        }
        sm.s_bcast = acc;
      }
      int pre = 0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const int c = sm.wcnt[0][w];
        if (w < warp) pre += c;
        n_a += c;
      }
      if (cand) {
        Entry en;
        en.key = f32_bits(e_mine);
        en.idx = tid;
        listA[pre + __popc(cb & ((1u << lane) - 1u))] = en;
      }
      __syncthreads();
      s = sm.s_bcast;
    }
    int buf = 0;
    constexpr bool kPrefetch = sizeof(T) == 2;  // 8 registers; fp32 chunks would need 16
    typename RowMath<T, S>::Raw raw_next;
    if (kPrefetch && kHead < vocab && rm.full(kHead + tid * kChunk)) rm.load_raw(kHead + tid * kChunk, &raw_next);
    for (int base = kHead; base < vocab; base += kTile) {
      const int i0 = base + tid * kChunk;
      float e[kChunk];
      if (kPrefetch) {
        if (rm.full(i0)) {
          const typename RowMath<T, S>::Raw raw = raw_next;
          const int inext = i0 + kTile;
          if (inext < vocab && rm.full(inext)) rm.load_raw(inext, &raw_next);
          rm.eval_raw(raw, sm, e);
        } else {
#pragma unroll
          for (int j = 0; j < kChunk; ++j) e[j] = rm.at(i0 + j, sm);
        }
      } else {
        rm.chunk(i0, sm, e);
      }
      // p_i >= cutoff needs e_i >= cutoff * S, and S is at least the running sum so far
      const float floor_now = use_topp ? fmaxf(e_floor, cutoff * s * 0.999999f) : e_floor;
      (void)exact_floor0;
      int cnt = 0, inc = 0;
      unsigned cmask = 0;  // bit j: e[j] is a candidate
      if (listing) {
        // entries beyond the row are 0 and the floor is > 0, so they never count.
        // e >= floor is e > f for the float f just below the floor; with B = 1 / ulp(f) the
        // fused e * B - f * B is >= 1 in the first case and <= 0 otherwise, so its saturation
        // is the indicator, and the indicators weighted by 2^j add up to the mask exactly:
        // float multiply-adds only, none of the scarce compare/logic instructions.
        const uint32_t fbits = f32_bits(floor_now) - 1u;  // floor_now >= 2^-100
        const float big = bits_f32((277u - (fbits >> 23)) << 23);
        const float neg_c = -__fmul_rn(bits_f32(fbits), big);
        float m4[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // interleaved: short dependency chains
#pragma unroll
        for (int j = 0; j < kChunk; ++j) {
          const float ind = __saturatef(__fmaf_rn(e[j], big, neg_c));
          m4[j & 3] = __fmaf_rn(ind, (float)(1u << j), m4[j & 3]);
        }
        cmask = (unsigned)((m4[0] + m4[1]) + (m4[2] + m4[3]));
        cnt = __popc(cmask);
        inc = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int o = __shfl_up_sync(0xffffffffu, inc, d);
          if (lane >= d) inc += o;
        }
        if (lane == 31) sm.wcnt[buf][warp] = inc;  // published by the barriers of seqsum_tile
      }
      int hp;
      float hs;
      const bool first_tile = base == kHead;  // block-uniform
      if (first_tile) {
        // The running sum leaves its binade every few hundred terms here, and every such
        // round would occupy the whole block: stage the tile's terms in shared memory and
        // let one warp sum them, 512 at a time, while the others list their candidates.
        stage_first_tile(sm, e);  // its barrier also publishes the candidate counts
      } else {
        seqsum_tile<false>(sm, e, s, rp, 0.0f, base, vocab, &hp, &hs);
      }
      if (listing) {
        // candidates of the warps in front of this one, and of the whole tile
        const int wc = lane < kWarps ? sm.wcnt[buf][lane] : 0;
        const int pre = __reduce_add_sync(0xffffffffu, lane < warp ? wc : 0);
        const int tot = __reduce_add_sync(0xffffffffu, wc);
        int off = n_a + pre + inc - cnt;
        // Candidates are rare (well under 1 % of the logits): visit only the groups of four
        // positions in which some lane of the warp has one.
        const unsigned any = __reduce_or_sync(0xffffffffu, cmask);
#pragma unroll
        for (int g = 0; g < kChunk; g += 4) {
          if (any & (0xFu << g)) {  // warp-uniform
#pragma unroll
            for (int j = g; j < g + 4; ++j) {
              if (cmask & (1u << j)) {
                Entry en;
                en.key = f32_bits(e[j]);
                en.idx = i0 + j;
                listA[off++] = en;
              }
            }
          }
        }
        n_a += tot;
        buf ^= 1;
        if constexpr (sizeof(T) == 2) {
          // n_a is the same in every thread; the flag was published by the barriers since pass 1
          // (sorting is the faster finish up to about kVcListCap candidates; candidates are
          // spread over the row, so a dense start tells early that there will be far more)
          const long long seen = (long long)base + kTile;
          if (n_a > kVcListProbe && (long long)n_a * vocab > (long long)kVcListCap * seen &&
              sm.vcc.class_ok != 0) {
            listing = false;
          }
        }
      }
      if (first_tile) sum_staged_tile<false>(sm, s, 0.0f, vocab, &hp, &hs);
    }
    }  // !have_sum
    const float sum = have_sum ? head.sum : s;
    __syncthreads();
    const float coin = sm.misc_f[0];
    int token;
    bool deferred = false;  // the row finishes in the value-class tail, after the row loop

    if (!use_list) {
      // ---- pass 3a: sample_mult (sampler.cpp:58-70): running float cdf of p_i = e_i / S
      token = vocab - 1;
      rm.sum = sum;
      rm.probs = true;
      if constexpr (kLut) {
        rm.build_lut(sm);  // the table now holds probabilities
      }
      float cdf = 0.0f;
      int hp;
      float hs;
      __syncthreads();
      const int cnt = vocab < kHead ? vocab : kHead;
      if (tid < kHead) sm.head[tid] = rm.at(tid, sm);
      bool hit = head_sum<true>(sm, cnt, cdf, coin, 0, &hp, &hs);
      for (int base = kHead; base < vocab && !hit; base += kTile) {
        float p[kChunk];
        rm.chunk(base + tid * kChunk, sm, p);
        if (base == kHead) {
          stage_first_tile(sm, p);
          hit = sum_staged_tile<true>(sm, cdf, coin, vocab, &hp, &hs);
        } else {
          hit = seqsum_tile<true>(sm, p, cdf, rp, coin, base, vocab, &hp, &hs);
        }
      }
      if (hit) token = hp;
    } else {
      // ---- pass 3b: sample_topp (sampler.cpp:122-171) or sample_topk (sampler.cpp:72-120)
      __threadfence_block();
      __syncthreads();
      // List A holds every entry with e >= max(exact floor, guess) ("complete" when the guess
      // was not above the exact floor). Each round: pick a value threshold from the bins,
      // compact, sort, and replay the reference's cumulative sums; a round that cannot
      // succeed first completes the list (regather with the exact floor, now that S is known)
      // and then widens the threshold to everything listed.
      const float exact_floor = use_topp ? cutoff * sum * 0.999999f : 1.4e-45f;
      bool complete = !have_sum && e_floor <= exact_floor;
      bool take_all = false;
      int n_b = 0, last_idx = 0;
      float cum = 0.0f;
      bool have = false, token_ready = false;
      token = 0;
      if constexpr (sizeof(T) == 2) {
        if (!listing) {
          // the list was abandoned: a long nucleus, finished without list or sort
          deferred = true;
          have = true;  // skips the rounds below
        }
      }
      if (have_sum && !have) {
        if constexpr (sizeof(T) == 2) {
          if (head.state == kRowLong && sm.vcc.class_ok != 0) {
            deferred = true;
            have = true;
          }
        }
        if (!have) {
          if constexpr (kLut) {
            if (head.state == kRowLong) {
              rm.build_lut(sm);
              __syncthreads();
            }
          }
          n_a = gather_candidates(rm, sm, listA, exact_floor);
          complete = true;
        }
      }
      for (int round = 0; round < 4 && !have; ++round) {
        int bin_lo = 0, kept = n_a;
        bool enough = true;
        if (!take_all) enough = pick_value_threshold(sm, listA, n_a, sum, topp, topk, use_topk, &bin_lo, &kept);
        if constexpr (sizeof(T) == 2) {
          if (!enough && !complete && sm.vcc.class_ok != 0) {
            // Every token that is not listed has e < e_floor, so the nucleus needs at least
            // (missing mass) / e_floor more of them: a long nucleus takes the class tail at once.
            const float missing = topp * sum - sm.misc_f[1];
            if ((float)n_a + missing / e_floor > (float)kVcMinNucleus) {
              deferred = true;
              break;
            }
          }
        }
        if (!enough && !complete) {
          guess = fmaxf(guess * 0.0625f, 1e-30f);  // later rows of this block start lower
          n_a = gather_candidates(rm, sm, listA, exact_floor);
          complete = true;
          continue;
        }
        if (!take_all && kept <= kRankSortMax) {
          // short nucleus (the usual case): finish in shared memory
          const uint32_t klo = bin_lo > 0 ? (uint32_t)(bin_lo + kBinBase) << kBinShift : 0u;
          int tk;
          if (small_tail(sm, listA, n_a, klo, sum, cutoff, topp, topk, use_topk, bin_lo == 0 && complete,
                         coin, &tk)) {
            token_ready = true;
            token = tk;
            break;
          }
        }
        // The radix sort ping-pongs into the free space behind list A. If the survivors may
        // not fit there, list A itself is the spare buffer, which is only allowed when list A
        // will not be needed again: make this the final round by taking everything listed
        // from a complete list.
        bool spare_is_list_a = false;
        if (n_a + kept > vocab) {
          if (!complete) {
            n_a = gather_candidates(rm, sm, listA, exact_floor);
            complete = true;
            continue;
          }
          if (!use_topk) bin_lo = 0;  // top-k's count threshold is exact: no later round either way
          spare_is_list_a = true;
        }
        const uint32_t key_lo = bin_lo > 0 ? (uint32_t)(bin_lo + kBinBase) << kBinShift : 0u;
        n_b = compact_candidates(sm, listA, n_a, listB, key_lo, sum, cutoff, use_topk);
        sort_candidates(sm, listB, n_b, spare_is_list_a ? listA : listA + n_a);
        int pos;
        float hs, total;
        if (use_topk) {
          // the k most probable entries (fewer if fewer have e > 0); their float sum in
          // sorted order is topk_sum (sampler.cpp:105-108)
          if (n_b >= topk || complete) {
            const int kk = topk < n_b ? topk : n_b;
            list_search(sm, listB, n_b, kk, INFINITY, rp, &pos, &hs, &total);
            have = true;
            last_idx = kk - 1;
            cum = total;
          } else {
            n_a = gather_candidates(rm, sm, listA, exact_floor);
            complete = true;
          }
        } else if (list_search(sm, listB, n_b, n_b, topp, rp, &pos, &hs, &total)) {
          have = true;
          last_idx = pos;
          cum = hs;
        } else if (bin_lo == 0 && complete) {
          // every candidate is in and the sum never exceeded topp: keep everything
          // (the "in case of rounding errors" branch, sampler.cpp:152)
          have = true;
          last_idx = n_b - 1;
          cum = total;
        } else if (!complete) {
          n_a = gather_candidates(rm, sm, listA, exact_floor);
          complete = true;
        } else {
          take_all = true;  // the value threshold was too optimistic: take all candidates
        }
      }
      if (deferred) {
        if (tid == 0) {
          VcControl::Pending pd;
          pd.row = (long long)r;
          pd.inv_t = inv_t;
          pd.mx = rm.mx;
          pd.sum = sum;
          pd.cutoff = cutoff;
          pd.topp = topp;
          pd.coin = coin;
          pd.raw_max = sm.vcc.raw_max;
          sm.vcc.pend[sm.vcc.n_pend] = pd;
          sm.vcc.n_pend += 1;  // read again behind the barrier that ends the row
        }
      } else if (token_ready) {
        // decided by small_tail
      } else if (n_b <= 0 || !have) {
        token = 0;  // no candidate at all (NaN rows): undefined in the reference
      } else {
        const float rr = __fmul_rn(coin, cum);  // sampler.cpp:162
        int pos;
        float hs, total;
        int j = last_idx;
        if (list_search(sm, listB, n_b, last_idx + 1, rr, rp, &pos, &hs, &total)) j = pos;
        token = listB[j].idx;
      }
    }
    if (!deferred) store_token(out_ids, peers, r, token);
    __syncthreads();
  }
  if constexpr (sizeof(T) == 2) {
    // ---- the deferred value-class tails
    const int n_pend = sm.vcc.n_pend;
    for (int k = 0; k < n_pend; ++k) {
      __syncthreads();
      const VcControl::Pending pd = sm.vcc.pend[k];
      RowMath<T, S> rm;
      rm.row = logits + pd.row * row_stride;
      rm.vocab = vocab;
      rm.vec_ok = (reinterpret_cast<uintptr_t>(rm.row) & 15u) == 0;
      rm.inv_t = pd.inv_t;
      rm.mx = pd.mx;
      rm.sum = 1.0f;
      rm.probs = false;
      if constexpr (kExt) rm.scale = ext.scale;
      int token = value_class_tail(sm, rm, pd.sum, pd.cutoff, pd.topp, pd.coin, pd.raw_max);
      if (token < 0) {
        // -1: no candidate at all, undefined in the reference (token 0 like the sorted path);
        // -2: counts that do not add up, which the host can read from the status word
        if (token == -2 && tid == 0 && status != nullptr) atomicMax(status, kStatusTailInconsistent);
        token = 0;
      }
      store_token(out_ids, peers, pd.row, token);
    }
    __syncthreads();
  }
  if (tid == 0) sm.vcc.n_pend = 0;
  __syncthreads();
  if (it >= n_todo) break;
  }
  peer_arrival_barrier(peers, status);
}

// ---------------------------------------------------------------------------------------
// Greedy kernel (temperature == 0): sample_argmax (sampler.cpp:44-56). Strict '>' in
// index order: the lowest index among equal maxima wins, -0 equals +0, a NaN never
// replaces the running maximum, and a NaN in element 0 is never replaced.
// ---------------------------------------------------------------------------------------
//
// Bound by HBM: every logit is read once. A cluster of blocks shares a row, so that small batches
// fill the chip, and the partial maxima meet in the first block's shared memory. A thread keeps eight 128-bit loads in flight, contiguous across the
// warp. A vector costs its packed maximum, a comparison and two selects; which of its elements it
// was is looked up for the winning vector alone. Vectors start at the 16-byte boundary at or in
// front of the row's first logit, whatever the row's alignment. Measured against one block per row with a
// comparison per logit and scalar loads for unaligned rows: one row of 128256 bf16 8.2 -> 3.7 us,
// 64 x 50257 fp16 10.3 -> 5.2 us, 256 x 128256 bf16 14.6 -> 13.1 us (5.0 TB/s).
constexpr int kArgVecs = 8;
constexpr int kArgMaxCluster = 16;

template <typename T>
__device__ __forceinline__ float arg_value(T x) {
  if constexpr (std::is_same<T, unsigned short>::value) return (float)x;  // sample<uint16_t> compares the raw integers
  else return to_f32(x);
}

// Largest value of a vector; NaNs count only if there is nothing else.
template <typename T>
__device__ __forceinline__ float vec_max(const uint4& raw) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
    const __nv_bfloat162 m = __hmax2(__hmax2(p[0], p[1]), __hmax2(p[2], p[3]));
    return fmaxf(__bfloat162float(m.x), __bfloat162float(m.y));
  } else if constexpr (std::is_same<T, __half>::value) {
    const __half2* p = reinterpret_cast<const __half2*>(&raw);
    const __half2 m = __hmax2(__hmax2(p[0], p[1]), __hmax2(p[2], p[3]));
    return fmaxf(__half2float(m.x), __half2float(m.y));
  } else if constexpr (std::is_same<T, float>::value) {
    return fmaxf(fmaxf(__uint_as_float(raw.x), __uint_as_float(raw.y)),
                 fmaxf(__uint_as_float(raw.z), __uint_as_float(raw.w)));
  } else {
    const unsigned m = __vmaxu2(__vmaxu2(raw.x, raw.y), __vmaxu2(raw.z, raw.w));
    return (float)max(m & 0xFFFFu, m >> 16);
  }
}

// The lanes' largest value and the lowest vector that holds it, in every lane.
__device__ __forceinline__ void arg_reduce(float* best, int* v) {
  const float m = warp_max_f32(*best);
  *v = __reduce_min_sync(0xffffffffu, *best == m ? *v : 0x7fffffff);
  *best = m;
}

template <typename T, int kArgThreads>
__global__ void __launch_bounds__(kArgThreads, 1024 / kArgThreads) argmax_rows_kernel(
    const T* __restrict__ logits, int64_t rows, int vocab, int64_t row_stride,
    int64_t* __restrict__ out_ids, PeerOut peers, int* __restrict__ status) {
  constexpr int kPerVec = 16 / sizeof(T);
  constexpr int kArgWarps = kArgThreads / 32;
  __shared__ float sv[kArgWarps], cv[kArgMaxCluster];
  __shared__ int si[kArgWarps], ci[kArgMaxCluster];
  __shared__ int answer;
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int csize = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  grid_launch_dependents();
  grid_dependency_wait();
  // (no row at all in a launch that only takes part in the arrival barrier)
  for (int64_t r = blockIdx.x / csize; r < rows; r += gridDim.x / csize) {
    const T* row = logits + r * row_stride;
    const int shift = (int)((reinterpret_cast<uintptr_t>(row) & 15u) / sizeof(T));
    const uint4* base4 = reinterpret_cast<const uint4*>(row - shift);
    // vectors [0, nvec) cover the row; [full0, full1) hold nothing but logits
    const int nvec = (int)(((int64_t)shift + vocab + kPerVec - 1) / kPerVec);
    const int full0 = shift > 0 ? 1 : 0, full1 = (int)(((int64_t)shift + vocab) / kPerVec);
    const int per = (nvec + csize - 1) / csize;
    const int beg = max(rank * per, full0), end = min((rank + 1) * per, full1);
    float best = -INFINITY;
    int bestv = 0x7fffffff;  // "nothing better than -inf seen"
    // A thread visits its vectors in increasing order, so strict '>' keeps the first of equal ones.
    for (int v0 = beg; v0 < end; v0 += kArgThreads * kArgVecs) {
      uint4 raw[kArgVecs];
#pragma unroll
      for (int q = 0; q < kArgVecs; ++q) {
        const int v = v0 + q * kArgThreads + tid;
        if (v < end) raw[q] = __ldg(base4 + v);
      }
#pragma unroll
      for (int q = 0; q < kArgVecs; ++q) {
        const int v = v0 + q * kArgThreads + tid;
        if (v < end) {
          const float x = vec_max<T>(raw[q]);
          if (x > best) {
            best = x;
            bestv = v;
          }
        }
      }
    }
    // the row's ragged ends, an element a thread
    if (rank == 0 && tid < 2 * kPerVec) {
      const int v = tid < kPerVec ? 0 : nvec - 1;
      const int i = v * kPerVec + (tid & (kPerVec - 1)) - shift;
      if ((v < full0 || v >= full1) && i >= 0 && i < vocab) {
        const float x = arg_value(row[i]);
        if (x > best || (x == best && x > -INFINITY && v < bestv)) {
          best = x;
          bestv = v;
        }
      }
    }
    arg_reduce(&best, &bestv);
    if (lane == 0) {
      sv[warp] = best;
      si[warp] = bestv;
    }
    __syncthreads();
    if (warp == 0) {
      best = lane < kArgWarps ? sv[lane] : -INFINITY;
      bestv = lane < kArgWarps ? si[lane] : 0x7fffffff;
      arg_reduce(&best, &bestv);
    }
    if (csize > 1) {
      cluster_arrive();  // the first block runs before its shared memory is written to
      cluster_wait();
      if (tid == 0) {
        *cluster.map_shared_rank(&cv[rank], 0) = best;
        *cluster.map_shared_rank(&ci[rank], 0) = bestv;
      }
      cluster_arrive();
      cluster_wait();
      if (warp == 0 && rank == 0) {
        best = lane < csize ? cv[lane] : -INFINITY;
        bestv = lane < csize ? ci[lane] : 0x7fffffff;
        arg_reduce(&best, &bestv);
      }
    }
    if (rank == 0) {
      if (warp == 0) {
        const float first = arg_value(row[0]);
        int i = 0x7fffffff;
        if (bestv != 0x7fffffff && lane < kPerVec) {
          const int j = bestv * kPerVec + lane - shift;
          if (j >= 0 && j < vocab && arg_value(row[j]) == best) i = j;
        }
        i = __reduce_min_sync(0xffffffffu, i);
        // Sequential semantics at the edges: the scan starts from element 0, so if nothing compares
        // greater than it (all -inf, or element 0 is NaN) the answer is 0.
        if (lane == 0) answer = (first != first || i == 0x7fffffff) ? 0 : i;
      }
      __syncthreads();
      store_token(out_ids, peers, r, answer);
      __syncthreads();
    }
  }
  peer_arrival_barrier(peers, status);
}

__global__ void expf_selftest_kernel(const float* __restrict__ x, float* __restrict__ y, int64_t n,
                                     ExpTable table) {
  __shared__ uint64_t tab[kExpTableSize];
  if (threadIdx.x < kExpTableSize) tab[threadIdx.x] = table.t[threadIdx.x];
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    y[i] = expf_ref(x[i], tab);
  }
}

}  // namespace

cudaError_t launch_expf_selftest(const float* x, float* y, int64_t n, const ExpTable& table,
                                 cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  expf_selftest_kernel<<<(int)blocks, 256, 0, stream>>>(x, y, n, table);
  return cudaGetLastError();
}

size_t sampler_scratch_bytes(int vocab, int blocks) {
  return (size_t)blocks * 2 * (size_t)vocab * sizeof(Entry);
}

int sampler_threads() { return kThreads; }

// Opts the kernel in to its dynamic shared-memory size (once per device would do; the call is
// cheap and idempotent).
template <typename T, bool kLut, bool kExt = false>
static cudaError_t prepare_sample_kernel() {
  static OncePerDevice once;
  return func_attr_once(once, reinterpret_cast<const void*>(sample_rows_kernel<T, kLut, kExt>),
                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Shared<kLut, kExt>));
}

template <typename T, bool kLut, bool kExt>
static cudaError_t launch_sample_t(
    const void* logits, int64_t rows, int vocab, int64_t row_stride, float inv_t, float topp,
    int topk, unsigned long long* rng_states, int64_t* out_ids, const PeerOut& peers, void* scratch,
    int blocks, const ExpTable& table, int* status, const RowSettings& settings, const RowPass& pass,
    cudaStream_t stream) {
  const cudaError_t attr = prepare_sample_kernel<T, kLut, kExt>();
  if (attr != cudaSuccess) return attr;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = sizeof(Shared<kLut, kExt>);
  cfg.stream = stream;
  cudaLaunchAttribute la[1];
  programmatic_launch(&la[0]);
  cfg.attrs = la;
  // the pass over the rows that the fast kernels hand on is resident early and waits for its
  // predecessor before it reads the list
  cfg.numAttrs = pass.row_list != nullptr ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, sample_rows_kernel<T, kLut, kExt>, static_cast<const T*>(logits), rows, vocab,
                            row_stride, inv_t, topp, topk, rng_states, out_ids, peers, static_cast<Entry*>(scratch),
                            table, status, pass.row_list, pass.row_count, pass.heads, settings);
}

template <bool kExt>
static cudaError_t launch_sample_dtype(
    int dtype, const void* logits, int64_t rows, int vocab, int64_t row_stride, float inv_t, float topp,
    int topk, unsigned long long* rng_states, int64_t* out_ids, const PeerOut& peers, void* scratch,
    int blocks, const ExpTable& table, int* status, const RowSettings& settings, const RowPass& pass,
    cudaStream_t stream) {
  switch (dtype) {
    case kDtypeFloat:
      return launch_sample_t<float, false, kExt>(logits, rows, vocab, row_stride, inv_t, topp, topk, rng_states,
                                                 out_ids, peers, scratch, blocks, table, status, settings, pass, stream);
    case kDtypeHalf:
      return launch_sample_t<__half, false, kExt>(logits, rows, vocab, row_stride, inv_t, topp, topk, rng_states,
                                                  out_ids, peers, scratch, blocks, table, status, settings, pass, stream);
    case kDtypeBFloat16:
      return launch_sample_t<__nv_bfloat16, true, kExt>(logits, rows, vocab, row_stride, inv_t, topp, topk, rng_states,
                                                        out_ids, peers, scratch, blocks, table, status, settings, pass,
                                                        stream);
    default:
      return cudaErrorInvalidValue;
  }
}

cudaError_t launch_sample_rows(
    int dtype, const void* logits, int64_t rows, int vocab, int64_t row_stride, float inv_t,
    float topp, int topk, unsigned long long* rng_states, int64_t* out_ids, const PeerOut& peers,
    void* scratch, int blocks, const ExpTable& table, int* status, cudaStream_t stream, const RowPass& pass) {
  return launch_sample_dtype<false>(dtype, logits, rows, vocab, row_stride, inv_t, topp, topk, rng_states, out_ids,
                                    peers, scratch, blocks, table, status, RowSettings{nullptr, nullptr, nullptr, 1.0f},
                                    pass, stream);
}

namespace {

// One thread per edit: logits[row][id] = T(float(logits[row][id]) + bias), what a mask or bias
// logit processor does in place (logit_processor.h:34-40).
template <typename T>
__global__ void apply_row_edits_kernel(T* logits, int64_t rows, int vocab, int64_t row_stride, RowEdits ed,
                                       long long total) {
  const long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (j >= total) return;
  int64_t row;
  long long e;
  if (ed.offsets == nullptr) {
    row = j / ed.n_shared;
    e = j % ed.n_shared;
  } else {
    // the row that owns entry j: the last row whose first entry is not behind j
    int64_t lo = 0, hi = rows - 1;
    while (lo < hi) {
      const int64_t mid = (lo + hi + 1) / 2;
      if (ed.offsets[mid] <= j) lo = mid; else hi = mid - 1;
    }
    row = lo;
    e = j;
  }
  const int id = ed.ids[e];
  if (id < 0 || id >= vocab) return;  // out of range: no-op, as the reference's processors
  T* p = logits + row * row_stride + id;
  const float v = to_f32(*p) + ed.bias[e];
  if constexpr (std::is_same<T, float>::value) {
    *p = v;
  } else if constexpr (std::is_same<T, __half>::value) {
    *p = __float2half_rn(v);
  } else {
    *p = __float2bfloat16_rn(v);
  }
}

}  // namespace

cudaError_t launch_row_edits(int dtype, void* logits, int64_t rows, int vocab, int64_t row_stride,
                             const RowEdits& edits, cudaStream_t stream) {
  // how many edits there are is known on the host: shared lists directly, per-row lists by
  // their last offset, which the caller passes in n_shared as well
  const long long n = edits.ids == nullptr ? 0 : (edits.offsets == nullptr ? edits.n_shared * rows : edits.n_shared);
  if (n <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)((n + 255) / 256);
  switch (dtype) {
    case kDtypeFloat:
      apply_row_edits_kernel<float><<<grid, 256, 0, stream>>>(static_cast<float*>(logits), rows, vocab, row_stride, edits, n);
      break;
    case kDtypeHalf:
      apply_row_edits_kernel<__half><<<grid, 256, 0, stream>>>(static_cast<__half*>(logits), rows, vocab, row_stride, edits, n);
      break;
    case kDtypeBFloat16:
      apply_row_edits_kernel<__nv_bfloat16>
          <<<grid, 256, 0, stream>>>(static_cast<__nv_bfloat16*>(logits), rows, vocab, row_stride, edits, n);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_sample_rows_ext(
    int dtype, const void* logits, int64_t rows, int vocab, int64_t row_stride, float inv_t, float topp,
    int topk, const RowSettings& settings, unsigned long long* rng_states, int64_t* out_ids, void* scratch, int blocks,
    const ExpTable& table, int* status, cudaStream_t stream, const RowPass& pass) {
  return launch_sample_dtype<true>(dtype, logits, rows, vocab, row_stride, inv_t, topp, topk, rng_states, out_ids,
                                   PeerOut{}, scratch, blocks, table, status, settings, pass, stream);
}

template <typename T, int kArgThreads>
static cudaError_t launch_argmax_t(
    const void* logits, int64_t rows, int vocab, int64_t row_stride, int64_t* out_ids, const PeerOut& peers,
    int csize, int* status, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  if (csize > 8) {
    static OncePerDevice once;
    const cudaError_t e = func_attr_once(once, reinterpret_cast<const void*>(argmax_rows_kernel<T, kArgThreads>),
                                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  const int64_t clusters = rows < 1 ? 1 : (rows < (1 << 30) ? rows : (1 << 30));
  cfg.gridDim = dim3((unsigned)(clusters * csize), 1, 1);
  cfg.blockDim = dim3(kArgThreads, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  programmatic_launch(&attr[1]);
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, argmax_rows_kernel<T, kArgThreads>, static_cast<const T*>(logits), rows, vocab, row_stride, out_ids,
                            peers, status);
}

// Blocks per row: as many as keep two blocks per SM, and leave each thread four loads to have in
// flight; more of them wait for one another longer than they stream (256 x 128256 bf16: 14.3 us with
// two blocks per row, 18.6 with eight; one row: 6.6 us with one block, 3.7 with eight). A row per block takes
// 512 threads while all rows run at once (13.1 us against 14.8 with 256 threads); beyond that smaller
// blocks make a shorter last wave (400 x 151936 bf16: 22.7 us against 23.8).
template <typename T>
static cudaError_t launch_argmax_dtype(
    const void* logits, int64_t rows, int vocab, int64_t row_stride, int64_t* out_ids, const PeerOut& peers,
    int sm_count, int* status, cudaStream_t stream) {
  const int64_t vecs = ((int64_t)vocab * (int64_t)sizeof(T) + 15) / 16;
  int csize = 1;
  while (csize < kArgMaxCluster && rows * 2 * csize <= 2 * (int64_t)sm_count && 2 * csize * 4 * 256 <= vecs) csize *= 2;
  if (csize == 1 && rows <= 2 * (int64_t)sm_count)
    return launch_argmax_t<T, 512>(logits, rows, vocab, row_stride, out_ids, peers, csize, status, stream);
  return launch_argmax_t<T, 256>(logits, rows, vocab, row_stride, out_ids, peers, csize, status, stream);
}

cudaError_t launch_argmax_rows(
    int dtype, const void* logits, int64_t rows, int vocab, int64_t row_stride, int64_t* out_ids,
    const PeerOut& peers, int sm_count, int* status, cudaStream_t stream) {
  switch (dtype) {
    case kDtypeFloat:
      return launch_argmax_dtype<float>(logits, rows, vocab, row_stride, out_ids, peers, sm_count, status, stream);
    case kDtypeHalf:
      return launch_argmax_dtype<__half>(logits, rows, vocab, row_stride, out_ids, peers, sm_count, status, stream);
    case kDtypeBFloat16:
      return launch_argmax_dtype<__nv_bfloat16>(logits, rows, vocab, row_stride, out_ids, peers, sm_count, status, stream);
    case kDtypeUInt16:
      return launch_argmax_dtype<unsigned short>(logits, rows, vocab, row_stride, out_ids, peers, sm_count, status, stream);
    default:
      return cudaErrorInvalidValue;
  }
}

int sample_kernel_max_blocks_per_sm(int dtype) {
  int n = 0;
  cudaError_t e;
  switch (dtype) {
    case kDtypeFloat:
      e = prepare_sample_kernel<float, false>();
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sample_rows_kernel<float, false>, kThreads,
                                                          sizeof(Shared<false>));
      break;
    case kDtypeHalf:
      e = prepare_sample_kernel<__half, false>();
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sample_rows_kernel<__half, false>, kThreads,
                                                          sizeof(Shared<false>));
      break;
    default:
      e = prepare_sample_kernel<__nv_bfloat16, true>();
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sample_rows_kernel<__nv_bfloat16, true>,
                                                          kThreads, sizeof(Shared<true>));
      break;
  }
  if (e != cudaSuccess || n < 1) n = 1;
  return n;
}

}  // namespace etb200
