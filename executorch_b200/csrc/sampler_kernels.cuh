// Launch interface of the sampling kernels (sampler_kernels.cu). Host-only declarations;
// the C ABI in c_api.cu is the only caller.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "exact_math.cuh"

namespace etb200 {

// dtype codes = the reference's ScalarType numbering
// (runtime/core/portable_type/scalar_type.h:98-125)
constexpr int kDtypeHalf = 5;
constexpr int kDtypeFloat = 6;
constexpr int kDtypeBFloat16 = 15;
constexpr int kDtypeUInt16 = 27;

// Optional destinations of the sampled ids: up to kMaxPeers int64 buffers (this GPU's and its
// peers' -- pointers obtained from symmetric / peer-mapped memory), each written at
// [offset + row]. n == 0 means "write out_ids[row] only".
constexpr int kMaxPeers = 16;
struct PeerOut {
  int64_t* ptr[kMaxPeers];
  int n;
  long long offset;
  // Optional arrival barrier at the end of the launch (epoch != 0): arrive[p] is rank p's
  // array of kMaxPeers 64-bit arrival marks. When the last block of this launch is done it
  // writes `epoch` into arrive[p][rank] of every rank p and then waits, at most wait_ns, until
  // arrive[rank][q] >= epoch for every q: when the launch completes, this GPU's buffer holds
  // the ids of all ranks. blocks_done is a counter of this GPU that is zero between launches.
  unsigned long long* arrive[kMaxPeers];
  unsigned long long epoch;
  int rank;
  int* blocks_done;
  unsigned long long wait_ns;  // limit of that wait, in nanoseconds of the GPU's global timer
};

// Per-row settings of the extended entry point (device arrays of `rows` entries, or null for
// "the handle's value"), and the scalar that multiplies every logit (1 = none).
struct RowSettings {
  const float* temperature;
  const float* topp;
  const int* topk;
  float scale;
};

// Sparse in-place edits of the logits before sampling (mask / bias logit processors): entry j
// adds bias[j] to logit ids[j] of its row (-inf masks the token; ids outside [0, vocab) are
// ignored). Row r owns entries [offsets[r], offsets[r + 1]) and n_shared is the total number of
// entries; with offsets == null the n_shared entries apply to every row. All pointers are
// device pointers; ids == null means "no edits".
struct RowEdits {
  const long long* offsets;
  const int* ids;
  const float* bias;
  long long n_shared;
};

// Bytes of candidate-list scratch the sampling kernel needs when launched with `blocks`
// thread blocks on rows of `vocab` logits.
size_t sampler_scratch_bytes(int vocab, int blocks);

// Resident thread blocks per SM of the sampling kernel for a dtype (occupancy query).
int sample_kernel_max_blocks_per_sm(int dtype);

int sampler_threads();

// What the fast path (launch_fast_rows) knows about a row that it hands on.
struct alignas(16) RowHead {
  float mx;       // largest scaled logit, as the reference has it
  float raw_max;  // largest logit
  float sum;      // exact softmax sum, when known
  int state;      // kRow...
};
constexpr int kRowUnknown = 0;  // nothing is known
constexpr int kRowSum = 1;      // mx, raw_max and sum are exact
constexpr int kRowLong = 2;     // the same, and the nucleus is long

// A pass over some of a batch's rows: the *row_count rows named in row_list, with what is known
// about each row r in heads[r]. All device pointers; null row_list means every row.
struct RowPass {
  const int* row_list;
  const int* row_count;
  const RowHead* heads;
};

// temperature != 0: top-k (0 < topk < vocab), else multinomial (topp outside (0,1)) or top-p
// sampling of every row. rng_states[r] is advanced once per row; out_ids[r] receives the
// token. Top-k and top-p need `scratch` (sampler_scratch_bytes).
cudaError_t launch_sample_rows(
    int dtype, const void* logits, int64_t rows, int vocab, int64_t row_stride, float inv_t,
    float topp, int topk, unsigned long long* rng_states, int64_t* out_ids, const PeerOut& peers,
    void* scratch, int blocks, const ExpTable& table, int* status, cudaStream_t stream,
    const RowPass& pass = RowPass{nullptr, nullptr, nullptr});

// The edits, applied to the logits in place (one thread per edit).
cudaError_t launch_row_edits(int dtype, void* logits, int64_t rows, int vocab, int64_t row_stride,
                             const RowEdits& edits, cudaStream_t stream);

// launch_sample_rows with every row's own settings; a row whose temperature is 0 takes the argmax.
cudaError_t launch_sample_rows_ext(
    int dtype, const void* logits, int64_t rows, int vocab, int64_t row_stride, float inv_t, float topp,
    int topk, const RowSettings& settings, unsigned long long* rng_states, int64_t* out_ids, void* scratch, int blocks,
    const ExpTable& table, int* status, cudaStream_t stream, const RowPass& pass = RowPass{nullptr, nullptr, nullptr});

// The fast path (fast_path.cu): a sweep by one thread-block cluster per row and a finishing
// kernel. It samples every row that it can decide; the others -- RNG state and output untouched --
// are appended to retry_rows (count in *retry_count, which must be zero at launch), with
// what is known about them in heads, and the caller runs launch_sample_rows[_ext] over that list
// on the same stream. *retry_count_next is cleared for the call after this one. *launches is
// increased by the number of kernels launched.
bool fast_rows_supported(int dtype, int64_t rows, int vocab, float inv_t);
size_t fast_rows_scratch_bytes(int vocab, int64_t rows);
cudaError_t launch_fast_rows(
    int dtype, const void* logits, int64_t rows, int vocab, int64_t row_stride, float inv_t, float topp, int topk,
    const RowSettings& settings, unsigned long long* rng_states, int64_t* out_ids, const PeerOut& peers,
    const ExpTable& table, void* scratch, RowHead* heads, int* retry_rows, int* retry_count, int* retry_count_next,
    int sm_count, cudaStream_t stream, unsigned long long* launches);

// temperature == 0: greedy argmax of every row.
cudaError_t launch_argmax_rows(
    int dtype, const void* logits, int64_t rows, int vocab, int64_t row_stride, int64_t* out_ids,
    const PeerOut& peers, int sm_count, int* status, cudaStream_t stream);

// Value stored into `status` when the arrival barrier of PeerOut gave up waiting for a rank.
constexpr int kStatusPeerTimeout = 2;
constexpr int kStatusTailInconsistent = 3;  // the long-nucleus tail's final lookup found its counts inconsistent

// y[i] = expf_ref(x[i]) on the device, for x <= 0: lets a test compare the device
// exponential with the host libm.
cudaError_t launch_expf_selftest(const float* x, float* y, int64_t n, const ExpTable& table,
                                 cudaStream_t stream);

}  // namespace etb200
