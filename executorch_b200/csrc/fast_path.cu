// Host side of the fast sampling path: row_sweep.cuh, then row_finish.cuh.
#include "sampler_device.cuh"

namespace etb200 {

namespace {

namespace cg = cooperative_groups;

#include "row_sweep.cuh"
#include "row_finish.cuh"

// Rows per launch pair: bounds the scratch (at most 8 KB of unit records per row).
constexpr int64_t kFastGroupRows = 4096;

int units_of(int vocab) { return (vocab + 7 + kUnit - 1) / kUnit; }  // whatever the row's alignment

template <typename T, int kUnitsPerWarp>
cudaError_t launch_sweep_t(const SweepArgs& args, int csize, int sm_count, cudaStream_t stream) {
  static OncePerDevice once_smem, once_np;
  const void* fn = reinterpret_cast<const void*>(row_sweep_kernel<T, kUnitsPerWarp>);
  constexpr int kSmem = (int)SweepLayout<T, kUnitsPerWarp>::kBytes;
  cudaError_t e = func_attr_once(once_smem, fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  if (e == cudaSuccess && csize > 8) e = func_attr_once(once_np, fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kSwThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // as many clusters as fit on the device at once (queried once per cluster size); each of them
  // takes every n-th row
  static std::atomic<int> resident[kSwMaxCluster + 1];
  int n_cl = resident[csize].load(std::memory_order_relaxed);
  if (n_cl == 0) {
    cfg.gridDim = dim3((unsigned)(csize * sm_count), 1, 1);
    e = cudaOccupancyMaxActiveClusters(&n_cl, row_sweep_kernel<T, kUnitsPerWarp>, &cfg);
    if (e != cudaSuccess) return e;
    if (n_cl < 1) n_cl = 1;
    resident[csize].store(n_cl, std::memory_order_relaxed);
  }
  const int64_t n = args.rows < n_cl ? args.rows : n_cl;
  cfg.gridDim = dim3((unsigned)(n * csize), 1, 1);
  programmatic_launch(&attr[1]);
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, row_sweep_kernel<T, kUnitsPerWarp>, args);
}

template <typename T, bool kMulti>
cudaError_t launch_finish_t(const FinishArgs& fin, const ExpTable& table, cudaStream_t stream) {
  static OncePerDevice once;
  const cudaError_t e = func_attr_once(once, reinterpret_cast<const void*>(row_finish_kernel<T, kMulti>),
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FinishShared));
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)fin.s.rows, 1, 1);
  cfg.blockDim = dim3(kFinThreads, 1, 1);
  cfg.dynamicSmemBytes = sizeof(FinishShared);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  programmatic_launch(&attr[0]);
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, row_finish_kernel<T, kMulti>, fin, table);
}

template <typename T>
cudaError_t launch_pair_t(SweepArgs args, const FinishArgs& fin, const ExpTable& table, int sm_count,
                          cudaStream_t stream) {
  const int units = units_of(args.vocab);
  // Four units per warp (64 logits per thread), or two: with fp32 logits because two slices of four
  // units would take the shared memory of a whole SM, and for few rows because smaller shares mean
  // more SMs per row. At most 16 blocks make a cluster.
  const int c2 = (units + 2 * kSwWarps - 1) / (2 * kSwWarps);
  const bool two = c2 <= kSwMaxCluster && (sizeof(T) == 4 || args.rows * c2 <= 3 * sm_count);
  const int csize = two ? c2 : (units + 4 * kSwWarps - 1) / (4 * kSwWarps);
  args.units_per_block = (units + csize - 1) / csize;
  cudaError_t e = two ? launch_sweep_t<T, 2>(args, csize, sm_count, stream)
                      : launch_sweep_t<T, 4>(args, csize, sm_count, stream);
  if (e != cudaSuccess) return e;
  FinishArgs f = fin;
  f.s = args;
  const bool multi = args.ext.temperature != nullptr || args.ext.topp != nullptr || args.ext.topk != nullptr ||
                     (args.topk == 0 && !(args.topp > 0.0f && args.topp < 1.0f));
  return multi ? launch_finish_t<T, true>(f, table, stream) : launch_finish_t<T, false>(f, table, stream);
}

}  // namespace

bool fast_rows_supported(int dtype, int64_t rows, int vocab, float inv_t) {
  if (dtype != kDtypeFloat && dtype != kDtypeHalf && dtype != kDtypeBFloat16) return false;
  if (!(inv_t > 0.0f) || !(inv_t < INFINITY)) return false;
  if (vocab < 256 || units_of(vocab) > kSwMaxUnits) return false;
  return rows >= 1 && rows <= (int64_t)0x7fffffff;
}

size_t fast_rows_scratch_bytes(int vocab, int64_t rows) {
  const int64_t group = rows < kFastGroupRows ? rows : kFastGroupRows;
  return (size_t)group * (size_t)units_of(vocab) * sizeof(UnitRec);
}

cudaError_t launch_fast_rows(
    int dtype, const void* logits, int64_t rows, int vocab, int64_t row_stride, float inv_t, float topp, int topk,
    const RowSettings& settings, unsigned long long* rng_states, int64_t* out_ids, const PeerOut& peers,
    const ExpTable& table, void* scratch, RowHead* heads, int* retry_rows, int* retry_count, int* retry_count_next,
    int sm_count, cudaStream_t stream, unsigned long long* launches) {
  SweepArgs args = {};
  args.logits = logits;
  args.row_stride = row_stride;
  args.vocab = vocab;
  args.units_pitch = units_of(vocab);
  args.inv_t = inv_t;
  args.topp = topp;
  args.topk = topk;
  args.ext = settings;
  args.units = static_cast<UnitRec*>(scratch);
  args.heads = heads;
  FinishArgs fin = {};
  fin.rng_states = rng_states;
  fin.out_ids = out_ids;
  fin.peers = peers;
  fin.retry_rows = retry_rows;
  fin.retry_count = retry_count;
  for (int64_t row0 = 0; row0 < rows; row0 += kFastGroupRows) {
    args.row0 = row0;
    args.rows = rows - row0 < kFastGroupRows ? rows - row0 : kFastGroupRows;
    fin.retry_count_next = row0 == 0 ? retry_count_next : nullptr;
    cudaError_t e;
    switch (dtype) {
      case kDtypeFloat:
        e = launch_pair_t<float>(args, fin, table, sm_count, stream);
        break;
      case kDtypeHalf:
        e = launch_pair_t<__half>(args, fin, table, sm_count, stream);
        break;
      default:
        e = launch_pair_t<__nv_bfloat16>(args, fin, table, sm_count, stream);
        break;
    }
    if (e != cudaSuccess) return e;
    *launches += 2;
  }
  return cudaSuccess;
}

}  // namespace etb200
