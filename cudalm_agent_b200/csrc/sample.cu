// Token sampling on the device over the candidate lists the vocabulary
// projection returns: CUDALM's sample_token (include/cudalm/sampling.h:131-234)
// for configurations with 1 <= top_k <= list length, where every token outside
// the first top_k candidates has probability zero.  What matters is that only a
// token id crosses PCIe instead of 497 KB of logits per row
// (src/runtime/scheduler.cpp:59-108).
//
// The arithmetic follows the reference operation for operation: logit / T, exp
// and all sums in double; top-p accumulates in candidate order (value
// descending, tie -> lower id); the normalising sum and the cumulative walk run
// in ascending token id; probabilities are rounded to float before the walk;
// one SplitMix64 draw per sampled row, none on the greedy path.
//
// Bound by latency: a row is at most 64 candidates.  One warp per row, a lane per two
// candidates: the exponentials (one per candidate instead of three), divisions, the sort
// by id (by counting) and the searches run side by side; only the three running sums,
// whose order the reference fixes, stay serial (a dependent double addition per
// candidate, read from shared memory).  With one thread per row every exponential and the
// insertion sort were part of that chain: 32 rows, top-k 50, top-p 0.95 took 150 us, now 10
// (as part of a token step: 221 -> 81 us).
#include "common.cuh"

namespace cb200 {
namespace {

constexpr int kMaxSampleK = 64;
constexpr int kPerLane = kMaxSampleK / 32;
constexpr unsigned kAll = 0xffffffffu;

// Running sums of v[0 .. n) in index order, left in place; returns the last one.  Every
// lane runs the same chain over the same words (broadcast reads), lane 0 writes.
__device__ __forceinline__ double running_sums(double* v, int n, int lane) {
  double sum = 0.0;
  for (int i0 = 0; i0 < n; i0 += 8) {
    double t[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) t[u] = v[i0 + u];  // past n: unused words of the array
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (i0 + u < n) sum += t[u];
      t[u] = sum;
    }
    __syncwarp();
    if (lane == 0) {
#pragma unroll
      for (int u = 0; u < 8; ++u) v[i0 + u] = t[u];
    }
    __syncwarp();
  }
  return sum;
}

// The first (kFirst) or last candidate index for which `hit` holds, -1 if there is none.
// hit[j] belongs to candidate lane + 32 j.
template <bool kFirst>
__device__ __forceinline__ int find_index(const bool (&hit)[kPerLane]) {
  int found = -1;
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) {
    const unsigned b = __ballot_sync(kAll, hit[j]);
    if (b != 0u && (!kFirst || found < 0)) found = 32 * j + (kFirst ? __ffs(b) - 1 : 31 - __clz(b));
  }
  return found;
}

__global__ void __launch_bounds__(32)
sample_topk_kernel(const std::int32_t* __restrict__ topk_idx, const std::uint16_t* __restrict__ topk_val,
                   int list_len, int M, float temperature, int top_k, float top_p,
                   unsigned long long* __restrict__ rng_state, std::int32_t* __restrict__ token_out) {
  __shared__ double sums[kMaxSampleK];
  __shared__ int ids[kMaxSampleK];
  __shared__ int by_id[kMaxSampleK];
  // the lists may come from a kernel launched just before
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int m = blockIdx.x, lane = threadIdx.x;
  const std::int32_t* idx = topk_idx + static_cast<std::size_t>(m) * list_len;
  const std::uint16_t* val = topk_val + static_cast<std::size_t>(m) * list_len;
  if (!(temperature > 0.0f)) {  // greedy: the argmax, no draw
    if (lane == 0) token_out[m] = idx[0];
    return;
  }
  const int k = top_k;
  const double max_f =
      static_cast<double>(bf16_bits_to_float(val[0])) / static_cast<double>(temperature);
  double e[kPerLane];
  int id[kPerLane];
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) {
    const int i = lane + 32 * j;
    e[j] = 0.0;
    id[j] = 0;
    if (i < k) {
      const double f = static_cast<double>(bf16_bits_to_float(val[i])) / static_cast<double>(temperature);
      e[j] = exp(f - max_f);
      id[j] = idx[i];
    }
    sums[i] = e[j];
    ids[i] = id[j];
  }
  __syncwarp();
  int kept = k;
  if (top_p < 1.0f) {
    const double total = running_sums(sums, k, lane);
    bool hit[kPerLane];
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      const int i = lane + 32 * j;
      hit[j] = i < k && (sums[i] >= static_cast<double>(top_p) * total || i + 1 == k);
    }
    kept = find_index<true>(hit) + 1;
    __syncwarp();
  }
  // ascending token id over the kept candidates, equal ids in list order
  int rank[kPerLane] = {};
  for (int o = 0; o < kept; ++o) {
    const int other = ids[o];
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) rank[j] += other < id[j] || (other == id[j] && o < lane + 32 * j);
  }
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) {
    if (lane + 32 * j < kept) {
      by_id[rank[j]] = id[j];
      sums[rank[j]] = e[j];
    }
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) e[j] = sums[lane + 32 * j];  // from here on in order of id
  __syncwarp();
  const double norm = running_sums(sums, kept, lane);
  // SplitMix64 (include/cudalm/sampling.h:99-116)
  unsigned long long z = rng_state[m] + 0x9E3779B97F4A7C15ull;
  __syncwarp();
  if (lane == 0) rng_state[m] = z;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z = z ^ (z >> 31);
  const double u = static_cast<double>(z >> 11) * 0x1.0p-53;
  // (a probability that rounds to zero leaves the cumulative sum as it is)
  float p[kPerLane];
  bool positive[kPerLane], reached[kPerLane];
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) {
    const int i = lane + 32 * j;
    p[j] = i < kept ? static_cast<float>(e[j] / norm) : 0.0f;
    positive[j] = p[j] > 0.0f;
    sums[i] = positive[j] ? static_cast<double>(p[j]) : 0.0;
  }
  __syncwarp();
  (void)running_sums(sums, kept, lane);
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) reached[j] = positive[j] && u < sums[lane + 32 * j];
  const int first = find_index<true>(reached);
  const int last = find_index<false>(positive);
  if (lane == 0) token_out[m] = first >= 0 ? by_id[first] : (last >= 0 ? by_id[last] : idx[0]);
}

}  // namespace
}  // namespace cb200

extern "C" int cudalm_b200_sample_topk(const int32_t* topk_idx, const uint16_t* topk_val,
                                       int list_len, int M, float temperature, int top_k,
                                       float top_p, uint64_t* rng_state, int32_t* token_out,
                                       void* stream) {
  using namespace cb200;
  if (!topk_idx || !topk_val || !token_out) return CUDALM_B200_ERR_NULL;
  if (list_len < 1 || M < 1) return CUDALM_B200_ERR_BAD_SHAPE;
  // the reference's validation (include/cudalm/sampling.h:73-91): values it rejects
  if (temperature != temperature || temperature - temperature != 0.0f) return CUDALM_B200_ERR_BAD_SHAPE;
  if (top_k < 0 || !(top_p > 0.0f) || top_p > 1.0f) return CUDALM_B200_ERR_BAD_SHAPE;
  const bool greedy = !(temperature > 0.0f);
  if (!greedy) {
    if (!rng_state) return CUDALM_B200_ERR_NULL;
    // top_k = 0 (or beyond the list) lets tokens outside the list keep a
    // non-zero probability: that needs the whole row of logits
    if (top_k < 1 || top_k > list_len) return CUDALM_B200_ERR_UNSUPPORTED;
    if (top_k > kMaxSampleK) return CUDALM_B200_ERR_TOO_LARGE;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(M));
  cfg.blockDim = dim3(32);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t le =
      cudaLaunchKernelEx(&cfg, sample_topk_kernel, topk_idx, topk_val, list_len, M, temperature, top_k,
                         top_p, reinterpret_cast<unsigned long long*>(rng_state), token_out);
  if (le != cudaSuccess) {
    g_last_cuda_error = static_cast<int>(le);
    (void)cudaGetLastError();
    return CUDALM_B200_ERR_CUDA;
  }
  return check_launch();
}
