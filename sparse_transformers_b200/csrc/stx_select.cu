// Per-row selection rules that need a whole score row, and the approximate top-k threshold.
//
//   statistical_topk  src/modeling_skip.py:197-202  scores > mean + std_pop * z   (per row)
//   topk              src/modeling_skip.py:208-211  scatter True at scores.topk(k)
//   approx_topk_threshold  sparse_transformers/csrc/approx_topk.h:10-87
//
// One block of 1024 threads per batch row; the per-row masks are OR-ed into the output bit
// words (mask.any(dim=0), src/modeling_skip.py:214).  All three are reproducible bit for bit
// by the CPU restatement (oracle/stx_oracle.c): exact k-th element by radix select, ties at
// the k-th value taken in ascending index order, and a fixed double-precision summation order
// for the mean and variance (1024 interleaved partial sums; XOR butterfly inside each group
// of 32 consecutive partials, then the 32 group sums added in ascending order).
#include "stx_common.cuh"

#include <algorithm>

namespace stx {

constexpr int SEL_THREADS = 1024;

__device__ __forceinline__ uint32_t order_key(float f) {  // ascending float order -> ascending uint order
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
  const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}

// Sum over the block in the documented order; every thread gets the result.
__device__ __forceinline__ double block_sum_fixed(double v, double* s_w /*[32]*/, double* s_out) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if (lane == 0) s_w[wid] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < 32; ++w) s += s_w[w];
    *s_out = s;
  }
  __syncthreads();
  const double r = *s_out;
  __syncthreads();
  return r;
}

// Keys of a score in the order of order_key: the 16-bit types need their own 16 bits only (widening to float keeps the
// order of all values), which halves the radix passes and lets a whole row of keys stay in shared memory.
template <typename T> struct SelKey {
  typedef uint16_t type;
  static constexpr int BITS = 16;
  static __device__ __forceinline__ uint32_t of(T v) {
    const uint32_t u = *reinterpret_cast<const uint16_t*>(&v);
    return (u & 0x8000u) ? (~u & 0xffffu) : (u | 0x8000u);
  }
  static __device__ __forceinline__ float value(uint32_t k) {
    const uint16_t u = static_cast<uint16_t>((k & 0x8000u) ? (k & 0x7fffu) : ~k);
    return DT<T>::to_f(*reinterpret_cast<const T*>(&u));
  }
};
template <> struct SelKey<float> {
  typedef uint32_t type;
  static constexpr int BITS = 32;
  static __device__ __forceinline__ uint32_t of(float v) { return order_key(v); }
  static __device__ __forceinline__ float value(uint32_t k) { return key_value(k); }
};

constexpr int SEL_HISTS = 8;  // histograms of a block: a warp adds to number warp & 7, scores crowd into a few bins

// k-th largest (k >= 1) of n keys of BITS bits produced by key_at(i), exact, by radix passes of 8 bits.
// All threads of the block must call it; returns the key.  s_hist: SEL_HISTS x 256 ints; s_pick: 2 ints.
// A pass: histogram, then warp 0 finds the bin (a lane sums 8 bins, a shuffle scan from the top finds the lane,
// that lane walks its 8 bins); one thread walking 256 bins took 3 us of a pass.
template <int BITS, typename KeyAt>
__device__ __forceinline__ uint32_t block_kth_largest(KeyAt key_at, int n, int k, int* s_hist, int* s_pick) {
  uint32_t prefix = 0u, mask = 0u;
  int kk = k;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int* hist = s_hist + (wid % SEL_HISTS) * 256;
  for (int shift = BITS - 8; shift >= 0; shift -= 8) {
    for (int i = threadIdx.x; i < SEL_HISTS * 256; i += blockDim.x) s_hist[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const uint32_t key = key_at(i);
      if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1);
    }
    __syncthreads();
    if (wid == 0) {
      int bin[8], sum = 0;  // bins 255 - 8 * lane - j, j = 0..7: the lanes go down from the top
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        bin[j] = 0;
#pragma unroll
        for (int q = 0; q < SEL_HISTS; ++q) bin[j] += s_hist[q * 256 + 255 - 8 * lane - j];
        sum += bin[j];
      }
      int inc = sum;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += v;
      }
      const int before = inc - sum;
      // the first lane whose running total reaches kk (the last lane if none does)
      const uint32_t reach = __ballot_sync(0xffffffffu, inc >= kk);
      const int owner = reach ? __ffs(reach) - 1 : 31;
      if (lane == owner) {
        int acc = before, j = 0;
#pragma unroll
        for (int q = 0; q < 7; ++q) {
          if (j == q && acc + bin[q] < kk) {
            acc += bin[q];
            ++j;
          }
        }
        s_pick[0] = 255 - 8 * lane - j;
        s_pick[1] = kk - acc;
      }
    }
    __syncthreads();
    prefix |= static_cast<uint32_t>(s_pick[0]) << shift;
    mask |= 255u << shift;
    kk = s_pick[1];
    __syncthreads();
  }
  return prefix;
}

template <typename T>
__global__ void __launch_bounds__(SEL_THREADS)
k_mask_statistical(const T* __restrict__ scores, int I, float z, uint32_t* __restrict__ bits) {
  __shared__ double s_w[32];
  __shared__ double s_out;
  const T* s = scores + static_cast<size_t>(blockIdx.x) * I;
  const int t = threadIdx.x;
  pdl_wait();
  pdl_launch_dependents();
  double a = 0.0;
  for (int i = t; i < I; i += SEL_THREADS) a += static_cast<double>(DT<T>::to_f(s[i]));
  const double mean_d = block_sum_fixed(a, s_w, &s_out) / static_cast<double>(I);
  a = 0.0;
  for (int i = t; i < I; i += SEL_THREADS) {
    const double d = static_cast<double>(DT<T>::to_f(s[i])) - mean_d;
    a += d * d;
  }
  const double var_d = block_sum_fixed(a, s_w, &s_out) / static_cast<double>(I);
  // rounding points of the reference's tensor arithmetic in the scores' dtype
  const float mean_r = DT<T>::round_f(static_cast<float>(mean_d));
  const float std_r = DT<T>::round_f(static_cast<float>(sqrt(var_d)));
  const float z_r = DT<T>::round_f(z);
  const float prod = DT<T>::round_f(__fmul_rn(std_r, z_r));
  const float cutoff = DT<T>::round_f(__fadd_rn(mean_r, prod));
  const int W = (I + 31) >> 5, lane = t & 31;
  for (int w = t >> 5; w < W; w += SEL_THREADS / 32) {
    const int i = w * 32 + lane;
    const uint32_t word = __ballot_sync(0xffffffffu, i < I && DT<T>::to_f(s[i]) > cutoff);
    if (lane == 0 && word) atomicOr(&bits[w], word);
  }
}

// Dynamic shared memory (KEYS_IN_SMEM): the row's keys.  A block reads its row once; the radix passes and the final
// compare run on the keys.
template <typename T, bool KEYS_IN_SMEM>
__global__ void __launch_bounds__(SEL_THREADS)
k_mask_topk(const T* __restrict__ scores, int I, int k, uint32_t* __restrict__ bits) {
  typedef typename SelKey<T>::type Key;
  extern __shared__ uint32_t s_keys[];
  __shared__ int s_hist[SEL_HISTS * 256];
  __shared__ int s_pick[2];
  __shared__ int s_wties[32];
  __shared__ int s_above;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int W = (I + 31) >> 5;
  Key* s_key = reinterpret_cast<Key*>(s_keys);
  pdl_wait();
  pdl_launch_dependents();
  const T* s = scores + static_cast<size_t>(blockIdx.x) * I;
  if (KEYS_IN_SMEM) {
    for (int i = t; i < I; i += SEL_THREADS) s_key[i] = static_cast<Key>(SelKey<T>::of(s[i]));
    __syncthreads();
  }
  auto key_at = [&](int i) -> uint32_t { return KEYS_IN_SMEM ? static_cast<uint32_t>(s_key[i]) : SelKey<T>::of(s[i]); };
  const float kth = SelKey<T>::value(block_kth_largest<SelKey<T>::BITS>(key_at, I, k, s_hist, s_pick));
  if (t == 0) s_above = 0;
  __syncthreads();
  // A warp owns a range of mask words.  First its scores above the k-th and equal to it are counted: ties are taken
  // in ascending index order, so a warp has to know how many lie in front of its range.
  const int per = (W + SEL_THREADS / 32 - 1) / (SEL_THREADS / 32);
  const int lo = min(W, wid * per), hi = min(W, lo + per);
  auto word_of = [&](int w, uint32_t& above, uint32_t& ties) {
    const int i = w * 32 + lane;
    const float v = i < I ? SelKey<T>::value(key_at(i)) : 0.f;
    above = __ballot_sync(0xffffffffu, i < I && v > kth);
    ties = __ballot_sync(0xffffffffu, i < I && v == kth);
  };
  int n_above = 0, n_ties = 0;
  for (int w = lo; w < hi; ++w) {
    uint32_t ab, ti;
    word_of(w, ab, ti);
    n_above += __popc(ab);
    n_ties += __popc(ti);
  }
  if (lane == 0) {
    atomicAdd(&s_above, n_above);
    s_wties[wid] = n_ties;
  }
  __syncthreads();
  int left = k - s_above;  // ties this warp may still take
  for (int w = 0; w < wid; ++w) left -= s_wties[w];
  for (int w = lo; w < hi; ++w) {
    uint32_t word, ti;
    word_of(w, word, ti);
    if (left > 0 && ti) {
      const bool take = ((ti >> lane) & 1u) && __popc(ti & ((1u << lane) - 1u)) < left;
      word |= __ballot_sync(0xffffffffu, take);
    }
    left -= __popc(ti);
    if (lane == 0 && word) atomicOr(&bits[w], word);
  }
}

// approx_topk.h:25-83.  Shared memory: 4 * width bucket keys.
template <typename T>
__global__ void __launch_bounds__(SEL_THREADS)
k_approx_topk(const T* __restrict__ scores, int I, int k, T* __restrict__ thr_out) {
  extern __shared__ uint32_t s_sk[];
  __shared__ int s_hist[SEL_HISTS * 256];
  __shared__ int s_pick[2];
  __shared__ int s_n;
  const T* s = scores + static_cast<size_t>(blockIdx.x) * I;
  const int t = threadIdx.x;
  const int S = 4;
  const int width = min(1024, I / 4);
  if (width <= 0) {
    if (t == 0) thr_out[blockIdx.x] = DT<T>::from_f(0.f);
    return;
  }
  const uint32_t neg_inf = order_key(-INFINITY);
  for (int i = t; i < S * width; i += SEL_THREADS) s_sk[i] = neg_inf;
  if (t == 0) s_n = 0;
  __syncthreads();
  for (int q = 0; q < S; ++q)
    for (int j = t; j < I; j += SEL_THREADS) {
      const long long key = static_cast<long long>(q) * I + j;  // std::hash<int64_t> is the identity
      const int pos = static_cast<int>(key % width);
      atomicMax(&s_sk[q * width + pos], order_key(DT<T>::to_f(s[j])));
    }
  __syncthreads();
  int mine = 0;
  for (int i = t; i < S * width; i += SEL_THREADS) mine += s_sk[i] != neg_inf;
  atomicAdd(&s_n, mine);
  __syncthreads();
  const int n = s_n;
  if (n == 0) {
    if (t == 0) thr_out[blockIdx.x] = DT<T>::from_f(0.f);
    return;
  }
  long long sketch_k = static_cast<long long>(k) * n / I;
  if (sketch_k < 1) sketch_k = 1;
  if (sketch_k > n) sketch_k = n;
  // the excluded -inf buckets sort last, so the rank among all buckets is the same
  const uint32_t key = block_kth_largest<32>([&](int i) { return s_sk[i]; }, S * width, static_cast<int>(sketch_k), s_hist, s_pick);
  if (t == 0) thr_out[blockIdx.x] = DT<T>::from_f(__fmul_rn(key_value(key), 0.9f));
}

template <typename T>
static int launch_topk(const void* scores, int64_t B, int64_t I, int k, uint32_t* bits, cudaStream_t s) {
  const size_t keys = static_cast<size_t>(I) * sizeof(typename SelKey<T>::type);
  constexpr size_t LIMIT = 200 * 1024;
  const dim3 grid(static_cast<unsigned>(B)), block(SEL_THREADS);
  const T* sc = static_cast<const T*>(scores);
  if (keys > LIMIT) {  // rows of more than 51200 fp32 (102400 16-bit) scores: the keys are made from the scores in every pass
    STX_CUDA(launch_pdl(k_mask_topk<T, false>, grid, block, 0, s, sc, static_cast<int>(I), k, bits));
    return STX_OK;
  }
  static bool attr_set[64] = {};
  int dev = 0;
  STX_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    STX_CUDA(cudaFuncSetAttribute(k_mask_topk<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(LIMIT)));
    attr_set[dev] = true;
  }
  STX_CUDA(launch_pdl(k_mask_topk<T, true>, grid, block, keys, s, sc, static_cast<int>(I), k, bits));
  return STX_OK;
}

// zeroed: `bits` was cleared by an earlier kernel of the same call
int mask_from_scores(const void* scores, int64_t B, int64_t I, int dtype, int method, float param,
                     uint32_t* bits_out, bool zeroed, cudaStream_t s) {
  const size_t W = static_cast<size_t>((I + 31) / 32);
  if (!zeroed) STX_CUDA(cudaMemsetAsync(bits_out, 0, W * sizeof(uint32_t), s));
  const dim3 grid(static_cast<unsigned>(B)), block(SEL_THREADS);
  const int ii = static_cast<int>(I);
  if (method == STX_MASK_STATISTICAL) {
    switch (dtype) {
      case STX_F32:
        STX_CUDA(launch_pdl(k_mask_statistical<float>, grid, block, 0, s, static_cast<const float*>(scores), ii, param, bits_out));
        break;
      case STX_F16:
        STX_CUDA(launch_pdl(k_mask_statistical<__half>, grid, block, 0, s, static_cast<const __half*>(scores), ii, param, bits_out));
        break;
      default:
        STX_CUDA(launch_pdl(k_mask_statistical<__nv_bfloat16>, grid, block, 0, s, static_cast<const __nv_bfloat16*>(scores), ii,
                            param, bits_out));
        break;
    }
    return STX_OK;
  }
  if (method == STX_MASK_TOPK) {
    int k = static_cast<int>(param);
    if (k < 1 || k > I) {
      set_error("topk rule: k=%d outside 1..%lld", k, static_cast<long long>(I));
      return STX_ERR_INVALID_ARG;
    }
    switch (dtype) {
      case STX_F32: return launch_topk<float>(scores, B, I, k, bits_out, s);
      case STX_F16: return launch_topk<__half>(scores, B, I, k, bits_out, s);
      default: return launch_topk<__nv_bfloat16>(scores, B, I, k, bits_out, s);
    }
  }
  set_error("mask rule %d needs no score pass", method);
  return STX_ERR_INVALID_ARG;
}

}  // namespace stx

using namespace stx;

extern "C" {

int stx_approx_topk_scratch_bytes(int64_t B, int64_t I, size_t* bytes_out) {
  STX_CHECK_ARG(bytes_out && B > 0 && I > 0, "stx_approx_topk_scratch_bytes: bad argument");
  *bytes_out = 256;  // the kernel works in shared memory; kept for interface stability
  return STX_OK;
}

int stx_approx_topk_threshold(const void* scores, int64_t B, int64_t I, int64_t k, int dtype, void* threshold_out,
                              void* scratch, void* stream) {
  (void)scratch;
  STX_CHECK_ARG(scores && threshold_out, "stx_approx_topk_threshold: null pointer");
  STX_CHECK_ARG(B > 0 && I > 0, "stx_approx_topk_threshold: sizes must be positive");
  STX_CHECK_ARG(k > 0, "k must be positive");
  STX_CHECK_ARG(k <= I, "k cannot be larger than feature size");
  STX_CHECK_ARG(dtype == STX_F32 || dtype == STX_F16 || dtype == STX_BF16, "stx_approx_topk_threshold: bad dtype %d", dtype);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int width = static_cast<int>(std::min<int64_t>(1024, I / 4));
  const size_t smem = static_cast<size_t>(4) * std::max(width, 1) * sizeof(uint32_t);
  const unsigned grid = static_cast<unsigned>(B);
  switch (dtype) {
    case STX_F32:
      k_approx_topk<float><<<grid, SEL_THREADS, smem, s>>>(static_cast<const float*>(scores), static_cast<int>(I), static_cast<int>(k), static_cast<float*>(threshold_out));
      break;
    case STX_F16:
      k_approx_topk<__half><<<grid, SEL_THREADS, smem, s>>>(static_cast<const __half*>(scores), static_cast<int>(I), static_cast<int>(k), static_cast<__half*>(threshold_out));
      break;
    default:
      k_approx_topk<__nv_bfloat16><<<grid, SEL_THREADS, smem, s>>>(static_cast<const __nv_bfloat16*>(scores), static_cast<int>(I), static_cast<int>(k), static_cast<__nv_bfloat16*>(threshold_out));
      break;
  }
  STX_LAUNCH_CHECK("k_approx_topk");
  return STX_OK;
}

}  // extern "C"
