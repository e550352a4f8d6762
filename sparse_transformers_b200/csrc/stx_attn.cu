// Decode-time glue of the LlamaSkip host around the sparse MLP (C ABI: stx_attn_decode,
// stx_add_rmsnorm): one query token against the KV cache, and residual add + RMSNorm.
//
//   k_attn_decode   grid = groups of query heads that share a cache head x splits of the keys.  A CTA
//                   rotates its q heads and the k head (rotate-half RoPE in fp32, rounded to the model
//                   dtype), one CTA per cache head appends k and v, and every CTA streams its share of
//                   the keys and values once for all of its query heads.  The position is read from
//                   device memory, so a captured CUDA graph can be replayed token after token.
//   k_add_rmsnorm   one CTA: h <- h + a (rounded to the model dtype), then
//                   x = round(h * rsqrt(mean(h^2) + eps)) * w, the order of operations of
//                   LlamaSkipRMSNorm (src/models/llama/modelling_llama_skip.py:39-44).
#include "stx_common.cuh"
#include "stx_tma.cuh"

#include <algorithm>
#include <cstdlib>
#include <cstring>

namespace stx {

constexpr int ATT_THREADS = 512;
constexpr int NORM_THREADS = 1024;

// Block-wide max / sum over the block's threads; `red` has 32 floats.  Every thread gets the result.
template <bool IS_MAX>
__device__ __forceinline__ float block_reduce(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float o = __shfl_xor_sync(0xffffffffu, v, off);
    v = IS_MAX ? fmaxf(v, o) : v + o;
  }
  __syncthreads();  // red may still be read from a previous call
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float r = IS_MAX ? -INFINITY : 0.f;
  for (int w = 0; w < nw; ++w) r = IS_MAX ? fmaxf(r, red[w]) : r + red[w];  // same order in every thread
  return r;
}

// Workspace of stx_attn_decode: one arrival counter per group of heads (zero between launches), then per head and
// split the unnormalised value sum [HD], the split's score maximum and its sum of exponentials.
constexpr size_t ATT_COUNTER_BYTES = 4096;  // up to 1024 heads
constexpr int ATT_MAX_SPLITS = 32;
// One block takes up to ATT_TILES_ALONE tiles of keys by itself, beyond that a split takes at least ATT_KEYS_PER_SPLIT: a
// second tile costs a block 0.5 to 1 us, the merge of splits 1.5 to 2.5 us whatever their number.
constexpr int ATT_TILES_ALONE = 2;
constexpr int ATT_KEYS_PER_SPLIT = 48;
__host__ __device__ inline int att_part_floats(int hd) { return hd + 2; }

// Sums of v[0..N) over groups of G neighbouring lanes (powers of two).  A stage halves the values a lane keeps, as long
// as there are two: about N + log2(G / N) shuffles instead of N log2(G).  Lane l of a group ends with value
// l / (G / N) when G >= N, else with the N / G values from (l * N / G) on, in v[0..).
template <int N, int G>
__device__ __forceinline__ void group_sum_many(float (&v)[N], int lane) {
  int n = N;
#pragma unroll
  for (int off = G / 2; off > 0; off >>= 1) {
    if (n > 1) {
      const bool hi = (lane & off) != 0;
#pragma unroll
      for (int j = 0; j < N / 2; ++j) {
        if (j < n / 2) {
          const float give = hi ? v[j] : v[j + n / 2];
          const float keep = hi ? v[j + n / 2] : v[j];
          v[j] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
      }
      n /= 2;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    }
  }
}

// Shapes of the key stream: a row of HD elements is LPK lanes x CPT 16-byte chunks; a thread has U rows of keys and U of
// values in flight, so a CTA takes TK keys at a time.
template <typename T, int HD, int REP> struct AttShape {
  static constexpr int V = DT<T>::V;
  static constexpr int CH = HD / V;                 // 16-byte chunks of a row
  static constexpr int LPK = CH < 32 ? CH : 32;
  static constexpr int CPT = CH / LPK;
  static constexpr int NG = ATT_THREADS / LPK;      // rows side by side
  static constexpr int U = (sizeof(T) == 4 ? 8 : REP == 1 ? 8 : REP == 4 ? 2 : 4) / CPT;  // what 128 registers hold
  static constexpr int TK = NG * U;
};

// What bounds it: the KV bytes at long contexts, a chain of dependent trips (position, rows, merge) at short ones.
// A CTA reads every key and value of its split once for its REP query heads (they share the cache head) with 16-byte
// loads, U keys and U values per thread requested before the first is used and the next tile's requested as soon as
// a tile's registers are free; each warp keeps a running soft-max of its own keys.
// 24 query heads on 8 cache heads of 128, 4000 tokens, fp16: four layers of norm, attention, projection and norm 136 -> 104.5 us
// (a warp per key and one batch of keys at a time before, every query head reading the cache for itself: 18.5 us a launch).
// The splits meet in the workspace: the last one to arrive at the group's counter merges.  Splits beyond what the
// position can use leave at once.  Between 64 and 1000 keys the ends of the chain are what counts: the warps' sums in
// lane order (no bank conflicts) with their weights formed once, one release per block instead of a fence per thread, and
// partial sums requested together with their weights took the same four layers from 78 to 74 us at 200 keys and from 103
// to 98 at 4000 (32 heads on 8: 103 to 97 and 126 to 116; before the heads of a cache head shared a block: 74 and 135,
// 96 and 167).
// Shared memory (floats): q_s[REP][HD] | kn_s[HD] | vn_s[HD] | red[16][REP][HD] | m[REP][16] | l[REP][16]
template <typename T, int HD, int REP>
__global__ void __launch_bounds__(ATT_THREADS, 1) k_attn_decode(const T* __restrict__ qkv, const float* __restrict__ cos_t,
                                                                 const float* __restrict__ sin_t,
                                                                 const long long* __restrict__ pos_dev, T* k_cache, T* v_cache,
                                                                 T* __restrict__ out, int nh, int nkv, long long max_len,
                                                                 float scale, unsigned char* workspace) {
  typedef AttShape<T, HD, REP> S;
  constexpr int V = S::V, LPK = S::LPK, CPT = S::CPT, NG = S::NG, U = S::U, TK = S::TK;
  constexpr int NW = ATT_THREADS / 32;
  extern __shared__ float sm[];
  float* q_s = sm;
  float* kn_s = q_s + REP * HD;
  float* vn_s = kn_s + HD;
  float* red = vn_s + HD;
  float* m_s = red + NW * REP * HD;
  float* l_s = m_s + NW * REP;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  pdl_launch_dependents();
  const long long pos = *pos_dev;
  if (pos < 0 || pos >= max_len) return;  // nothing sensible to do; the output is left as it was
  const int h0 = blockIdx.x * REP, g = h0 / (nh / nkv);
  const int np = static_cast<int>(pos);   // cached keys
  const int NSP = np <= ATT_TILES_ALONE * TK ? 1 : min(static_cast<int>(gridDim.y), np / ATT_KEYS_PER_SPLIT + 1);
  const int sp = blockIdx.y;
  if (sp >= NSP) return;
  T* kc = k_cache + static_cast<size_t>(g) * max_len * HD;
  T* vc = v_cache + static_cast<size_t>(g) * max_len * HD;
  const int chunk = (np + NSP - 1) / NSP;
  const int lo = min(sp * chunk, np), n = min(lo + chunk, np) - lo;  // key j of the split is cached key lo + j
  const bool own = sp == NSP - 1;                                    // this split also takes the token's own key
  const T* ks = kc + static_cast<size_t>(lo) * HD;
  const T* vs = vc + static_cast<size_t>(lo) * HD;
  const int ch = tid % LPK, grp = tid / LPK;

  uint4 kr[U][CPT], vr[U][CPT];
  auto load_tile = [&](const T* src, int j0, uint4 (&r)[U][CPT]) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + grp + NG * u;
#pragma unroll
      for (int c = 0; c < CPT; ++c)
        r[u][c] = j < n ? ld_cached16(src + static_cast<size_t>(j) * HD + (ch + LPK * c) * V) : make_uint4(0, 0, 0, 0);
    }
  };
  load_tile(ks, 0, kr);
  load_tile(vs, 0, vr);

  for (int i = tid; i < (REP + 1) * HD; i += ATT_THREADS) {
    constexpr int half = HD / 2;
    const int r = i / HD, d = i - r * HD;
    const int dp = d < half ? d + half : d - half;
    const float sign = d < half ? -1.f : 1.f;
    const float c = cos_t[pos * HD + d], s = sin_t[pos * HD + d];
    const T* row = qkv + static_cast<size_t>(r < REP ? h0 + r : nh + g) * HD;
    // x * cos + rotate_half(x) * sin: two rounded products, one rounded sum, then the model dtype
    const T y = DT<T>::from_f(__fadd_rn(__fmul_rn(DT<T>::to_f(row[d]), c), __fmul_rn(sign * DT<T>::to_f(row[dp]), s)));
    q_s[i] = DT<T>::to_f(y);  // row REP is kn_s
    if (r == REP) {
      const T v = qkv[static_cast<size_t>(nh + nkv + g) * HD + d];
      vn_s[d] = DT<T>::to_f(v);
      if (sp == 0 && h0 == g * (nh / nkv)) {  // one writer per cache head; the others use their own copy
        kc[pos * HD + d] = y;
        vc[pos * HD + d] = v;
      }
    }
  }
  __syncthreads();

  // Every warp runs its own soft-max over the keys that it loads (no barrier inside the loop); in the last split warp 0
  // starts from the token's own key.
  float qf[REP][CPT * V], acc[REP][CPT * V], m_run[REP], l_run[REP];
#pragma unroll
  for (int r = 0; r < REP; ++r) {
#pragma unroll
    for (int c = 0; c < CPT; ++c)
#pragma unroll
      for (int v = 0; v < V; ++v) {
        qf[r][c * V + v] = q_s[r * HD + (ch + LPK * c) * V + v];
        acc[r][c * V + v] = own && grp == 0 ? vn_s[(ch + LPK * c) * V + v] : 0.f;
      }
    m_run[r] = -INFINITY;
    l_run[r] = 0.f;
    if (own && warp == 0) {
      float dot = 0.f;
      for (int d = lane; d < HD; d += 32) dot = fmaf(q_s[r * HD + d], kn_s[d], dot);
      m_run[r] = warp_sum_xor(dot) * scale;
      l_run[r] = 1.f;
    }
  }

  for (int j0 = 0; j0 < n; j0 += TK) {
    float p[REP][U];
#pragma unroll
    for (int r = 0; r < REP; ++r) {
      float dot[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        dot[u] = 0.f;
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          float f[V];
          Unpack<T>::run(kr[u][c], f);
#pragma unroll
          for (int v = 0; v < V; ++v) dot[u] = fmaf(qf[r][c * V + v], f[v], dot[u]);
        }
      }
      group_sum_many<U, LPK>(dot, lane);
      constexpr int LPV = LPK / U;  // lanes of a row group that hold the same key's sum (LPK >= U in every instance)
      float mx = m_run[r];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float s = __shfl_sync(0xffffffffu, dot[0], (lane & ~(LPK - 1)) + u * LPV) * scale;
        p[r][u] = j0 + grp + NG * u < n ? s : -INFINITY;
        mx = fmaxf(mx, p[r][u]);
      }
#pragma unroll
      for (int off = LPK; off < 32; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      float sum = 0.f;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        p[r][u] = p[r][u] == -INFINITY ? 0.f : __expf(p[r][u] - mx);
        sum += p[r][u];
      }
#pragma unroll
      for (int off = LPK; off < 32; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
      const float corr = mx == m_run[r] ? 1.f : __expf(m_run[r] - mx);  // 0 where nothing came before
      m_run[r] = mx;
      l_run[r] = fmaf(l_run[r], corr, sum);
#pragma unroll
      for (int k = 0; k < CPT * V; ++k) acc[r][k] *= corr;
    }
    if (j0 + TK < n) load_tile(ks, j0 + TK, kr);
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        float f[V];
        Unpack<T>::run(vr[u][c], f);
#pragma unroll
        for (int r = 0; r < REP; ++r)
#pragma unroll
          for (int v = 0; v < V; ++v) acc[r][c * V + v] = fmaf(p[r][u], f[v], acc[r][c * V + v]);
      }
    if (j0 + TK < n) load_tile(vs, j0 + TK, vr);
  }

  // ---- the warps' results meet in shared memory: sum_w e^(m_w - M) acc_w in warp order.  Until the result is written, a
  // row's elements stand in the order of the lanes that hold them (element `slot` = k * LPK + ch), so that neighbouring
  // lanes touch neighbouring banks.
#pragma unroll
  for (int r = 0; r < REP; ++r) {
#pragma unroll
    for (int k = 0; k < CPT * V; ++k) {
      float a = acc[r][k];
#pragma unroll
      for (int off = LPK; off < 32; off <<= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
      if (lane < LPK) red[(warp * REP + r) * HD + k * LPK + lane] = a;
    }
    if (lane == 0) {
      m_s[r * NW + warp] = m_run[r];
      l_s[r * NW + warp] = l_run[r];
    }
  }
  __shared__ float s_M[REP], s_l[REP];
  __shared__ __align__(16) float s_w[REP][NW];
  __syncthreads();
  if (warp < REP) {
    const float mw = lane < NW ? m_s[warp * NW + lane] : -INFINITY;
    float M = mw;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
    const float f = mw == -INFINITY ? 0.f : __expf(mw - M);  // 0 for a warp without keys
    const float l = warp_sum_xor(lane < NW ? f * l_s[warp * NW + lane] : 0.f);
    if (lane < NW) s_w[warp][lane] = f;
    if (lane == 0) {
      s_M[warp] = M;
      s_l[warp] = l;
    }
  }
  __syncthreads();
  int* counter = reinterpret_cast<int*>(workspace) + blockIdx.x;
  float* part = reinterpret_cast<float*>(workspace + ATT_COUNTER_BYTES);
  auto part_of = [&](int split, int r) { return part + (static_cast<size_t>(h0 + r) * ATT_MAX_SPLITS + split) * att_part_floats(HD); };
  auto element = [&](int slot) {  // element of the head that stands in this slot
    const int k = slot / LPK;
    return (slot % LPK + LPK * (k / V)) * V + k % V;
  };
  for (int i = tid; i < REP * HD; i += ATT_THREADS) {
    const int r = i / HD, slot = i - r * HD;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < NW; w += 4) {
      const float4 f = *reinterpret_cast<const float4*>(&s_w[r][w]);
      s = fmaf(f.x, red[w * REP * HD + i], s);
      s = fmaf(f.y, red[(w + 1) * REP * HD + i], s);
      s = fmaf(f.z, red[(w + 2) * REP * HD + i], s);
      s = fmaf(f.w, red[(w + 3) * REP * HD + i], s);
    }
    if (NSP == 1) {
      out[static_cast<size_t>(h0 + r) * HD + element(slot)] = DT<T>::from_f(s / s_l[r]);
    } else {
      float* mine = part_of(sp, r);
      __stcg(mine + slot, s);
      if (slot == 0) {
        __stcg(mine + HD, s_M[r]);
        __stcg(mine + HD + 1, s_l[r]);
      }
    }
  }
  if (NSP == 1) return;
  // ---- the split that arrives last merges: out = sum_s e^(m_s - M) acc_s / sum_s e^(m_s - M) l_s
  __shared__ int s_last;
  __syncthreads();  // the block's partial results precede thread 0's release
  if (tid == 0) {
    int t;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(t) : "l"(counter) : "memory");
    s_last = t == NSP - 1;
    if (s_last) *counter = 0;  // every other split has arrived: ready for the next launch
  }
  __syncthreads();
  if (!s_last) return;
  float v[ATT_MAX_SPLITS];  // all loads in flight together, next to those of the weights
  auto load_parts = [&](int i) {
    const int r = i / HD;
    const float* pk = part_of(0, r) + (i - r * HD);
#pragma unroll
    for (int k = 0; k < ATT_MAX_SPLITS; ++k) v[k] = k < NSP ? __ldcg(pk + static_cast<size_t>(k) * att_part_floats(HD)) : 0.f;
  };
  if (tid < REP * HD) load_parts(tid);
  float* wgt = red;  // [REP][ATT_MAX_SPLITS] weights; behind them the sums of exponentials
  float* den_s = red + REP * ATT_MAX_SPLITS;
  if (warp < REP) {
    const float* pk = part_of(lane, warp);
    const float pm = lane < NSP ? __ldcg(pk + HD) : -INFINITY, pl = lane < NSP ? __ldcg(pk + HD + 1) : 0.f;
    float M = pm;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
    const float w = lane < NSP && pm != -INFINITY ? __expf(pm - M) : 0.f;  // 0 for a split without keys
    wgt[warp * ATT_MAX_SPLITS + lane] = w;
    const float den = warp_sum_xor(w * pl);
    if (lane == 0) den_s[warp] = den;
  }
  __syncthreads();
  for (int i = tid; i < REP * HD; i += ATT_THREADS) {
    const int r = i / HD;
    if (i != tid) load_parts(i);
    float num = 0.f;
#pragma unroll
    for (int k = 0; k < ATT_MAX_SPLITS; ++k) num = fmaf(wgt[r * ATT_MAX_SPLITS + k], v[k], num);  // weight 0 beyond NSP
    out[static_cast<size_t>(h0 + r) * HD + element(i - r * HD)] = DT<T>::from_f(num / den_s[r]);
  }
}

// h_out = round(h + a) (a may be null: h_out = h, nothing written unless write_h), then
// x = round(h_out * rsqrt(mean(h_out^2) + eps)) * w.  Thread t owns elements t, t + blockDim.x, ...
// (at most MAXPT of them, kept in registers).  `store_x(i, value)` receives x.
constexpr int NORM_MAX_H = 8192;
template <int MAXPT> struct NormRegs {
  float v[MAXPT], wv[MAXPT];
};
// Part 1: the loads (and the add).  Kernels that also stream bulk copies call this BEFORE they
// request the copies: small loads issued behind hundreds of KB of bulk traffic of the same SM
// come back only when that traffic has drained.
template <typename T, int MAXPT>
__device__ __forceinline__ void norm_load(const T* h, const T* __restrict__ a, const T* __restrict__ w, int H,
                                          NormRegs<MAXPT>& r) {
  const int tid = threadIdx.x, nt = blockDim.x;
#pragma unroll
  for (int k = 0; k < MAXPT; ++k) {
    const int i = tid + k * nt;
    r.v[k] = 0.f;
    r.wv[k] = 0.f;
    if (i < H) {
      r.v[k] = DT<T>::to_f(h[i]);
      if (a) r.v[k] = DT<T>::round_f(r.v[k] + DT<T>::to_f(a[i]));
      r.wv[k] = DT<T>::to_f(w[i]);
    }
  }
}
// Part 2: h_out, the sum of squares, x.
template <typename T, int MAXPT, typename StoreX>
__device__ __forceinline__ void norm_finish(const NormRegs<MAXPT>& r, float eps, T* h_out, int H, float* red, StoreX store_x) {
  const int tid = threadIdx.x, nt = blockDim.x;
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < MAXPT; ++k) {
    const int i = tid + k * nt;
    if (i < H && h_out) h_out[i] = DT<T>::from_f(r.v[k]);
    ss = fmaf(r.v[k], r.v[k], ss);
  }
  const float tot = block_reduce<false>(ss, red);
  const float inv = rsqrtf(tot / static_cast<float>(H) + eps);
#pragma unroll
  for (int k = 0; k < MAXPT; ++k) {
    const int i = tid + k * nt;
    if (i < H) store_x(i, DT<T>::from_f(DT<T>::round_f(r.v[k] * inv) * r.wv[k]));
  }
}
template <typename T, int MAXPT, typename StoreX>
__device__ __forceinline__ void add_rmsnorm_block(const T* h, const T* __restrict__ a, const T* __restrict__ w, float eps,
                                                  T* h_out, int H, float* red, StoreX store_x) {
  NormRegs<MAXPT> r;
  norm_load<T, MAXPT>(h, a, w, H, r);
  norm_finish<T, MAXPT>(r, eps, h_out, H, red, store_x);
}

template <typename T>
__global__ void __launch_bounds__(NORM_THREADS) k_add_rmsnorm(const T* h, const T* __restrict__ a, const T* __restrict__ w,
                                                               float eps, T* h_out, T* __restrict__ x_out, int H) {
  __shared__ float red[32];
  pdl_wait();
  pdl_launch_dependents();
  add_rmsnorm_block<T, NORM_MAX_H / NORM_THREADS>(h, a, w, eps, a ? h_out : nullptr, H, red, [&](int i, T x) { x_out[i] = x; });
}

// y[n] = W[n,:] . x for a row-major W [N,H], with x either given (w_norm == null: x = h) or made
// on the fly as x = RMSNorm(h + a) * w_norm in every CTA (the vector is a few KB; recomputing it
// costs less than a kernel boundary).  CTA 0 also writes h + a to h_out and x to x_out (either
// may be null).  h_out must not alias h: other CTAs still read h.  A warp per output row, 16-byte
// loads, two batches of eight per lane in flight, the first of them while the norm is computed.
constexpr int GEMV_THREADS = 512;
constexpr int GEMV_BATCH = 8;  // 16-byte loads per lane and item
template <typename T>
__global__ void __launch_bounds__(GEMV_THREADS) k_norm_gemv(const T* __restrict__ h, const T* __restrict__ a,
                                                             const T* __restrict__ w_norm, float eps,
                                                             const T* __restrict__ W, T* __restrict__ y, T* h_out,
                                                             T* x_out, int H, int N) {
  constexpr int V = DT<T>::V;
  extern __shared__ __align__(128) unsigned char gsm[];
  T* x_s = reinterpret_cast<T*>(gsm);
  __shared__ float red[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nchunk = H / V;
  const int wpg = (GEMV_THREADS / 32) * gridDim.x;  // warps in the grid
  const int row0 = blockIdx.x * (GEMV_THREADS / 32) + warp;
  // A warp's work is a sequence of items: item it = (its row number it / nb, batch it % nb of that
  // row), a batch being GEMV_BATCH x 32 consecutive 16-byte chunks.  Two items are in flight.
  const int nb = (nchunk + 32 * GEMV_BATCH - 1) / (32 * GEMV_BATCH);
  const int nrows = row0 < N ? (N - 1 - row0) / wpg + 1 : 0;
  const int nitems = nrows * nb;
  auto load_item = [&](int it, uint4 (&buf)[GEMV_BATCH]) {
    const int r = it / nb, bi = it - r * nb;
    const uint4* wr = reinterpret_cast<const uint4*>(W + static_cast<size_t>(row0 + r * wpg) * H) + bi * 32 * GEMV_BATCH + lane;
    const int left = nchunk - bi * 32 * GEMV_BATCH - lane;
#pragma unroll
    for (int i = 0; i < GEMV_BATCH; ++i)
      if (32 * i < left) buf[i] = ld_stream16(wr + 32 * i);
  };
  float acc0 = 0.f, acc1 = 0.f;
  auto compute_item = [&](int it, const uint4 (&buf)[GEMV_BATCH]) {
    const int r = it / nb, bi = it - r * nb;
    const uint4* xs = reinterpret_cast<const uint4*>(x_s) + bi * 32 * GEMV_BATCH + lane;
    const int left = nchunk - bi * 32 * GEMV_BATCH - lane;
#pragma unroll
    for (int i = 0; i < GEMV_BATCH; ++i) {
      if (32 * i < left) {
        float wf[V], xf[V];
        Unpack<T>::run(buf[i], wf);
        Unpack<T>::run(xs[32 * i], xf);
        float t = 0.f;
#pragma unroll
        for (int v = 0; v < V; ++v) t = fmaf(xf[v], wf[v], t);
        if (i & 1) acc1 += t; else acc0 += t;
      }
    }
    if (bi == nb - 1) {  // the row is complete
      const float dot = warp_sum_xor(acc0 + acc1);
      if (lane == 0) y[row0 + r * wpg] = DT<T>::from_f(dot);
      acc0 = 0.f;
      acc1 = 0.f;
    }
  };
  uint4 bufa[GEMV_BATCH], bufb[GEMV_BATCH];
  pdl_wait();  // the preceding kernel may have written W
  pdl_launch_dependents();
  if (nitems > 0) load_item(0, bufa);  // in flight while the norm is computed
  if (w_norm) {
    const bool first = blockIdx.x == 0;
    add_rmsnorm_block<T, NORM_MAX_H / GEMV_THREADS>(h, a, w_norm, eps, first ? h_out : nullptr, H, red, [&](int i, T x) {
      x_s[i] = x;
      if (first && x_out) x_out[i] = x;
    });
  } else {
    for (int i = tid; i < nchunk; i += GEMV_THREADS) reinterpret_cast<uint4*>(x_s)[i] = reinterpret_cast<const uint4*>(h)[i];
  }
  __syncthreads();
  for (int it = 0; it < nitems; it += 2) {
    if (it + 1 < nitems) load_item(it + 1, bufb);
    compute_item(it, bufa);
    if (it + 2 < nitems) load_item(it + 2, bufa);
    if (it + 1 < nitems) compute_item(it + 1, bufb);
  }
}

// The same product when the CTA's share of W fits in shared memory (N * H elements over one CTA
// per SM, e.g. a 5120 x 3072 fp16 projection: 35 rows, 215 KB): every row is requested by a bulk
// copy before the norm is computed, so the whole matrix is in flight while the norm is
// computed, and each warp then reads its rows from shared memory.
// Dynamic shared memory: [0,128) one mbarrier per warp | x_s [H] | rows [rows_per_cta][H].
template <typename T>
__global__ void __launch_bounds__(GEMV_THREADS) k_norm_gemv_tma(const T* __restrict__ h, const T* __restrict__ a,
                                                                 const T* __restrict__ w_norm, float eps,
                                                                 const T* __restrict__ W, T* __restrict__ y, T* h_out,
                                                                 T* x_out, int H, int N, int rows_per_cta) {
  constexpr int V = DT<T>::V;
  constexpr int NW = GEMV_THREADS / 32;
  extern __shared__ __align__(128) unsigned char gsm[];
  __shared__ float red[32];
  uint64_t* bar = reinterpret_cast<uint64_t*>(gsm);
  T* x_s = reinterpret_cast<T*>(gsm + 128);
  const size_t row_bytes = static_cast<size_t>(H) * sizeof(T);
  unsigned char* rows = gsm + 128 + (row_bytes + 127) / 128 * 128;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nchunk = H / V;
  const int r0 = blockIdx.x * rows_per_cta;
  const int nr = max(0, min(rows_per_cta, N - r0));
  const int mine = warp < nr ? (nr - 1 - warp) / NW + 1 : 0;  // local rows warp, warp + NW, ...
  if (tid == 0) {
    for (int w = 0; w < NW; ++w) mbar_init(&bar[w], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // The preceding kernel may have written W, or write it still, so the rows are read behind the wait; until then they are
  // on their way into the L2, where they meet such writes.  Four layers of norm, attention, projection and norm (24 heads
  // of 128, 4000 tokens, fp16): 106.7 us without the prefetch, 104.5 with it (102.5 with the reads themselves ahead).
  for (int k = lane; k < mine; k += 32) bulk_prefetch_l2(W + static_cast<size_t>(r0 + warp + k * NW) * H, static_cast<uint32_t>(row_bytes));
  pdl_wait();
  pdl_launch_dependents();
  // the small loads of the prologue go first: behind the bulk copies they would come back last
  constexpr int MAXPT = NORM_MAX_H / GEMV_THREADS;
  NormRegs<MAXPT> nr_regs;
  uint4 xr[MAXPT / 4 + 1];
  if (w_norm) {
    norm_load<T, MAXPT>(h, a, w_norm, H, nr_regs);
  } else {
#pragma unroll
    for (int k = 0; k < MAXPT / 4 + 1; ++k)
      if (tid + k * GEMV_THREADS < nchunk) xr[k] = reinterpret_cast<const uint4*>(h)[tid + k * GEMV_THREADS];
  }
  if (mine > 0) {
    if (lane == 0) mbar_expect_tx(&bar[warp], static_cast<uint32_t>(mine * row_bytes));
    __syncwarp();
    for (int k = lane; k < mine; k += 32) {
      const int lr = warp + k * NW;
      bulk_load(rows + static_cast<size_t>(lr) * row_bytes, W + static_cast<size_t>(r0 + lr) * H, static_cast<uint32_t>(row_bytes),
                &bar[warp]);
    }
  }
  if (w_norm) {
    const bool first = blockIdx.x == 0;
    norm_finish<T, MAXPT>(nr_regs, eps, first ? h_out : nullptr, H, red, [&](int i, T x) {
      x_s[i] = x;
      if (first && x_out) x_out[i] = x;
    });
  } else {
#pragma unroll
    for (int k = 0; k < MAXPT / 4 + 1; ++k)
      if (tid + k * GEMV_THREADS < nchunk) reinterpret_cast<uint4*>(x_s)[tid + k * GEMV_THREADS] = xr[k];
  }
  __syncthreads();
  if (mine == 0) return;
  const bool ok = mbar_wait_bounded(&bar[warp], 0);
  for (int k = 0; k < mine; ++k) {
    const int lr = warp + k * NW;
    const uint4* wr = reinterpret_cast<const uint4*>(rows + static_cast<size_t>(lr) * row_bytes);
    float acc0 = 0.f, acc1 = 0.f;
    int c = lane;
    for (; c + 32 < nchunk; c += 64) {
      float w0[V], w1[V], x0[V], x1[V];
      Unpack<T>::run(wr[c], w0);
      Unpack<T>::run(wr[c + 32], w1);
      Unpack<T>::run(reinterpret_cast<const uint4*>(x_s)[c], x0);
      Unpack<T>::run(reinterpret_cast<const uint4*>(x_s)[c + 32], x1);
#pragma unroll
      for (int v = 0; v < V; ++v) {
        acc0 = fmaf(x0[v], w0[v], acc0);
        acc1 = fmaf(x1[v], w1[v], acc1);
      }
    }
    for (; c < nchunk; c += 32) {
      float w0[V], x0[V];
      Unpack<T>::run(wr[c], w0);
      Unpack<T>::run(reinterpret_cast<const uint4*>(x_s)[c], x0);
#pragma unroll
      for (int v = 0; v < V; ++v) acc0 = fmaf(x0[v], w0[v], acc0);
    }
    const float dot = warp_sum_xor(acc0 + acc1);
    // a copy that did not arrive within the wait limit must not pass for a result
    if (lane == 0) y[r0 + lr] = DT<T>::from_f(ok ? dot : __int_as_float(0x7fc00000));
  }
}

// Logits to fp32 and their argmax over the whole chip; the block that arrives last moves the decode state on.  A key is
// the value in ascending unsigned order with the complemented index below it, so one 64-bit maximum finds the first of
// the largest.  128256 fp16 logits: torch's conversion, copy, one-block argmax (30 us) and four small ops were 43 us of a
// token, the kernel takes 5.7.
constexpr int FIN_THREADS = 256;
template <typename T>
__global__ void __launch_bounds__(FIN_THREADS) k_decode_finish(const T* logits, long long V, float* logits_out, long long* token,
                                                                long long* pos, const long long* __restrict__ gen_base,
                                                                long long* generated, long long max_len,
                                                                unsigned long long* __restrict__ ws) {
  __shared__ unsigned long long s_best[FIN_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  pdl_launch_dependents();
  unsigned long long best = 0;
  for (long long i = static_cast<long long>(blockIdx.x) * FIN_THREADS + tid; i < V; i += static_cast<long long>(gridDim.x) * FIN_THREADS) {
    const float v = DT<T>::to_f(logits[i]);
    logits_out[i] = v;
    const uint32_t u = __float_as_uint(v == 0.f ? 0.f : v);  // -0 equals +0
    const uint32_t key = v != v ? 0xffffffffu : (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    const unsigned long long k = (static_cast<unsigned long long>(key) << 32) | static_cast<uint32_t>(~static_cast<uint32_t>(i));
    best = k > best ? k : best;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, best, off);
    best = o > best ? o : best;
  }
  if (lane == 0) s_best[warp] = best;
  __syncthreads();
  if (tid != 0) return;
#pragma unroll
  for (int w = 1; w < FIN_THREADS / 32; ++w) best = s_best[w] > best ? s_best[w] : best;
  atomicMax(ws, best);
  __threadfence();
  unsigned int* arrived = reinterpret_cast<unsigned int*>(ws + 1);
  if (atomicAdd(arrived, 1u) != gridDim.x - 1) return;
  __threadfence();
  const long long t = static_cast<uint32_t>(~static_cast<uint32_t>(__ldcg(ws)));
  *ws = 0ull;
  *arrived = 0u;
  const long long p = *pos + 1;
  *pos = p;
  *token = t;
  const long long at = p - *gen_base;
  if (at >= 0 && at < max_len) generated[at] = t;
}
template <typename T>
static int launch_decode_finish(const void* logits, long long V, float* logits_out, long long* token, long long* pos,
                                const long long* gen_base, long long* generated, long long max_len, void* ws, cudaStream_t s) {
  const unsigned grid = static_cast<unsigned>(std::min<long long>(num_sms(), (V + FIN_THREADS - 1) / FIN_THREADS));
  STX_CUDA(launch_pdl(k_decode_finish<T>, dim3(grid), dim3(FIN_THREADS), 0, s, static_cast<const T*>(logits), V, logits_out,
                      token, pos, gen_base, generated, max_len, static_cast<unsigned long long*>(ws)));
  return STX_OK;
}

template <typename T>
static int launch_add_rmsnorm(const void* h, const void* a, const void* w, float eps, void* h_out, void* x_out, int H, cudaStream_t s) {
  STX_CUDA(launch_pdl(k_add_rmsnorm<T>, dim3(1), dim3(NORM_THREADS), 0, s, static_cast<const T*>(h), static_cast<const T*>(a),
                      static_cast<const T*>(w), eps, static_cast<T*>(h_out), static_cast<T*>(x_out), H));
  return STX_OK;
}

template <typename T>
static int launch_norm_gemv(const void* h, const void* a, const void* w_norm, float eps, const void* W, void* y, void* h_out,
                            void* x_out, int H, int N, cudaStream_t s) {
  const int warps = GEMV_THREADS / 32;
  const int sms = num_sms();
  // A CTA of this size needs an SM to itself; a few SMs are left to kernels that run beside it on
  // other streams (the weight cache's upkeep), or one CTA would wait for a second wave.
  const int target = std::max(1, sms - 4);
  const int rows_per_cta = (N + target - 1) / target;
  const size_t row_bytes = static_cast<size_t>(H) * sizeof(T);
  const size_t smem_tma = 128 + (row_bytes + 127) / 128 * 128 + static_cast<size_t>(rows_per_cta) * row_bytes;
  const size_t budget = 227 * 1024 - 1024;  // per-block limit less the kernel's static shared memory
  if (smem_tma <= budget) {
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
      STX_CUDA(cudaFuncSetAttribute(k_norm_gemv_tma<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(budget)));
      attr_set[dev] = true;
    }
    const unsigned grid = static_cast<unsigned>((N + rows_per_cta - 1) / rows_per_cta);
    STX_CUDA(launch_pdl(k_norm_gemv_tma<T>, dim3(grid), dim3(GEMV_THREADS), smem_tma, s, static_cast<const T*>(h), static_cast<const T*>(a),
                        static_cast<const T*>(w_norm), eps, static_cast<const T*>(W), static_cast<T*>(y), static_cast<T*>(h_out),
                        static_cast<T*>(x_out), H, N, rows_per_cta));
  } else {
    const int want = (N + warps - 1) / warps;
    const unsigned grid = static_cast<unsigned>(std::min(want, sms));  // one CTA per SM: the norm is made once per CTA
    STX_CUDA(launch_pdl(k_norm_gemv<T>, dim3(grid), dim3(GEMV_THREADS), row_bytes, s, static_cast<const T*>(h), static_cast<const T*>(a),
                        static_cast<const T*>(w_norm), eps, static_cast<const T*>(W), static_cast<T*>(y), static_cast<T*>(h_out),
                        static_cast<T*>(x_out), H, N));
  }
  return STX_OK;
}

template <typename T, int HD, int REP>
static int launch_attn(const void* qkv, const float* cos_t, const float* sin_t, const long long* pos, void* k_cache, void* v_cache,
                       void* out, int nh, int nkv, long long max_len, float scale, void* workspace, cudaStream_t s) {
  constexpr int smem = static_cast<int>(sizeof(float) * ((REP + 2) * HD + ATT_THREADS / 32 * REP * (HD + 2)));
  if (smem > 48 * 1024) {
    static bool attr_set[64] = {};
    int dev = 0;
    STX_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
      STX_CUDA(cudaFuncSetAttribute(k_attn_decode<T, HD, REP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      attr_set[dev] = true;
    }
  }
  const int groups = nh / REP;
  const int nsp = std::max(1, std::min(ATT_MAX_SPLITS, num_sms() / groups));  // one CTA per SM
  STX_CUDA(launch_pdl(k_attn_decode<T, HD, REP>, dim3(groups, nsp), dim3(ATT_THREADS), smem, s, static_cast<const T*>(qkv), cos_t, sin_t,
                      pos, static_cast<T*>(k_cache), static_cast<T*>(v_cache), static_cast<T*>(out), nh, nkv, max_len, scale,
                      static_cast<unsigned char*>(workspace)));
  return STX_OK;
}

// Query heads of a CTA: the largest divisor of the heads per cache head up to 4, four only where eight groups are left.  With
// fewer, the work of a tile for four heads is what a CTA waits for, and reading a cache head once more costs less: 16 heads
// on 2 of 128, four layers of the glue at 200 tokens 70 -> 60 us, at 4000 76 -> 72; 16 on 4 of 64 59.7 -> 51.4 and 63.8 -> 60.
template <typename T, int HD>
static int launch_attn_rep(const void* qkv, const float* cos_t, const float* sin_t, const long long* pos, void* k_cache, void* v_cache,
                           void* out, int nh, int nkv, long long max_len, float scale, void* ws, cudaStream_t s) {
  const int rep = nh / nkv;
  if (rep % 4 == 0 && nh >= 32) return launch_attn<T, HD, 4>(qkv, cos_t, sin_t, pos, k_cache, v_cache, out, nh, nkv, max_len, scale, ws, s);
  if (rep % 3 == 0) return launch_attn<T, HD, 3>(qkv, cos_t, sin_t, pos, k_cache, v_cache, out, nh, nkv, max_len, scale, ws, s);
  if (rep % 2 == 0) return launch_attn<T, HD, 2>(qkv, cos_t, sin_t, pos, k_cache, v_cache, out, nh, nkv, max_len, scale, ws, s);
  return launch_attn<T, HD, 1>(qkv, cos_t, sin_t, pos, k_cache, v_cache, out, nh, nkv, max_len, scale, ws, s);
}

}  // namespace stx

using namespace stx;

extern "C" {

int stx_attn_decode_workspace_bytes(int n_heads, int head_dim, int64_t* bytes_out) {
  STX_CHECK_ARG(bytes_out, "stx_attn_decode_workspace_bytes: null pointer");
  STX_CHECK_ARG(n_heads > 0 && n_heads <= 1024 && head_dim > 0, "stx_attn_decode_workspace_bytes: bad shape");
  *bytes_out = static_cast<int64_t>(ATT_COUNTER_BYTES + sizeof(float) * static_cast<size_t>(n_heads) * ATT_MAX_SPLITS * att_part_floats(head_dim));
  return STX_OK;
}

int stx_attn_decode(const void* qkv, const float* cos_table, const float* sin_table, const int64_t* pos_dev, void* k_cache,
                    void* v_cache, void* out, int n_heads, int n_kv_heads, int head_dim, int64_t max_len, int dtype,
                    void* workspace, void* stream) {
  STX_CHECK_ARG(qkv && cos_table && sin_table && pos_dev && k_cache && v_cache && out && workspace,
                "stx_attn_decode: null pointer");
  STX_CHECK_ARG(n_heads <= 1024, "stx_attn_decode: more than 1024 heads");
  STX_CHECK_ARG(dtype == STX_F32 || dtype == STX_F16 || dtype == STX_BF16, "stx_attn_decode: bad dtype %d", dtype);
  STX_CHECK_ARG(head_dim == 64 || head_dim == 128 || head_dim == 256, "stx_attn_decode: head_dim %d is not 64, 128 or 256",
                head_dim);
  STX_CHECK_ARG(n_heads > 0 && n_kv_heads > 0 && n_heads % n_kv_heads == 0,
                "stx_attn_decode: %d query heads do not divide into %d key/value heads", n_heads, n_kv_heads);
  STX_CHECK_ARG(max_len > 0 && max_len <= 8192, "stx_attn_decode: max_len %lld outside 1..8192", static_cast<long long>(max_len));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float scale = 1.0f / sqrtf(static_cast<float>(head_dim));
  const long long* pos = reinterpret_cast<const long long*>(pos_dev);
#define STX_ATT_ARGS qkv, cos_table, sin_table, pos, k_cache, v_cache, out, n_heads, n_kv_heads, static_cast<long long>(max_len), scale, workspace, s
#define STX_ATT_HD(T)                                                                  \
  (head_dim == 64 ? launch_attn_rep<T, 64>(STX_ATT_ARGS)                               \
                  : head_dim == 128 ? launch_attn_rep<T, 128>(STX_ATT_ARGS) : launch_attn_rep<T, 256>(STX_ATT_ARGS))
  switch (dtype) {
    case STX_F32: return STX_ATT_HD(float);
    case STX_F16: return STX_ATT_HD(__half);
    default: return STX_ATT_HD(__nv_bfloat16);
  }
#undef STX_ATT_HD
#undef STX_ATT_ARGS
}

int stx_add_rmsnorm(const void* h, const void* a, const void* w, float eps, void* h_out, void* x_out, int64_t H, int dtype,
                    void* stream) {
  STX_CHECK_ARG(h && w && x_out, "stx_add_rmsnorm: null pointer");
  STX_CHECK_ARG(!a || h_out, "stx_add_rmsnorm: h_out is required when a is given");
  STX_CHECK_ARG(dtype == STX_F32 || dtype == STX_F16 || dtype == STX_BF16, "stx_add_rmsnorm: bad dtype %d", dtype);
  STX_CHECK_ARG(H > 0 && H <= NORM_MAX_H, "stx_add_rmsnorm: H=%lld outside 1..%d", static_cast<long long>(H), NORM_MAX_H);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int Hi = static_cast<int>(H);
  switch (dtype) {
    case STX_F32: return launch_add_rmsnorm<float>(h, a, w, eps, h_out, x_out, Hi, s);
    case STX_F16: return launch_add_rmsnorm<__half>(h, a, w, eps, h_out, x_out, Hi, s);
    default: return launch_add_rmsnorm<__nv_bfloat16>(h, a, w, eps, h_out, x_out, Hi, s);
  }
}

int stx_decode_finish(const void* logits, int64_t V, int dtype, float* logits_out, int64_t* token, int64_t* pos,
                      const int64_t* gen_base, int64_t* generated, int64_t max_len, void* workspace, void* stream) {
  STX_CHECK_ARG(logits && logits_out && token && pos && gen_base && generated && workspace, "stx_decode_finish: null pointer");
  STX_CHECK_ARG(V > 0 && V <= 0x7fffffff, "stx_decode_finish: V=%lld out of range", static_cast<long long>(V));
  STX_CHECK_ARG(dtype == STX_F32 || dtype == STX_F16 || dtype == STX_BF16, "stx_decode_finish: bad dtype %d", dtype);
  STX_CHECK_ARG((reinterpret_cast<uintptr_t>(workspace) & 7) == 0, "stx_decode_finish: workspace must be 8-byte aligned");
  static_assert(sizeof(int64_t) == sizeof(long long), "token and position types");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  long long* t = reinterpret_cast<long long*>(token);
  long long* p = reinterpret_cast<long long*>(pos);
  const long long* g = reinterpret_cast<const long long*>(gen_base);
  long long* out = reinterpret_cast<long long*>(generated);
  switch (dtype) {
    case STX_F32: return launch_decode_finish<float>(logits, V, logits_out, t, p, g, out, max_len, workspace, s);
    case STX_F16: return launch_decode_finish<__half>(logits, V, logits_out, t, p, g, out, max_len, workspace, s);
    default: return launch_decode_finish<__nv_bfloat16>(logits, V, logits_out, t, p, g, out, max_len, workspace, s);
  }
}

int stx_norm_gemv(const void* h, const void* a, const void* w_norm, float eps, const void* W, void* y, void* h_out,
                  void* x_out, int64_t H, int64_t N, int dtype, void* stream) {
  STX_CHECK_ARG(h && W && y, "stx_norm_gemv: null pointer");
  STX_CHECK_ARG(w_norm || (!a && !h_out && !x_out), "stx_norm_gemv: a, h_out and x_out need w_norm");
  STX_CHECK_ARG(!h_out || h_out != h, "stx_norm_gemv: h_out must not alias h");
  STX_CHECK_ARG(dtype == STX_F32 || dtype == STX_F16 || dtype == STX_BF16, "stx_norm_gemv: bad dtype %d", dtype);
  const int64_t V = 16 / static_cast<int64_t>(dtype_size(dtype));
  STX_CHECK_ARG(H > 0 && H <= NORM_MAX_H && H % V == 0, "stx_norm_gemv: H=%lld must be a multiple of %lld, at most %d",
                static_cast<long long>(H), static_cast<long long>(V), NORM_MAX_H);
  STX_CHECK_ARG(N > 0 && N <= (1 << 30), "stx_norm_gemv: N=%lld out of range", static_cast<long long>(N));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int Hi = static_cast<int>(H), Ni = static_cast<int>(N);
  switch (dtype) {
    case STX_F32: return launch_norm_gemv<float>(h, a, w_norm, eps, W, y, h_out, x_out, Hi, Ni, s);
    case STX_F16: return launch_norm_gemv<__half>(h, a, w_norm, eps, W, y, h_out, x_out, Hi, Ni, s);
    default: return launch_norm_gemv<__nv_bfloat16>(h, a, w_norm, eps, W, y, h_out, x_out, Hi, Ni, s);
  }
}

}  // extern "C"
