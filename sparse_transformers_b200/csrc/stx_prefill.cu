// Sparse gated MLP over packed active rows for row blocks (9 rows and more) in fp16/bf16: here the
// gathered weights form a dense contraction, so it runs on the 5th-generation tensor cores.
//
//   GEMM 1   [G ; U] = [Wg ; Wu] · X^T      M = neurons (gate and up rows), N = tokens, k = H
//            epilogue: A = act(G) * U -> fp16/bf16 scratch [tokens, K8] (and combined_buf)
//   GEMM 2   out^T  = Wd^T · A^T            M = H, N = tokens, k = neurons
//
// The weights are the M side and the tokens the N side: a few dozen tokens then cost an N of 32..128
// and not a 128-row tile, an odd number of tokens is padded to the next 32 and not to 256, and the
// packed down rows [K, H] are an M-major operand as they lie (the k-major form needs a transposed
// copy of them on every call: 26 us of a 166 us layer at 64 tokens and K = 8700, 90 MB at K = 11008).
//
// One kernel, k_pair_gemm<T, MODE>: a cluster of two CTAs (one SM pair) works on tiles of 256 M rows
// x N tokens with tcgen05.mma.cta_group::2 (M = 256): each CTA holds its 128 M rows of A and half of
// the tokens, so the token operand crosses into shared memory once per pair.  The grid is one pair
// per SM pair; a pair walks the tiles, two accumulators of 256 TMEM columns alternate, so that the
// epilogue of a tile runs while the next one is multiplied.
//   MODE 0: a CTA's 128 M rows are the gate rows (0..63) and the up rows (64..127) of the same 64
//           neurons (fewer when the neurons are shared out evenly, see pf_plan())
//   MODE 1: 128 columns of H, loaded as two [64 neurons][64 columns] boxes, M-major
//   warps 0, 6, 7  producers: TMA tiled loads (128-byte swizzle) of a 64-wide k block per stage, one
//               box of the stage each (gate / up rows or the two column boxes / tokens): a warp
//               issues about one box per 85 ns, and three in a row made the issue the bottleneck
//               (64 tokens, 8700 neurons of 4096: GEMM 1 57 -> 44 us).  Both CTAs' copies complete on the
//               even CTA's barrier
//   warp 1      even CTA: issues the MMAs from one lane; tcgen05.commit (multicast to both CTAs)
//               releases a stage / publishes an accumulator.  Allocates and frees tensor memory.
//   warps 2..5 and 8..11  epilogue, every other 32 tokens each: tcgen05.ld 32 lanes x 32 tokens; a
//               warp's 32 lanes are neighbouring columns of the result, so every store is one contiguous
//               64- or 128-byte piece whatever the alignment of the row.
// Edges are handled by TMA zero fill on loads and by masked stores; no load is multicast.
// Every mbarrier wait is bounded; a role whose wait expired records DEV_TIMEOUT, stops, and the
// others run out of their own waits in turn, so that TMEM is always freed.
#include "stx_common.cuh"

#include <cuda.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>

namespace stx {

constexpr int PF_BK = 64;
constexpr int PF_THREADS = 384;
constexpr int PF_TW = 128;                               // neurons of a MODE 0 tile (64 per CTA)
constexpr int PF_HW = 256;                               // columns of H of a MODE 1 tile (128 per CTA)
constexpr int PF_MAX_N = 256;                            // tokens of a tile
constexpr int PF_MAX_STAGES = 12;
constexpr uint32_t PF_A_BYTES = 128 * PF_BK * 2;         // a CTA's A tile of one stage
constexpr uint32_t PF_XCH_BYTES = 2 * 2 * 2 * 16 * 32 * 4;  // [epilogue set][warp pair][g|u][16 tokens][32 lanes] fp32
constexpr uint32_t PF_SMEM = 226 * 1024;
constexpr uint32_t PF_SMEM_FEW = 148 * 1024;
constexpr uint32_t PF_WAIT_LIMIT = 1u << 22;
constexpr int PF_GROUP = 8;                              // token tiles that walk the weights together

struct PfArgs {
  int M;               // tokens
  int N;               // MODE 0: neurons K ; MODE 1: columns H
  int Kd;              // contraction length: H ; K
  int n_tok;           // tokens of a tile (multiple of 32)
  int tok_tiles;
  int pairs;           // SM pairs the tiles are shared out over
  int even;            // MODE 0: share the neurons out evenly over whole waves (one token tile)
  int splits;          // MODE 1: contraction splits
  int stages;
  void* a_out;         // MODE 0: activations [M, ld_out] or null; MODE 1: output [M, ld_out]
  int ld_out;
  void* combined;      // MODE 0, optional: [M, 2K]
  int act;
  int* status;
  // Optional device-side count of valid rows of the packed weights (a weight cache's K): MODE 0
  // covers *k_dev neurons rounded up to a k-block, zeros beyond *k_dev; MODE 1 stops its contraction there.
  const int* k_dev;
  int early;           // MODE 1: the weights do not depend on the preceding kernel, fetch them while it ends
  int tmem_cols;       // two accumulators of n_tok columns, as a power of two
  float* part;         // MODE 1 with splits: part[split][M][ld_out], summed by the caller in split order
};

__device__ __forceinline__ uint32_t pf_smem(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void pf_mbar_init(uint64_t* b, uint32_t n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(pf_smem(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void pf_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(pf_smem(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t pf_mapa(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(pf_smem(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void pf_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool pf_try_wait(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(pf_smem(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool pf_wait(uint64_t* b, uint32_t parity) {
  for (uint32_t it = 0; it < PF_WAIT_LIMIT; ++it) {
    if (pf_try_wait(b, parity)) return true;
    if (it > 1024) __nanosleep(64);
  }
  return false;
}
// bar: shared::cluster address of the even CTA's barrier
__device__ __forceinline__ void pf_tma_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          pf_smem(dst)),
      "l"(map), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
// Operand tile with 128-byte swizzle.  K-major: rows of 64 k elements, 8-row groups 1024 bytes apart (lbo unused).
// M-major: [64 k][64 m elements] boxes, 8-k groups 1024 bytes apart, the next 64 m elements lbo bytes further.
__device__ __forceinline__ uint64_t pf_smem_desc(uint32_t addr, uint32_t lbo) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3ffffu) >> 4);   // start address
  d |= static_cast<uint64_t>(lbo >> 4) << 16;            // leading byte offset
  d |= static_cast<uint64_t>(1024 >> 4) << 32;           // stride byte offset
  d |= static_cast<uint64_t>(1) << 46;                   // descriptor version (Blackwell)
  d |= static_cast<uint64_t>(2) << 61;                   // SWIZZLE_128B
  return d;
}
__device__ __forceinline__ void pf_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at this offset in both CTAs once the MMAs issued so far are done.
__device__ __forceinline__ void pf_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(pf_smem(bar)),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}
__device__ __forceinline__ void pf_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Boxes of 64, 32, 16 and 8 rows of the same weights.
struct PfWeightMaps {
  CUtensorMap m[4];
};

// Box (index in PfWeightMaps) of at least `rows` rows.  It may fetch rows beyond the CTA's share (its neighbour's, on
// their way through the L2 anyway); their products land in accumulator lanes that nobody reads.  A CTA without rows
// fetches eight as well: every producer has a part in every stage, so the ring can never run past one of them (a
// producer that nothing waits for can fall two uses of a stage behind, where the parity of its barrier reads as pending).
__device__ __forceinline__ int pf_box(int rows) { return rows > 32 ? 0 : rows > 16 ? 1 : rows > 8 ? 2 : 3; }

// One tile of a pair's walk.
struct PfTile {
  int m0, m_rows0, m_rows1;  // first M row of the tile (neuron / column); neurons of the even and the odd CTA
  int tok0;                  // first token
  int zi, kb_lo, nkb;        // contraction split and its k-blocks
};

// How the tiles of a launch are laid out.  Host-visible sizes give the grid; the device-side K decides here.
struct PfPlan {
  int w_tiles, tw, cover, tiles;  // M tiles, M rows per tile, M rows to cover, tiles in all
  int nkb_all, splits, tok_tiles, n_tok;
};

template <int MODE>
__device__ __forceinline__ PfPlan pf_plan(const PfArgs& p, int k_valid) {
  PfPlan q;
  q.splits = MODE == 1 ? max(1, p.splits) : 1;
  q.tok_tiles = p.tok_tiles;
  q.n_tok = p.n_tok;
  if (MODE == 0) {
    // with a device-side K the rows up to the end of its k-block are GEMM 2's operand too: zeros
    q.cover = p.k_dev ? min(p.N, (k_valid + PF_BK - 1) / PF_BK * PF_BK) : p.N;
    q.w_tiles = (q.cover + PF_TW - 1) / PF_TW;
    q.tw = PF_TW;
    if (p.even && q.cover > 0) {
      // One token tile: every weight row is read once and the launch is bound by HBM, so all pairs
      // take the same number of neurons (in 8s) instead of full tiles and a nearly empty last wave.
      const int want = (q.w_tiles + p.pairs - 1) / p.pairs * p.pairs;
      q.tw = max(16, ((q.cover + want - 1) / want + 7) / 8 * 8);
      q.w_tiles = (q.cover + q.tw - 1) / q.tw;
    }
    q.nkb_all = (p.Kd + PF_BK - 1) / PF_BK;
  } else {
    q.cover = p.N;
    q.tw = PF_HW;
    q.w_tiles = (p.N + PF_HW - 1) / PF_HW;
    q.nkb_all = ((p.k_dev ? min(p.Kd, k_valid) : p.Kd) + PF_BK - 1) / PF_BK;
  }
  q.tiles = q.w_tiles * q.tok_tiles * q.splits;
  return q;
}

template <int MODE>
__device__ __forceinline__ PfTile pf_tile(const PfPlan& q, int it) {
  PfTile t;
  const int per_split = q.w_tiles * q.tok_tiles;
  t.zi = it / per_split;
  const int i = it - t.zi * per_split;
  // PF_GROUP token tiles walk the weights together: what is in flight shares both operands in the L2
  const int g = i / (PF_GROUP * q.w_tiles);
  const int gn = min(PF_GROUP, q.tok_tiles - g * PF_GROUP);
  const int rem = i - g * PF_GROUP * q.w_tiles;
  const int w = rem / gn;
  t.tok0 = (g * PF_GROUP + rem - w * gn) * q.n_tok;
  t.m0 = w * q.tw;
  if (MODE == 0) {
    const int n8 = (min(q.tw, q.cover - t.m0) + 7) / 8;  // groups of 8 neurons
    t.m_rows0 = (n8 + 1) / 2 * 8;
    t.m_rows1 = n8 / 2 * 8;
  } else {
    t.m_rows0 = t.m_rows1 = 128;
  }
  t.kb_lo = static_cast<int>(static_cast<long long>(q.nkb_all) * t.zi / q.splits);
  t.nkb = static_cast<int>(static_cast<long long>(q.nkb_all) * (t.zi + 1) / q.splits) - t.kb_lo;
  return t;
}

// tmA[i]: weights, box 64 k x (64 >> i) rows (MODE 0) / [0] only, 64 columns x 64 k rows (MODE 1); tmB: tokens, box
// 64 x n_tok/2.  Dynamic shared memory (1024-byte aligned): stages x (A tile | token tile), exchange buffers of the
// epilogue, then full[S], empty[S], acc_full[2], acc_empty[2], TMEM base address.
template <typename T, int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PF_THREADS, 1)
k_pair_gemm(const __grid_constant__ PfWeightMaps tmA, const __grid_constant__ CUtensorMap tmB, const PfArgs p) {
  extern __shared__ unsigned char pf_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(pf_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int S = p.stages;
  const uint32_t b_bytes = static_cast<uint32_t>(p.n_tok / 2) * (PF_BK * 2);
  const uint32_t stage_bytes = PF_A_BYTES + b_bytes;  // n_tok/2 is a multiple of 16: 1024-byte aligned stages
  float* xch = reinterpret_cast<float*>(smem + static_cast<size_t>(S) * stage_bytes);
  uint64_t* full = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(xch) + PF_XCH_BYTES);
  uint64_t* empty = full + S;
  uint64_t* acc_full = empty + S;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      pf_mbar_init(&full[s], 1);
      pf_mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      pf_mbar_init(&acc_full[b], 1);
      pf_mbar_init(&acc_empty[b], 16);  // eight epilogue warps of either CTA
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // tensor memory: this warp of both CTAs allocates, the same warps free
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(pf_smem(tmem_slot)), "r"(p.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  if (!(MODE == 1 && p.early && (warp == 0 || warp == 6))) {
    pdl_wait();
    pdl_launch_dependents();
  }

  const uint32_t full0 = pf_mapa(full, 0);  // the even CTA's barriers
  const int k_valid = p.k_dev ? min(__ldcg(p.k_dev), MODE == 0 ? p.N : p.Kd) : (MODE == 0 ? p.N : p.Kd);
  const PfPlan plan = pf_plan<MODE>(p, k_valid);
  bool timed_out = false;

  if (warp == 0 || warp == 6 || warp == 7) {
    // ------------------------------------------------------------------ TMA producers
    if (lane == 0) {
      const int part = warp == 0 ? 0 : warp - 5;  // 0, 1: the halves of the A tile, 2: tokens
      int s = 0;
      uint32_t phase = 1;  // the first round finds every stage free
      for (int it = pair; it < plan.tiles && !timed_out; it += npairs) {
        const PfTile t = pf_tile<MODE>(plan, it);
        const int box0 = pf_box(t.m_rows0), box1 = pf_box(t.m_rows1);
        const uint32_t bytes = (MODE == 0 ? ((64u >> box0) + (64u >> box1)) * (2 * PF_BK * 2) : 2 * PF_A_BYTES) + 2 * b_bytes;
        const int box = rank ? box1 : box0;
        const int m0 = MODE == 0 ? t.m0 + (rank ? t.m_rows0 : 0) + (part == 1 ? p.N : 0)
                                 : t.m0 + static_cast<int>(rank) * 128 + part * 64;
        const int tok = t.tok0 + static_cast<int>(rank) * (p.n_tok / 2);
        const CUtensorMap* map = part == 2 ? &tmB : &tmA.m[MODE == 0 ? box : 0];
        // One token tile: all pairs stream weights at once, and rows of a power of two of bytes would have every one of
        // them ask for the same columns at the same time; each starts at another k block instead (GEMM 1 of 64 tokens,
        // 8700 neurons of 4096: 44.4 -> 41.5 us)
        int k = (MODE == 0 && p.even ? (it * 37) % t.nkb : t.kb_lo) * PF_BK;
        for (int kb = 0; kb < t.nkb; ++kb) {
          if (!pf_wait(&empty[s], phase)) {
            timed_out = true;
            break;
          }
          unsigned char* dst = smem + static_cast<size_t>(s) * stage_bytes + (part == 2 ? PF_A_BYTES : part * 8192u);
          if (rank == 0 && part == 0) pf_expect_tx(&full[s], bytes);
          if (part == 2) pf_tma_2d(dst, map, k, tok, full0 + s * 8);
          else if (MODE == 0) pf_tma_2d(dst, map, k, m0, full0 + s * 8);
          else pf_tma_2d(dst, map, m0, k, full0 + s * 8);
          k += PF_BK;
          if (MODE == 0 && k >= t.nkb * PF_BK) k = 0;
          if (++s == S) {
            s = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (even CTA)
    if (rank == 0 && lane == 0) {
      // instruction descriptor: D = f32, A/B = f16 or bf16, A M-major in MODE 1, M = 256
      const uint32_t fmt = DT<T>::id == STX_BF16 ? 1u : 0u;
      const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((MODE == 1 ? 1u : 0u) << 15) |
                             (static_cast<uint32_t>(p.n_tok >> 3) << 17) | (static_cast<uint32_t>(256 >> 4) << 24);
      constexpr uint32_t A_STEP = MODE == 0 ? 32 : 2048;  // bytes of 16 k elements inside the A tile
      int s = 0, na = 0;
      uint32_t phase = 0;
      for (int it = pair; it < plan.tiles && !timed_out; it += npairs) {
        const PfTile t = pf_tile<MODE>(plan, it);
        if (t.nkb == 0) continue;
        const int buf = na & 1;
        if (na >= 2 && !pf_wait(&acc_empty[buf], ((na >> 1) - 1) & 1)) {
          timed_out = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int kb = 0; kb < t.nkb; ++kb) {
          if (!pf_wait(&full[s], phase)) {
            timed_out = true;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t st = pf_smem(smem + static_cast<size_t>(s) * stage_bytes);
          const uint64_t da = pf_smem_desc(st, MODE == 0 ? 16 : 8192), db = pf_smem_desc(st + PF_A_BYTES, 16);
#pragma unroll
          for (int kk = 0; kk < PF_BK / 16; ++kk)
            pf_mma(tmem_base + buf * p.n_tok, da + (kk * A_STEP >> 4), db + (kk * 32 >> 4), idesc, (kb | kk) != 0);
          pf_commit(&empty[s]);
          if (++s == S) {
            s = 0;
            phase ^= 1;
          }
        }
        if (timed_out) break;
        pf_commit(&acc_full[buf]);
        ++na;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps 2..5, 8..11
    const int lg = warp & 3;  // TMEM lane group this warp may read
    const int set = warp >> 3;
    const int pair_bar = 1 + (lg & 1) + 2 * set;  // the gate and the up warp of the same neurons
    T* out = static_cast<T*>(p.a_out);
    T* comb = static_cast<T*>(p.combined);
    const uint32_t acc_empty0[2] = {pf_mapa(&acc_empty[0], 0), pf_mapa(&acc_empty[1], 0)};
    int na = 0;
    for (int it = pair; it < plan.tiles && !timed_out; it += npairs) {
      const PfTile t = pf_tile<MODE>(plan, it);
      const int buf = na & 1;
      const int ntok = min(p.n_tok, p.M - t.tok0);
      if (t.nkb > 0) {
        timed_out = __any_sync(0xffffffffu, !pf_wait(&acc_full[buf], (na >> 1) & 1));
        if (MODE == 0) {  // the two warps of a pair leave the loop together
          int dead = timed_out;
          asm volatile(
              "{\n\t.reg .pred a, b;\n\tsetp.ne.s32 a, %1, 0;\n\t"
              "barrier.cta.red.or.pred b, %2, 64, a;\n\tselp.s32 %0, 1, 0, b;\n\t}"
              : "=r"(dead)
              : "r"(dead), "r"(pair_bar)
              : "memory");
          timed_out = dead != 0;
        }
        if (timed_out) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(lg * 32) << 16) + buf * p.n_tok;
      if (MODE == 0) {
        const int nl = (lg & 1) * 32 + lane;  // neuron inside the CTA's share
        const int j = t.m0 + (rank ? t.m_rows0 : 0) + nl;
        const bool mine = nl < (rank ? t.m_rows1 : t.m_rows0) && j < plan.cover;
        const bool is_up = lg >= 2;
        float* xp = xch + (2 * set + (lg & 1)) * 1024;
        float* give = xp + (is_up ? 512 : 0);
        const float* take = xp + (is_up ? 0 : 512);
        // gate warps finish tokens 0..15 of a chunk, up warps tokens 16..31: each hands the other half over
#pragma unroll 1
        for (int c = 32 * set; c < ntok; c += 64) {
          float v[32];
          pf_ld32(taddr + c, v);
          if (c >= 64) asm volatile("barrier.cta.sync %0, 64;" ::"r"(pair_bar) : "memory");  // the last chunk has been read
          if (is_up) {
#pragma unroll
            for (int e = 0; e < 16; ++e) give[e * 32 + lane] = v[e];
          } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) give[e * 32 + lane] = v[16 + e];
          }
          asm volatile("barrier.cta.sync %0, 64;" ::"r"(pair_bar) : "memory");
          if (mine) {
            const int tb = c + (is_up ? 16 : 0);
            const size_t row0 = static_cast<size_t>(t.tok0 + tb);
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const float other = take[e * 32 + lane];
              const float g = is_up ? other : v[e], u = is_up ? v[16 + e] : other;
              if (tb + e < ntok) {
                const T a = DT<T>::from_f(j < k_valid ? apply_act(p.act, g) * u : 0.f);
                if (out) out[(row0 + e) * p.ld_out + j] = a;
                if (comb) {
                  T* cr = comb + (row0 + e) * (2 * static_cast<size_t>(p.N)) + j;
                  cr[0] = a;
                  cr[p.N] = DT<T>::from_f(u);
                }
              }
            }
          }
        }
      } else {
        const int col = t.m0 + static_cast<int>(rank) * 128 + lg * 32 + lane;
#pragma unroll 1
        for (int c = 32 * set; c < ntok; c += 64) {
          float v[32];
          if (t.nkb > 0) {
            pf_ld32(taddr + c, v);
          } else {  // empty contraction: the accumulator was never written
#pragma unroll
            for (int e = 0; e < 32; ++e) v[e] = 0.f;
          }
          if (col < p.N) {
            const size_t row0 = static_cast<size_t>(t.tok0 + c);
            if (p.part) {
              float* dst = p.part + (static_cast<size_t>(t.zi) * p.M + row0) * p.ld_out + col;
#pragma unroll
              for (int e = 0; e < 32; ++e)
                if (c + e < ntok) dst[static_cast<size_t>(e) * p.ld_out] = v[e];
            } else {
              T* dst = out + row0 * p.ld_out + col;
#pragma unroll
              for (int e = 0; e < 32; ++e)
                if (c + e < ntok) dst[static_cast<size_t>(e) * p.ld_out] = DT<T>::from_f(v[e]);
            }
          }
        }
      }
      if (t.nkb > 0) {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) pf_arrive_cluster(acc_empty0[buf]);
        ++na;
      }
    }
  }
  __syncwarp();  // the producing lanes are back: what follows is executed by whole warps
  if (timed_out && p.status && lane == 0) atomicOr(p.status, DEV_TIMEOUT);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // neither CTA leaves (or frees tensor memory) while the other's copies and commits may still reach its barriers
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(p.tmem_cols) : "memory");
  }
}

// ---------------------------------------------------------------------------------- host
typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static PFN_encodeTiled encode_fn() {
  static PFN_encodeTiled fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_encodeTiled>(p);
  }
  return fn;
}

// 2-D operand [rows, cols] of 16-bit elements with row stride ld (elements), 128-byte swizzle.
static int make_map(CUtensorMap* m, const void* base, int dtype, int64_t rows, int64_t cols, int64_t ld, int box_rows) {
  PFN_encodeTiled enc = encode_fn();
  if (!enc) {
    set_error("prefill path: cuTensorMapEncodeTiled is not available from this driver");
    return STX_ERR_CUDA;
  }
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  const cuuint32_t box[2] = {PF_BK, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(m, dtype == STX_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                         const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("prefill path: cuTensorMapEncodeTiled failed with %d (rows=%lld cols=%lld ld=%lld)", static_cast<int>(r),
              static_cast<long long>(rows), static_cast<long long>(cols), static_cast<long long>(ld));
    return STX_ERR_CUDA;
  }
  return STX_OK;
}

static int sm_pairs() { return std::max(1, num_sms() / 2); }

template <typename T, int MODE>
static int launch_pair(const PfWeightMaps& a, const CUtensorMap& b, PfArgs p, int tiles, bool pdl, cudaStream_t s) {
  static bool attr_set[64] = {};
  int dev = 0;
  STX_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    STX_CUDA(cudaFuncSetAttribute(k_pair_gemm<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, PF_SMEM));
    attr_set[dev] = true;
  }
  const uint32_t stage_bytes = PF_A_BYTES + static_cast<uint32_t>(p.n_tok / 2) * (PF_BK * 2);
  const uint32_t fixed = 1024 + PF_XCH_BYTES + (2 * PF_MAX_STAGES + 4) * 8 + 16;
  // Few tokens: HBM-bound, and five or six stages per SM are enough in flight (120 KB x 148 against 6.6 TB/s x 1.5 us;
  // four stages, which would let the next GEMM's CTA in, cost 4 %).  The rest of the shared memory is for kernels that
  // run beside the CTA: the next layer's predictor and cache upkeep in a stack.
  const uint32_t room = p.tok_tiles == 1 && p.n_tok <= 128 ? PF_SMEM_FEW : PF_SMEM;
  p.stages = static_cast<int>(std::min<uint32_t>(PF_MAX_STAGES, (room - fixed) / stage_bytes));
  p.pairs = sm_pairs();
  p.tmem_cols = 64;
  while (p.tmem_cols < 2 * p.n_tok) p.tmem_cols *= 2;
  const size_t smem = fixed + static_cast<size_t>(p.stages) * stage_bytes;
  const unsigned grid = 2u * static_cast<unsigned>(std::max(1, std::min(tiles, p.pairs)));
  STX_CUDA(launch_pdl_if(pdl, k_pair_gemm<T, MODE>, dim3(grid), dim3(PF_THREADS), smem, s, a, b, p));
  return STX_OK;
}

// Tokens of a tile and contraction splits of one launch, by an estimate of its time: a k-block of a
// tile takes the pair 2 clocks per token of the tile on the tensor pipe, and 0.37 us for its 32 KB of
// weights at an even share of HBM when no other token tile reads the same ones; whole waves of tiles
// count.  Splits (partial sums in fp32, added by one more kernel) pay where the tiles are too few.
struct PfShape {
  int n_tok, tok_tiles, splits;
};
constexpr int64_t PF_SPLIT_ROWS = 2048;  // splits x tokens of the partial sums
static PfShape pair_shape(int64_t B, int64_t m_tiles, int64_t nkb, int64_t H, bool may_split, bool even) {
  PfShape best = {0, 0, 1};
  double best_t = 1e30;
  const int64_t t_min = (B + PF_MAX_N - 1) / PF_MAX_N;
  for (int64_t tt = t_min; tt <= t_min + std::max<int64_t>(2, t_min / 4); ++tt) {
    const int64_t n = ((B + tt - 1) / tt + 31) / 32 * 32;
    const int64_t tiles_t = (B + n - 1) / n;
    if (tiles_t > 1 && n < 96) break;
    const double kb_us = std::max(0.37 / static_cast<double>(std::min<int64_t>(tiles_t, PF_GROUP)), 0.0011 * static_cast<double>(n));
    for (int64_t z = 1; z <= (may_split ? 16 : 1); ++z) {
      if (z > 1 && (z * B > PF_SPLIT_ROWS || z > nkb)) break;
      const double tiles = static_cast<double>(m_tiles * tiles_t * z), pairs = sm_pairs();
      const double waves =
          even && tiles_t == 1 ? tiles / pairs : static_cast<double>((m_tiles * tiles_t * z + sm_pairs() - 1) / sm_pairs());
      double t = waves * static_cast<double>((nkb + z - 1) / z) * kb_us;
      if (z > 1) t += 3.0 + 8.0 * static_cast<double>(z * B * H) / 5e6;
      if (t < best_t * 0.999) {
        best_t = t;
        best = {static_cast<int>(n), static_cast<int>(tiles_t), static_cast<int>(z)};
      }
    }
  }
  return best;
}

size_t prefill_scratch_bytes(int64_t B, int64_t H, int64_t K) {
  const int64_t K8 = (K + 7) / 8 * 8;
  // activations [B, K8], partial sums of a split GEMM 2 (at most 16 splits and PF_SPLIT_ROWS rows in all): grows with B
  return 1024 + align_up(static_cast<size_t>(B) * K8 * 2, 1024) +
         align_up(static_cast<size_t>(std::min<int64_t>(16 * B, PF_SPLIT_ROWS)) * H * sizeof(float), 1024);
}

// Implemented in stx_mlp_row.cu: out[i] = sum over g < G of partial[g][i], g ascending (n % 128 == 0).
int partial_sum(const float* partial, int G, int64_t n, void* out, int dtype, cudaStream_t s);

// Row blocks of STX_GEMM_MIN_ROWS and more (16-bit, gated) run as tensor-core GEMMs.
bool prefill_wanted(int64_t B, int64_t H, int64_t K, int dtype, int has_gate) {
  return dtype != STX_F32 && has_gate && B >= STX_GEMM_MIN_ROWS && (H % 64) == 0 && K >= 64;
}

template <typename T>
static int prefill_run(const PfWeightMaps& mw, const CUtensorMap& mx, const PfArgs& g1, int tiles1, const PfWeightMaps& md,
                       const CUtensorMap& ma, const PfArgs& g2, int tiles2, bool pdl, cudaStream_t s) {
  const int rc = launch_pair<T, 0>(mw, mx, g1, tiles1, pdl, s);
  return rc != STX_OK ? rc : launch_pair<T, 1>(md, ma, g2, tiles2, true, s);
}

// x [B,H], concat [2K,H] (gate rows then up rows), down_packed [K,H]; scratch: prefill_scratch_bytes().
// k_dev (optional): device count of valid packed rows, <= K; the work then follows *k_dev while all
// shapes, tensor maps and grids are built for K, so the call needs no host read-back.
// pdl: the first kernel may overlap the end of its predecessor (no dependency on other streams).
int prefill_forward(const void* x, int64_t B, int64_t H, const void* concat, const void* down_packed, int64_t K,
                    void* out, void* combined, int act, int dtype, void* scratch, int* status, const int* k_dev,
                    bool pdl, cudaStream_t s) {
  const int64_t K8 = (K + 7) / 8 * 8;
  const uintptr_t base = (reinterpret_cast<uintptr_t>(scratch) + 1023) & ~static_cast<uintptr_t>(1023);
  void* a_scr = reinterpret_cast<void*>(base);                                                   // [B, K8]
  float* part = reinterpret_cast<float*>(base + align_up(static_cast<size_t>(B) * K8 * 2, 1024));
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(concat) | reinterpret_cast<uintptr_t>(down_packed)) & 15) {
    set_error("prefill path: x, concat_w and down_packed must be 16-byte aligned");
    return STX_ERR_INVALID_ARG;
  }
  const int64_t w_tiles = (K + PF_TW - 1) / PF_TW, h_tiles = (H + PF_HW - 1) / PF_HW;
  const PfShape s1 = pair_shape(B, w_tiles, (H + PF_BK - 1) / PF_BK, H, false, true);
  const PfShape s2 = pair_shape(B, h_tiles, (K + PF_BK - 1) / PF_BK, H, (B * H) % 128 == 0, false);
  // the activations are GEMM 2's token operand: read them straight from combined_buf[:, :K] when its
  // row stride is TMA-compatible (a multiple of 16 bytes), else from the scratch copy
  const bool a_in_combined = combined != nullptr && (K % 4) == 0 && (reinterpret_cast<uintptr_t>(combined) & 15) == 0;
  CUtensorMap mx, ma;
  PfWeightMaps mw, md = {};
  int rc = make_map(&mx, x, dtype, B, H, H, s1.n_tok / 2);
  for (int i = 0; i < 4 && rc == STX_OK; ++i) rc = make_map(&mw.m[i], concat, dtype, 2 * K, H, H, 64 >> i);
  if (rc == STX_OK)
    rc = a_in_combined ? make_map(&ma, combined, dtype, B, K, 2 * K, s2.n_tok / 2) : make_map(&ma, a_scr, dtype, B, K, K8, s2.n_tok / 2);
  if (rc == STX_OK) rc = make_map(&md.m[0], down_packed, dtype, K, H, H, PF_BK);
  if (rc != STX_OK) return rc;
  PfArgs g1{};
  g1.M = static_cast<int>(B);
  g1.N = static_cast<int>(K);
  g1.Kd = static_cast<int>(H);
  g1.n_tok = s1.n_tok;
  g1.tok_tiles = s1.tok_tiles;
  g1.even = s1.tok_tiles == 1;
  g1.a_out = a_in_combined ? nullptr : a_scr;
  g1.ld_out = static_cast<int>(K8);
  g1.combined = combined;
  g1.act = act;
  g1.status = status;
  g1.k_dev = k_dev;
  PfArgs g2{};
  g2.M = static_cast<int>(B);
  g2.N = static_cast<int>(H);
  g2.Kd = static_cast<int>(K);
  g2.n_tok = s2.n_tok;
  g2.tok_tiles = s2.tok_tiles;
  g2.splits = s2.splits;
  g2.a_out = out;
  g2.ld_out = static_cast<int>(H);
  g2.act = act;
  g2.status = status;
  g2.k_dev = k_dev;
  if (s2.splits > 1) g2.part = part;
  g2.early = 1;
  // evenly shared neurons fill all pairs even where full tiles would not
  const int tiles1 = g1.even ? sm_pairs() : static_cast<int>(w_tiles * s1.tok_tiles);
  const int tiles2 = static_cast<int>(h_tiles * s2.tok_tiles * s2.splits);
  rc = dtype == STX_F16 ? prefill_run<__half>(mw, mx, g1, tiles1, md, ma, g2, tiles2, pdl, s)
                        : prefill_run<__nv_bfloat16>(mw, mx, g1, tiles1, md, ma, g2, tiles2, pdl, s);
  if (rc == STX_OK && g2.part) rc = partial_sum(part, s2.splits, B * H, out, dtype, s);
  return rc;
}

}  // namespace stx
