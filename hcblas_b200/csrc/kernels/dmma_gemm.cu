/*
 * dmma_gemm.cu -- native FP64 DGEMM on the FP64 tensor path of sm_100a
 * (warp-level mma.sync .f64, m16n8k16), the plain DGEMM of this library
 * (reference: lib/src/blas/dgemm/dgemm_*kernels*.cpp, one HCC tile kernel per
 * layout and size bucket).
 *
 * Why the tensor path for FP64: B200's FP64 rate is the same on the CUDA
 * cores and through DMMA, but one m16n8k4 instruction does 512 multiply-adds
 * from 3 operand registers per lane where the CUDA-core form needs 16 DFMA
 * instructions and 32 register reads; the shared-memory traffic per flop
 * drops 4x, which leaves issue slots for loads.
 *
 * Design: 64 x 64 CTA tiles, four CTAs of two warps per SM, each warp a
 * 64 x 32 block = 4 x 4 m16n8 accumulators (64 doubles per lane), multiplied
 * with m16n8k16 DMMAs (one instruction per 16 K where m16n8k4 needs four).
 * Small CTAs fill each other's ramps and barriers and waste less on edges and
 * the last wave than one CTA of eight warps on 128 x 128 (measured, B200:
 * 4096 x 4096 x 2048 NN 2149 against 2320 us, 8378 x 777 x 1133 531 / 870,
 * 2047 x 2047 x 333 TT 115 / 168, 3000 x 3000 x 32 35.2 / 37.3).  K advances
 * in slabs of 16 through a ring of shared-memory stages filled by cp.async
 * (16-byte copies where the operand is 16-byte aligned with an even leading
 * dimension, 8-byte copies otherwise; zero fill outside the matrix): an
 * MN-contiguous operand is kept as [k][mn], a K-contiguous one as [mn][k], so that each is copied
 * along its contiguous dimension and the 16 lanes of a half-warp reading a
 * fragment hit 16 distinct bank pairs in either layout.  Few tiles: the CTAs
 * of a cluster share a tile's K and add up their partial tiles over the
 * cluster's shared memory, ranks in order (100 x 100 x 5000 797 -> 64 us,
 * 1024^3 170 -> 94).  Any shape, leading dimension, offset and alignment runs
 * here; batches (strided or pointer arrays) take blockIdx.y.  Epilogue:
 * alpha * acc + beta * C in registers, beta == 0 never reads C.
 *
 * Fragment layout of mma.sync.aligned.m16n8k4.row.col.f64 (PTX ISA, "matrix
 * fragments for mma.m16n8k4 .f64"): lane = 4 g + t; A (16 x 4, row):
 * a0 = A[g][t], a1 = A[g + 8][t]; B (4 x 8, col): b0 = B[t][g];
 * C (16 x 8): c0, c1 = C[g][2t], C[g][2t + 1]; c2, c3 = C[g + 8][2t],
 * C[g + 8][2t + 1].
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <type_traits>

#include "hcbk.h"

namespace hcbk {
namespace {

constexpr int WM = 64, WN = 32; /* warp tile */
constexpr int MT = WM / 16, NTL = WN / 8; /* m16 x n8 accumulators per warp */
constexpr int BM = 64, BN = 64, BK = 16;
constexpr int DNT = 64, DPER_SM = 4; /* two warps per CTA, four CTAs per SM */
constexpr int LDS = BM + 4; /* doubles per [k][mn] row, */
constexpr int LDK = BK + 4; /* per [mn][k] row: a half-warp's fragment loads hit 16 banks */
constexpr int MAX_SPLIT = 8; /* CTAs of a cluster sharing a tile's K (the portable size) */
/* the ring: doubles of an operand's stage; two stages, the other CTAs' slabs
 * cover a slab's latency (three gained nothing) */
template <bool A_MN, bool B_MN> struct DRing {
  static constexpr int OPA = A_MN ? BK * LDS : BM * LDK, OPB = B_MN ? BK * LDS : BN * LDK;
  static constexpr int STAGES = 2;
  static constexpr int SMEM = STAGES * (OPA + OPB) * 8;
  static_assert(SMEM >= BM * BN * 8, "a split tile meets in the ring's memory");
  static_assert((SMEM + 1024) * DPER_SM <= 233472, "resident CTAs");
};

struct DmmaParams {
  int64_t m, n, k;
  const double *a;
  int64_t lda, sa, a_off;
  const double *b;
  int64_t ldb, sb, b_off;
  double *c;
  int64_t ldc, sc, c_off;
  const double *const *a_arr;
  const double *const *b_arr;
  double *const *c_arr;
  int64_t batch;
  double alpha, beta;
  int beta_nonzero;
  int split; /* CTAs per tile (cluster size) */
};

/* m16n8k16: a[2i] = A[g][t + 4i], a[2i + 1] = A[g + 8][t + 4i], b[i] = B[t + 4i][g]
 * (the m16n8k4 fragments of the four K quarters side by side; checked lane
 * by lane against a CPU product on B200) */
__device__ __forceinline__ void dmma16(double (&c)[4], const double (&a)[8], const double (&b)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, "
      "{%4, %5, %6, %7, %8, %9, %10, %11}, {%12, %13, %14, %15}, {%0, %1, %2, %3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]),
        "d"(b[0]), "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

struct alignas(16) D2 {
  double v[2];
};

/* shared-memory address of a generic pointer */
__device__ __forceinline__ uint32_t sptr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
/* asynchronous global -> shared copies; `bytes` of the source are read and
 * the rest of the destination is zero-filled (bytes = 0: nothing is read) */
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes)
               : "memory");
}
/* Tile `lin` of tiles_m x tiles_n in bands of 8 tile rows, walked column by
 * column, for L2 reuse of B panels. */
__device__ __forceinline__ void tile_of(unsigned lin, unsigned tiles_m, unsigned tiles_n,
                                        unsigned &tm, unsigned &tn) {
  const unsigned band = lin / (8 * tiles_n), in_band = lin - band * 8 * tiles_n;
  const unsigned h = tiles_m - band * 8 < 8 ? tiles_m - band * 8 : 8;
  tn = in_band / h;
  tm = band * 8 + in_band - tn * h;
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
/* two doubles at shared-memory address `addr` of the cluster's CTA `rank` */
__device__ __forceinline__ double2 ld_cluster2(uint32_t addr, int rank) {
  double2 v;
  asm volatile(
      "{\n\t.reg .b32 r;\n\t"
      "mapa.shared::cluster.u32 r, %2, %3;\n\t"
      "ld.shared::cluster.v2.f64 {%0, %1}, [r];\n\t}"
      : "=d"(v.x), "=d"(v.y)
      : "r"(addr), "r"(rank)
      : "memory");
  return v;
}

/* The CTAs of a cluster, each with a partial tile of `vecs` 16-byte pairs per
 * column at `tile`, add up columns [c0, c1) in rank order into this CTA's own
 * copy.  Ends with an arrival that the caller answers with cluster_wait(). */
__device__ __forceinline__ void cluster_sum(double2 *tile, int vecs, int c0, int c1, int split,
                                            int tid, int threads) {
  cluster_arrive();
  cluster_wait(); /* every rank's partial tile is in place */
  const uint32_t base = sptr(tile);
  for (int u = c0 * vecs + tid; u < c1 * vecs; u += threads) {
    double2 part[MAX_SPLIT];
#pragma unroll
    for (int r = 0; r < MAX_SPLIT; ++r)
      if (r < split) part[r] = ld_cluster2(base + 16u * (uint32_t)u, r);
    double2 sum = part[0];
#pragma unroll
    for (int r = 1; r < MAX_SPLIT; ++r)
      if (r < split) {
        sum.x += part[r].x;
        sum.y += part[r].y;
      }
    tile[u] = sum; /* only this rank reads its columns of its own tile */
  }
  cluster_arrive();
  __syncthreads();
}

/* One operand's side of the ring, this thread's copies: an MN-contiguous
 * operand as [k][mn] (pitch LDS), a K-contiguous one as [mn][k] (pitch LDK);
 * either is copied along its contiguous dimension, two doubles per copy
 * (16-byte copies when the operand allows, else two 8-byte ones), zero
 * outside the matrix.  Eight copies per slab, a constant number of rows or k
 * apart, so that a slab costs a few additions beside its copies (short K and
 * many tiles are bound by instructions: 3000 x 3000 x 32 took 3600 per warp
 * with every position computed from its index). */
template <bool MN> struct DCopy {
  static constexpr int STEP = MN ? DNT / (BM / 2) : DNT / (BK / 2); /* k or rows per copy */
  static constexpr int COPIES = (MN ? BK : BM) / STEP;
  const double *p; /* first source of the next slab */
  uint32_t dst;    /* its place in stage 0 (shared-memory address) */
  int64_t ld;
  int left; /* valid rows from this thread's first on */
  int k0;   /* its first k in a slab */
  bool vec;

  __device__ __forceinline__ DCopy(const double *src, int64_t ld_, double *stage, int rows, int tid)
      : ld(ld_) {
    vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0 && (ld & 1) == 0;
    const int r0 = MN ? (tid % (BM / 2)) * 2 : tid / (BK / 2);
    k0 = MN ? tid / (BM / 2) : (tid % (BK / 2)) * 2;
    p = MN ? src + r0 + k0 * ld : src + k0 + r0 * ld;
    dst = sptr(stage + (MN ? k0 * LDS + r0 : r0 * LDK + k0));
    left = rows - r0;
  }
  /* the slab at p, of which kc k are valid, into the stage `at` bytes on */
  __device__ __forceinline__ void slab(uint32_t at, int kc) const {
    const double *s = p;
    const uint32_t d = dst + at;
    const int n_mn = left >= 2 ? 2 : left > 0 ? left : 0;
    const int n_k = kc - k0 >= 2 ? 2 : kc > k0 ? kc - k0 : 0;
#pragma unroll
    for (int v = 0; v < COPIES; ++v) {
      const int n = MN ? (k0 + v * STEP < kc ? n_mn : 0) : (v * STEP < left ? n_k : 0);
      const uint32_t to = d + 8 * v * STEP * (MN ? LDS : LDK);
      if (vec) {
        cp_async16(to, s, n * 8);
      } else {
        cp_async8(to, s, n >= 1 ? 8 : 0);
        cp_async8(to + 8, s + 1, n >= 2 ? 8 : 0);
      }
      s += STEP * ld;
    }
  }
};

/*
 * OP_A / OP_B: 0 = N, 1 = T (column-major canonical; FP64 has no conjugate).
 *   op(A) MN-contiguous iff OP_A == N;  op(B) K-contiguous iff OP_B == N.
 * K slabs go through a ring of shared-memory stages filled by
 * cp.async: while one slab is multiplied, the next STAGES - 1 are in flight,
 * and one barrier per slab both publishes the landed slab and frees the stage
 * that the next copies overwrite.
 */
template <int OP_A, int OP_B, bool SPLIT>
__global__ void __launch_bounds__(DNT, DPER_SM) dmma_gemm_kernel(const __grid_constant__ DmmaParams p) {
  constexpr bool A_MN = (OP_A == HCBK_OP_N);
  constexpr bool B_MN = (OP_B != HCBK_OP_N);
  using Ring = DRing<A_MN, B_MN>;
  constexpr int DSTAGES = Ring::STAGES;
  extern __shared__ __align__(16) double dmma_smem[];

  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm = 0, wn = warp * WN;

  /* the cluster's tile and this CTA's share of its K slabs */
  const unsigned split = SPLIT ? (unsigned)p.split : 1u;
  const int rank = SPLIT ? (int)(blockIdx.x % split) : 0;
  unsigned tm, tn;
  tile_of(blockIdx.x / split, (unsigned)((p.m + BM - 1) / BM), (unsigned)((p.n + BN - 1) / BN), tm,
          tn);
  const int64_t m0 = (int64_t)tm * BM, n0 = (int64_t)tn * BN;
  const int rows = (int)(p.m - m0 < BM ? p.m - m0 : BM);
  const int cols = (int)(p.n - n0 < BN ? p.n - n0 : BN);
  const unsigned slabs = (unsigned)((p.k + BK - 1) / BK);
  const int s0 = SPLIT ? (int)(slabs * (uint64_t)rank / split) : 0;
  const int ktiles = SPLIT ? (int)(slabs * (uint64_t)(rank + 1) / split) - s0 : (int)slabs;

  for (int64_t bidx = blockIdx.y; bidx < p.batch; bidx += gridDim.y) {
    const double *A = (p.a_arr ? p.a_arr[bidx] : p.a) + p.a_off + bidx * p.sa;
    const double *B = (p.b_arr ? p.b_arr[bidx] : p.b) + p.b_off + bidx * p.sb;
    double *C = (p.c_arr ? p.c_arr[bidx] : p.c) + p.c_off + bidx * p.sc;
    const int64_t step_a = A_MN ? BK * p.lda : BK, step_b = B_MN ? BK * p.ldb : BK;
    DCopy<A_MN> ca(A + (A_MN ? m0 : m0 * p.lda) + s0 * step_a, p.lda, dmma_smem, rows, tid);
    DCopy<B_MN> cb(B + (B_MN ? n0 : n0 * p.ldb) + s0 * step_b, p.ldb, dmma_smem + Ring::OPA, cols,
                   tid);
    int64_t kleft = p.k - (int64_t)s0 * BK; /* k from the next slab on */
    auto load_stage = [&](int slot) {
      const uint32_t at = 8u * (Ring::OPA + Ring::OPB) * (uint32_t)slot;
      const int kc = kleft < BK ? (int)kleft : BK;
      ca.slab(at, kc);
      cb.slab(at, kc);
      ca.p += step_a;
      cb.p += step_b;
      kleft -= BK;
    };

    double acc[MT][NTL][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NTL; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;

#pragma unroll
    for (int s = 0; s < DSTAGES - 1; ++s) {
      if (s < ktiles) load_stage(s);
      cp_async_commit();
    }
    int slot = 0;
    for (int kt = 0; kt < ktiles; ++kt) {
      cp_async_wait<DSTAGES - 2>(); /* this thread's copies of slab kt have landed */
      __syncthreads();              /* everyone's; and slab kt - 1 is no longer read */
      if (kt + DSTAGES - 1 < ktiles)
        load_stage(slot == 0 ? DSTAGES - 1 : slot - 1);
      cp_async_commit();
      const double *As = dmma_smem + slot * (Ring::OPA + Ring::OPB), *Bs = As + Ring::OPA;
      {
        double af[MT][8];
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          const int r = wm + 16 * i + g;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int kk = t + 4 * q;
            af[i][2 * q] = A_MN ? As[kk * LDS + r] : As[r * LDK + kk];
            af[i][2 * q + 1] = A_MN ? As[kk * LDS + r + 8] : As[(r + 8) * LDK + kk];
          }
        }
#pragma unroll
        for (int j = 0; j < NTL; ++j) {
          const int c = wn + 8 * j + g;
          double bf[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int kk = t + 4 * q;
            bf[q] = B_MN ? Bs[kk * LDS + c] : Bs[c * LDK + kk];
          }
#pragma unroll
          for (int i = 0; i < MT; ++i) dmma16(acc[i][j], af[i], bf);
        }
      }
      slot = slot + 1 == DSTAGES ? 0 : slot + 1;
    }
    cp_async_wait<0>(); /* only empty groups remain */

    const bool rd = p.beta_nonzero != 0;
    double *Ct = C + m0 + n0 * p.ldc;
    if constexpr (!SPLIT) {
      /* c0, c1 at (g, 2t), (g, 2t + 1); c2, c3 at row g + 8; every element of C
       * of an m16 block row is read before the first is written */
      double *Cg = Ct + wm + g + (wn + 2 * t) * p.ldc;
      const int rl = rows - wm - g, cl = cols - wn - 2 * t; /* rows and columns left from there */
      auto write = [&](auto whole) {
        constexpr bool WHOLE = decltype(whole)::value;
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          double old[NTL][4];
          if (rd) {
#pragma unroll
            for (int j = 0; j < NTL; ++j)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int r = 16 * i + (e >> 1) * 8, c = 8 * j + (e & 1);
                old[j][e] = WHOLE || (r < rl && c < cl) ? Cg[r + c * p.ldc] : 0.0;
              }
          }
#pragma unroll
          for (int j = 0; j < NTL; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int r = 16 * i + (e >> 1) * 8, c = 8 * j + (e & 1);
              const double o = p.alpha * acc[i][j][e];
              if (WHOLE || (r < rl && c < cl))
                Cg[r + c * p.ldc] = rd ? fma(p.beta, old[j][e], o) : o;
            }
        }
      };
      if (rows == BM && cols == BN) write(std::true_type());
      else write(std::false_type());
      if (p.batch > 1) __syncthreads(); /* the stages are reused by the next entry */
      continue;
    }

    /* split K: the partial tiles meet in the ring's memory, column-major */
    __syncthreads(); /* the stages are no longer read */
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NTL; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          dmma_smem[(wn + 8 * j + 2 * t + (e & 1)) * BM + wm + 16 * i + g + (e >> 1) * 8] =
              acc[i][j][e];
    const int c0 = cols * rank / (int)split, c1 = cols * (rank + 1) / (int)split;
    cluster_sum(reinterpret_cast<double2 *>(dmma_smem), BM / 2, c0, c1, split, tid, DNT);
    constexpr int UN = 8; /* elements of C in flight per thread */
    for (int u0 = c0 * BM + tid; u0 < c1 * BM; u0 += UN * DNT) {
      double old[UN];
#pragma unroll
      for (int i = 0; i < UN; ++i) {
        const int u = u0 + i * DNT, r = u % BM;
        old[i] = rd && u < c1 * BM && r < rows ? Ct[r + (u / BM) * p.ldc] : 0.0;
      }
#pragma unroll
      for (int i = 0; i < UN; ++i) {
        const int u = u0 + i * DNT, r = u % BM;
        if (u < c1 * BM && r < rows) {
          const double o = p.alpha * dmma_smem[u];
          Ct[r + (u / BM) * p.ldc] = rd ? fma(p.beta, old[i], o) : o;
        }
      }
    }
    cluster_wait(); /* no rank reads this CTA's memory any more */
    /* nor does this CTA: the arrivals above came before its reads of the sums */
    if (p.batch > 1) __syncthreads();
  }
}

/*
 * Native ZGEMM on the same FP64 tensor path: the complex product is four
 * real products per fragment set, Re += Ar Br - Ai Bi, Im += Ar Bi + Ai Br
 * (the 4M form), on m16n8k16 DMMAs.  64 x 64 CTA tiles, two per SM, 4 warps as
 * 2 x 2, warp tiles 32 x 32 = 2 x 4 m16n8 accumulator pairs (one 128 x 64 tile
 * of 8 warps per SM: CN 2048 x 2048 x 512 710 us, two of 64 x 64 608; 3000 x
 * 300 x 100 47 and 41).  K advances in slabs of 16 complex elements through a
 * 2-stage ring filled by cp.async (the other CTA covers a slab's latency), one
 * 16-byte copy per element (two 8-byte ones for an operand that is only
 * 8-byte aligned), complex values kept interleaved: an MN-contiguous operand
 * as [k][mn] (pitch 66 elements), a K-contiguous one as
 * [mn][k] (pitch 20), so that each quarter-warp's 16-byte fragment loads --
 * real and imaginary part together -- hit 8 distinct bank groups.
 * Conjugation is applied to the fragments.
 */
constexpr int ZBK = 16;
constexpr int ZLDK = ZBK + 4; /* [mn][k] pitch (complex elements) */
constexpr int ZWM = 32, ZWN = 32, ZMT = ZWM / 16, ZNT = ZWN / 8;
constexpr int ZBM = 64, ZBN = 64, ZTHREADS = 128, ZPER_SM = 2, ZSTAGES = 2;
constexpr int ZLD = ZBM + 2; /* [k][mn] pitch */
constexpr int ZOP = ZBK * ZLD > ZBM * ZLDK ? ZBK * ZLD : ZBM * ZLDK; /* per operand and stage */
constexpr int ZSMEM = ZSTAGES * 2 * ZOP * 16;
static_assert(ZSMEM >= ZBM * ZBN * 16, "a split tile meets in the ring's memory");
static_assert((ZSMEM + 1024) * ZPER_SM <= 233472, "resident CTAs");

struct ZmmaParams {
  int64_t m, n, k;
  const double2 *a;
  int64_t lda, sa, a_off;
  const double2 *b;
  int64_t ldb, sb, b_off;
  double2 *c;
  int64_t ldc, sc, c_off;
  const double2 *const *a_arr;
  const double2 *const *b_arr;
  double2 *const *c_arr;
  int64_t batch;
  double2 alpha, beta;
  int beta_nonzero;
  int split; /* CTAs per tile (cluster size) */
};

/* one operand's slab of complex elements into a stage: [k][mn] or [mn][k] as
 * stored, one copy per element, zeros outside the matrix */
template <bool MN, int ROWS, int NT>
__device__ __forceinline__ void zload_slab(double2 *dst, const double2 *X, int64_t ld,
                                           int64_t rows, int64_t K, int64_t r0, int64_t k0,
                                           bool vec, int tid) {
  constexpr int PITCH_MN = ROWS + 2;
#pragma unroll
  for (int v = 0; v < (ROWS * ZBK) / NT; ++v) {
    const int idx = tid + v * NT;
    int mn, kk, off;
    if (MN) {
      mn = idx % ROWS;
      kk = idx / ROWS;
      off = kk * PITCH_MN + mn;
    } else {
      mn = idx / ZBK;
      kk = idx % ZBK;
      off = mn * ZLDK + kk;
    }
    const int64_t grow = r0 + mn, gk = k0 + kk;
    const bool ok = grow < rows && gk < K;
    const double2 *src = ok ? (MN ? X + grow + gk * ld : X + gk + grow * ld) : X;
    if (vec) {
      cp_async16(sptr(dst + off), src, ok ? 16 : 0);
    } else {
      const double *s = reinterpret_cast<const double *>(src);
      double *d = reinterpret_cast<double *>(dst + off);
      cp_async8(sptr(d), s, ok ? 8 : 0);
      cp_async8(sptr(d + 1), ok ? s + 1 : s, ok ? 8 : 0);
    }
  }
}

template <int OP_A, int OP_B, bool SPLIT>
__global__ void __launch_bounds__(ZTHREADS, ZPER_SM)
zmma_gemm_kernel(const __grid_constant__ ZmmaParams p) {
  constexpr int NT = ZTHREADS;
  constexpr bool A_MN = (OP_A == HCBK_OP_N);
  constexpr bool B_MN = (OP_B != HCBK_OP_N);
  constexpr bool CJ_A = (OP_A == HCBK_OP_C);
  constexpr bool CJ_B = (OP_B == HCBK_OP_C);
  extern __shared__ __align__(16) double zmma_smem[];
  double2 *zs = reinterpret_cast<double2 *>(zmma_smem);

  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm = (warp & 1) * ZWM, wn = (warp >> 1) * ZWN;

  const unsigned split = SPLIT ? (unsigned)p.split : 1u;
  const int rank = SPLIT ? (int)(blockIdx.x % split) : 0;
  unsigned tm, tn;
  tile_of(blockIdx.x / split, (unsigned)((p.m + ZBM - 1) / ZBM), (unsigned)((p.n + ZBN - 1) / ZBN),
          tm, tn);
  const int64_t m0 = (int64_t)tm * ZBM, n0 = (int64_t)tn * ZBN;
  const int rows = (int)(p.m - m0 < ZBM ? p.m - m0 : ZBM);
  const int cols = (int)(p.n - n0 < ZBN ? p.n - n0 : ZBN);
  const unsigned slabs = (unsigned)((p.k + ZBK - 1) / ZBK);
  const int64_t s0 = SPLIT ? (int64_t)(slabs * (uint64_t)rank / split) : 0;
  const int ktiles = SPLIT ? (int)(slabs * (uint64_t)(rank + 1) / split - s0) : (int)slabs;

  for (int64_t bidx = blockIdx.y; bidx < p.batch; bidx += gridDim.y) {
    const double2 *A = (p.a_arr ? p.a_arr[bidx] : p.a) + p.a_off + bidx * p.sa;
    const double2 *B = (p.b_arr ? p.b_arr[bidx] : p.b) + p.b_off + bidx * p.sb;
    double2 *C = (p.c_arr ? p.c_arr[bidx] : p.c) + p.c_off + bidx * p.sc;
    const bool vec_a = (reinterpret_cast<uintptr_t>(A) & 15) == 0;
    const bool vec_b = (reinterpret_cast<uintptr_t>(B) & 15) == 0;

    auto load_stage = [&](int slot, int kt) {
      double2 *sa = zs + slot * 2 * ZOP, *sb = sa + ZOP;
      zload_slab<A_MN, ZBM, NT>(sa, A, p.lda, p.m, p.k, m0, (s0 + kt) * ZBK, vec_a, tid);
      zload_slab<B_MN, ZBN, NT>(sb, B, p.ldb, p.n, p.k, n0, (s0 + kt) * ZBK, vec_b, tid);
    };

    double cr[ZMT][ZNT][4], ci[ZMT][ZNT][4];
#pragma unroll
    for (int i = 0; i < ZMT; ++i)
#pragma unroll
      for (int j = 0; j < ZNT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) cr[i][j][e] = ci[i][j][e] = 0.0;

#pragma unroll
    for (int s = 0; s < ZSTAGES - 1; ++s) {
      if (s < ktiles) load_stage(s, s);
      cp_async_commit();
    }
    int slot = 0;
    for (int kt = 0; kt < ktiles; ++kt) {
      cp_async_wait<ZSTAGES - 2>();
      __syncthreads();
      if (kt + ZSTAGES - 1 < ktiles)
        load_stage(slot == 0 ? ZSTAGES - 1 : slot - 1, kt + ZSTAGES - 1);
      cp_async_commit();
      const double2 *As = zs + slot * 2 * ZOP, *Bs = As + ZOP;
#pragma unroll
      for (int i = 0; i < ZMT; ++i) {
        const int r = wm + 16 * i + g;
        /* real parts, and the imaginary parts both ways round: ai for the
         * imaginary accumulator, -ai for the real one */
        double ar[8], ai[8], nai[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int kk = t + 4 * q;
          const double2 x0 = A_MN ? As[kk * ZLD + r] : As[r * ZLDK + kk];
          const double2 x1 = A_MN ? As[kk * ZLD + r + 8] : As[(r + 8) * ZLDK + kk];
          ar[2 * q] = x0.x;
          ar[2 * q + 1] = x1.x;
          ai[2 * q] = CJ_A ? -x0.y : x0.y;
          ai[2 * q + 1] = CJ_A ? -x1.y : x1.y;
          nai[2 * q] = -ai[2 * q];
          nai[2 * q + 1] = -ai[2 * q + 1];
        }
#pragma unroll
        for (int j = 0; j < ZNT; ++j) {
          const int c = wn + 8 * j + g;
          double br[4], bi[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int kk = t + 4 * q;
            const double2 y = B_MN ? Bs[kk * ZLD + c] : Bs[c * ZLDK + kk];
            br[q] = y.x;
            bi[q] = CJ_B ? -y.y : y.y;
          }
          dmma16(cr[i][j], ar, br);
          dmma16(cr[i][j], nai, bi);
          dmma16(ci[i][j], ar, bi);
          dmma16(ci[i][j], ai, br);
        }
      }
      slot = slot + 1 == ZSTAGES ? 0 : slot + 1;
    }
    cp_async_wait<0>();

    const bool rd = p.beta_nonzero != 0;
    double2 *Ct = C + m0 + n0 * p.ldc;
    auto out = [&](double re, double im, double2 cv) {
      double2 o;
      o.x = p.alpha.x * re - p.alpha.y * im;
      o.y = p.alpha.x * im + p.alpha.y * re;
      if (rd) {
        o.x += p.beta.x * cv.x - p.beta.y * cv.y;
        o.y += p.beta.x * cv.y + p.beta.y * cv.x;
      }
      return o;
    };
    if constexpr (!SPLIT) {
#pragma unroll
      for (int i = 0; i < ZMT; ++i) {
        double2 old[ZNT][4];
#pragma unroll
        for (int j = 0; j < ZNT; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int row = wm + 16 * i + g + (e >> 1) * 8, col = wn + 8 * j + 2 * t + (e & 1);
            old[j][e] = rd && row < rows && col < cols ? Ct[row + col * p.ldc]
                                                       : make_double2(0.0, 0.0);
          }
#pragma unroll
        for (int j = 0; j < ZNT; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int row = wm + 16 * i + g + (e >> 1) * 8, col = wn + 8 * j + 2 * t + (e & 1);
            if (row < rows && col < cols)
              Ct[row + col * p.ldc] = out(cr[i][j][e], ci[i][j][e], old[j][e]);
          }
      }
      if (p.batch > 1) __syncthreads(); /* the stages are reused by the next entry */
      continue;
    }

    __syncthreads(); /* the stages are no longer read: the partial tiles meet there */
#pragma unroll
    for (int i = 0; i < ZMT; ++i)
#pragma unroll
      for (int j = 0; j < ZNT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          zs[(wn + 8 * j + 2 * t + (e & 1)) * ZBM + wm + 16 * i + g + (e >> 1) * 8] =
              make_double2(cr[i][j][e], ci[i][j][e]);
    const int c0 = cols * rank / (int)split, c1 = cols * (rank + 1) / (int)split;
    cluster_sum(zs, ZBM, c0, c1, split, tid, NT);
    constexpr int UN = 4; /* elements of C in flight per thread */
    for (int u0 = c0 * ZBM + tid; u0 < c1 * ZBM; u0 += UN * NT) {
      double2 old[UN];
#pragma unroll
      for (int i = 0; i < UN; ++i) {
        const int u = u0 + i * NT, r = u % ZBM;
        old[i] = rd && u < c1 * ZBM && r < rows ? Ct[r + (u / ZBM) * p.ldc]
                                                : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int i = 0; i < UN; ++i) {
        const int u = u0 + i * NT, r = u % ZBM;
        if (u < c1 * ZBM && r < rows)
          Ct[r + (u / ZBM) * p.ldc] = out(zs[u].x, zs[u].y, old[i]);
      }
    }
    cluster_wait(); /* no rank reads this CTA's memory any more */
    /* nor does this CTA: the arrivals above came before its reads of the sums */
    if (p.batch > 1) __syncthreads();
  }
}

}  // namespace
}  // namespace hcbk

using namespace hcbk;

namespace hcbk {
namespace {

/* one CTA per tile and split, clusters of `split` along x */
template <class K, class P>
int launch_split(K kern, int smem, int threads, int64_t tiles, const P &p, cudaStream_t st) {
  if (tiles * p.split > 0x7fffffffLL) return HCBK_ERR_ARGS;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(tiles * p.split), (unsigned)(p.batch < 65535 ? p.batch : 65535), 1);
  cfg.blockDim = dim3((unsigned)threads, 1, 1);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = p.split > 1 ? 1 : 0;
  if (cudaLaunchKernelEx(&cfg, kern, p) != cudaSuccess) {
    cudaGetLastError();
    return HCBK_ERR_LAUNCH;
  }
  return HCBK_OK;
}

template <int OP_A, int OP_B, bool SPLIT> int launch_dmma(const DmmaParams &p, cudaStream_t st) {
  constexpr int smem = DRing<OP_A == HCBK_OP_N, OP_B != HCBK_OP_N>::SMEM;
  auto kern = dmma_gemm_kernel<OP_A, OP_B, SPLIT>;
  static bool attr_set[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return HCBK_ERR_LAUNCH;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
        cudaSuccess)
      return HCBK_ERR_LAUNCH;
    attr_set[dev] = true;
  }
  const int64_t tiles = ((p.m + BM - 1) / BM) * ((p.n + BN - 1) / BN);
  return launch_split(kern, smem, DNT, tiles, p, st);
}

template <bool SPLIT> int launch_dmma_ops(const DmmaParams &p, int op_a, int op_b, cudaStream_t st) {
  if (op_a == HCBK_OP_N)
    return op_b == HCBK_OP_N ? launch_dmma<0, 0, SPLIT>(p, st) : launch_dmma<0, 1, SPLIT>(p, st);
  return op_b == HCBK_OP_N ? launch_dmma<1, 0, SPLIT>(p, st) : launch_dmma<1, 1, SPLIT>(p, st);
}

template <bool SPLIT> int launch_zmma(const ZmmaParams &p, int op_a, int op_b, cudaStream_t st) {
  using K = void (*)(const ZmmaParams);
  static const K table[3][3] = {
      {zmma_gemm_kernel<0, 0, SPLIT>, zmma_gemm_kernel<0, 1, SPLIT>, zmma_gemm_kernel<0, 2, SPLIT>},
      {zmma_gemm_kernel<1, 0, SPLIT>, zmma_gemm_kernel<1, 1, SPLIT>, zmma_gemm_kernel<1, 2, SPLIT>},
      {zmma_gemm_kernel<2, 0, SPLIT>, zmma_gemm_kernel<2, 1, SPLIT>, zmma_gemm_kernel<2, 2, SPLIT>}};
  static bool attr_set[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return HCBK_ERR_LAUNCH;
  if (!attr_set[dev]) {
    for (int x = 0; x < 3; ++x)
      for (int y = 0; y < 3; ++y)
        if (cudaFuncSetAttribute(table[x][y], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 ZSMEM) != cudaSuccess)
          return HCBK_ERR_LAUNCH;
    attr_set[dev] = true;
  }
  const int64_t tiles = ((p.m + ZBM - 1) / ZBM) * ((p.n + ZBN - 1) / ZBN);
  return launch_split(table[op_a][op_b], ZSMEM, ZTHREADS, tiles, p, st);
}

}  // namespace
}  // namespace hcbk

extern "C" int hcbk_dgemm_dmma(const hcbk_gemm_args *a, int split, void *stream) {
  if (a->dtype != HCBK_D || a->m <= 0 || a->n <= 0 || a->k <= 0 || a->batch <= 0 ||
      a->op_a == HCBK_OP_C || a->op_b == HCBK_OP_C || a->batch_select || split < 1 ||
      split > MAX_SPLIT)
    return HCBK_ERR_ARGS;
  DmmaParams p;
  p.m = a->m;
  p.n = a->n;
  p.k = a->k;
  p.a = static_cast<const double *>(a->a);
  p.lda = a->lda;
  p.sa = a->stride_a;
  p.a_off = a->a_off;
  p.b = static_cast<const double *>(a->b);
  p.ldb = a->ldb;
  p.sb = a->stride_b;
  p.b_off = a->b_off;
  p.c = static_cast<double *>(a->c);
  p.ldc = a->ldc;
  p.sc = a->stride_c;
  p.c_off = a->c_off;
  p.a_arr = reinterpret_cast<const double *const *>(a->a_array);
  p.b_arr = reinterpret_cast<const double *const *>(a->b_array);
  p.c_arr = reinterpret_cast<double *const *>(a->c_array);
  p.batch = a->batch;
  p.alpha = a->alpha_re;
  p.beta = a->beta_re;
  p.beta_nonzero = a->beta_re != 0.0;
  const int64_t slabs = (a->k + BK - 1) / BK;
  p.split = split < slabs ? split : (int)slabs;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return p.split > 1 ? launch_dmma_ops<true>(p, a->op_a, a->op_b, st)
                     : launch_dmma_ops<false>(p, a->op_a, a->op_b, st);
}

extern "C" int hcbk_zgemm_zmma(const hcbk_gemm_args *a, int split, void *stream) {
  if (a->dtype != HCBK_Z || a->m <= 0 || a->n <= 0 || a->k <= 0 || a->batch <= 0 ||
      a->batch_select || split < 1 || split > MAX_SPLIT || a->op_a < 0 || a->op_a > 2 ||
      a->op_b < 0 || a->op_b > 2)
    return HCBK_ERR_ARGS;
  ZmmaParams p;
  p.m = a->m;
  p.n = a->n;
  p.k = a->k;
  p.a = static_cast<const double2 *>(a->a);
  p.lda = a->lda;
  p.sa = a->stride_a;
  p.a_off = a->a_off;
  p.b = static_cast<const double2 *>(a->b);
  p.ldb = a->ldb;
  p.sb = a->stride_b;
  p.b_off = a->b_off;
  p.c = static_cast<double2 *>(a->c);
  p.ldc = a->ldc;
  p.sc = a->stride_c;
  p.c_off = a->c_off;
  p.a_arr = reinterpret_cast<const double2 *const *>(a->a_array);
  p.b_arr = reinterpret_cast<const double2 *const *>(a->b_array);
  p.c_arr = reinterpret_cast<double2 *const *>(a->c_array);
  p.batch = a->batch;
  p.alpha = make_double2(a->alpha_re, a->alpha_im);
  p.beta = make_double2(a->beta_re, a->beta_im);
  p.beta_nonzero = a->beta_re != 0.0 || a->beta_im != 0.0;
  const int64_t slabs = (a->k + ZBK - 1) / ZBK;
  p.split = split < slabs ? split : (int)slabs;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return p.split > 1 ? launch_zmma<true>(p, a->op_a, a->op_b, st)
                     : launch_zmma<false>(p, a->op_a, a->op_b, st);
}

/* The split from an estimate of the busiest SM's cycles: the slabs of its
 * CTAs at the rate that many resident CTAs reach, plus each CTA's prologue and
 * epilogue (dearer when a cluster adds up its tile).  Rates and costs are read
 * off measured times (DGEMM 64^3 to 8378 x 777 x 1133, ZGEMM 64^3 to
 * 2048^2 x 512). */
extern "C" int hcbk_gemm_f64_split(int complex, int64_t m, int64_t n, int64_t k, int64_t batch) {
  static const double eff[2][4] = {{.28, .50, .68, .80}, {.70, .80}};
  static const double cta[2][2] = {{1000, 4000}, {3000, 10000}}; /* whole K, split */
  const int z = complex ? 1 : 0;
  const int sms = hcbk_sm_count(), res = z ? ZPER_SM : DPER_SM;
  const int64_t slabs = (k + BK - 1) / BK;
  static_assert(ZBM == BM && ZBN == BN && ZBK == BK, "one tile shape");
  const int64_t tiles = ((m + BM - 1) / BM) * ((n + BN - 1) / BN) * batch;
  const double slab = z ? 4096 : 1024; /* FMA cycles */
  double best = 0;
  int choice = 1;
  for (int split = 1; split <= MAX_SPLIT && split <= slabs; split *= 2) {
    const double work = (double)((slabs + split - 1) / split) * slab;
    const double extra = cta[z][split > 1];
    const int64_t ctas = tiles * split, full = ctas / ((int64_t)sms * res);
    const int64_t rem = ctas - full * sms * res, last = (rem + sms - 1) / sms;
    double t = (double)(full * res) * (work / eff[z][res - 1] + extra);
    if (last) t += (double)last * (work / eff[z][last - 1] + extra);
    if (split > 1) t += 3000; /* the cluster's launch and barriers (60 x 9 x 20: 10.3 -> 12.3 us) */
    if (best == 0 || t < best) {
      best = t;
      choice = split;
    }
  }
  return choice;
}
