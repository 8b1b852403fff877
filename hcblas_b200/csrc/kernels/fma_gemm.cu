/*
 * fma_gemm.cu -- plain SGEMM and CGEMM on the FP32 FMA pipe of sm_100a.
 *
 * Bound by the FP32 pipe (128 FMAs per clock and SM, packed as fma.rn.f32x2:
 * a row's value against a pair of columns).  A complex value meets a pair
 * (br, bi) as two rows, ar and ai: row ar collects (ar br, ar bi), row ai
 * (ai br, ai bi), so CGEMM is the same loop on pairs, and conjugation only
 * changes the signs with which the two rows are put together at the end.
 *
 * Tiles: 64 floats x 4 TN floats per warp (8 x TN per thread, lanes 8 x 4, so
 * that every fragment load is one wavefront), 128 x 128 floats per CTA with
 * eight warps (TN = 8) or four (TN = 16, complex), or 64 x 64 with two.
 * Fragments are loaded one k ahead.  K advances in slabs of 16 through a ring
 * of shared-memory stages kept as [k][mn] and filled by cp.async: 16-byte
 * copies for an aligned MN-contiguous operand, element copies otherwise (a
 * K-contiguous operand is transposed by them: eight k by four rows per warp
 * instruction is one 32-byte sector per row and free of bank conflicts).  No
 * operand passes through registers, and a leading dimension off 16 bytes
 * costs only the smaller copies.  The main loop is instantiated per copy mode
 * (with one loop for all modes, predicated-off copies took 8 % of the issued
 * instructions and their address arithmetic 10 % of the FMA pipe).
 *
 * Split K: the CTAs of a cluster share one tile, each with its range of slabs;
 * the partial tiles meet in shared memory over the cluster (each CTA adds up
 * its share of the columns, ranks in order, so that results repeat), without
 * workspace, second launch or atomics.  hcbk_gemm_f32_plan chooses tile and
 * split.
 *
 * Measured (B200), TFLOP/s of this kernel against the 8 x 8-per-thread kernel
 * with register-staged loads (simt_gemm.cu): 4096^3 NT 58.4 against 58.1,
 * NN 58.1 / 54.4, TN 56.5 / 54.1; 4095 x 4095 x 2047 TN 51.8 / 49.1; complex
 * CN 2048^3 59.4 / 45.0; with split K 1024^3 33.8 / 28.3, 777 x 1133 x 14522
 * 34.0 / 15.6, 64 x 64 x 4096 1.0 / 0.2.
 *
 * Reference: lib/src/blas/{s,c}gemm/ *kernels*.cpp, one HCC tile kernel per
 * layout and size bucket.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <type_traits>

#include "hcbk.h"

namespace hcbk {
namespace {

constexpr int BK = 16;
constexpr int MAX_SPLIT = 8; /* the portable cluster size */

struct F32Params {
  int64_t m, n, k; /* elements (float or float2) */
  const float *a;
  int64_t lda, sa; /* floats */
  const float *b;
  int64_t ldb, sb;
  float *c;
  int64_t ldc, sc;
  const float *const *a_arr;
  const float *const *b_arr;
  float *const *c_arr;
  int64_t a_off, b_off, c_off;
  int64_t batch;
  float alpha_re, alpha_im, beta_re, beta_im;
  int beta_nonzero;
  int conj_a, conj_b;
  int split; /* CTAs per tile (cluster size) */
};

/* WM x WN warps of 64 x 4 TN floats */
template <int TN, int WM, int WN> struct F32Cfg {
  static constexpr int BM = 64 * WM, BN = 4 * TN * WN;
  static constexpr int NT = 32 * WM * WN;
  static constexpr int PA = BM + 4, PB = BN + 4; /* floats per k row */
  static constexpr int STAGE = BK * (PA + PB);   /* floats */
  /* at least three stages, and room for the tile itself (split K, staged C) */
  static constexpr int STAGES = 3 * STAGE >= BM * BN ? 3 : 4;
  static constexpr int SMEM = STAGES * STAGE * 4;
  static constexpr int PER_SM = 128 / TN / (WM * WN);
  static_assert(STAGES * STAGE >= BM * BN, "the tile fits the stages");
};

__device__ __forceinline__ uint32_t sptr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
/* BYTES from global to shared memory, of which `valid` are read and the rest
 * are zeros (valid = 0: nothing is read) */
template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const float *src, int valid) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;" ::"r"(dst), "l"(src), "r"(valid),
                 "n"(BYTES)
                 : "memory");
}

/* How the operands' slabs are copied.  Tests of the rows cost instructions in
 * the main loop (4096 x 4096 x 512 NN 308 us without, 324 with), so that whole
 * tiles have a loop without; edge tiles keep the wide copies (with element
 * copies there 3000 x 3000 x 512 NT took 193 us, now 179). */
enum CopyMode {
  COPY_WHOLE, /* 16-byte copies along MN where it is contiguous, no row to test */
  COPY_VEC,   /* the same, zeros outside the tile's valid rows */
  COPY_ELEM,  /* one element per copy, zeros outside the tile's valid rows */
};

/* One operand's side of the ring: this thread's copies of a slab of 16 k x
 * ROWS floats (E floats per element) into [k][mn].  A K-contiguous operand is
 * transposed by its copies, lane = k + 8 * row. */
template <int E, int ROWS, int PITCH, int NT, bool MN, int MODE, bool SPREAD> struct SlabCopy {
  static constexpr bool VEC = MODE != COPY_ELEM && MN;
  static constexpr bool ALL = MODE == COPY_WHOLE; /* every row is valid */
  static constexpr int U = VEC ? 4 : E; /* floats per copy */
  /* MN: copies per k row, k rows per pass, passes per k row */
  static constexpr int PER = ROWS / U;
  static constexpr int STEP = NT > PER ? NT / PER : 1;
  static constexpr int PARTS = NT > PER ? 1 : PER / NT;
  static constexpr int RPP = NT / 8; /* K: rows per pass */
  static constexpr int PASSES = MN ? BK / STEP : ROWS / E / RPP;
  const float *p;   /* this thread's first source of the next slab */
  uint32_t dst;     /* and its place in stage 0 */
  int64_t ld;
  int left;         /* valid rows (K-contiguous) or floats from this thread's first on */
  int k0;

  /* src: the operand's first element of the tile at k = 0 */
  __device__ __forceinline__ SlabCopy(const float *src, int64_t ld_, uint32_t stage, int rows)
      : ld(ld_) {
    const int tid = threadIdx.x;
    if constexpr (MN) {
      const int r0 = (tid % PER) * U;
      k0 = tid / PER;
      p = src + r0 + k0 * ld;
      dst = stage + 4 * (k0 * PITCH + r0);
      left = rows * E - r0;
    } else {
      k0 = tid & 7;
      const int r0 = tid >> 3;
      p = src + k0 * E + r0 * ld;
      dst = stage + 4 * (k0 * PITCH + r0 * E);
      left = rows - r0;
    }
  }

  /* pass v of the slab whose first source is s (kc valid k: 16 unless
   * GUARD_K) into the stage at byte offset `at` */
  template <bool GUARD_K>
  __device__ __forceinline__ void pass(const float *s, uint32_t at, int v, int kc) const {
    const uint32_t d = dst + at;
    if constexpr (MN) {
      s += v * (STEP * ld);
#pragma unroll
      for (int h = 0; h < PARTS; ++h) {
        int n = ALL ? U : left - h * NT * U;
        n = n < 0 || (GUARD_K && k0 + v * STEP >= kc) ? 0 : n > U ? U : n;
        cp_async<4 * U>(d + 4 * (v * STEP * PITCH + h * NT * U), s + h * NT * U, 4 * n);
      }
    } else {
      s += v * (RPP * ld);
#pragma unroll
      for (int h = 0; h < BK / 8; ++h) {
        const bool ok = (ALL || v * RPP < left) && (!GUARD_K || k0 + 8 * h < kc);
        cp_async<4 * E>(d + 4 * (8 * h * PITCH + v * RPP * E), s + 8 * h * E, ok ? 4 * E : 0);
      }
    }
  }
  template <bool GUARD_K>
  __device__ __forceinline__ void slab(const float *s, uint32_t at, int kc) const {
#pragma unroll
    for (int v = 0; v < PASSES; ++v) pass<GUARD_K>(s, at, v, kc);
  }
  /* the passes that go with step kk of 16 (all by step 14).  SPREAD: evenly,
   * so that they do not hold up the warp's FMAs in one burst (TN = 8: NN 52.2
   * -> 57.1, TN 48.5 -> 52.5, complex 52.6 -> 57.0 TFLOP/s; TN = 16: TN 52.2
   * -> 54.5); else all with the first step (TN = 16 with 8-byte copies: 57.8
   * spread, 60.8 at once) */
  __device__ __forceinline__ void step(const float *s, uint32_t at, int kk) const {
#pragma unroll
    for (int v = 0; v < PASSES; ++v)
      if ((SPREAD ? v * (BK - 1) / PASSES : 0) == kk) pass<false>(s, at, v, BK);
  }
};

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float lo2(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi2(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ void fma2(uint64_t &c, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

/* v = alpha * v + beta * o, N floats of E per element (o is not looked at
 * when beta == 0) */
template <int E, int N>
__device__ __forceinline__ void scale_add(const F32Params &p, float (&v)[N], const float (&o)[N]) {
#pragma unroll
  for (int e = 0; e < N; e += E) {
    if constexpr (E == 1) {
      v[e] *= p.alpha_re;
      if (p.beta_nonzero) v[e] = fmaf(p.beta_re, o[e], v[e]);
    } else {
      const float x = v[e], y = v[e + 1];
      v[e] = p.alpha_re * x - p.alpha_im * y;
      v[e + 1] = p.alpha_re * y + p.alpha_im * x;
      if (p.beta_nonzero) {
        v[e] += p.beta_re * o[e] - p.beta_im * o[e + 1];
        v[e + 1] += p.beta_re * o[e + 1] + p.beta_im * o[e];
      }
    }
  }
}

/* N floats at 4 * N byte alignment */
template <int N> struct alignas(4 * N) Run {
  float v[N];
};

template <int E, int TN, int WM, int WN, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(F32Cfg<TN, WM, WN>::NT, F32Cfg<TN, WM, WN>::PER_SM)
f32_gemm_kernel(const __grid_constant__ F32Params p) {
  using Cfg = F32Cfg<TN, WM, WN>;
  constexpr bool SPREAD = TN == 8 || E == 1;
  constexpr int BM = Cfg::BM, BN = Cfg::BN, PA = Cfg::PA, PB = Cfg::PB, NT = Cfg::NT;
  constexpr int BME = BM / E, BNE = BN / E; /* elements */
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = lane & 7, ty = lane >> 3;
  const int wm = (warp % WM) * 64, wn = (warp / WM) * 4 * TN;

  /* the cluster's tile (bands of 8 tile rows for L2 reuse) and this CTA's
   * share of its K slabs */
  const int split = p.split;
  const int rank = split > 1 ? (int)(blockIdx.x % (unsigned)split) : 0;
  const int64_t lin = blockIdx.x / (unsigned)split;
  const int64_t tiles_m = (p.m + BME - 1) / BME, tiles_n = (p.n + BNE - 1) / BNE;
  const int64_t per_band = 8 * tiles_n;
  const int64_t band = lin / per_band;
  const int64_t band_h = tiles_m - band * 8 < 8 ? tiles_m - band * 8 : 8;
  const int64_t in_band = lin - band * per_band;
  const int64_t m0 = (band * 8 + in_band % band_h) * BME;
  const int64_t n0 = (in_band / band_h) * BNE;
  const int rows = (int)(p.m - m0 < BME ? p.m - m0 : BME);
  const int cols = (int)(p.n - n0 < BNE ? p.n - n0 : BNE);
  const int64_t slabs = (p.k + BK - 1) / BK;
  const int64_t s0 = slabs * rank / split, s1 = slabs * (rank + 1) / split;
  const int nslab = (int)(s1 - s0);

  for (int64_t bidx = blockIdx.y; bidx < p.batch; bidx += gridDim.y) {
    const float *A = (p.a_arr ? p.a_arr[bidx] : p.a) + p.a_off + bidx * p.sa;
    const float *B = (p.b_arr ? p.b_arr[bidx] : p.b) + p.b_off + bidx * p.sb;
    float *C = (p.c_arr ? p.c_arr[bidx] : p.c) + p.c_off + bidx * p.sc;
    /* 16-byte copies run along the MN dimension only */
    const bool vec_a = !A_MN || (!(reinterpret_cast<uintptr_t>(A) & 15) && !(p.lda & 3));
    const bool vec_b = !B_MN || (!(reinterpret_cast<uintptr_t>(B) & 15) && !(p.ldb & 3));
    const int64_t step_a = A_MN ? BK * p.lda : BK * E, step_b = B_MN ? BK * p.ldb : BK * E;
    const float *pa = A + (A_MN ? m0 * E : m0 * p.lda), *pb = B + (B_MN ? n0 * E : n0 * p.ldb);

    uint64_t acc[8][TN / 2]; /* float row i of the thread x float column pair j */
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

    /* fragments of one k: loaded one k ahead of their use, across slabs too */
    float fa[2][8];
    uint64_t fb[2][TN / 2];
    auto fragment = [&](int x, int slot, int kk) {
      const float *as = smem + slot * Cfg::STAGE + kk * PA + wm + tx * 4;
      const float *bs = smem + slot * Cfg::STAGE + BK * PA + kk * PB + wn + ty * 4;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const float4 v = *reinterpret_cast<const float4 *>(as + 32 * g);
        fa[x][4 * g] = v.x;
        fa[x][4 * g + 1] = v.y;
        fa[x][4 * g + 2] = v.z;
        fa[x][4 * g + 3] = v.w;
      }
#pragma unroll
      for (int g = 0; g < TN / 4; ++g) {
        const float4 v = *reinterpret_cast<const float4 *>(bs + 16 * g);
        fb[x][2 * g] = pack2(v.x, v.y);
        fb[x][2 * g + 1] = pack2(v.z, v.w);
      }
    };
    /* the main loop for one copy mode.  The range's last slab, when K ends
     * inside it, goes first, so that the loop's copies need no test of k. */
    auto run = [&](auto mode) {
      constexpr int MODE = decltype(mode)::value;
      const SlabCopy<E, BM, PA, NT, A_MN, MODE, SPREAD> ca(pa, p.lda, sptr(smem), rows);
      const SlabCopy<E, BN, PB, NT, B_MN, MODE, SPREAD> cb(pb, p.ldb, sptr(smem + BK * PA), cols);
      const int kc = (int)(p.k - (s1 - 1) * BK < BK ? p.k - (s1 - 1) * BK : BK);
      const float *sa = ca.p + s0 * step_a, *sb = cb.p + s0 * step_b; /* the next slab */
      int left = nslab;
      uint32_t at = 0;
      auto next_stage = [&] {
        asm volatile("cp.async.commit_group;" ::: "memory");
        at = at == 4u * (Cfg::STAGES - 1) * Cfg::STAGE ? 0u : at + 4u * Cfg::STAGE;
        sa += step_a;
        sb += step_b;
        --left;
      };
      if (kc < BK) {
        ca.template slab<true>(ca.p + (s1 - 1) * step_a, at, kc);
        cb.template slab<true>(cb.p + (s1 - 1) * step_b, at, kc);
        sa -= step_a;
        sb -= step_b;
        next_stage();
      }
#pragma unroll 1
      for (int s = kc < BK ? 1 : 0; s < Cfg::STAGES - 1; ++s) {
        if (left > 0) {
          ca.template slab<false>(sa, at, BK);
          cb.template slab<false>(sb, at, BK);
        }
        next_stage();
      }
      asm volatile("cp.async.wait_group %0;" ::"n"(Cfg::STAGES - 2) : "memory");
      __syncthreads();
      int slot = 0;
      fragment(0, 0, 0);
#pragma unroll 1
      for (int s = 0; s < nslab; ++s) {
        const int next = slot + 1 == Cfg::STAGES ? 0 : slot + 1;
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
          /* slab s - 1 is no longer read: its stage takes slab s + STAGES - 1,
           * the copies spread over the steps */
          if (left > 0) {
            ca.step(sa, at, kk);
            cb.step(sb, at, kk);
          }
          if (kk == BK - 1) { /* slab s + 1 has landed for everyone */
            next_stage();
            asm volatile("cp.async.wait_group %0;" ::"n"(Cfg::STAGES - 2) : "memory");
            __syncthreads();
            fragment(0, next, 0);
          } else {
            fragment((kk + 1) & 1, slot, kk + 1);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint64_t aa = pack2(fa[kk & 1][i], fa[kk & 1][i]);
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], aa, fb[kk & 1][j]);
          }
        }
        slot = next;
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory"); /* only empty groups remain */
    };
    if constexpr (A_MN || B_MN) {
      if (!vec_a || !vec_b)
        run(std::integral_constant<int, COPY_ELEM>());
      else if (rows == BME && cols == BNE)
        run(std::integral_constant<int, COPY_WHOLE>());
      else
        run(std::integral_constant<int, COPY_VEC>());
    } else {
      run(std::integral_constant<int, COPY_ELEM>());
    }

    /* four consecutive floats of a column: rows 32 g + 4 tx .. + 3 of the
     * warp tile, element column j of the thread */
    auto run4 = [&](int g, int j) {
      Run<4> r;
      if constexpr (E == 1) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          r.v[e] = j & 1 ? hi2(acc[4 * g + e][j >> 1]) : lo2(acc[4 * g + e][j >> 1]);
      } else {
        /* rows ar, ai of acc against the pair (br, bi):
         * re = ar br -+ ai bi, im = +-ai br +- ar bi */
        const float sr = p.conj_a != p.conj_b ? 1.f : -1.f;
        const float si = p.conj_a ? -1.f : 1.f, sj = p.conj_b ? -1.f : 1.f;
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          const uint64_t x = acc[4 * g + e][j], y = acc[4 * g + e + 1][j];
          r.v[e] = fmaf(sr, hi2(y), lo2(x));
          r.v[e + 1] = fmaf(si, lo2(y), sj * hi2(x));
        }
      }
      return r;
    };
    constexpr int TC = TN / E; /* element columns per thread */
    auto col_of = [&](int j) { /* tile column of the thread's element column j */
      return E == 1 ? wn + (j >> 2) * 16 + ty * 4 + (j & 3)
                    : wn / 2 + (j >> 1) * 8 + ty * 2 + (j & 1);
    };
    float *Ct = C + m0 * E + n0 * p.ldc;
    const bool vec_c = !(reinterpret_cast<uintptr_t>(C) & 15) && !(p.ldc & 3);
    const bool rd = p.beta_nonzero != 0;

    if (split == 1 && vec_c) {
      /* eight 16-byte runs of C are read before the first is written */
#pragma unroll
      for (int jb = 0; jb < TC; jb += 4) {
        Run<4> old[4][2];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const int col = col_of(jb + j), r = wm + 32 * g + 4 * tx;
            const float *src = Ct + r + col * p.ldc;
#pragma unroll
            for (int e = 0; e < 4; ++e) old[j][g].v[e] = 0.f;
            if (rd && col < cols) {
              if (r + 4 <= rows * E) {
                old[j][g] = *reinterpret_cast<const Run<4> *>(src);
              } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                  if (r + e < rows * E) old[j][g].v[e] = src[e];
              }
            }
          }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const int col = col_of(jb + j), r = wm + 32 * g + 4 * tx;
            float *dst = Ct + r + col * p.ldc;
            Run<4> v = run4(g, jb + j);
            scale_add<E, 4>(p, v.v, old[j][g].v);
            if (col < cols) {
              if (r + 4 <= rows * E) {
                *reinterpret_cast<Run<4> *>(dst) = v;
              } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                  if (r + e < rows * E) dst[e] = v.v[e];
              }
            }
          }
      }
      if (p.batch > 1) __syncthreads(); /* the stages are filled again */
      continue;
    }

    /* through shared memory, column by column: split K, and a C that 16-byte
     * vectors cannot address (its columns are then written by consecutive
     * lanes instead of four scattered stores per thread) */
    __syncthreads(); /* the stages are no longer read */
#pragma unroll
    for (int j = 0; j < TC; ++j)
#pragma unroll
      for (int g = 0; g < 2; ++g)
        *reinterpret_cast<Run<4> *>(smem + col_of(j) * BM + wm + 32 * g + 4 * tx) = run4(g, j);
    int c0 = 0, c1 = cols;
    if (split > 1) {
      cluster_arrive();
      cluster_wait(); /* every rank's partial tile is in place */
      c0 = cols * rank / split;
      c1 = cols * (rank + 1) / split;
      const uint32_t base = sptr(smem);
      constexpr int V = BM / 4;
      for (int u = c0 * V + tid; u < c1 * V; u += NT) {
        float4 part[MAX_SPLIT];
#pragma unroll
        for (int r = 0; r < MAX_SPLIT; ++r)
          if (r < split) {
            uint32_t remote;
            asm("mapa.shared::cluster.u32 %0, %1, %2;"
                : "=r"(remote)
                : "r"(base + 16u * (uint32_t)u), "r"(r));
            part[r] = ld_cluster4(remote);
          }
        float4 sum = part[0];
#pragma unroll
        for (int r = 1; r < MAX_SPLIT; ++r)
          if (r < split) {
            sum.x += part[r].x;
            sum.y += part[r].y;
            sum.z += part[r].z;
            sum.w += part[r].w;
          }
        /* only this rank reads its columns of its own tile */
        *reinterpret_cast<float4 *>(smem + 4 * u) = sum;
      }
      cluster_arrive();
    }
    __syncthreads();
    constexpr int UN = 8; /* elements of C in flight per thread */
    for (int u0 = c0 * BME + tid; u0 < c1 * BME; u0 += UN * NT) {
      Run<E> old[UN];
#pragma unroll
      for (int i = 0; i < UN; ++i) {
        const int u = u0 + i * NT, r = u % BME;
        if (rd && u < c1 * BME && r < rows)
          old[i] = *reinterpret_cast<const Run<E> *>(Ct + r * E + (u / BME) * p.ldc);
      }
#pragma unroll
      for (int i = 0; i < UN; ++i) {
        const int u = u0 + i * NT, r = u % BME;
        if (u < c1 * BME && r < rows) {
          Run<E> v = *reinterpret_cast<const Run<E> *>(smem + u * E);
          scale_add<E, E>(p, v.v, old[i].v);
          *reinterpret_cast<Run<E> *>(Ct + r * E + (u / BME) * p.ldc) = v;
        }
      }
    }
    if (split > 1) cluster_wait(); /* no rank reads this CTA's memory any more */
    /* nor does this CTA: the arrivals above came before its reads of the sums */
    if (p.batch > 1) __syncthreads();
  }
}

template <int E, int TN, int WM, int WN, bool A_MN, bool B_MN>
int launch_f32(const F32Params &p, int batch_blocks, cudaStream_t st) {
  using Cfg = F32Cfg<TN, WM, WN>;
  auto kern = f32_gemm_kernel<E, TN, WM, WN, A_MN, B_MN>;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return HCBK_ERR_LAUNCH;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM) !=
        cudaSuccess) {
      cudaGetLastError();
      return HCBK_ERR_LAUNCH;
    }
    attr_set[dev] = true;
  }
  const int64_t tiles = ((p.m * E + Cfg::BM - 1) / Cfg::BM) * ((p.n * E + Cfg::BN - 1) / Cfg::BN);
  if (tiles * p.split > 0x7fffffffLL) return HCBK_ERR_ARGS;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(tiles * p.split), (unsigned)batch_blocks, 1);
  cfg.blockDim = dim3(Cfg::NT, 1, 1);
  cfg.dynamicSmemBytes = Cfg::SMEM;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = p.split > 1 ? 1 : 0;
  if (cudaLaunchKernelEx(&cfg, kern, p) != cudaSuccess) {
    cudaGetLastError();
    return HCBK_ERR_LAUNCH;
  }
  return HCBK_OK;
}

template <int E, int TN, int WM, int WN>
int launch_ops(const F32Params &p, bool a_mn, bool b_mn, int by, cudaStream_t st) {
  if (a_mn && b_mn) return launch_f32<E, TN, WM, WN, true, true>(p, by, st);
  if (a_mn) return launch_f32<E, TN, WM, WN, true, false>(p, by, st);
  if (b_mn) return launch_f32<E, TN, WM, WN, false, true>(p, by, st);
  return launch_f32<E, TN, WM, WN, false, false>(p, by, st);
}

}  // namespace
}  // namespace hcbk

using namespace hcbk;

extern "C" int hcbk_gemm_f32(const hcbk_gemm_args *a, hcbk_f32_cfg cfg, void *stream) {
  if (a->dtype != HCBK_S && a->dtype != HCBK_C) return HCBK_ERR_ARGS;
  if (a->m <= 0 || a->n <= 0 || a->k <= 0 || a->batch <= 0 || a->batch_select || cfg.split < 1 ||
      cfg.split > MAX_SPLIT)
    return HCBK_ERR_ARGS;
  const int E = a->dtype == HCBK_C ? 2 : 1;
  F32Params p;
  memset(&p, 0, sizeof(p));
  p.m = a->m;
  p.n = a->n;
  p.k = a->k;
  p.a = static_cast<const float *>(a->a);
  p.b = static_cast<const float *>(a->b);
  p.c = static_cast<float *>(a->c);
  p.lda = a->lda * E;
  p.ldb = a->ldb * E;
  p.ldc = a->ldc * E;
  p.sa = a->stride_a * E;
  p.sb = a->stride_b * E;
  p.sc = a->stride_c * E;
  p.a_off = a->a_off * E;
  p.b_off = a->b_off * E;
  p.c_off = a->c_off * E;
  p.a_arr = reinterpret_cast<const float *const *>(a->a_array);
  p.b_arr = reinterpret_cast<const float *const *>(a->b_array);
  p.c_arr = reinterpret_cast<float *const *>(a->c_array);
  p.batch = a->batch;
  p.alpha_re = (float)a->alpha_re;
  p.alpha_im = (float)a->alpha_im;
  p.beta_re = (float)a->beta_re;
  p.beta_im = (float)a->beta_im;
  p.beta_nonzero = a->beta_re != 0.0 || a->beta_im != 0.0;
  p.conj_a = a->op_a == HCBK_OP_C;
  p.conj_b = a->op_b == HCBK_OP_C;
  const int64_t slabs = (a->k + BK - 1) / BK;
  p.split = cfg.split < slabs ? cfg.split : (int)slabs;
  const bool a_mn = a->op_a == HCBK_OP_N, b_mn = a->op_b != HCBK_OP_N;
  const int by = (int)(a->batch < 65535 ? a->batch : 65535);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  /* both operands K-contiguous and 16-byte aligned: the wider thread tile
   * (4096 x 4096 x 1024 TN 54.5 against 52.5 TFLOP/s; misaligned 50.5 / 51.1) */
  const bool aligned = a->batch == 1 && !a->a_array && !((p.lda | p.ldb) & 3) &&
                       !((reinterpret_cast<uintptr_t>(p.a + p.a_off) |
                          reinterpret_cast<uintptr_t>(p.b + p.b_off)) & 15);
  if (E == 1 && cfg.tile == 0 && !a_mn && !b_mn && aligned)
    return launch_f32<1, 16, 2, 2, false, false>(p, by, st);
  if (E == 1)
    return cfg.tile == 0 ? launch_ops<1, 8, 2, 4>(p, a_mn, b_mn, by, st)
                         : launch_ops<1, 8, 1, 2>(p, a_mn, b_mn, by, st);
  return cfg.tile == 0 ? launch_ops<2, 16, 2, 2>(p, a_mn, b_mn, by, st)
                       : launch_ops<2, 8, 1, 2>(p, a_mn, b_mn, by, st);
}

/* Tile and split from an estimate of the busiest SM's cycles: the slabs of
 * its CTAs at the rate that many resident CTAs reach, plus each CTA's prologue
 * and epilogue (dearer when a cluster adds up its tile, dearest when clusters
 * queue for more than one wave).  Rates and costs were fitted to measured
 * times of every (tile, split) on 26 shapes each of SGEMM (256^2 x 4000 to
 * 2048^3) and CGEMM; the choice is within 1.8 % of the fastest on average,
 * 18 % at worst.  Splits that are not powers of two pack badly into the GPCs
 * and were never much better. */
extern "C" int hcbk_gemm_f32_plan(int complex, int64_t m, int64_t n, int64_t k, int64_t batch,
                                  hcbk_f32_cfg *cfg, double *us) {
  static const double eff[3][8] = {
      {.72, .83},                                /* 128 x 128, real */
      {.56, .82},                                /* complex */
      {.33, .52, .54, .62, .62, .62, .62, .70}}; /* 64 x 64 */
  static const int resident[2] = {2, 8};
  static const double slab[2] = {2048, 512}; /* FMA cycles of a slab */
  /* per CTA: whole K, split in one wave, split in several */
  static const double cta[2][3] = {{1200, 4800, 20000}, {300, 640, 1100}};
  const int sms = hcbk_sm_count();
  const int64_t slabs = (k + BK - 1) / BK;
  double best = 0;
  cfg->tile = 0;
  cfg->split = 1;
  for (int tile = 0; tile < 2; ++tile) {
    const int64_t b = (tile == 0 ? 128 : 64) / (complex ? 2 : 1);
    const int64_t tiles = ((m + b - 1) / b) * ((n + b - 1) / b) * batch;
    const int res = resident[tile];
    const double *rate = eff[tile ? 2 : complex ? 1 : 0];
    for (int split = 1; split <= MAX_SPLIT && split <= slabs; split *= 2) {
      const double work = (double)((slabs + split - 1) / split) * slab[tile];
      const int64_t ctas = tiles * split, full = ctas / ((int64_t)sms * res);
      const int64_t rem = ctas - full * sms * res, last = (rem + sms - 1) / sms;
      const double extra = cta[tile][split == 1 ? 0 : ctas <= (int64_t)sms * res ? 1 : 2];
      double t = (double)(full * res) * (work / rate[res - 1] + extra);
      if (last) t += (double)last * (work / rate[last - 1] + extra);
      if (split > 1) t += 4400;
      if (best == 0 || t < best) {
        best = t;
        cfg->tile = tile;
        cfg->split = split;
      }
    }
  }
  if (us) *us = 7.0 + best / 1965.0; /* launch, first fetches of the loop's code; at 1965 MHz */
  return HCBK_OK;
}
