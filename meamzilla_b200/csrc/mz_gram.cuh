// FP64 products of row sets over a long shared axis, for Powell's normal
// equations: out[i][j] = sum_k A[i][k] * B[j][k] (i < na, j < nb, k < n).
//
// Powell's linear system is lineqsys = gamma^T gamma and p = -gamma^T e
// (OptPowell::lineqsys_init, opt_powell.cpp:438-472) with one row and p
// redone after each secant update (OptPowell::lineqsys_update,
// opt_powell.cpp:476-493).  gamma is esize x ncoeff; here its columns are
// the rows of A (ncoeff rows of esize doubles, one per coefficient, which is
// how the forward-difference residual vectors come out of the evaluator), so
// every read walks a row and is coalesced.  The reference sums k in one
// sequential loop; here k is cut into S contiguous ranges (one per CTA
// column of the grid), each summed in a fixed order, and k_gram_sum adds the
// S partials in rank order: the result is bit-reproducible for a given
// (na, nb, n, S), and S depends only on the shapes and the SM count.
//
//   k_gram_tile  nb > GRAM_VEC: 64 x 64 output tiles on the FP64 matrix
//                instruction (mma m8n8k4), k streamed through a four-stage
//                cp.async ring of 32-k slices.  When A and B are the same rows
//                only tiles on or above the diagonal run, a diagonal tile
//                loads its rows once and forms its 36 blocks of 8 x 8 on or
//                above the diagonal (the rest is mirrored by k_gram_sum).
//   k_gram_vec   nb <= GRAM_VEC (the update's one or two columns): chunks of
//                1024 k with B's chunk in shared memory, one warp per A row,
//                lanes striding k, a fixed shuffle tree per row and chunk.
//   k_gram_sum   a warp per run of partials, 32 outputs per CTA, the runs in
//                order; k_gram_sum_few a thread per output.
//
// Bytes: k_gram_vec reads A once; k_gram_tile reads each 64-row block of A
// once per output tile it takes part in (ceil(nb / 64) times in all).  The
// vector form is HBM-bound, the square form bound by the FP64 pipe (a 64 x 64
// tile costs an SM 4 cycles per 8 x 8 x 4 step).  The register-tile form
// (4 x 4 per thread, 16 shared-memory wavefronts per 9 cycles of FMA, 510
// partials added by one thread per output) took 126 us for a call with 56 rows
// of 65 k, from host to host; this 46 (one or two CTAs per SM alike, three 4 us
// more).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

namespace mzb {

constexpr int GRAM_T = 64;      // output tile edge of k_gram_tile
constexpr int GRAM_BK = 32;     // k slice staged per step
constexpr int GRAM_VEC = 4;     // largest nb served by k_gram_vec
constexpr int GRAM_FEW = 32;    // ranges up to which k_gram_sum_few adds them
constexpr int GRAM_VK = 1024;   // k chunk of k_gram_vec

struct GramArgs {
  const double *A;
  const double *B;
  int64_t lda, ldb, n;
  int na, nb;
  int sym;      // A and B are the same rows: upper tiles only
  int S;        // k ranges (grid.y of k_gram_tile, grid.x of k_gram_vec)
  int64_t kper; // k per range (multiple of GRAM_BK / GRAM_VK)
  double *partial;  // [S][na][nb]
  double *out;      // [na][nb]
};

// Tile index t of the upper triangle (row-major over tile rows) -> (bi, bj).
__device__ __forceinline__ void gram_upper_tile(int t, int T, int &bi, int &bj) {
  bi = 0;
  int rowlen = T;
  while (t >= rowlen) {
    t -= rowlen;
    ++bi;
    --rowlen;
  }
  bj = bi + t;
}

// D += A B on the FP64 tensor pipe: lane l holds A[l / 4][l % 4],
// B[l % 4][l / 4] and D[l / 4][2 (l % 4)], D[l / 4][2 (l % 4) + 1].
__device__ __forceinline__ void gram_mma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// Rows lie GRAM_LD doubles apart (32 bytes modulo 128: the 4 rows x 4 k that a
// half warp reads are 16 different banks pairs).
constexpr int GRAM_LD = GRAM_BK + 4;
constexpr int GRAM_STAGES = 4;
constexpr size_t GRAM_SMEM_SIDE = sizeof(double) * GRAM_T * GRAM_LD;  // one operand's slice
constexpr size_t gram_smem(bool sym_only) { return GRAM_STAGES * (sym_only ? 1 : 2) * GRAM_SMEM_SIDE; }

// One operand's slice of 64 rows x 32 k; rows and k past the end are zero.
// WIDE: two k per copy (16-byte aligned rows).
template <bool WIDE>
__device__ __forceinline__ void gram_load(double *dst, const double *src, int64_t ld, int rows, int64_t k0, int64_t k1) {
  constexpr int W = WIDE ? 2 : 1, PER = GRAM_BK / W;
  const int k = (threadIdx.x % PER) * W, left = (int)min((int64_t)W, max((int64_t)0, k1 - k0 - k));
#pragma unroll
  for (int r = threadIdx.x / PER; r < GRAM_T; r += 256 / PER) {
    const int bytes = r < rows ? 8 * left : 0;
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst + r * GRAM_LD + k);
    const double *p = bytes ? src + (int64_t)r * ld + k0 + k : src;
    if (WIDE) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(p), "r"(bytes));
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(p), "r"(bytes));
  }
}

template <bool WIDE>
__global__ void __launch_bounds__(256) k_gram_tile(GramArgs g) {
  extern __shared__ __align__(16) double gsm_[];
  const int T = (g.nb + GRAM_T - 1) / GRAM_T;
  int bi, bj;
  if (g.sym) {
    gram_upper_tile(blockIdx.x, T, bi, bj);
  } else {
    bi = blockIdx.x / T;
    bj = blockIdx.x % T;
  }
  const bool diag = g.sym && bi == bj;
  const int s = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t k0 = (int64_t)s * g.kper, k1 = min(g.n, k0 + g.kper);
  const int i0 = bi * GRAM_T, j0 = bj * GRAM_T;
  const int nsl = (int)((k1 - k0 + GRAM_BK - 1) / GRAM_BK);
  const int side = GRAM_T * GRAM_LD, stage = diag ? side : 2 * side;
  auto load = [&](int q) {
    if (q < nsl) {
      double *d = gsm_ + (q % GRAM_STAGES) * stage;
      const int64_t kb = k0 + (int64_t)q * GRAM_BK;
      gram_load<WIDE>(d, g.A + (int64_t)i0 * g.lda, g.lda, g.na - i0, kb, k1);
      if (!diag) gram_load<WIDE>(d + side, g.B + (int64_t)j0 * g.ldb, g.ldb, g.nb - j0, kb, k1);
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  // Blocks of 8 x 8.  A diagonal tile: block rows w and nr - 1 - w to warps w
  // and w + 4 (so that each pair has about as many blocks on or above the
  // diagonal), each of the two half of every slice's k.  Else block row `warp`.
  const int nr = min(8, (g.na - i0 + 7) / 8), nc = min(8, (g.nb - j0 + 7) / 8);
  const int half = warp >> 2, r0 = diag ? (warp & 3) : warp, r1 = nr - 1 - r0;
  const int fr = lane >> 2, fk = lane & 3;
  double acc[12][2];  // blocks (r0, r0 + q) (else (r0, q)), q < 8, and (r1, r1 + q - 8)
#pragma unroll
  for (int q = 0; q < 12; ++q) acc[q][0] = acc[q][1] = 0.0;
  for (int q = 0; q < GRAM_STAGES - 1; ++q) load(q);
  for (int q = 0; q < nsl; ++q) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(GRAM_STAGES - 2));
    __syncthreads();  // slice q is there, and every warp is done with slice q - 1
    load(q + GRAM_STAGES - 1);
    const double *As = gsm_ + (q % GRAM_STAGES) * stage, *Bs = diag ? As : As + side;
    if (diag) {
      if (r0 > r1) continue;
#pragma unroll
      for (int k4 = 0; k4 < GRAM_BK / 8; ++k4) {
        const int k = half * (GRAM_BK / 2) + 4 * k4 + fk;
        const double a0 = As[(8 * r0 + fr) * GRAM_LD + k];
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (r0 + c < nc) gram_mma(acc[c], a0, As[(8 * (r0 + c) + fr) * GRAM_LD + k]);
        if (r1 > r0) {
          const double a1 = As[(8 * r1 + fr) * GRAM_LD + k];
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (r1 + c < nc) gram_mma(acc[8 + c], a1, As[(8 * (r1 + c) + fr) * GRAM_LD + k]);
        }
      }
    } else if (r0 < nr) {
#pragma unroll
      for (int k4 = 0; k4 < GRAM_BK / 4; ++k4) {
        const int k = 4 * k4 + fk;
        const double a = As[(8 * r0 + fr) * GRAM_LD + k];
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (c < nc) gram_mma(acc[c], a, Bs[(8 * c + fr) * GRAM_LD + k]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  if (diag) {  // the second half of k onto the first
    double *x = gsm_ + (size_t)(warp & 3) * 24 * 32 + lane;
    if (half)
#pragma unroll
      for (int q = 0; q < 12; ++q) {
        x[(2 * q) * 32] = acc[q][0];
        x[(2 * q + 1) * 32] = acc[q][1];
      }
    __syncthreads();
    if (half) return;
#pragma unroll
    for (int q = 0; q < 12; ++q) {
      acc[q][0] += x[(2 * q) * 32];
      acc[q][1] += x[(2 * q + 1) * 32];
    }
  }
  double *P = g.partial + (size_t)s * g.na * g.nb;
  auto put = [&](int r, int c, const double (&v)[2]) {
    const int i = i0 + 8 * r + fr, j = j0 + 8 * c + 2 * fk;
    if (i >= g.na) return;
    if (j < g.nb) P[(size_t)i * g.nb + j] = v[0];
    if (j + 1 < g.nb) P[(size_t)i * g.nb + j + 1] = v[1];
  };
  if (diag) {
    if (r0 > r1) return;
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (r0 + c < nc) put(r0, r0 + c, acc[c]);
    if (r1 > r0)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (r1 + c < nc) put(r1, r1 + c, acc[8 + c]);
  } else if (r0 < nr) {
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (c < nc) put(r0, c, acc[c]);
  }
}

__global__ void __launch_bounds__(256) k_gram_vec(GramArgs g) {
  __shared__ double Bs[GRAM_VEC][GRAM_VK];
  const int s = blockIdx.x;
  const int64_t k0 = (int64_t)s * g.kper;
  const int64_t k1 = min(g.n, k0 + g.kper);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // this CTA's sums, row i owned by warp i % nw (its lane 0 alone adds)
  double *P = g.partial + (size_t)s * g.na * g.nb;
  for (int i = warp; i < g.na; i += nw)
    if (lane < g.nb) P[(size_t)i * g.nb + lane] = 0.0;
  for (int64_t kb = k0; kb < k1; kb += GRAM_VK) {
    const int len = (int)min((int64_t)GRAM_VK, k1 - kb);
    __syncthreads();  // the previous chunk's reads of Bs are done
    for (int j = 0; j < g.nb; ++j)
      for (int t = threadIdx.x; t < GRAM_VK; t += blockDim.x)
        Bs[j][t] = t < len ? __ldg(g.B + (int64_t)j * g.ldb + kb + t) : 0.0;
    __syncthreads();
    for (int i = warp; i < g.na; i += nw) {
      const double *a = g.A + (int64_t)i * g.lda + kb;
      double acc[GRAM_VEC] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
      for (int t = lane; t < GRAM_VK; t += 32) {
        const double av = t < len ? __ldg(a + t) : 0.0;
#pragma unroll
        for (int j = 0; j < GRAM_VEC; ++j)
          if (j < g.nb) acc[j] = fma(av, Bs[j][t], acc[j]);
      }
#pragma unroll
      for (int j = 0; j < GRAM_VEC; ++j) {
        double v = acc[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0 && j < g.nb) P[(size_t)i * g.nb + j] += v;
      }
    }
  }
}

// where output t's partials start: of its mirror where only that was computed
__device__ __forceinline__ const double *gram_partials(const GramArgs &g, int t) {
  int i = t / g.nb, j = t % g.nb;
  if (g.sym && j < i) {
    const int x = i;
    i = j;
    j = x;
  }
  return g.partial + (size_t)i * g.nb + j;
}

// Many ranges (few outputs)
__global__ void __launch_bounds__(1024) k_gram_sum(GramArgs g) {
  __shared__ double part[32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = blockIdx.x * 32 + lane, outs = g.na * g.nb;
  const int per = (g.S + 31) / 32, s1 = min(g.S, (warp + 1) * per);
  double v = 0.0;
  if (t < outs) {
    const double *p = gram_partials(g, t);
#pragma unroll 8
    for (int s = warp * per; s < s1; ++s) v += p[(size_t)s * outs];
  }
  part[warp][lane] = v;
  __syncthreads();
  // lane w of warp q: run w of output q, a fixed tree
  v = part[lane][warp];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int q = blockIdx.x * 32 + warp;
  if (lane == 0 && q < outs) g.out[q] = v;
}

// Few ranges, many outputs: a thread per output.  (A CTA of 1024 threads per 32
// outputs made 1000 rows of 5000, one range, a call of 382 us; this 256.)
__global__ void __launch_bounds__(256) k_gram_sum_few(GramArgs g) {
  const int t = blockIdx.x * 256 + threadIdx.x, outs = g.na * g.nb;
  if (t >= outs) return;
  const double *p = gram_partials(g, t);
  double v = 0.0;
#pragma unroll 8
  for (int s = 0; s < g.S; ++s) v += p[(size_t)s * outs];
  g.out[t] = v;
}

// Ranges of k that k_gram_tile's `ntiles` tiles are cut into: an SM runs one
// CTA at a time (eight warps keep its FP64 pipe busy), so the time is that of
// ceil(ntiles S / nsm) rounds of ceil(units / S) slices, plus about three
// slices a round for the pipeline's start and the partials' store, plus
// reading the partials back (a slice takes 1.55 us).  At most four CTAs' worth
// of ranges per SM, which bounds the workspace.  With nsm / ntiles ranges
// 760 rows of 5000 (78 tiles, one range) took 326 us on half of the SMs and
// 1200 rows (190 tiles, a short second round) 677; this rule 166 and 350.
inline int64_t gram_ranges(int64_t ntiles, int64_t units, int64_t outs, int nsm) {
  const int64_t most = std::min(units, (4 * (int64_t)nsm + ntiles - 1) / ntiles);
  int64_t best = 1;
  double t = 1e300;
  for (int64_t rounds = (ntiles + nsm - 1) / nsm, S = 0; S < most; ++rounds) {
    S = std::min(most, rounds * nsm / ntiles);  // the most ranges in this many rounds
    const double x = rounds * ((double)((units + S - 1) / S) + 3.0) + 2.6e-6 * (double)(S * outs);
    if (x < t) {
      t = x;
      best = S;
    }
  }
  return best;
}

}  // namespace mzb
