// FP64 products of the band space on the FP64 tensor cores (DMMA,
// mma.sync.m16n8k8.f64), fed by TMA: the FP64 path's overlap S = 2 C0^T C0
// (ortho_gs DSYRK, wfn_initialize.f90:481), Lambda = 2 C2^T C0 (OVLAP_D,
// wfn_initialize.f90:234-263), the projections nl = 2 P^T C0
// (pseudopotential.f90:211-213) and dfnl = 2 tpiba Q^T C0
// (nuclear_grad.f90:135,359), and the rotations C2 -= C0 Lambda
// (gradient.f90:31) and C0 U^{-1} (ortho_gs DTRMM, wfn_initialize.f90:485).
// tcgen05 has no FP64 kind, so these are warp-level MMAs; every product is
// exact FP64 arithmetic (a fused multiply-add chain per output in a fixed
// order), like the DGEMM calls of the reference.
//
// TN (out = alpha A^T B over the long real index K; A is K x m and B is
// K x n, both column-major with leading dimension K): output tiles of 64 x 64,
// the (tile, 16-wide k tile) units split evenly over two blocks per SM; one
// copy warp streams the k tiles of A and B (128-byte swizzled TMA boxes of
// 16 x 64) through a 4-stage mbarrier pipeline, four MMA warps each own a
// 32 x 32 quarter of the tile.  The partial tiles go to a buffer that
// k_dgemm_tn_sum adds up in block order (deterministic).  With sym only the
// tiles on and above the diagonal are formed and the sum mirrors them (S is
// symmetric).
//
// NN (out = alpha A G + beta out; A is K x n1 column-major, G is n1 x n
// column-major): persistent blocks over work items of 64 rows of the long
// index x 128 output columns, eight warps each owning 32 rows x 32 columns;
// per 16-band step, A arrives in four TMA boxes and G in two, through a
// 4-stage mbarrier pipeline.
//
// Fragment layout (PTX ISA, mma.m16n8k8 with .f64): A (16 x 8) a0, a1 at rows
// lane/4, lane/4 + 8 of column lane%4, a2, a3 the same of column lane%4 + 4; B
// (8 x 8) rows lane%4, lane%4 + 4 of column lane/4; C (16 x 8) as two 8 x 8
// blocks, rows lane/4 and lane/4 + 8, columns 2 (lane%4) + {0, 1}.
// Each thread reads 16 bytes of shared memory at a time: in TN the two values
// are consecutive k and serve k = t and t + 4 of an MMA (half kb takes the k
// tile's 4 t + 2 kb + {0, 1}, the same set for A and B, so that the eight lanes
// of a quarter warp read eight different 16-byte bank groups of the swizzled
// rows).
//
// Waits are bounded as in the integer-slice kernels: a pipeline wait gives up
// after plim polls, sets *err and the shared abort flag; the block then runs
// its loops to the end without waiting (so every warp reaches the same
// barriers), the copy warp waits (SG_SPIN polls) for its own copies in
// flight, and the results are written as NaN.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "slicegemm.cuh"

namespace amdk {

constexpr int DG_T = 64;    // TN output tile
constexpr int DG_KT = 16;   // doubles per TN k tile (one 128-byte row)
constexpr int DG_ST = 4;    // TN stages
constexpr int DG_THREADS = 160;  // TN: 4 MMA warps + 1 copy warp
constexpr int DG_TN_BPS = 2;     // TN blocks per SM (one: 110 us, two: 83, three: 83 for 128 x 128, K = 64 000)
constexpr int DG_TN_STAGE = 2 * DG_T * DG_KT * 8;  // A and B boxes, 16 KB
constexpr int DG_TN_SMEM = DG_ST * DG_TN_STAGE + 1024 + 2 * DG_ST * 8;
constexpr int DG_NN_R = 64;    // NN: rows of the long index per work item
constexpr int DG_NN_J = 128;   // output columns per work item
constexpr int DG_NN_K = 16;    // bands per pipeline step
constexpr int DG_NN_ST = 4;
constexpr int DG_NN_THREADS = 256;             // 8 MMA warps (thread 0 also issues the TMA copies)
constexpr int DG_NN_A = DG_NN_R * DG_NN_K * 8;  // 4 TMA boxes of 16 rows x 16 bands, 8 KB
constexpr int DG_NN_STAGE = DG_NN_A + DG_NN_J * DG_NN_K * 8;
constexpr int DG_NN_SMEM = DG_NN_ST * DG_NN_STAGE + 1024 + 2 * DG_NN_ST * 8;

// 16 bytes (16-byte chunk `chunk` of row `row`) of a 128-byte-swizzled tile
// of 128-byte rows (the tile 1024-byte aligned)
__device__ __forceinline__ double2 dg_ld_sw(const unsigned char *tile, int row, int chunk) {
  return *reinterpret_cast<const double2 *>(tile + row * 128 + ((chunk ^ (row & 7)) << 4));
}
__device__ __forceinline__ unsigned char *dg_align1k(unsigned char *p) {
  return reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(p) + 1023) & ~(uintptr_t)1023);
}
// tile index -> (it, jt): column-major over mt x nt, or the upper triangle
// (it <= jt) enumerated column by column when sym
__host__ __device__ inline void dg_tile(int tile, int mt, int sym, int &it, int &jt) {
  if (sym) {
    jt = 0;
    while (tile > jt) {
      tile -= jt + 1;
      ++jt;
    }
    it = tile;
  } else {
    it = tile % mt;
    jt = tile / mt;
  }
}

__device__ __forceinline__ void dg_mma16(double (&d)[4], const double2 &a0, const double2 &a1, double b0, double b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0.x), "d"(a1.x), "d"(a0.y), "d"(a1.y), "d"(b0), "d"(b1));
}

// The (tile, k tile) units of a product, tile-major, are split into equal
// contiguous ranges over nb blocks (all resident: every SM gets the same share
// of the work); block b takes [b U / nb, (b+1) U / nb), U = ntile ktiles, and
// leaves one partial tile per output tile it touches, in slots of its own:
// part[(b seg + s) 4096 + i + 64 j], s the tile's place in its range.
__host__ __device__ __forceinline__ int dg_first(int b, long U, int nb) { return (int)(b * U / nb); }
// the block that holds unit u
__host__ __device__ __forceinline__ int dg_block(long u, long U, int nb) {
  const unsigned long x = (unsigned long)(u + 1) * nb - 1;
  return (x >> 32) == 0 ? (int)((unsigned)x / (unsigned)U) : (int)(x / U);
}
// What bounds it: the FP64 tensor pipe (84% active where a block runs).  K =
// 64 000, 128 x 128: 85 -> 83 us, symmetric 68 -> 66 us; K = 256 000,
// 512 x 512: 6.6 -> 4.3 ms, symmetric 3.7 -> 2.4 ms (a grid of tiles x K
// splits before, uneven over the SMs: 320 blocks of three resident per SM).
__global__ void __launch_bounds__(DG_THREADS, 3) k_dgemm_tn(const __grid_constant__ CUtensorMap ta,
                                                                    const __grid_constant__ CUtensorMap tb, int m, int n,
                                                                    int mt, int sym, int ntile, int ktiles, int seg,
                                                                    double *part, int *err, long plim) {
  extern __shared__ unsigned char dg_raw[];
  unsigned char *sm = dg_align1k(dg_raw);
  uint64_t *full = reinterpret_cast<uint64_t *>(sm + DG_ST * DG_TN_STAGE);
  uint64_t *empty = full + DG_ST;
  __shared__ int aborted;
  volatile int *ab = &aborted;
  const long U = (long)ntile * ktiles;
  const int u0 = dg_first(blockIdx.x, U, gridDim.x), u1 = dg_first(blockIdx.x + 1, U, gridDim.x), nk = u1 - u0;
  const int tile0 = u0 / ktiles, kk0 = u0 - tile0 * ktiles;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    aborted = 0;
    for (int s = 0; s < DG_ST; ++s) {
      sg_bar_init(sg_smem(full + s), 1);
      sg_bar_init(sg_smem(empty + s), 4);
    }
    sg_bar_fence_init();
  }
  __syncthreads();
  if (warp == 4) {
    if (lane == 0) {
      int issued = 0, tile = tile0, k = kk0, it, jt;
      dg_tile(tile, mt, sym, it, jt);
      for (int q = 0; q < nk; ++q) {
        const int s = q % DG_ST;
        if (q >= DG_ST && !*ab && !sg_bar_wait(sg_smem(empty + s), ((q / DG_ST) - 1) & 1, err, 31, plim)) *ab = 1;
        if (*ab) break;
        unsigned char *st = sm + s * DG_TN_STAGE;
        sg_bar_expect_tx(sg_smem(full + s), DG_TN_STAGE);
        sg_tma_2d(sg_smem(st), &ta, k * DG_KT, it * DG_T, sg_smem(full + s));
        sg_tma_2d(sg_smem(st + DG_TN_STAGE / 2), &tb, k * DG_KT, jt * DG_T, sg_smem(full + s));
        issued = q + 1;
        if (++k == ktiles) {
          k = 0;
          if (++tile < ntile) dg_tile(tile, mt, sym, it, jt);
        }
      }
      // no copy of this block may land after it exits
      for (int q = max(0, issued - DG_ST); q < issued; ++q)
        sg_bar_wait(sg_smem(full + q % DG_ST), (q / DG_ST) & 1, err, 32);
    }
    return;
  }
  const int wr = warp & 1, wc = warp >> 1, g = lane >> 2, t = lane & 3;
  int q = 0;
  for (int tile = tile0, k = kk0; q < nk; ++tile, k = 0) {
    int it, jt;
    dg_tile(tile, mt, sym, it, jt);
    const int qe = min(nk, q + ktiles - k);
    // a 16 x 8 piece entirely outside m x n (few bands or projectors) has nothing to form
    const int ilive = min(2, (m - it * DG_T - wr * 32 + 15) / 16), jlive = min(4, (n - jt * DG_T - wc * 32 + 7) / 8);
    double acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;
    for (; q < qe; ++q) {
      const int s = q % DG_ST;
      if (!*ab && !sg_bar_wait(sg_smem(full + s), (q / DG_ST) & 1, err, 33, plim)) *ab = 1;
      __syncwarp();
      if (!*ab && ilive > 0 && jlive > 0) {
        const unsigned char *A = sm + s * DG_TN_STAGE, *B = A + DG_TN_STAGE / 2;
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
          double2 a[4], b[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) a[i] = dg_ld_sw(A, wr * 32 + i * 8 + g, 2 * t + kb);
#pragma unroll
          for (int j = 0; j < 4; ++j) b[j] = dg_ld_sw(B, wc * 32 + j * 8 + g, 2 * t + kb);
          if (ilive == 2 && jlive == 4) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
              for (int i = 0; i < 2; ++i) dg_mma16(acc[i][j], a[2 * i], a[2 * i + 1], b[j].x, b[j].y);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (j < jlive)
#pragma unroll
                for (int i = 0; i < 2; ++i)
                  if (i < ilive) dg_mma16(acc[i][j], a[2 * i], a[2 * i + 1], b[j].x, b[j].y);
          }
        }
      }
      __syncwarp();
      if (lane == 0) sg_bar_arrive(sg_smem(empty + s));
    }
    const bool bad = *ab != 0;
    double *p = part + ((long)blockIdx.x * seg + (tile - tile0)) * (DG_T * DG_T);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int r = wr * 32 + i * 16 + 8 * (e >> 1) + g, col = wc * 32 + j * 8 + 2 * t + (e & 1);
          if (i < ilive && j < jlive) p[r + DG_T * col] = bad ? __longlong_as_double(0x7ff8000000000000LL) : acc[i][j][e];
        }
  }
}

// out[i + ldo j] = alpha times the sum of the partial tiles of its tile (i < m,
// j < n).  A block takes 32 consecutive elements of a tile; each of its 8 warps
// sums a contiguous range of the blocks that hold the tile, in order (four
// loads in flight), and warp 0 adds the 8 results in order (deterministic).
// With sym, an element of a tile above the diagonal is written at (i, j) and
// (j, i).
__global__ void __launch_bounds__(256) k_dgemm_tn_sum(const double *part, int nb, int seg, int ntile, int ktiles, int mt,
                                                      int sym, int m, int n, double alpha, double *out, int ldo,
                                                      G0Term g0) {
  __shared__ double red[8][32];
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const long tot = (long)ntile * (DG_T * DG_T), U = (long)ntile * ktiles;
  for (long base = (long)blockIdx.x * 32; base < tot; base += (long)gridDim.x * 32) {
    const int tile = (int)(base / (DG_T * DG_T)), loc = (int)(base % (DG_T * DG_T)) + lane;
    int it, jt;
    dg_tile(tile, mt, sym, it, jt);
    const int i = it * DG_T + loc % DG_T, j = jt * DG_T + loc / DG_T;
    if (jt * DG_T + loc / DG_T >= n) continue;  // the same column for the whole block (32 divides 64)
    const int b0 = dg_block((long)tile * ktiles, U, nb), b1 = dg_block((long)(tile + 1) * ktiles - 1, U, nb) + 1;
    const int qn = (b1 - b0 + 7) / 8, q0 = b0 + grp * qn, q1 = min(b1, q0 + qn);
    double s = 0.0;
    if (i < m) {
      // the tile is the first of every block's range but b0's, which may begin before it
      const long bs = (long)seg * (DG_T * DG_T);
      const double *p = part + loc;
      int q = q0;
      if (grp == 0 && q < q1) s = p[(q++) * bs + (long)(tile - dg_first(b0, U, nb) / ktiles) * (DG_T * DG_T)];
      auto at = [&](int b) { return p[b * bs]; };
      for (; q + 3 < q1; q += 4) {
        const double v0 = at(q), v1 = at(q + 1), v2 = at(q + 2), v3 = at(q + 3);
        s += v0;
        s += v1;
        s += v2;
        s += v3;
      }
      for (; q < q1; ++q) s += at(q);
    }
    red[grp][lane] = s;
    __syncthreads();
    if (grp == 0 && i < m) {
      double v = red[0][lane];
#pragma unroll
      for (int k = 1; k < 8; ++k) v += red[k][lane];
      out[i + (long)ldo * j] = g0(alpha * v, i, j);
      if (sym && it != jt) out[j + (long)ldo * i] = g0(alpha * v, j, i);
    }
    __syncthreads();
  }
}

// out (K x n, leading dimension ldo) = alpha A G + beta out (beta 0: out is
// only written).  ta maps A (K x n1, boxes of 16 rows x 16 bands, 128-byte
// swizzled), tg maps G (n1 x n, boxes of 8 bands x 128 columns).  With upper,
// G is upper triangular (its lower part holds zeros) and the products with the
// lower part are skipped 16 columns at a time.  With g0twice the product's
// rows 0 and 1 (G = 0 of a projector matrix that holds half its value there)
// count twice; with zclean row 1 of out, Im c(G=0), is set to zero (ZCLEAN,
// wfn_initialize.f90:531-558).
// A warp's MMAs take the columns j as the M index and the long index r as N,
// with the n index of two adjacent N tiles interleaved (r = 2n, 2n + 1), so
// that a lane reads 16 bytes of every operand at a time, free of bank
// conflicts (band k = t, t + 4 of an MMA step are 2t, 2t + 1 of a box's
// eight), and owns four consecutive rows of an output column.
// What bounds it: the FP64 tensor pipe.  Two blocks per SM, so that one's
// epilogue (and its reads of the old outputs) runs under the other's MMAs; no
// block-wide barrier in the loop: a warp waits for a stage's copies, and thread
// 0 issues a stage's next copies once every warp has released it.  128 bands,
// K = 64 000: C2 -= C0 Lambda 124 -> 108 us, C0 U^-1 86 -> 72 us; 512 bands,
// K = 256 000: 8.6 -> 4.7 and 8.2 -> 2.5 ms (one block per SM, 64-band steps,
// G copied in 8-byte pieces by all threads, a barrier per step, before).
__global__ void __launch_bounds__(DG_NN_THREADS, 2) k_dgemm_nn(const __grid_constant__ CUtensorMap ta,
                                                               const __grid_constant__ CUtensorMap tg, long K, int n1,
                                                               int n, double alpha, double beta, int upper,
                                                               int g0twice, int zclean, double *out, long ldo, int *err,
                                                               long plim) {
  extern __shared__ unsigned char dg_raw[];
  unsigned char *sm = dg_align1k(dg_raw);
  uint64_t *full = reinterpret_cast<uint64_t *>(sm + DG_NN_ST * DG_NN_STAGE), *empty = full + DG_NN_ST;
  __shared__ int aborted;
  volatile int *ab = &aborted;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int wj = warp >> 1, wr = warp & 1;  // 32 columns x 32 rows of the block's 128 x 64
  const int nrt = (int)((K + DG_NN_R - 1) / DG_NN_R), njt = (n + DG_NN_J - 1) / DG_NN_J, items = nrt * njt;
  auto steps = [&](int jt) {  // 16-band steps of a column tile
    const int nb = upper ? min(n1, (jt + 1) * DG_NN_J) : n1;
    return (nb + DG_NN_K - 1) / DG_NN_K;
  };
  // the block's work is a sequence of steps; thread 0's load cursor runs up to
  // DG_NN_ST - 1 of them ahead
  int lw = blockIdx.x, lk = 0, copies = 0;
  auto load = [&]() {
    const int lrt = lw / njt, ljt = lw - lrt * njt, st = copies % DG_NN_ST;
    unsigned char *As = sm + st * DG_NN_STAGE, *Gs = As + DG_NN_A;
    sg_bar_expect_tx(sg_smem(full + st), DG_NN_STAGE);
#pragma unroll
    for (int i = 0; i < DG_NN_R / 16; ++i)
      sg_tma_2d(sg_smem(As + i * 2048), &ta, lrt * DG_NN_R + 16 * i, lk * DG_NN_K, sg_smem(full + st));
#pragma unroll
    for (int i = 0; i < DG_NN_K / 8; ++i)
      sg_tma_2d(sg_smem(Gs + i * DG_NN_J * 64), &tg, lk * DG_NN_K + 8 * i, ljt * DG_NN_J, sg_smem(full + st));
    ++copies;
    if (++lk >= steps(ljt)) {
      lk = 0;
      lw += gridDim.x;
    }
  };
  if (threadIdx.x == 0) {
    aborted = 0;
    for (int s = 0; s < DG_NN_ST; ++s) {
      sg_bar_init(sg_smem(full + s), 1);
      sg_bar_init(sg_smem(empty + s), DG_NN_THREADS / 32);
    }
    sg_bar_fence_init();
    for (int s = 0; s < DG_NN_ST - 1 && lw < items; ++s) load();
  }
  __syncthreads();
  int q = 0;
  for (int w = blockIdx.x; w < items; w += gridDim.x) {
    const int rt = w / njt, jt = w - rt * njt, j0 = jt * DG_NN_J + 32 * wj, nk = steps(jt);
    // the item's old outputs towards the L2 while its products run
    if (beta != 0.0)
      for (int i = threadIdx.x; i < DG_NN_J * (DG_NN_R / 16); i += DG_NN_THREADS) {
        const int j = jt * DG_NN_J + i / (DG_NN_R / 16);
        const long r = (long)rt * DG_NN_R + 16 * (i % (DG_NN_R / 16));
        if (j < n && r < K) asm volatile("prefetch.global.L2 [%0];" ::"l"(out + r + ldo * j));
      }
    double acc[2][2][2][4];  // [16 columns][16 rows][row parity][fragment]
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[m][p][h][e] = 0.0;
    for (int k = 0; k < nk; ++k, ++q) {
      const int st = q % DG_NN_ST;
      // the load DG_NN_ST - 1 steps ahead goes to the previous step's stage,
      // once every warp has released it
      if (threadIdx.x == 0 && lw < items && !*ab) {
        if (q > 0 && !sg_bar_wait(sg_smem(empty + (q - 1) % DG_NN_ST), ((q - 1) / DG_NN_ST) & 1, err, 34, plim)) *ab = 1;
        else load();
      }
      __syncwarp();
      if (!*ab && !sg_bar_wait(sg_smem(full + st), (q / DG_NN_ST) & 1, err, 36, plim)) *ab = 1;
      __syncwarp();
      const unsigned char *As = sm + st * DG_NN_STAGE + wr * 4096;
      const unsigned char *Gs = sm + st * DG_NN_STAGE + DG_NN_A + (32 * wj + g) * 64 + t * 16;
      // live 16-column tiles: below n and, with upper, not left of these bands
      const int jmin = upper ? k * DG_NN_K : 0;
      const bool on0 = j0 < n && j0 + 15 >= jmin, on1 = j0 + 16 < n && j0 + 31 >= jmin;
      if (!*ab && (on0 || on1)) {
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
          double2 a[2][2], b[2][2];
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              a[m][h] = *reinterpret_cast<const double2 *>(Gs + (kb * DG_NN_J + 16 * m + 8 * h) * 64);
#pragma unroll
          for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
              const int band = 8 * kb + 2 * t + s;
              b[p][s] = *reinterpret_cast<const double2 *>(As + p * 2048 + band * 128 + ((g ^ (band & 7)) << 4));
            }
#pragma unroll
          for (int m = 0; m < 2; ++m)
            if (m == 0 ? on0 : on1)
#pragma unroll
              for (int p = 0; p < 2; ++p) {
                dg_mma16(acc[m][p][0], a[m][0], a[m][1], b[p][0].x, b[p][1].x);
                dg_mma16(acc[m][p][1], a[m][0], a[m][1], b[p][0].y, b[p][1].y);
              }
        }
      }
      __syncwarp();
      if (lane == 0) sg_bar_arrive(sg_smem(empty + st));
    }
    // the eight old values of a 16-column tile are read before its stores
    const bool bad = *ab != 0;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const long r0 = (long)rt * DG_NN_R + 32 * wr + 4 * t;
      double *o = out + r0 + ldo * (j0 + 16 * m + g);
      double2 old[2][2][2];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            old[h][p][e] = beta != 0.0 && j0 + 16 * m + 8 * h + g < n && r0 + 16 * p + 2 * e < K
                               ? *reinterpret_cast<const double2 *>(o + ldo * (8 * h) + 16 * p + 2 * e)
                               : make_double2(0.0, 0.0);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (j0 + 16 * m + 8 * h + g >= n || r0 + 16 * p + 2 * e >= K) continue;
            const double f = g0twice && r0 + 16 * p + e == 0 ? 2.0 * alpha : alpha;
            double2 v = make_double2(f * acc[m][p][0][2 * h + e] + beta * old[h][p][e].x,
                                     f * acc[m][p][1][2 * h + e] + beta * old[h][p][e].y);
            if (zclean && r0 + 16 * p + e == 0) v.y = 0.0;
            if (bad) v.x = v.y = __longlong_as_double(0x7ff8000000000000LL);
            *reinterpret_cast<double2 *>(o + ldo * (8 * h) + 16 * p + 2 * e) = v;
          }
    }
  }
  // no copy of this block may land after it exits
  if (threadIdx.x == 0 && *ab)
    for (int p = max(0, copies - DG_NN_ST); p < copies; ++p)
      sg_bar_wait(sg_smem(full + p % DG_NN_ST), (p / DG_NN_ST) & 1, err, 35);
}

}  // namespace amdk
