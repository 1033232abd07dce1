// "Pencil" path for the band-pair transforms of vpsi and eval_density
// (wfn_initialize.f90:283-362, density.f90:19-90) on cubic grids.
//
// The x pass writes the ray buffer transposed, RT[t][kx][ray], so that one
// block can take one x-plane of one band pair: the first y phase reads the
// plane's rays straight from the buffer into the registers of its
// sub-transforms and leaves the slab plane P[zi][ky] in shared memory, then
// per tile of columns the z transform, V(r)*psi and the inverse z transform
// (or the |psi|^2 accumulation), the inverse y transforms, and the last phase
// stores the rays.  Every line transform is the two-level register FFT of
// fft.cuh; the backward y transform leaves its output in the permuted order
// the forward one takes, so no pass reorders data.  No slab or grid buffer
// goes through HBM: the only HBM traffic is the ray buffer (read and written
// once per pass), V (L2 resident) and the coefficients.
#pragma once
#include <type_traits>

#include "fft.cuh"

namespace amdk {

struct PencilGeom {
  int n1, n2, n3, nray;  // n1: x planes of the buffers the plane kernels read
  const int *cols;   // [n2] rays of ky (ray_pack): ray of kz (signed, lo..hi) = off + kz
  const int2 *seg;   // [n2][slab rows] slab decomposition: {seg_r0, position in the segment | segment rays << 16}, {., 0} no ray
  const int *gmapt;  // [n1][nray] G code of (ray, kx): +(ig+1) at +G, -(ig+1) at -G, 0 empty
  // x passes: element kx of the line (pair t, ray r) at t*xt_t + kx*xt_x + r
  long xt_t, xt_x;
  // plane kernels: the rays of plane kx of pair t form row pr = t*pr_t +
  // kx*pr_x.  One GPU: row pr = t*n1 + kx of nray rays.  Slab decomposition:
  // one segment of rays per source rank, as the all-to-all leaves them; the
  // segment whose first ray is r0 and which holds c rays has its row pr at
  // seg_mul*r0 + pr*c.
  int pr_t, pr_x;
  long seg_mul;
};
// ray table entry of a ky: first ray minus lo (17 bits), lo + 64 and hi + 64
// (|kz| < N/4 <= 40); hi < lo: no ray
__host__ __device__ __forceinline__ int ray_pack(int off, int lo, int hi) { return off << 14 | (lo + 64) << 7 | (hi + 64); }
__device__ __forceinline__ int ray_off(int e) { return e >> 14; }
__device__ __forceinline__ int ray_lo(int e) { return ((e >> 7) & 127) - 64; }
__device__ __forceinline__ int ray_hi(int e) { return (e & 127) - 64; }
// the one-GPU layout RT[t][kx][ray]
inline PencilGeom pencil_geom_1gpu(int n1, int n2, int n3, int nray, const int *cols, const int *gmapt) {
  PencilGeom g{};
  g.n1 = n1;
  g.n2 = n2;
  g.n3 = n3;
  g.nray = nray;
  g.cols = cols;
  g.gmapt = gmapt;
  g.xt_t = (long)n1 * nray;
  g.xt_x = nray;
  g.pr_t = n1;
  g.pr_x = 1;
  return g;
}

// Shared-memory rows (slab plane P, column tile S) have odd strides so that
// threads taking consecutive rows hit distinct banks.

constexpr int XL = 32;  // lines per x-pass block
// Backward x pass with the band-pair pack (psi_a + i psi_b, the pack of
// vpsi and eval_density), output transposed: RT[t][kx][r] on one GPU, the
// slab decomposition's send layout [kx][t][r] (strides xt_t, xt_x).  Block = XL lines
// (consecutive rays) x N2 threads; thread (l, j2) gathers the N1 elements
// kx = j2 + N2*j1 of its ray straight from the coefficients, the second
// phase writes kx = k1 + N1*k2 back with consecutive threads on consecutive
// rays.
template <typename C, int N>
__global__ void __launch_bounds__(512) k_xt_bwd_pair(const double2 *__restrict__ c0, int ngpw, int nstate, int band0,
                                                     int T, PencilGeom pg, Plan<C> p, C *__restrict__ rt) {
  typedef decltype(C().x) Rl;
  constexpr int N1 = fft_n1(N), N2 = N / N1, NP = N + 1;
  extern __shared__ unsigned char smraw[];
  C *S = reinterpret_cast<C *>(smraw);
  C *tw = S + XL * NP;
  load_tw<C, N>(tw, p);
  __syncthreads();
  const int R = pg.nray;
  const long line0 = (long)blockIdx.x * XL;
  const long nlines = (long)T * R;
  {
    const int l = threadIdx.x % XL, j2 = threadIdx.x / XL;
    const long line = line0 + l;
    C v[N1];
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) v[j1] = czero<C>();
    if (line < nlines) {
      const int t = (int)(line / R), r = (int)(line % R);
      const int ba = band0 + 2 * t, bb = ba + 1;
      const double2 *ca = c0 + (long)ba * ngpw;
      const double2 *cb = c0 + (long)bb * ngpw;
      const bool hb = bb < nstate;
#pragma unroll
      for (int j1 = 0; j1 < N1; ++j1) {
        const int code = pg.gmapt[(long)(j2 + N2 * j1) * R + r];
        const int ig = (code > 0 ? code : -code) - 1;
        if (code != 0 && ig < ngpw) {
          const double2 a = ca[ig];
          const double2 b = hb ? cb[ig] : make_double2(0.0, 0.0);
          if (code > 0) v[j1] = mk((Rl)(a.x - b.y), (Rl)(a.y + b.x));
          else v[j1] = mk((Rl)(a.x + b.y), (Rl)(-a.y + b.x));
        }
      }
    }
    Dft<C, N1, 1>::run(v);
    twiddle_tab<C, N, N1, 1, 0>(v, j2, tw);
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) S[l * NP + k1 * N2 + j2] = v[k1];
  }
  __syncthreads();
  if (threadIdx.x < XL * N1) {
    const int l = threadIdx.x % XL, k1 = threadIdx.x / XL;
    const long line = line0 + l;
    C u[N2];
#pragma unroll
    for (int j2 = 0; j2 < N2; ++j2) u[j2] = S[l * NP + k1 * N2 + j2];
    Dft<C, N2, 1>::run(u);
    if (line < nlines) {
      const int t = (int)(line / R), r = (int)(line % R);
      C *o = rt + t * pg.xt_t + r;
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) o[(long)(k1 + N1 * k2) * pg.xt_x] = u[k2];
    }
  }
}

// Forward x pass in place on the transposed ray buffer (same blocking)
template <typename C, int N>
__global__ void __launch_bounds__(512) k_xt_fwd(int T, PencilGeom pg, Plan<C> p, C *__restrict__ rt) {
  constexpr int N1 = fft_n1(N), N2 = N / N1, NP = N + 1;
  extern __shared__ unsigned char smraw[];
  C *S = reinterpret_cast<C *>(smraw);
  C *tw = S + XL * NP;
  load_tw<C, N>(tw, p);
  __syncthreads();
  const int R = pg.nray;
  const long line0 = (long)blockIdx.x * XL;
  const long nlines = (long)T * R;
  {
    const int l = threadIdx.x % XL, j2 = threadIdx.x / XL;
    const long line = line0 + l;
    C v[N1];
    if (line < nlines) {
      const int t = (int)(line / R), r = (int)(line % R);
      const C *in = rt + t * pg.xt_t + r;
#pragma unroll
      for (int j1 = 0; j1 < N1; ++j1) v[j1] = in[(long)(j2 + N2 * j1) * pg.xt_x];
    } else {
#pragma unroll
      for (int j1 = 0; j1 < N1; ++j1) v[j1] = czero<C>();
    }
    Dft<C, N1, -1>::run(v);
    twiddle_tab<C, N, N1, -1, 0>(v, j2, tw);
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) S[l * NP + k1 * N2 + j2] = v[k1];
  }
  __syncthreads();
  if (threadIdx.x < XL * N1) {
    const int l = threadIdx.x % XL, k1 = threadIdx.x / XL;
    const long line = line0 + l;
    C u[N2];
#pragma unroll
    for (int j2 = 0; j2 < N2; ++j2) u[j2] = S[l * NP + k1 * N2 + j2];
    Dft<C, N2, -1>::run(u);
    if (line < nlines) {
      const int t = (int)(line / R), r = (int)(line % R);
      C *o = rt + t * pg.xt_t + r;
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) o[(long)(k1 + N1 * k2) * pg.xt_x] = u[k2];
    }
  }
}

// The wavefunction sphere reaches |k| < N/4 on every axis of an N-point grid
// that holds the density sphere (twice the radius), so a slab of H = (N-1)/4
// planes on each side of kz = 0 holds every ray, and of the N1
// elements k = j2 + N2 j1 of a first-phase sub-transform only j1 < LO (k >= 0)
// and j1 >= HI (k < 0) can be inside it: the others are neither stored, read
// nor added.
template <int N, int M1 = fft_n1(N)> struct Sphere {
  static constexpr int N1 = M1, N2 = N / N1;
  static constexpr int H = (N - 1) / 4, NZ = 2 * H + 1;   // the slab: kz = -H .. H
  static constexpr int LO = H / N2 + 1;                   // k <= H lies in j1 < LO
  static constexpr int HI = (N - H) / N2;                 // k >= N - H lies in j1 >= HI
  // slab plane of kz = j2 + N2 j1: zi = kz, or kz - (N - NZ) for kz < 0
  __host__ __device__ static constexpr int row(int j1) { return N2 * j1 - (j1 >= HI ? N - NZ : 0); }
  // whether j1's element is in the slab (a test of j2 only where j1 straddles its edge)
  static __device__ __forceinline__ bool in(int j1, int j2) {
    if (j1 < LO) return N2 * j1 + N2 - 1 <= H || j2 <= H - N2 * j1;
    if (j1 >= HI) return N2 * j1 >= N - H || j2 >= N - H - N2 * j1;
    return false;
  }
};

// Rays of a slab plane.  SEG = false (one GPU): the rays of a ky are those of
// kz = lo .. hi (signed), consecutive in the buffer; SEG = true (the segments
// of a slab decomposition): looked up per (ky, zi).  Each thread (row zi, j2)
// of the first y phase takes its elements ky = j2 + N2 j1 straight from the
// ray buffer (consecutive threads, consecutive kz), and the last y phase
// stores them there: no scatter into or gather from the shared plane, and no
// zero fill.
template <typename C, int N, bool SEG> struct PlaneRays {
  typedef Sphere<N> Sp;
  static constexpr int N1 = fft_n1(N), N2 = N / N1;
  template <bool LOAD> static __device__ __forceinline__ void each(C *rt, const PencilGeom &pg, const int *cols, long pr,
                                                                   int zi, int j2, C (&v)[N1]) {
    const int kz = zi <= Sp::H ? zi : zi - Sp::NZ;  // signed
    C *base = rt + pr * pg.nray + kz;
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) {
      if (j1 >= Sp::LO && j1 < Sp::HI) {
        if (LOAD) v[j1] = czero<C>();
        continue;
      }
      const int ky = j2 + N2 * j1;
      C *at = nullptr;
      if constexpr (SEG) {
        const int2 e = pg.seg[ky * Sp::NZ + zi];
        if (e.y) at = rt + pg.seg_mul * e.x + pr * (e.y >> 16) + (e.y & 0xffff);
      } else {
        const int e = cols[ky];
        if (kz >= ray_lo(e) && kz <= ray_hi(e)) at = base + ray_off(e);
      }
      if (LOAD) v[j1] = at ? *at : czero<C>();
      else if (at) *at = v[j1];
    }
  }
};

// The same elements in a block's own dense scratch plane [ky][zi] (NZ x NZ)
template <typename C, int N> struct PartRays {
  typedef Sphere<N> Sp;
  static constexpr int N1 = fft_n1(N), N2 = N / N1;
  template <bool LOAD> static __device__ __forceinline__ void each(C *part, int zi, int j2, C (&v)[N1]) {
    C *at = part + zi + j2 * Sp::NZ;
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) {
      if (LOAD) v[j1] = czero<C>();
      if (Sp::in(j1, j2)) {
        if (LOAD) v[j1] = at[Sp::row(j1) * Sp::NZ];
        else at[Sp::row(j1) * Sp::NZ] = v[j1];
      }
    }
  }
};

// Length-N transforms of the rows of a shared plane P (row stride NP), each in
// two phases whose sub-transforms read and write the same positions, one
// barrier between them.  The outer phases (y1, y4) exchange with the ray
// buffer; the inner ones:
//   y2: X[k1 + N1*k2] left at position i*N2 + k2 for the NK k1 = ga*i + gr
//   y3: that order in, the first phase of the transform back
template <typename C, int N, int NT, int NP, int NK, int SG, bool TW>
__device__ __forceinline__ void rows_inner(C *P, const C *tw, int ga, int gr) {
  constexpr int N1 = fft_n1(N), N2 = N / N1, NZ = Sphere<N>::NZ;
  for (int idx = threadIdx.x; idx < NZ * NK; idx += NT) {
    const int i = idx / NZ, r = idx - i * NZ;
    C *row = P + r * NP + i * N2;
    C u[N2];
#pragma unroll
    for (int j = 0; j < N2; ++j) u[j] = row[j];
    Dft<C, N2, SG>::run(u);
    if constexpr (TW) twiddle_tab<C, N, N2, SG, 1>(u, ga * i + gr, tw);
#pragma unroll
    for (int j = 0; j < N2; ++j) row[j] = u[j];
  }
}
// Backward z transform of a column, first phase: thread (column, j2) takes
// the slab planes kz = j2 + N2 j1 and leaves W_N^(j2 k1) DFT_N1 in the
// column's tile row (N = N1 N2 as fft_n1 splits it, or the other way round:
// twiddle table 1 holds the rows of that split).
template <typename C, int N, int NP, int N1>
__device__ __forceinline__ void zcol_first(const C *Pq, C *srow, int j2, const C *tw) {
  typedef Sphere<N, N1> Sp;
  constexpr int N2 = N / N1, TAB = N1 == fft_n1(N) ? 0 : 1;
  const C *Pj = Pq + j2 * NP;
  C v[N1];
#pragma unroll
  for (int j1 = 0; j1 < N1; ++j1) v[j1] = Sp::in(j1, j2) ? Pj[Sp::row(j1) * NP] : czero<C>();
  Dft<C, N1, 1>::template run_in<Sp::LO, Sp::HI>(v);
  twiddle_tab<C, N, N1, 1, TAB>(v, j2, tw);
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1) srow[k1 * N2 + j2] = v[k1];
}

// The k1's of a y transform fall into GA groups, group r holding k1 = r mod
// GA: the radix-GA first stage of a backward transform (last stage of a
// forward one) separates them at no extra arithmetic, so a block can take the
// columns of one group at a time with 1/GA of the slab plane in shared memory.
__host__ __device__ constexpr int col_groups(int n) { return fft_n1(n) % 2 == 0 ? 2 : 3; }
// first phase of a row's backward y transform, the outputs k1 = R mod GA only
// (R a template argument, so that the other groups' sub-transforms are dropped)
template <typename C, int N, int GA, int R>
__device__ __forceinline__ void y1_group(C (&v)[fft_n1(N)], C *row, const C *tr) {
  constexpr int N1 = fft_n1(N), N2 = N / N1;
  Dft<C, N1, 1>::template run_in<Sphere<N>::LO, Sphere<N>::HI>(v);
#pragma unroll
  for (int i = 0; i < N1 / GA; ++i) {
    C tv = tr[GA * i + R];
    tv.y = -tv.y;
    row[i * N2] = R + i == 0 ? v[0] : cmul(v[GA * i + R], tv);
  }
}
template <typename C, int N, int GA>
__device__ __forceinline__ void y1_store(C (&v)[fft_n1(N)], int r, C *row, const C *tr) {
  if (GA == 1 || r == 0) y1_group<C, N, GA, 0>(v, row, tr);
  else if (r == 1) y1_group<C, N, GA, GA == 1 ? 0 : 1>(v, row, tr);
  else y1_group<C, N, GA, GA - 1>(v, row, tr);
}
// last phase of a row's forward y transform from the k1 = R mod GA inputs
// (the other groups' share is added by the caller)
template <typename C, int N, int GA, int R>
__device__ __forceinline__ void y4_group(C (&x)[fft_n1(N)], const C *row) {
  constexpr int N1 = fft_n1(N), N2 = N / N1;
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1) x[k1] = k1 % GA == R ? row[(k1 / GA) * N2] : czero<C>();
  Dft<C, N1, -1>::template run_out<GA, R>(x);
}
template <typename C, int N, int GA>
__device__ __forceinline__ void y4_load(C (&x)[fft_n1(N)], int r, const C *row) {
  if (GA == 1 || r == 0) y4_group<C, N, GA, 0>(x, row);
  else if (r == 1) y4_group<C, N, GA, GA == 1 ? 0 : 1>(x, row);
  else y4_group<C, N, GA, GA - 1>(x, row);
}

// Launch shape of the pencil kernels for a length and a precision, all fixed
// at compile time (strides and offsets are then immediates).  NT threads per
// block; the registers of a sub-transform (up to 128 in FP64, 64 to 80 in
// FP32) allow 16 FP64 or 24 to 32 FP32 warps per SM, as one block of 512 or
// two of 256 threads in FP64, two of 512 or three of 256 in FP32.  A tile of
// w columns is w N2 tasks, one per thread at most; of the two block sizes the
// one whose tiles keep clearly more threads busy is taken, else the larger.
constexpr size_t PENCIL_SMEM = 227 * 1024;
constexpr size_t pencil_smem_bytes(size_t csize, int n, int np, int w) {
  return (size_t)(n * 4 + 15) / 16 * 16 + csize * ((size_t)(2 * ((n - 1) / 4) + 1) * np + (size_t)w * (n + 1));
}
// widest equal tiles of nc columns with w n2 <= nt and `blocks` blocks per SM (0: none)
constexpr int pencil_width(size_t csize, int n, int nc, int nt, int blocks, int n2) {
  for (int t = 1; t <= nc; ++t) {
    const int w = (nc + t - 1) / t;
    if (w * n2 <= nt && (pencil_smem_bytes(csize, n, nc | 1, w) + 1024) * blocks <= PENCIL_SMEM + 1024) return w;
  }
  return 0;
}
constexpr int pencil_blocks(size_t csize, int nt) { return csize == 16 ? 512 / nt : (nt == 256 ? 3 : 2); }
constexpr int pencil_tiles(int nc, int w) { return w > 0 ? (nc + w - 1) / w : 4096; }
// V(r)psi.  The whole plane (GA = 1) where a tile then still keeps half of a
// block's threads busy, else one group of its columns at a time.
// Both sides of the rules, 64 pairs, us a launch, the rule's choice first:
//   whole plane | groups   FP64 100^3 473 | 580, 128^3 1001 | 1225; FP32 100^3
//     241 | 296, 160^3 1099 | 1222; at every length the whole plane is faster,
//     by 2% (48^3 FP64) to 77% (108^3 FP32).  FP64 160^3: groups 3155 | 4548.
//   256 threads | 512   FP64 36^3 30 | 41, 60^3 115 | 134, 72^3 185 | 223,
//     96^3 431 | 430; FP32 36^3 19 | 24, 60^3 70 | 76, 72^3 100 | 109, 96^3
//     235 | 217
//   512 threads | 256   FP64 48^3 71 | 60, 64^3 123 | 107, 80^3 269 | 252, 90^3
//     395 | 391, 100^3 473 | 494, 108^3 639 | 685; FP32 48^3 40 | 36, 64^3
//     66 | 60, 80^3 137 | 139, 90^3 205 | 209, 100^3 241 | 255, 108^3 340 | 357,
//     120^3 434 | 479, 128^3 497 | 687.  The count of busy threads misses what
//     else the smaller blocks bring at 48, 64 and 80 and cost at 96.
//   FP32 of 512 threads: two blocks at 144^3 745 | one 797, one at 160^3 1099 |
//     two 1775
template <typename C, int N> struct VpsiShape {
  static constexpr int N1 = fft_n1(N), N2 = N / N1;
  static constexpr size_t cs = sizeof(C);
  static constexpr int whole = pencil_width(cs, N, N, 512, 1, N2);
  static constexpr int GA = 2 * whole * N2 >= 512 || 2 * whole >= N ? 1 : col_groups(N), GC = N / GA;
  static constexpr int w2 = pencil_width(cs, N, GC, 512, pencil_blocks(cs, 512), N2),
                       w1 = pencil_width(cs, N, GC, 512, 1, N2),
                       ws = pencil_width(cs, N, GC, 256, pencil_blocks(cs, 256), N2);
  static constexpr int wl = 2 * w2 >= w1 ? w2 : w1;  // 512 threads: one block per SM only for tiles over twice as wide
  // share of busy threads: N*N2 tasks over tiles x threads
  static constexpr bool small = ws > 0 && 10 * pencil_tiles(GC, wl) * 512 > 11 * pencil_tiles(GC, ws) * 256;
  static constexpr int NT = small ? 256 : 512, W = small ? ws : wl;
  static constexpr int MINB = small ? pencil_blocks(cs, 256) : (wl == w2 ? pencil_blocks(cs, 512) : 1);
  static constexpr size_t smem = pencil_smem_bytes(cs, N, GC | 1, W);
};
// Density: one column group at a time, or the whole plane where three groups
// would read and transform its rays three times and the whole plane's sums are
// no more than 20.  The sums stay in registers, NS tiles x Z2 values per thread:
// long second phases take the split of the z transform the other way round
// (Z1 x Z2), where the sums take more than 20 registers a block of 512 FP32
// threads has the SM to itself, and blocks of 256 take more than 20 only where
// a larger block would leave over two fifths of its threads idle (96 points).
// Both sides of the rules, 64 pairs, us a launch with its reduction, the rule's
// choice first:
//   256 threads | 512   FP64 36^3 32 | 44, 48^3 46 | 65, 64^3 73 | 93, 96^3
//     286 | 341; FP32 36^3 26 | 30, 48^3 34 | 41, 64^3 49 | 58, 96^3 166 | 247
//   512 threads | 256   FP64 60^3 96 | 91, 72^3 141 | 144, 80^3 180 | 178, 100^3
//     305 | 307, 108^3 537 | 486, 120^3 630 | 564, 128^3 660 | 675, 144^3
//     945 | 1114, 160^3 1734 | 5494; FP32 60^3 61 | 61, 72^3 85 | 83, 80^3
//     105 | 101, 100^3 181 | 185, 108^3 285 | 300, 120^3 409 | 337, 128^3
//     338 | 363, 144^3 575 | 612, 160^3 997 | 804 (with 4 pairs 256 threads take
//     2 to 8% more at 120 and 160)
//   the whole density call: whole plane | three groups   90^3 FP64 64 pairs
//     316 | 408, 16 pairs 120 | 137, 4 pairs 68 | 69; FP32 198 | 255, 87 | 97,
//     61 | 60.  Three groups | whole plane   108^3 FP64 736 | 625, 229 | 211,
//     110 | 107; FP32 387 | 341, 141 | 145, 77 | 97
//   two FP32 blocks of 512 | one   60^3 61 | 71, 72^3 85 | 96, 80^3 105 | 120,
//     100^3 181 | 197, 108^3 285 | 392, 128^3 338 | 433
//   one FP32 block of 512 | two   120^3 409 | 355, 144^3 575 | 521, 160^3
//     997 | 854: above 20 sums two blocks spill and are faster all the same where
//     there are many pairs
//   z split swapped | as it is   128^3 FP64 660 | 665, FP32 338 | 430; 160^3
//     1734 | 1915, 997 | 1012
//   z split as it is | swapped   FP64 72^3 141 | 146, 120^3 630 | 636; FP32 72^3
//     85 | 85, 108^3 285 | 288, 120^3 409 | 346 (there the swap also takes the
//     sums from 24 to 20)
template <typename C, int N> struct DensShape {
  static constexpr size_t cs = sizeof(C);
  static constexpr bool swap = N / fft_n1(N) > 12;
  static constexpr int Z1 = swap ? N / fft_n1(N) : fft_n1(N), Z2 = N / Z1, ZM = Z1 > Z2 ? Z1 : Z2;
  static constexpr int whole = pencil_width(cs, N, N, 512, pencil_blocks(cs, 512), ZM);
  static constexpr int GA = col_groups(N) == 3 && pencil_tiles(N, whole) * Z2 <= 20 ? 1 : col_groups(N), GC = N / GA;
  static constexpr int w2 = pencil_width(cs, N, GC, 512, pencil_blocks(cs, 512), ZM),
                       ws = pencil_width(cs, N, GC, 256, pencil_blocks(cs, 256), ZM);
  static constexpr bool two = w2 > 0 && (cs == 16 || pencil_tiles(GC, w2) * Z2 <= 20);
  static constexpr int wl = two ? w2 : pencil_width(cs, N, GC, 512, 1, ZM);
  static constexpr bool small = ws > 0 && (pencil_tiles(GC, ws) * Z2 <= 20 || 5 * wl * ZM < 3 * 512) &&
                                20 * pencil_tiles(GC, wl) * 512 >= 21 * pencil_tiles(GC, ws) * 256;
  static constexpr int NT = small ? 256 : 512, W = small ? ws : wl, NS = pencil_tiles(GC, W);
  static constexpr int MINB = small ? pencil_blocks(cs, 256) : (two ? pencil_blocks(cs, 512) : 1);
  static constexpr size_t smem = pencil_smem_bytes(cs, N, GC | 1, W);
};

// shared memory of a pencil block: the ray table of the ky's, P[NZ][NP],
// S[w][N+1]
template <typename C, int N> struct PencilSmem {
  int *cols;
  C *P, *S;
  __device__ __forceinline__ PencilSmem(unsigned char *raw, int NP) {
    cols = reinterpret_cast<int *>(raw);
    P = reinterpret_cast<C *>(raw + (N * 4 + 15) / 16 * 16);
    S = P + Sphere<N>::NZ * NP;
  }
  __device__ __forceinline__ void load(const PencilGeom &pg) {
    if (pg.cols)
      for (int i = threadIdx.x; i < N; i += blockDim.x) cols[i] = pg.cols[i];
  }
};

// V(r) psi (vpsi, wfn_initialize.f90:311-340): x-planes of band pairs through
// y, z, V(r), z, y.  Persistent blocks, each taking the (pair, plane) units
// blockIdx.x, + gridDim.x, ..., and of each unit the GA column groups in turn.
// P[zi][c] holds the slab plane; after the backward y transform column
// c = i*N2 + k2 of group r carries ky = k1 + N1*k2, k1 = r + GA*i, and the
// position q = k1*N2 + k2.  vp[kx][k'][q] is V at that ky and at
// kz = k'/N2 + N1*(k'%N2), the order in which the z transform leaves psi
// (consecutive threads, consecutive q).
// Column tiles are W wide; a thread keeps its (column, j2) from tile to tile,
// so a tile's last phase and the next tile's first one touch the same
// positions of S and need no barrier between them; the same holds for a
// group's last y phase and the next one's first, which is also where the next
// rays are loaded.  With GA > 1 the groups' shares of a unit's rays are summed
// in `scratch` (nray elements per block, L2 resident) and stored with the
// last one, after every read of the unit's rays.
// What bounds it: shared-memory bandwidth (60-80% of the LSU data pipe) and,
// in FP64, the FP64 pipe (45%) with 16 warps per SM to overlap them; HBM 5%.
// Tables read from the constant bank, no zero fill, scatter or gather pass
// through the plane, transforms pruned at their zero inputs and unused
// outputs, strides and tiles known at compile time.  64 pairs on 100^3: FP64
// 814 -> 485 us, FP32 402 -> 262 us; on 72^3 FP32 165 -> 110 us; on 160^3 FP32
// 2537 -> 1074 us, FP64 (8 pairs) 675 -> 400 us (one block per (plane, pair),
// the plane scattered, zero filled and gathered in shared memory, before).
// LSD (open shell): pair gp0 + t takes the spin-2 potential vp2 from pair
// psplit on, and the pair pstraddle (whose first band is the last of spin 1)
// multiplies its real part by V_1 and its imaginary part by V_2
// (wfn_initialize.f90:313-326).
template <typename C, int N, bool SEG, bool LSD>
__global__ void __launch_bounds__(VpsiShape<C, N>::NT, VpsiShape<C, N>::MINB)
    k_pencil_vpsi(const PencilGeom pg, const __grid_constant__ FftTw<C, N> p, C *__restrict__ rt,
                  const decltype(C().x) *__restrict__ vp, int units, C *__restrict__ scratch,
                  const decltype(C().x) *__restrict__ vp2, int gp0, int psplit, int pstraddle) {
  typedef decltype(C().x) Rl;
  typedef VpsiShape<C, N> Sh;
  typedef PlaneRays<C, N, SEG> Rays;
  typedef Sphere<N> Sp;
  constexpr int N1 = fft_n1(N), N2 = N / N1, NT = Sh::NT, W = Sh::W, GA = Sh::GA, GC = Sh::GC, NK = N1 / GA;
  constexpr int NP = GC | 1, NS = N + 1, NZ = Sp::NZ;
  extern __shared__ __align__(16) unsigned char smraw[];
  PencilSmem<C, N> sm(smraw, NP);
  C *P = sm.P, *S = sm.S;
  sm.load(pg);
  const C *tw = p.t;
  __syncthreads();
  auto row_of = [&](int u) {
    const int t = u / pg.n1, kx = u - t * pg.n1;
    return (long)t * pg.pr_t + (long)kx * pg.pr_x;
  };
  if ((int)blockIdx.x < units) {
    const long pr = row_of(blockIdx.x);
    for (int idx = threadIdx.x; idx < NZ * N2; idx += NT) {
      const int j2 = idx / NZ, zi = idx - j2 * NZ;
      C v[N1];
      Rays::template each<true>(rt, pg, sm.cols, pr, zi, j2, v);
      y1_store<C, N, GA>(v, 0, P + zi * NP + j2, tw + j2 * N1);
    }
  }
  C *part = GA > 1 ? scratch + (long)blockIdx.x * NZ * NZ : nullptr;
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    const int t = u / pg.n1, kx = u - t * pg.n1;
    const long pr = (long)t * pg.pr_t + (long)kx * pg.pr_x;
    const Rl *V = vp + (long)kx * N * N;
    const Rl *V2 = nullptr;
    bool straddle = false;
    if constexpr (LSD) {
      const int gp = gp0 + t;
      if (gp == pstraddle) {
        straddle = true;
        V2 = vp2 + (long)kx * N * N;
      } else if (gp >= psplit) {
        V = vp2 + (long)kx * N * N;
      }
    }
    for (int r = 0; r < GA; ++r) {
      // position q of group r's column c
      auto vcol = [&](int c) {
        if constexpr (GA == 1) return c;
        const int i = c / N2;
        return (r + GA * i) * N2 + c - i * N2;
      };
      __syncthreads();
      rows_inner<C, N, NT, NP, NK, 1, false>(P, tw, GA, r);
      __syncthreads();
      const int a0 = threadIdx.x / W, qq0 = threadIdx.x - a0 * W;  // this thread's first (k1, column) of a tile
      for (int idx = threadIdx.x; idx < W * N2; idx += NT) {
        const int j2 = idx / W, qq = idx - j2 * W;
        zcol_first<C, N, NP, N1>(P + qq, S + qq * NS, j2, tw);
      }
      for (int q0 = 0; q0 < GC; q0 += W) {
        const int ct = min(W, GC - q0);
        // V of this thread's first middle task, in flight across the barrier
        const bool has0 = a0 < N1 && qq0 < ct;
        Rl v0[N2];
        {
          const Rl *vv = V + (long)(a0 * N2) * N + vcol(q0 + qq0);
#pragma unroll
          for (int k2 = 0; k2 < N2; ++k2) v0[k2] = has0 ? vv[k2 * N] : (Rl)0;
        }
        __syncthreads();
        // DFT_N2 -> psi(kz = k1 + N1*k2), times V, then the first phase of the
        // forward z transform, in registers
        for (int idx = threadIdx.x; idx < W * N1; idx += NT) {
          const int k1 = idx / W, qq = idx - k1 * W;
          if (qq >= ct) continue;
          if (idx != threadIdx.x) {
            const Rl *vv = V + (long)(k1 * N2) * N + vcol(q0 + qq);
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) v0[k2] = vv[k2 * N];
          }
          C *row = S + qq * NS + k1 * N2;
          C x[N2];
#pragma unroll
          for (int j2 = 0; j2 < N2; ++j2) x[j2] = row[j2];
          Dft<C, N2, 1>::run(x);
          if (LSD && straddle) {
            const Rl *vg2 = V2 + (long)(k1 * N2) * N + vcol(q0 + qq);
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) {
              x[k2].x = x[k2].x * v0[k2];
              x[k2].y = x[k2].y * vg2[k2 * N];
            }
          } else {
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) x[k2] = cscale(x[k2], v0[k2]);
          }
          Dft<C, N2, -1>::run(x);
          twiddle_tab<C, N, N2, -1, 1>(x, k1, tw);
#pragma unroll
          for (int n2 = 0; n2 < N2; ++n2) row[n2] = x[n2];
        }
        __syncthreads();
        // second phase: x(kz = n2 + N2*n1) for the slab planes only; then the
        // first phase of the next tile's column
        for (int idx = threadIdx.x; idx < W * N2; idx += NT) {
          const int n2 = idx / W, qq = idx - n2 * W;
          C *srow = S + qq * NS;
          if (qq < ct) {
            C x[N1];
#pragma unroll
            for (int k1 = 0; k1 < N1; ++k1) x[k1] = srow[k1 * N2 + n2];
            Dft<C, N1, -1>::template run_out<1, 0>(x);
            C *Pj = P + q0 + qq + n2 * NP;
#pragma unroll
            for (int n1 = 0; n1 < N1; ++n1)
              if (Sp::in(n1, n2)) Pj[Sp::row(n1) * NP] = x[n1];
          }
          if (q0 + W + qq < GC) zcol_first<C, N, NP, N1>(P + q0 + W + qq, srow, n2, tw);
        }
      }
      __syncthreads();
      rows_inner<C, N, NT, NP, NK, -1, true>(P, tw, GA, r);
      __syncthreads();
      const bool last = r == GA - 1;
      const int un = last ? u + (int)gridDim.x : u, rn = last ? 0 : r + 1;
      const long prn = un < units ? row_of(un) : 0;
      for (int idx = threadIdx.x; idx < NZ * N2; idx += NT) {
        const int n2 = idx / NZ, zi = idx - n2 * NZ;
        C v[N1];
        if (un < units) Rays::template each<true>(rt, pg, sm.cols, prn, zi, n2, v);
        {
          C x[N1];
          if constexpr (GA > 1) {
            C q[N1];
            if (r > 0) PartRays<C, N>::template each<true>(part, zi, n2, q);
            y4_load<C, N, GA>(x, r, P + zi * NP + n2);
            if (r > 0)
#pragma unroll
              for (int n1 = 0; n1 < N1; ++n1) x[n1] = cadd(x[n1], q[n1]);
          } else {
            y4_load<C, N, GA>(x, r, P + zi * NP + n2);
          }
          if (GA == 1 || last) Rays::template each<false>(rt, pg, sm.cols, pr, zi, n2, x);
          else PartRays<C, N>::template each<false>(part, zi, n2, x);
        }
        if (un < units) y1_store<C, N, GA>(v, rn, P + zi * NP + n2, tw + n2 * N1);
      }
    }
  }
}

// Density (density.f90:49-86): rho_part += wa_t Re^2 + wb_t Im^2 over band
// pairs, in the permuted (ky, kz) order, one column group of an x-plane at a
// time.  The (plane, group, pair) units, plane-major, are split into equal
// contiguous ranges over one wave of blocks; a block keeps the sums of its
// current (plane, group) in registers (a thread's (column, k1) is the same for
// every pair: NS column tiles of W, Z2 values each) in the data's precision
// and stores them, FP64, in the partial grid k when it is the k-th of the
// consecutive blocks sharing that (plane, group): part[k][kx][k'][r GC + c],
// c the column of the group.  Each element has one writer: no atomics.  FP32
// sums are carried over to the FP64 grid every 32 pairs.  Bound as the V(r)psi
// kernel is; 64 pairs on 100^3: FP64 353 -> 295 us, FP32 205 -> 165 us against
// whole planes, 160^3 FP64 (8 pairs) 280 us against 460 through HBM slabs.
__host__ __device__ __forceinline__ int bal_block(long u, long U, int nblk) {
  return (int)(((u + 1) * nblk - 1) / U);  // the largest b with floor(b U / nblk) <= u
}
__host__ __device__ __forceinline__ int bal_slots(int kx, int T, long U, int nblk) {
  return bal_block((long)kx * T + T - 1, U, nblk) - bal_block((long)kx * T, U, nblk) + 1;
}
template <typename C, int N, bool SEG>
__global__ void __launch_bounds__(DensShape<C, N>::NT, DensShape<C, N>::MINB)
    k_pencil_density(const PencilGeom pg, const __grid_constant__ FftTw<C, N> p, const C *__restrict__ rt, int T,
                     const double *__restrict__ wa, const double *__restrict__ wb, double *__restrict__ rho_part) {
  typedef decltype(C().x) Rl;
  typedef DensShape<C, N> Sh;
  typedef PlaneRays<C, N, SEG> Rays;
  constexpr int N1 = fft_n1(N), N2 = N / N1, NZ = Sphere<N>::NZ, NSR = N + 1, NT = Sh::NT, W = Sh::W, NS = Sh::NS;
  constexpr int GA = Sh::GA, NK = N1 / GA, GC = Sh::GC, NP = GC | 1, Z1 = Sh::Z1, Z2 = Sh::Z2;
  extern __shared__ __align__(16) unsigned char smraw[];
  PencilSmem<C, N> sm(smraw, NP);
  C *P = sm.P, *S = sm.S;
  sm.load(pg);
  const C *tw = p.t;
  const int U = pg.n1 * GA * T, nb = gridDim.x, b = blockIdx.x;  // within an int: more units would have more rays than the card holds
  const int u0 = (int)((long)b * U / nb), u1 = (int)((long)(b + 1) * U / nb);
  const int k1t = threadIdx.x / W, qqt = threadIdx.x - k1t * W;
  Rl acc[NS][Z2];
  auto row_of = [&](int pgq, int t) { return (long)t * pg.pr_t + (long)(pgq / GA) * pg.pr_x; };
  auto y1_tasks = [&](int pgq, int t, bool first) {
    const long pr = row_of(pgq, t);
    const int r = pgq % GA;
    for (int idx = threadIdx.x + (first ? 0 : NT); idx < NZ * N2; idx += NT) {
      const int j2 = idx / NZ, zi = idx - j2 * NZ;
      C v[N1];
      Rays::template each<true>(const_cast<C *>(rt), pg, sm.cols, pr, zi, j2, v);
      y1_store<C, N, GA>(v, r, P + zi * NP + j2, tw + j2 * N1);
    }
  };
  __syncthreads();
  if (u0 < u1) y1_tasks(u0 / T, u0 % T, true);
  const int j20 = threadIdx.x / NZ, zi0 = threadIdx.x - j20 * NZ;
  for (int u = u0; u < u1;) {
    const int pgq = u / T;
    const bool more = u > u0 && u > pgq * T;  // adds to this block's sums of the same (plane, group)
    int ue = min(u1, (pgq + 1) * T);
    if (sizeof(C) == 8) ue = min(ue, u + 32);
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
      for (int k2 = 0; k2 < Z2; ++k2) acc[s][k2] = (Rl)0;
    for (; u < ue; ++u) {
      const int t = u - pgq * T;
      __syncthreads();
      rows_inner<C, N, NT, NP, NK, 1, false>(P, tw, GA, 0);
      const Rl fa = (Rl)wa[t], fb = (Rl)wb[t];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const int q0 = s * W, ct = min(W, GC - q0);
        __syncthreads();
        for (int idx = threadIdx.x; idx < W * Z2; idx += NT) {
          const int j2 = idx / W, qq = idx - j2 * W;
          if (qq < ct) zcol_first<C, N, NP, Z1>(P + q0 + qq, S + qq * NSR, j2, tw);
        }
        __syncthreads();
        // the plane is free after the last tile's first phase: the next
        // unit's rays are loaded here and transformed after this tile's sums
        const bool nxt = s == NS - 1 && u + 1 < u1;
        const int tn = t + 1 < T ? t + 1 : 0, pn = pgq + (t + 1 < T ? 0 : 1);
        C v[N1];
        if (nxt && j20 < N2) Rays::template each<true>(const_cast<C *>(rt), pg, sm.cols, row_of(pn, tn), zi0, j20, v);
        if (k1t < Z1 && qqt < ct) {
          const C *row = S + qqt * NSR + k1t * Z2;
          C x[Z2];
#pragma unroll
          for (int j2 = 0; j2 < Z2; ++j2) x[j2] = row[j2];
          Dft<C, Z2, 1>::run(x);
#pragma unroll
          for (int k2 = 0; k2 < Z2; ++k2) {
            const Rl re = x[k2].x, im = x[k2].y;
            acc[s][k2] += fa * re * re + fb * im * im;
          }
        }
        if (nxt) {
          if (j20 < N2) y1_store<C, N, GA>(v, pn % GA, P + zi0 * NP + j20, tw + j20 * N1);
          y1_tasks(pn, tn, false);
        }
      }
    }
    const int slot = b - bal_block((long)pgq * T, U, nb), kx = pgq / GA;
    double *out = rho_part + ((long)slot * pg.n1 + kx) * N * N + (pgq - kx * GA) * GC;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const int q = s * W + qqt;
      if (k1t < Z1 && qqt < min(W, GC - s * W)) {
#pragma unroll
        for (int k2 = 0; k2 < Z2; ++k2) {
          double *o = out + (long)(k1t * Z2 + k2) * N + q;
          *o = more ? *o + (double)acc[s][k2] : (double)acc[s][k2];
        }
      }
    }
  }
}

// position <-> index of the permuted (ky, kz) order: position a*N2 + b holds
// index a + N1*b
__host__ __device__ __forceinline__ int perm_index(int pos, int n1f, int n2f) { return pos / n2f + n1f * (pos % n2f); }

// rho[kz][ky][kx] (=, or += with add) the sum of the partial grids
// part[g][kx][k'][c] of the density kernel (c = group r, column), for nx x
// planes (n on one GPU, a rank's planes in the slab decomposition); z1: the
// density kernel's split of z; nblk, T: the schedule.  grid ((n+31)/32, (nx+31)/32, n), block (32, 8): a 32 (c) x 32
// (kx) tile of plane k'; a thread adds the grids of its four rows together
// (four loads in flight; each element's sum keeps the block order), the tile
// is transposed through shared memory.
__global__ void k_rho_reduce_p(int n, int nx, int n1f, int n2f, int z1, int ga, const double *__restrict__ part,
                               double *__restrict__ rho, int add, int T, int nblk) {
  __shared__ double tile[32][33];
  __shared__ int slots[32 * 3];  // of (kx0 + i, group) at i*ga + group; ga <= 3
  const int kp = blockIdx.z, gc = n / ga;
  const int c0 = blockIdx.x * 32, kx0 = blockIdx.y * 32;
  const long gstride = (long)nx * n * n;
  const int c = c0 + threadIdx.x, tid = threadIdx.y * 32 + threadIdx.x;
  if (tid < 32 * ga && kx0 + tid / ga < nx) slots[tid] = bal_slots(kx0 * ga + tid, T, (long)nx * ga * T, nblk);
  __syncthreads();
  long off[4];
  int ng[4];
  double s[4];
  int gmax = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int kx = kx0 + threadIdx.y + 8 * i;
    const bool ok = kx < nx && c < n;
    ng[i] = ok ? slots[(threadIdx.y + 8 * i) * ga + c / gc] : 0;
    gmax = max(gmax, ng[i]);
    off[i] = ok ? ((long)kx * n + kp) * n + c : 0;
    s[i] = 0.0;
  }
#pragma unroll 2
  for (int g = 0; g < gmax; ++g) {
    const double *pg = part + g * gstride;
    double v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = g < ng[i] ? pg[off[i]] : 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] += v[i];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) tile[threadIdx.y + 8 * i][threadIdx.x] = s[i];
  __syncthreads();
  const int kz = perm_index(kp, z1, n / z1);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int cc = c0 + threadIdx.y + 8 * i, kx = kx0 + threadIdx.x;
    if (kx < nx && cc < n) {
      const int r = cc / gc, x = cc - r * gc;
      const int ky = r + ga * (x / n2f) + n1f * (x % n2f);
      double *o = rho + ((long)kz * n + ky) * nx + kx;
      const double t = tile[threadIdx.x][threadIdx.y + 8 * i];
      *o = add ? *o + t : t;
    }
  }
}

// vp[kx][k'][q] (working precision) from V[kz][ky][kx] (FP64), permuted
// order, for nx x planes
template <typename Rl>
__global__ void k_v_permute(int n, int nx, int n1f, int n2f, const double *__restrict__ v, Rl *__restrict__ vp) {
  __shared__ double tile[32][33];
  const int kp = blockIdx.z;
  const int kz = perm_index(kp, n1f, n2f);
  const int kx0 = blockIdx.x * 32, q0 = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int q = q0 + j, kx = kx0 + threadIdx.x;
    tile[j][threadIdx.x] = (kx < nx && q < n) ? v[((long)kz * n + perm_index(q, n1f, n2f)) * nx + kx] : 0.0;
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int kx = kx0 + j, q = q0 + threadIdx.x;
    if (kx < nx && q < n) vp[((long)kx * n + kp) * n + q] = (Rl)tile[threadIdx.x][j];
  }
}

// Slab decomposition: the +G / -G positions of a rank's G vectors in its
// send/return buffer [kx][t][local ray] for T pairs (row = T * local rays),
// from the planes and local rays of the two positions
__global__ void k_slab_pos(int ng, const int *__restrict__ kxp, const int *__restrict__ rlp,
                           const int *__restrict__ kxm, const int *__restrict__ rlm, long row, int *__restrict__ pp,
                           int *__restrict__ pm) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g < ng) {
    pp[g] = (int)(kxp[g] * row + rlp[g]);
    pm[g] = (int)(kxm[g] * row + rlm[g]);
  }
}

}  // namespace amdk
