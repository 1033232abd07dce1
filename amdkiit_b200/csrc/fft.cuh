// Pruned, batched 3D FFT engine for the G-sphere (sm_100a).
//
// Replaces do_fft (fft_interface.f90:33-148), which runs three FFTW passes
// with two full-grid work arrays per transform.  Here a transform is split in
// three passes whose extents follow the sphere:
//   X pass : the x-rays that carry G vectors (ngrays of the wavefunction
//            sphere, nhrays of the density sphere; PW rays are a prefix of
//            the density rays, in the reference's numbering), layout
//            R[t][ray][kx]
//   Y pass : the z planes that contain rays (the slab), layout S[t][zi][ky][kx]
//   Z pass : every (kx,ky) column of the full grid
// For the specialised lengths a thread takes the elements of its
// sub-transforms straight from global memory (x-fastest, coalesced) and stores
// them from registers, with one exchange through shared memory between the
// two phases; run-time lengths load a tile of lines into shared memory and
// transform it with a Stockham mixed-radix (4,2,3,5) FFT.  The Z pass of band
// pairs carries the fused consumers: |psi|^2 density accumulation, and
// V(r)*psi between the backward and forward z transforms (the full grid is
// never written for H|psi>).  The band-pair transforms of cubic grids take the
// pencil path of pencil.cuh instead; these kernels serve the density-sphere
// fields and the other grids.
//
// Index convention: grid index k = (Miller index) mod N, x fastest.  The
// backward transform is sum_G c(G) exp(+iG.r) (FFTW_BACKWARD, unscaled); the
// forward one is exp(-iG.r), and the 1/N of fft_interface.f90:121 is applied
// by the gather kernels.  The reference's centred layout and its (-1)^(i+j+k)
// phasen (fft_interface.f90:515-532) are the same transform in a shifted index
// and are not needed here.
#pragma once
#include <cuda_runtime.h>

namespace amdk {

// ---------------------------------------------------------------- complex
template <typename R> struct CT;
template <> struct CT<double> { typedef double2 T; };
template <> struct CT<float> { typedef float2 T; };

__host__ __device__ __forceinline__ double2 mk(double x, double y) { return make_double2(x, y); }
__host__ __device__ __forceinline__ float2 mk(float x, float y) { return make_float2(x, y); }
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { a.x += b.x; a.y += b.y; return a; }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { a.x -= b.x; a.y -= b.y; return a; }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  C r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
template <typename C, typename R> __device__ __forceinline__ C cscale(C a, R s) { a.x *= s; a.y *= s; return a; }
// i*sg*a
template <typename C> __device__ __forceinline__ C cimul(C a, int sg) {
  C r;
  if (sg > 0) { r.x = -a.y; r.y = a.x; }
  else { r.x = a.y; r.y = -a.x; }
  return r;
}
template <typename C> __device__ __forceinline__ C czero() { C r; r.x = 0; r.y = 0; return r; }
// a*s + b, s real
template <typename C, typename R> __device__ __forceinline__ C cfmas(C a, R s, C b) {
  b.x += a.x * s;
  b.y += a.y * s;
  return b;
}

// float2 arithmetic on the packed FP32x2 instructions of sm_100 (one
// instruction for both components)
__device__ __forceinline__ unsigned long long f2pack(float2 v) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v.x), "f"(v.y));
  return r;
}
__device__ __forceinline__ float2 f2unpack(unsigned long long u) {
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(u));
  return v;
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2pack(a)), "l"(f2pack(b)));
  return f2unpack(r);
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2pack(a)), "l"(f2pack(b)));
  return f2unpack(r);
}
__device__ __forceinline__ float2 cscale(float2 a, float s) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2pack(a)), "l"(f2pack(make_float2(s, s))));
  return f2unpack(r);
}
__device__ __forceinline__ float2 cfmas(float2 a, float s, float2 b) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(f2pack(a)), "l"(f2pack(make_float2(s, s))), "l"(f2pack(b)));
  return f2unpack(r);
}

// ---------------------------------------------------------------- plans
constexpr int MAXF = 8;
template <typename C> struct Plan {
  int n, nf;
  int f[MAXF];
  const C *w;   // w[k] = exp(-2 pi i k/n), k < n (device)
};

// a + i sg b and its scaled form a + i sg s b: the quarter turn is folded into
// the two scalar additions (FMAs) instead of forming i b
template <typename C> __device__ __forceinline__ C caddi(C a, C b, int sg) {
  C r;
  r.x = sg > 0 ? a.x - b.y : a.x + b.y;
  r.y = sg > 0 ? a.y + b.x : a.y - b.x;
  return r;
}
template <typename C, typename R> __device__ __forceinline__ C cfmai(C a, R s, C b) {  // a + i s b
  C r;
  r.x = a.x - s * b.y;
  r.y = a.y + s * b.x;
  return r;
}
template <typename C> __device__ __forceinline__ C cneg(C a) {
  a.x = -a.x;
  a.y = -a.y;
  return a;
}
// x + y and x - y where zx / zy say (at compile time, after unrolling) that a term is zero
template <typename C> __device__ __forceinline__ C addz(C x, bool zx, C y, bool zy) {
  return zx ? y : (zy ? x : cadd(x, y));
}
template <typename C> __device__ __forceinline__ C subz(C x, bool zx, C y, bool zy) {
  return zy ? x : (zx ? cneg(y) : csub(x, y));
}
// radix-r DFT as dft_r with z[q] set where input q is known to be zero
template <typename C> __device__ __forceinline__ void dft_rz(C *a, const bool *z, int r, int sg) {
  typedef decltype(a[0].x) R;
  if (r == 2) {
    const C t = a[0];
    a[0] = addz(t, z[0], a[1], z[1]);
    a[1] = subz(t, z[0], a[1], z[1]);
  } else if (r == 4) {
    const bool z02 = z[0] && z[2], z13 = z[1] && z[3];
    const C t0 = addz(a[0], z[0], a[2], z[2]), t1 = subz(a[0], z[0], a[2], z[2]);
    const C t2 = addz(a[1], z[1], a[3], z[3]), t3 = subz(a[1], z[1], a[3], z[3]);
    a[0] = addz(t0, z02, t2, z13);
    a[2] = subz(t0, z02, t2, z13);
    a[1] = z13 ? t1 : (z02 ? cimul(t3, sg) : caddi(t1, t3, sg));
    a[3] = z13 ? t1 : (z02 ? cimul(t3, -sg) : caddi(t1, t3, -sg));
  } else if (r == 3) {
    const R s3 = (R)0.86602540378443864676 * (R)sg;
    const C t1 = addz(a[1], z[1], a[2], z[2]), d = subz(a[1], z[1], a[2], z[2]);
    const C m = z[0] ? cscale(t1, (R)-0.5) : cfmas(t1, (R)-0.5, a[0]);
    a[0] = addz(a[0], z[0], t1, z[1] && z[2]);
    a[1] = cfmai(m, s3, d);
    a[2] = cfmai(m, -s3, d);
  } else {  // r == 5 (no zero inputs: it is never a first stage)
    const R c1 = (R)0.30901699437494742410, c2 = (R)-0.80901699437494742410;
    const R s1 = (R)0.95105651629515357212, s2 = (R)0.58778525229247312917;
    const C t1 = cadd(a[1], a[4]), t2 = cadd(a[2], a[3]);
    const C t3 = csub(a[1], a[4]), t4 = csub(a[2], a[3]);
    const C m1 = cfmas(t2, c2, cfmas(t1, c1, a[0]));
    const C m2 = cfmas(t2, c1, cfmas(t1, c2, a[0]));
    const C n1 = cfmas(t4, s2, cscale(t3, s1));
    const C n2 = cfmas(t4, -s1, cscale(t3, s2));
    a[0] = cadd(a[0], cadd(t1, t2));
    a[1] = caddi(m1, n1, sg);
    a[4] = caddi(m1, n1, -sg);
    a[2] = caddi(m2, n2, sg);
    a[3] = caddi(m2, n2, -sg);
  }
}
// y_p = sum_q a_q exp(sg 2 pi i p q / r)
template <typename C> __device__ __forceinline__ void dft_r(C *a, int r, int sg) {
  const bool z[5] = {false, false, false, false, false};
  dft_rz(a, z, r, sg);
}

// Stockham FFT of L lines held in shared memory, element k of line l at
// buf[k*es + l].  Ping-pong between a and b; returns the buffer holding the
// result.  Must be called by all threads of the block.
template <typename C>
__device__ C *smem_fft(C *a, C *b, int L, int es, const Plan<C> &p, int sg) {
  const int n = p.n;
  int s = 1;
  for (int st = 0; st < p.nf; ++st) {
    const int r = p.f[st];
    const int m = n / (s * r);
    const int nbf = L * (n / r);
    for (int idx = threadIdx.x; idx < nbf; idx += blockDim.x) {
      const int l = idx % L;
      const int bf = idx / L;
      const int k = bf % s;
      const int j = bf / s;
      C v[5];
#pragma unroll 5
      for (int q = 0; q < 5; ++q)
        if (q < r) v[q] = a[(k + s * j + s * m * q) * es + l];
      dft_r(v, r, sg);
#pragma unroll 5
      for (int q = 0; q < 5; ++q)
        if (q < r) {
          int e = (s * j * q) % n;
          C w = p.w[e];
          if (sg > 0) w.y = -w.y;
          b[(k + s * q + s * r * j) * es + l] = (q == 0) ? v[q] : cmul(v[q], w);
        }
    }
    __syncthreads();
    C *t = a;
    a = b;
    b = t;
    s *= r;
  }
  return a;
}


// ---------------------------------------------------------------- register FFT
// Small DFTs held in registers (R <= 16 with factors 2, 3, 4, 5) and the
// two-level line transform N = N1*N2 built on them: each thread loads the N1
// (or N2) elements of one sub-transform, works in registers and writes back,
// so a length-N line costs two shared-memory round trips.  Twiddles
// W_R^m = exp(-2 pi i m/R) of the small DFTs (R = 2..16) sit in constant
// memory at ctw_off(R) + m and are filled by the host.
__host__ __device__ constexpr int ctw_off(int R) { return R * (R - 1) / 2 - 1; }
constexpr int CTW_LEN = ctw_off(17);
__constant__ double2 c_twd[CTW_LEN];
__constant__ float2 c_twf[CTW_LEN];
template <typename C> __device__ __forceinline__ C ctw(int i);
template <> __device__ __forceinline__ double2 ctw<double2>(int i) { return c_twd[i]; }
template <> __device__ __forceinline__ float2 ctw<float2>(int i) { return c_twf[i]; }

__host__ __device__ constexpr int reg_radix(int r) { return (r % 4 == 0) ? 4 : (r % 2 == 0) ? 2 : (r % 3 == 0) ? 3 : 5; }
// N = N1 * N2 with N1 <= N2 <= 16 and N1 as large as possible (0: none)
__host__ __device__ constexpr int fft_n1(int n) {
  int best = 0;
  for (int d = 2; d <= 16; ++d)
    if (n % d == 0 && n / d <= 16 && d <= n / d) best = d;
  return best;
}

// a W_R^(T m), W_R = exp(-2 pi i / R), for an m known after unrolling:
// quarter turns cost no multiplication
template <typename C, int R, int T> __device__ __forceinline__ C ctw_mul(C a, int m) {
  m %= R;
  if (m == 0) return a;
  if (2 * m == R) return cneg(a);
  if (4 * m == R) return cimul(a, -T);
  if (4 * m == 3 * R) return cimul(a, T);
  C w = ctw<C>(ctw_off(R) + m);
  if (T < 0) w.y = -w.y;
  return cmul(a, w);
}

__host__ __device__ constexpr int dft_gcd(int a, int b) { return b == 0 ? a : dft_gcd(b, a % b); }
// the e < A*B with e = 1 mod A and e = 0 mod B (A, B coprime)
__host__ __device__ constexpr int crt_unit(int A, int B) {
  for (int e = 0; e < A * B; e += B)
    if (e % A == 1 % A) return e;
  return 0;
}

// y_k = sum_j v_j exp(SG 2 pi i jk/R), natural order in and out.  R > 5 is
// A x B; coprime factors (6, 10, 12) are indexed as Good (1958) and Thomas
// (1963) do, which needs no twiddles between the stages.
//   run       every input and output
//   run_in    inputs LO <= j < HI are zero (and not read): radix A first, on
//             inputs B apart, so that most of its terms are copies
//   run_out   radix A last: outputs the caller does not use cost nothing (the
//             unused half of the last butterflies is dead code); only inputs
//             j = GR (mod GA) are read, the others are zero (GA divides A)
template <typename C, int R, int SG> struct Dft {
  static constexpr int A = R <= 5 ? 1 : reg_radix(R), B = R <= 5 ? R : R / A;
  static constexpr bool PFA = R > 5 && dft_gcd(A, B) == 1;
  template <int LO, int HI> static __device__ __forceinline__ void run_in(C (&v)[R]) {
    if constexpr (R <= 5) {
      bool z[R];
#pragma unroll
      for (int j = 0; j < R; ++j) z[j] = false;
      dft_rz(v, z, R, SG);
    } else {
      constexpr int eA = crt_unit(A, B), eB = crt_unit(B, A);
      C t[R];  // t[b + B*ka]
#pragma unroll
      for (int b = 0; b < B; ++b) {
        C a[A];
        bool z[A];
#pragma unroll
        for (int i = 0; i < A; ++i) {
          const int j = PFA ? (B * i + A * b) % R : b + B * i;
          a[i] = v[j];
          z[i] = j >= LO && j < HI;
        }
        dft_rz(a, z, A, SG);
#pragma unroll
        for (int ka = 0; ka < A; ++ka) t[b + B * ka] = PFA ? a[ka] : ctw_mul<C, R, -SG>(a[ka], b * ka);
      }
#pragma unroll
      for (int ka = 0; ka < A; ++ka) {
        C u[B];
#pragma unroll
        for (int b = 0; b < B; ++b) u[b] = t[b + B * ka];
        Dft<C, B, SG>::run(u);
#pragma unroll
        for (int kb = 0; kb < B; ++kb) v[PFA ? (ka * eA + kb * eB) % R : ka + A * kb] = u[kb];
      }
    }
  }
  static __device__ __forceinline__ void run(C (&v)[R]) { run_in<R, R>(v); }
  template <int GA, int GR> static __device__ __forceinline__ void run_out(C (&v)[R]) {
    if constexpr (R <= 5) {
      run(v);
    } else {
      constexpr int eA = crt_unit(A, B), eB = crt_unit(B, A);
      C t[R];  // t[kb + B*i]
#pragma unroll
      for (int i = 0; i < A; ++i) {
        // the inputs of sub-transform i are all = i (mod GA) (GA divides A), up
        // to the unit B of the coprime index map
        if ((PFA ? B * i : i) % GA != GR) continue;
        C u[B];
#pragma unroll
        for (int b = 0; b < B; ++b) u[b] = v[PFA ? (B * i + A * b) % R : i + A * b];
        Dft<C, B, SG>::run(u);
#pragma unroll
        for (int kb = 0; kb < B; ++kb) t[kb + B * i] = PFA ? u[kb] : ctw_mul<C, R, -SG>(u[kb], i * kb);
      }
#pragma unroll
      for (int kb = 0; kb < B; ++kb) {
        C a[A];
        bool z[A];
#pragma unroll
        for (int i = 0; i < A; ++i) {
          z[i] = (PFA ? B * i : i) % GA != GR;
          if (!z[i]) a[i] = t[kb + B * i];
        }
        dft_rz(a, z, A, SG);
#pragma unroll
        for (int ka = 0; ka < A; ++ka) v[PFA ? (ka * eA + kb * eB) % R : kb + B * ka] = a[ka];
      }
    }
  }
};

// Twiddles of the two-level transform of a specialised length N = N1*N2,
// built per block in shared memory (2N entries) from the plan's
// w[e] = exp(-2 pi i e/N): tw[j2*N1 + k1] = W_N^(j2 k1) (table 0, the
// twiddles of a natural-order-in transform's first phase) and
// tw[N + k1*N2 + k2] = W_N^(k1 k2) (table 1, those of a permuted-order-in
// transform's first phase).  A thread reads its row with constant offsets,
// so no exponent arithmetic is left in the butterflies.
template <typename C, int N> __device__ __forceinline__ void load_tw(C *tw, const Plan<C> &p) {
  if constexpr (N > 0) {
    constexpr int N1 = fft_n1(N), N2 = N / N1;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
      tw[i] = p.w[(i / N1) * (i % N1) % N];
      tw[N + i] = p.w[(i / N2) * (i % N2) % N];
    }
  }
}
// v[k] *= W_N^(SG j k), k = 1..R-1, from row j of twiddle table TAB (table 0
// for R = N1, j = j2; table 1 for R = N2, j = k1).
template <typename C, int N, int R, int SG, int TAB>
__device__ __forceinline__ void twiddle_tab(C (&v)[R], int j, const C *tw) {
  const C *row = tw + TAB * N + j * R;
#pragma unroll
  for (int k = 1; k < R; ++k) {
    C w = row[k];
    if (SG > 0) w.y = -w.y;
    v[k] = cmul(v[k], w);
  }
}

// The twiddle tables of a specialised length as a kernel parameter (read from
// the constant bank): t[j2*N1 + k1] = W_N^(j2 k1), t[N + k1*N2 + k2] =
// W_N^(k1 k2).  N = 0 (run-time lengths): unused.
template <typename C, int N> struct FftTw {
  C t[N > 0 ? 2 * N : 1];
};
// Two-level transform of lines that come from and go to global memory, one
// line per l: load(k) and store(k, value) move element k of the calling
// thread's line.  Thread (l, h), h < N2: phase A loads its N1 elements straight
// into registers and leaves them in s[k*ES + l*EL]; after one barrier phase B
// (h < N1) stores its N2 outputs from registers.  The field transforms are
// short launches bound by latency (7% of the copy rate): one shared tile and
// one barrier, where staging the tile in and out took two tiles and three.
// 100^3 FP64, per launch: y 18.6 -> 10.8 us, forward x 16.1 -> 11.3, backward x
// 24 -> 12 (gradients 23), z 17-22 -> 8-13.
template <typename C, int N, int SG, int ES, int EL, typename Load, typename Store>
__device__ __forceinline__ void line_fft_direct(C *s, int l, int h, bool on, const C *tw, Load &&load, Store &&store) {
  constexpr int N1 = fft_n1(N), N2 = N / N1;
  C *line = s + l * EL;
  if (on && h < N2) {
    C v[N1];
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) v[j1] = load(h + N2 * j1);
    Dft<C, N1, SG>::run(v);
    twiddle_tab<C, N, N1, SG, 0>(v, h, tw);
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) line[(k1 * N2 + h) * ES] = v[k1];
  }
  __syncthreads();
  if (on && h < N1) {
    C u[N2];
#pragma unroll
    for (int j2 = 0; j2 < N2; ++j2) u[j2] = line[(h * N2 + j2) * ES];
    Dft<C, N2, SG>::run(u);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) store(h + N1 * k2, u[k2]);
  }
}

// Two-level register FFT of a tile of L lines (element k of line l at
// a[k*ES + l]), natural order in a, natural order out in b: phase A in place
// in a (thread (l, j2): DFT_N1 of elements j2 + N2*j1, twiddle, back to
// k1*N2 + j2), phase B from a to b (thread (l, k1): DFT_N2 of the N2
// contiguous elements, out to k1 + N1*k2).
template <typename C, int N, int L, int ES, int SG>
__device__ __forceinline__ void tile_reg_fft(C *a, C *b, const C *tw) {
  constexpr int N1 = fft_n1(N), N2 = N / N1;
  for (int idx = threadIdx.x; idx < L * N2; idx += blockDim.x) {
    const int l = idx % L, j2 = idx / L;
    C v[N1];
#pragma unroll
    for (int j1 = 0; j1 < N1; ++j1) v[j1] = a[(j2 + N2 * j1) * ES + l];
    Dft<C, N1, SG>::run(v);
    twiddle_tab<C, N, N1, SG, 0>(v, j2, tw);
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) a[(k1 * N2 + j2) * ES + l] = v[k1];
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < L * N1; idx += blockDim.x) {
    const int l = idx % L, k1 = idx / L;
    C u[N2];
#pragma unroll
    for (int j2 = 0; j2 < N2; ++j2) u[j2] = a[(k1 * N2 + j2) * ES + l];
    Dft<C, N2, SG>::run(u);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) b[(k1 + N1 * k2) * ES + l] = u[k2];
  }
  __syncthreads();
}

// FFT of a tile of L lines (element k of line l at buf[k*ES + l]); returns
// the buffer that holds the result.  N = 0 is the run-time-length Stockham
// path; a specialised N uses the register FFT (tw: shared copy of p.w).
template <typename C, int N, int L, int ES>
__device__ __forceinline__ C *fft_tile(C *a, C *b, const Plan<C> &p, const C *tw, int sg) {
  if constexpr (N == 0) {
    return smem_fft(a, b, L, ES, p, sg);
  } else {
    if (sg > 0) tile_reg_fft<C, N, L, ES, 1>(a, b, tw);
    else tile_reg_fft<C, N, L, ES, -1>(a, b, tw);
    return b;
  }
}

// ---------------------------------------------------------------- geometry
struct Geom {
  int n1, n2, n3;
  int ngpw, ngrho;
  int nray[2];            // rays of the PW (0) / density (1) sphere
  const int *gmap;        // [nhrays*n1]: +(ig+1) at +G, -(ig+1) at -G, 0 empty
  const int *pos_p;       // [ngrho] ray*n1 + kx of +G
  const int *pos_m;       // [ngrho] ray*n1 + kx of -G
  int nz[2];              // slab planes per sphere
  const int *zlist[2];    // [nz] kz of each slab plane
  const int *rayidx[2];   // [nz*n2] ray of (zi, ky) or -1
  const int *zinv[2];     // [n3] slab plane of kz or -1
};

constexpr int TX = 16;    // x-extent of a Y/Z tile (16 complex = 256 B in FP64)
constexpr int LX = 8;     // lines per X-pass block
constexpr int LXD = 16;   // lines per X-pass block of the density-sphere fields (specialised lengths)
// threads and shared memory of the direct field kernels of length n
constexpr int direct_threads(int n, int lines) { return lines * (n / fft_n1(n)); }

// ---------------------------------------------------------------- X pass
// Backward X pass with the band-pair pack fused (vpsi/eval_density pack,
// wfn_initialize.f90:286-308, density.f90:26-47): psi_a + i psi_b.
template <typename C, int N = 0>
__global__ void __launch_bounds__(256) k_x_bwd_pair(const double2 *__restrict__ c0, int ngpw, int nstate, int band0, int T,
                                                    Geom g, Plan<C> p, C *__restrict__ rb) {
  extern __shared__ unsigned char smraw[];
  C *sa = reinterpret_cast<C *>(smraw);
  const int n1 = g.n1, R = g.nray[0];
  const int es = LX + 1;
  C *sb = sa + n1 * es;
  C *tw = sb + n1 * es;
  load_tw<C, N>(tw, p);
  const long line0 = (long)blockIdx.x * LX;
  const long nlines = (long)T * R;
  for (int idx = threadIdx.x; idx < LX * n1; idx += blockDim.x) {
    const int l = idx / n1, k = idx % n1;
    const long line = line0 + l;
    C v = czero<C>();
    if (line < nlines) {
      const int t = (int)(line / R), r = (int)(line % R);
      const int code = g.gmap[(long)r * n1 + k];
      const int ig = (code > 0 ? code : -code) - 1;
      if (code != 0 && ig < ngpw) {
        const int ba = band0 + 2 * t, bb = ba + 1;
        double2 a = c0[(long)ba * ngpw + ig];
        double2 b = (bb < nstate) ? c0[(long)bb * ngpw + ig] : make_double2(0.0, 0.0);
        if (code > 0) v = mk((decltype(v.x))(a.x - b.y), (decltype(v.x))(a.y + b.x));
        else v = mk((decltype(v.x))(a.x + b.y), (decltype(v.x))(-a.y + b.x));
      }
    }
    sa[k * es + l] = v;
  }
  __syncthreads();
  C *res = fft_tile<C, N, LX, LX + 1>(sa, sb, p, tw, +1);
  for (int idx = threadIdx.x; idx < LX * n1; idx += blockDim.x) {
    const int l = idx / n1, k = idx % n1;
    const long line = line0 + l;
    if (line < nlines) rb[line * n1 + k] = res[k * es + l];
  }
}

// Backward X pass of real fields given at +G (-G: the conjugate), the t-th
// field at f + t*ngmax (FS_REAL), or of the packed fields rho + i d_x rho
// (t = 0) and d_y rho + i d_z rho (t = 1) of GRAD_CAL (xc.f90:471-487), formed
// from rho(G) = f and G as they are gathered (FS_GRAD).
enum { FS_REAL = 0, FS_GRAD = 1 };
template <typename C, int N, int SRC>
__global__ void __launch_bounds__(256) k_x_bwd_field(const double2 *__restrict__ f, const double *__restrict__ gvec,
                                                     double tpiba, int ngmax,
                                                     int sphere, int T, Geom g, Plan<C> p,
                                                     const __grid_constant__ FftTw<C, N> ft, C *__restrict__ rb) {
  extern __shared__ unsigned char smraw[];
  C *sa = reinterpret_cast<C *>(smraw);
  const int n1 = g.n1, R = sphere ? g.nray[1] : g.nray[0];
  const long nlines = (long)T * R;
  auto gather = [&](long line, int k) {
    C v = czero<C>();
    if (line < nlines) {
      const int t = (int)(line / R), r = (int)(line % R);
      const int code = g.gmap[(long)r * n1 + k];
      const int ig = (code > 0 ? code : -code) - 1;
      if (code != 0 && ig < ngmax) {
        const double sg = code > 0 ? 1.0 : -1.0;
        double2 a = f[(SRC == FS_REAL ? (long)t * ngmax : 0L) + ig];
        a.y *= sg;
        if (SRC == FS_GRAD) {
          // f + i (i G_x f) and i G_y f + i (i G_z f), of f(G) or its conjugate at -G
          if (t == 0) {
            const double gx = sg * (tpiba * gvec[3 * ig]);
            a = make_double2(a.x - gx * a.x, a.y - gx * a.y);
          } else {
            const double ax = -(sg * tpiba) * gvec[3 * ig + 2], ay = (sg * tpiba) * gvec[3 * ig + 1];
            a = make_double2(ax * a.x - ay * a.y, ax * a.y + ay * a.x);
          }
        }
        v = mk((decltype(v.x))a.x, (decltype(v.x))a.y);
      }
    }
    return v;
  };
  if constexpr (N > 0) {
    constexpr int N2 = N / fft_n1(N);
    const int l = threadIdx.x / N2, h = threadIdx.x - l * N2;
    const long line = (long)blockIdx.x * LXD + l;
    C *o = rb + line * N;
    line_fft_direct<C, N, 1, 1, N + 1>(
        sa, l, h, line < nlines, ft.t, [&](int k) { return gather(line, k); }, [&](int k, const C &v) { o[k] = v; });
  } else {
    const int es = LX + 1;
    C *sb = sa + n1 * es;
    const long line0 = (long)blockIdx.x * LX;
    for (int idx = threadIdx.x; idx < LX * n1; idx += blockDim.x)
      sa[(idx % n1) * es + idx / n1] = gather(line0 + idx / n1, idx % n1);
    __syncthreads();
    C *res = smem_fft(sa, sb, LX, es, p, +1);
    for (int idx = threadIdx.x; idx < LX * n1; idx += blockDim.x) {
      const int l = idx / n1, k = idx % n1;
      const long line = line0 + l;
      if (line < nlines) rb[line * n1 + k] = res[k * es + l];
    }
  }
}

// Forward X pass in place on the ray buffer.
template <typename C, int N = 0>
__global__ void __launch_bounds__(256) k_x_fwd(int sphere, int T, Geom g, Plan<C> p,
                                               const __grid_constant__ FftTw<C, N> ft, C *__restrict__ rb) {
  extern __shared__ unsigned char smraw[];
  C *sa = reinterpret_cast<C *>(smraw);
  const int n1 = g.n1, R = sphere ? g.nray[1] : g.nray[0];
  const long nlines = (long)T * R;
  if constexpr (N > 0) {
    constexpr int N2 = N / fft_n1(N);
    const int l = threadIdx.x / N2, h = threadIdx.x - l * N2;
    const long line = (long)blockIdx.x * LXD + l;
    C *o = rb + line * N;
    line_fft_direct<C, N, -1, 1, N + 1>(
        sa, l, h, line < nlines, ft.t, [&](int k) { return o[k]; }, [&](int k, const C &v) { o[k] = v; });
  } else {
    const int es = LX + 1;
    C *sb = sa + n1 * es;
    const long line0 = (long)blockIdx.x * LX;
    for (int idx = threadIdx.x; idx < LX * n1; idx += blockDim.x) {
      const int l = idx / n1, k = idx % n1;
      const long line = line0 + l;
      sa[k * es + l] = (line < nlines) ? rb[line * n1 + k] : czero<C>();
    }
    __syncthreads();
    C *res = smem_fft(sa, sb, LX, es, p, -1);
    for (int idx = threadIdx.x; idx < LX * n1; idx += blockDim.x) {
      const int l = idx / n1, k = idx % n1;
      const long line = line0 + l;
      if (line < nlines) rb[line * n1 + k] = res[k * es + l];
    }
  }
}

// ---------------------------------------------------------------- Y pass
// grid: (ceil(n1/TX), nz[sphere], T).  DIR=+1 backward (rays -> slab),
// DIR=-1 forward (slab -> rays).
template <typename C, int N, int DIR>
__global__ void __launch_bounds__(256) k_y(int sphere, Geom g, Plan<C> p, const __grid_constant__ FftTw<C, N> ft,
                                           C *__restrict__ rb, C *__restrict__ sbuf, long rstride, long sstride) {
  extern __shared__ unsigned char smraw[];
  C *sa = reinterpret_cast<C *>(smraw);
  const int n1 = g.n1, n2 = g.n2;
  const int kx0 = blockIdx.x * TX, zi = blockIdx.y, t = blockIdx.z;
  const int *ri = (sphere ? g.rayidx[1] : g.rayidx[0]) + (long)zi * n2;
  C *R = rb + (long)t * rstride;
  C *S = sbuf + (long)t * sstride + (long)zi * n2 * n1;
  auto fetch = [&](int kx, int ky) {
    C v = czero<C>();
    if (DIR > 0) {
      const int r = ri[ky];
      if (r >= 0) v = R[(long)r * n1 + kx];
    } else {
      v = S[(long)ky * n1 + kx];
    }
    return v;
  };
  auto put = [&](int kx, int ky, const C &v) {
    if (DIR > 0) {
      S[(long)ky * n1 + kx] = v;
    } else {
      const int r = ri[ky];
      if (r >= 0) R[(long)r * n1 + kx] = v;
    }
  };
  if constexpr (N > 0) {
    const int l = threadIdx.x % TX, h = threadIdx.x / TX, kx = kx0 + l;
    line_fft_direct<C, N, DIR, TX, 1>(
        sa, l, h, kx < n1, ft.t, [&](int k) { return fetch(kx, k); }, [&](int k, const C &v) { put(kx, k, v); });
  } else {
    C *sb = sa + n2 * TX;
    for (int idx = threadIdx.x; idx < TX * n2; idx += blockDim.x) {
      const int kx = kx0 + idx % TX;
      sa[idx] = kx < n1 ? fetch(kx, idx / TX) : czero<C>();
    }
    __syncthreads();
    C *res = smem_fft(sa, sb, TX, TX, p, DIR);
    for (int idx = threadIdx.x; idx < TX * n2; idx += blockDim.x) {
      const int kx = kx0 + idx % TX;
      if (kx < n1) put(kx, idx / TX, res[idx]);
    }
  }
}

// ---------------------------------------------------------------- Z pass
enum { Z_TO_GRID = 0, Z_FROM_GRID_REAL = 1, Z_FROM_GRID_CPLX = 2, Z_VPSI = 3, Z_DENSITY = 4, Z_TO_REAL = 5 };

// grid: (ceil(n1/TX), n2, T) for TO_GRID/FROM_GRID/VPSI; (ceil(n1/TX), n2, 1)
// for DENSITY, which loops over the T transforms of the batch.
//   TO_GRID          slab -> complex grid (double2)                    backward
//   TO_REAL          slab -> real part, a real grid (double)           backward
//   FROM_GRID_REAL   real grid (double) -> slab                        forward
//   FROM_GRID_CPLX   complex grid (double2) -> slab                    forward
//   VPSI             slab -> (bwd) * V(r) -> (fwd) -> slab  (vpsi, wfn_initialize.f90:311-340)
//   DENSITY          slab -> (bwd) -> rho += f_a/Omega Re^2 + f_b/Omega Im^2 (density.f90:49-86)
// The field modes of specialised lengths move their lines directly between
// global memory and registers (k_z_field below); k_z has the pair modes and
// the run-time lengths.
template <typename C, int MODE, int N>
__global__ void __launch_bounds__(256) k_z_field(int sphere, Geom g, const __grid_constant__ FftTw<C, N> ft,
                                                 C *__restrict__ sbuf, long sstride, double2 *__restrict__ cgrid,
                                                 double *__restrict__ rgrid, long gstride) {
  typedef decltype(C().x) R;
  extern __shared__ unsigned char smraw[];
  const int n1 = g.n1, n2 = g.n2;
  const int l = threadIdx.x % TX, h = threadIdx.x / TX, kx = blockIdx.x * TX + l, ky = blockIdx.y;
  const int *zinv = sphere ? g.zinv[1] : g.zinv[0];
  const long plane = (long)n2 * n1, at = (long)ky * n1 + kx;
  C *S = sbuf + (long)blockIdx.z * sstride + at;
  double2 *G = cgrid + (long)blockIdx.z * gstride + at;
  double *Q = rgrid + (long)blockIdx.z * gstride + at;
  constexpr bool BWD = MODE == Z_TO_GRID || MODE == Z_TO_REAL;
  line_fft_direct<C, N, BWD ? 1 : -1, TX, 1>(
      reinterpret_cast<C *>(smraw), l, h, kx < n1, ft.t,
      [&](int kz) {
        C v = czero<C>();
        if (BWD) {
          const int zi = zinv[kz];
          if (zi >= 0) v = S[zi * plane];
        } else if (MODE == Z_FROM_GRID_REAL) {
          v.x = (R)Q[kz * plane];
        } else {
          const double2 c = G[kz * plane];
          v = mk((R)c.x, (R)c.y);
        }
        return v;
      },
      [&](int kz, const C &v) {
        if (MODE == Z_TO_GRID) G[kz * plane] = make_double2((double)v.x, (double)v.y);
        else if (MODE == Z_TO_REAL) Q[kz * plane] = (double)v.x;
        else {
          const int zi = zinv[kz];
          if (zi >= 0) S[zi * plane] = v;
        }
      });
}

template <typename C, int MODE, int N = 0>
__global__ void __launch_bounds__(256) k_z(int sphere, int T, Geom g, Plan<C> p, C *__restrict__ sbuf, long sstride,
                                           double2 *__restrict__ cgrid, double *__restrict__ rgrid, long gstride,
                                           const double *__restrict__ vpot, double *__restrict__ rho,
                                           const double *__restrict__ wa, const double *__restrict__ wb) {
  static_assert(N == 0 || MODE == Z_VPSI || MODE == Z_DENSITY, "k_z_field has the other modes of a known length");
  typedef decltype(C().x) R;
  extern __shared__ unsigned char smraw[];
  C *sa = reinterpret_cast<C *>(smraw);
  const int n1 = g.n1, n2 = g.n2, n3 = g.n3, nz = sphere ? g.nz[1] : g.nz[0];
  C *sb = sa + n3 * TX;
  C *tw = sb + n3 * TX;
  load_tw<C, N>(tw, p);
  const int kx0 = blockIdx.x * TX, ky = blockIdx.y;
  const int *zl = sphere ? g.zlist[1] : g.zlist[0];
  const long plane = (long)n2 * n1;
  double acc[16];  // TX*n3 <= 16*blockDim (checked at setup)
  if (MODE == Z_DENSITY)
    for (int i = 0; i < 16; ++i) acc[i] = 0.0;
  const int tb = (MODE == Z_DENSITY) ? 0 : blockIdx.z;
  const int te = (MODE == Z_DENSITY) ? T : blockIdx.z + 1;
  for (int t = tb; t < te; ++t) {
    C *S = sbuf + (long)t * sstride;
    if (MODE == Z_TO_GRID || MODE == Z_TO_REAL || MODE == Z_VPSI || MODE == Z_DENSITY) {
      if constexpr (N > 0) {
        // the slab loads are issued before the clearing barrier (256 threads per block)
        constexpr int CNT = (TX * N + 255) / 256;
        C v[CNT];
        int dst[CNT];
#pragma unroll
        for (int i = 0; i < CNT; ++i) {
          const int idx = threadIdx.x + 256 * i;
          dst[i] = -1;
          if (idx < TX * nz) {
            const int zi = idx / TX, tx = idx % TX, kx = kx0 + tx;
            if (kx < n1) {
              v[i] = S[(long)zi * plane + (long)ky * n1 + kx];
              dst[i] = zl[zi] * TX + tx;
            }
          }
        }
        for (int idx = threadIdx.x; idx < TX * n3; idx += blockDim.x) sa[idx] = czero<C>();
        __syncthreads();
#pragma unroll
        for (int i = 0; i < CNT; ++i)
          if (dst[i] >= 0) sa[dst[i]] = v[i];
      } else {
        for (int idx = threadIdx.x; idx < TX * n3; idx += blockDim.x) sa[idx] = czero<C>();
        __syncthreads();
        for (int idx = threadIdx.x; idx < TX * nz; idx += blockDim.x) {
          const int zi = idx / TX, tx = idx % TX, kx = kx0 + tx;
          if (kx < n1) sa[zl[zi] * TX + tx] = S[(long)zi * plane + (long)ky * n1 + kx];
        }
      }
      __syncthreads();
      C *res = fft_tile<C, N, TX, TX>(sa, sb, p, tw, +1);
      if (MODE == Z_TO_GRID) {
        double2 *G = cgrid + (long)t * gstride;
        for (int idx = threadIdx.x; idx < TX * n3; idx += blockDim.x) {
          const int kz = idx / TX, tx = idx % TX, kx = kx0 + tx;
          if (kx < n1) {
            C v = res[idx];
            G[(long)kz * plane + (long)ky * n1 + kx] = make_double2((double)v.x, (double)v.y);
          }
        }
        __syncthreads();
      } else if (MODE == Z_TO_REAL) {
        double *G = rgrid + (long)t * gstride;
        for (int idx = threadIdx.x; idx < TX * n3; idx += blockDim.x) {
          const int kz = idx / TX, tx = idx % TX, kx = kx0 + tx;
          if (kx < n1) G[(long)kz * plane + (long)ky * n1 + kx] = (double)res[idx].x;
        }
        __syncthreads();
      } else if (MODE == Z_DENSITY) {
        const double fa = wa[t], fb = wb[t];
        int i = 0;
        for (int idx = threadIdx.x; idx < TX * n3; idx += blockDim.x, ++i) {
          C v = res[idx];
          double re = (double)v.x, im = (double)v.y;
          acc[i] += fa * re * re + fb * im * im;
        }
        __syncthreads();
      } else {  // VPSI
        C *other = (res == sa) ? sb : sa;
        for (int idx = threadIdx.x; idx < TX * n3; idx += blockDim.x) {
          const int kz = idx / TX, tx = idx % TX, kx = kx0 + tx;
          R v = (kx < n1) ? (R)vpot[(long)kz * plane + (long)ky * n1 + kx] : (R)0;
          res[idx] = cscale(res[idx], v);
        }
        __syncthreads();
        C *out = fft_tile<C, N, TX, TX>(res, other, p, tw, -1);
        for (int idx = threadIdx.x; idx < TX * nz; idx += blockDim.x) {
          const int zi = idx / TX, tx = idx % TX, kx = kx0 + tx;
          if (kx < n1) S[(long)zi * plane + (long)ky * n1 + kx] = out[zl[zi] * TX + tx];
        }
        __syncthreads();
      }
    } else {  // FROM_GRID
      auto fetch = [&](int idx) {
        const int kz = idx / TX, tx = idx % TX, kx = kx0 + tx;
        C v = czero<C>();
        if (kx < n1) {
          const long o = (long)t * gstride + (long)kz * plane + (long)ky * n1 + kx;
          if (MODE == Z_FROM_GRID_REAL) v.x = (R)rgrid[o];
          else { double2 c = cgrid[o]; v.x = (R)c.x; v.y = (R)c.y; }
        }
        return v;
      };
      for (int idx = threadIdx.x; idx < TX * n3; idx += blockDim.x) sa[idx] = fetch(idx);
      __syncthreads();
      C *res = fft_tile<C, N, TX, TX>(sa, sb, p, tw, -1);
      for (int idx = threadIdx.x; idx < TX * nz; idx += blockDim.x) {
        const int zi = idx / TX, tx = idx % TX, kx = kx0 + tx;
        if (kx < n1) S[(long)zi * plane + (long)ky * n1 + kx] = res[zl[zi] * TX + tx];
      }
      __syncthreads();
    }
  }
  if (MODE == Z_DENSITY) {
    int i = 0;
    for (int idx = threadIdx.x; idx < TX * n3; idx += blockDim.x, ++i) {
      const int kz = idx / TX, tx = idx % TX, kx = kx0 + tx;
      if (kx < n1) rho[(long)kz * plane + (long)ky * n1 + kx] += acc[i];
    }
  }
}

}  // namespace amdk
