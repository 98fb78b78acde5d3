// bdg_eig.cu -- largest eigenpairs of the small symmetric matrix of the
// Rayleigh-Ritz step (real, k <= 192), in five kernels.
//
// cuSOLVER's syevd takes 0.42 ms at k = 48, 1.15 ms at 96 and 1.7 ms at 192, most
// of it in a chain of 2k launches that apply one reflector each.  bdgd_eig_top
// takes 0.13, 0.26 and 1.04 ms for the k / 3 largest pairs.  Here:
//
//   k_tridiag   Householder tridiagonalisation, the lower triangle in the
//               registers of one block
//   k_bisect    all eigenvalues of the tridiagonal matrix, one warp each:
//               33-section by Sturm counts
//   k_invit     eigenvectors of the nv largest by inverse iteration, one thread
//               each, from random starts
//   k_backtr    the reflectors applied to them, one warp each
//   (caller)    their Gram matrix, its Cholesky factor, one product: vectors of
//               close eigenvalues come out orthonormal
//
// Inverse iteration gives each vector a residual of a few eps ||T||, and
// vectors of eigenvalues a gap g apart an overlap of eps ||T|| / g; within a
// cluster the random starts give independent combinations.  Orthonormalising
// mixes vectors by their overlaps, which leaves the residuals as they are.  The
// caller checks the residuals (d_check) and the smallest pivot of the Gram
// matrix and falls back to syevd.  The residuals are those of the tridiagonal
// matrix, so a matrix whose squares leave the range of a double would pass the
// check with a wrong reduction: k_tridiag scales by a power of two.
#include <cuda_runtime.h>
#include <math.h>

#include "bdg_blas.h"
#include "bdg_dev.h"
#include "bdg_dft.cuh"

#define EIG_THREADS 512
#define EIG_MAXK 192

// sum over the 32 lanes of each of the N values of v (N a power of two <= 16);
// lane l returns the sum of value fold_index<N>(l).  Each step sends the half of
// the values that the partner keeps, so N values take N + 4 - log2 N exchanges.
template <int N, int OFF = 16>
__device__ __forceinline__ double fold_sum(double (&v)[N], int lane) {
  if constexpr (N == 1) {
    double s = v[0];
#pragma unroll
    for (int o = OFF; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
  } else {
    const bool hi = lane & OFF;
    double h[N / 2];
#pragma unroll
    for (int q = 0; q < N / 2; ++q) {
      const double keep = hi ? v[q + N / 2] : v[q], send = hi ? v[q] : v[q + N / 2];
      h[q] = keep + __shfl_xor_sync(0xffffffffu, send, OFF);
    }
    return fold_sum<N / 2, OFF / 2>(h, lane);
  }
}
template <int N>
__device__ __forceinline__ int fold_index(int lane) {
  int idx = 0, off = 16;
#pragma unroll
  for (int n = N; n > 1; n >>= 1, off >>= 1)
    if (lane & off) idx += n / 2;
  return idx;
}
// the one lane of those holding value fold_index<N> that writes it
template <int N>
__device__ __forceinline__ bool fold_writer(int lane) {
  return (lane & (32 / N - 1)) == 0;
}

__device__ __forceinline__ double warp_sum(double s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// ---------------------------------------------------------------------------
// A (k x k, column-major, symmetric) = Q T Q^T: diagonal d, off-diagonal e, and
// the reflectors H_j = 1 - tau_j v_j v_j^T in the columns of V (rows > j).
// Thread (ty, tx) of 16 x 32 holds the elements i = ty (mod 16), c = tx (mod 32),
// c <= i; a seventeenth warp does the scalars.  With x the column below the
// diagonal and beta = -+|x| the reflector is v = x - beta e_1, tau = 1 / (beta
// (beta - x_1)), not scaled to v_1 = 1, so A v = A x - beta A e_1 starts before
// beta is known and the square root and the division run beside it.  A step:
// columns j and j + 1 to shared memory; A x from the lower triangle, row sums
// folded within a warp, column sums through shared memory; p = tau A v;
// A -= v w^T + w v^T.  Three barriers a step; bound by the latency of a step's
// chain of FP64 operations (about 40 cycles each).
// ---------------------------------------------------------------------------
// threads: the scalar warp is the seventeenth up to 96 columns; above, 96
// registers a thread would spill the matrix, and the sixteenth does both
template <int NB> constexpr int tri_threads() { return EIG_THREADS + (NB <= 3 ? 32 : 0); }

// exponent of the largest element by its high word, 0 where that needs no scaling
__device__ __forceinline__ int tri_scale(unsigned top) {
  const int ex = (int)(top >> 20) - 1023;
  return (ex > 256 || ex < -256) && ex < 1024 && top != 0 ? ex : 0;
}

template <int NB>
__global__ void __launch_bounds__(tri_threads<NB>()) k_tridiag(const double *__restrict__ A, int k, double *__restrict__ V,
                                                              double *__restrict__ tau, double *__restrict__ d,
                                                              double *__restrict__ e) {
  constexpr int K = 32 * NB, NR = 2 * NB, NF = NR <= 2 ? 2 : NR <= 4 ? 4 : NR <= 8 ? 8 : 16;
  __shared__ double xs[2][K], ys[2][K], ps[K], pf[K], vs[K], part[16][K], red[NB], par[2];
  __shared__ unsigned top;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  if (threadIdx.x == 0) top = 0;
  double a[NR][NB];
  unsigned big = 0;  // largest high word without its sign: the exponent, in order of magnitude
#pragma unroll
  for (int r = 0; r < NR; ++r)
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int i = 16 * r + ty, c = 32 * b + tx;
      a[r][b] = (ty < 16 && i < k && c <= i) ? A[(long long)c * k + i] : 0.0;
      big = max(big, (unsigned)__double2hiint(a[r][b]) & 0x7fffffffu);
    }
  for (int i = threadIdx.x; i < K; i += tri_threads<NB>()) xs[0][i] = xs[1][i] = ys[0][i] = ys[1][i] = ps[i] = pf[i] = vs[i] = 0.0;
  __syncthreads();
  big = __reduce_max_sync(0xffffffffu, big);
  if (tx == 0) atomicMax(&top, big);
  __syncthreads();
  // far from one: the largest element to [1, 2), d and e scaled back at the end
  // (by two factors, as 2^ex may leave the range).  Infinities and NaN stay
  if (const int ex = tri_scale(top)) {
    const int e1 = ex / 2, e2 = ex - e1;
    const double f1 = __hiloint2double((1023 - e1) << 20, 0), f2 = __hiloint2double((1023 - e2) << 20, 0);
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
      for (int b = 0; b < NB; ++b) a[r][b] = a[r][b] * f1 * f2;
  }
  for (int j = 0; j < k - 2; ++j) {
    double *x = xs[j & 1], *y = ys[j & 1];
    if (ty < 16) {
      // rows up to j are published as zeros, so what follows needs no masks
      sfor<0, NB>([&](auto B) {
        constexpr int b = CV(B);
        if (b == (j >> 5) && tx == (j & 31)) {
#pragma unroll
          for (int r = 0; r < NR; ++r) {
            const int i = 16 * r + ty;
            x[i] = i > j ? a[r][b] : 0.0;
            if (i == j) d[j] = a[r][b];
          }
        }
        if (b == ((j + 1) >> 5) && tx == ((j + 1) & 31)) {
#pragma unroll
          for (int r = 0; r < NR; ++r) y[16 * r + ty] = 16 * r + ty > j ? a[r][b] : 0.0;
        }
      });
    }
    __syncthreads();
    constexpr int SW = tri_threads<NB>() / 32 - 1;
    if (ty == SW) {
      double t[NB];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int c = 32 * b + tx;
        t[b] = c > j + 1 ? x[c] * x[c] : 0.0;
      }
#pragma unroll
      for (int b = 1; b < NB; ++b) t[0] += t[b];
      const double s = warp_sum(t[0]), alpha = x[j + 1];
      double beta = alpha, tj = 0.0;
      if (s > 0.0) {
        beta = sqrt(alpha * alpha + s);
        if (alpha > 0.0) beta = -beta;
        tj = 1.0 / (beta * (beta - alpha));
      }
      if (tx == 0) {
        par[0] = tj;
        par[1] = beta;
        tau[j] = tj;
        e[j] = beta;
      }
    }
    if (ty < 16) {
      // A x
      double pr[NF], xi[NR];
#pragma unroll
      for (int r = 0; r < NF; ++r) pr[r] = 0.0;
#pragma unroll
      for (int r = 0; r < NR; ++r) xi[r] = x[16 * r + ty];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const double xc = x[32 * b + tx];
        double p0 = 0.0, p1 = 0.0;
#pragma unroll
        for (int r = 0; r < NR; ++r)
          if (16 * r + 15 >= 32 * b) {
            pr[r] += a[r][b] * xc;
            // blocks that cross the diagonal count their diagonal elements once
            const double t = 16 * r >= 32 * b + 32 || 16 * r + ty > 32 * b + tx ? xi[r] : 0.0;
            if (r & 1) p1 += a[r][b] * t;
            else p0 += a[r][b] * t;
          }
        part[ty][32 * b + tx] = p0 + p1;
      }
      const double sum = fold_sum<NF>(pr, tx);
      const int r = fold_index<NF>(tx);
      if (fold_writer<NF>(tx) && r < NR) ps[16 * r + ty] = sum;
    }
    __syncthreads();
    const double tj = par[0], beta = par[1];
    if (ty < NB) {
      const int c = 32 * ty + tx;
      double q[16];
#pragma unroll
      for (int w = 0; w < 16; ++w) q[w] = part[w][c];
#pragma unroll
      for (int h = 8; h > 0; h >>= 1)
#pragma unroll
        for (int w = 0; w < h; ++w) q[w] += q[w + h];
      const double p = c > j ? tj * ((q[0] + ps[c]) - beta * y[c]) : 0.0;
      const double v = c == j + 1 ? x[c] - beta : x[c];
      pf[c] = p;
      vs[c] = v;
      if (c < k) V[(long long)j * k + c] = v;
      const double dot = warp_sum(p * v);
      if (tx == 0) red[ty] = dot;
    }
    __syncthreads();
    if (ty < 16) {
      double h = 0.0;
#pragma unroll
      for (int b = 0; b < NB; ++b) h += red[b];
      h *= 0.5 * tj;
      double vc[NB], wc[NB];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        vc[b] = vs[32 * b + tx];
        wc[b] = pf[32 * b + tx] - h * vc[b];
      }
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int i = 16 * r + ty;
        const double vi = vs[i], wi = pf[i] - h * vi;
#pragma unroll
        for (int b = 0; b < NB; ++b)
          if (16 * r + 15 >= 32 * b) {
            if (16 * r >= 32 * b + 32) {
              a[r][b] -= vi * wc[b] + wi * vc[b];
            } else {  // elements above the diagonal stay zero
              const double u = vi * wc[b] + wi * vc[b];
              a[r][b] -= 32 * b + tx <= i ? u : 0.0;
            }
          }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < NR; ++r)
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int i = 16 * r + ty, c = 32 * b + tx;
      if (ty < 16 && 16 * r + 15 >= 32 * b && i < k) {
        if (i == c && i >= k - 2) d[i] = a[r][b];
        if (i == k - 1 && c == k - 2) e[c] = a[r][b];
      }
    }
  if (const int ex = tri_scale(top)) {
    __syncthreads();
    const int e1 = ex / 2, e2 = ex - e1;
    const double f1 = __hiloint2double((1023 + e1) << 20, 0), f2 = __hiloint2double((1023 + e2) << 20, 0);
    for (int i = threadIdx.x; i < k; i += tri_threads<NB>()) {
      d[i] = d[i] * f1 * f2;
      if (i + 1 < k) e[i] = e[i] * f1 * f2;
    }
  }
}

// Gershgorin bounds of the tridiagonal matrix, by one warp
__device__ __forceinline__ void gersh(const double *d, const double *e, int k, int lane, double &lo, double &hi) {
  lo = 1e300;
  hi = -1e300;
  for (int i = lane; i < k; i += 32) {
    const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < k ? fabs(e[i]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
}

// ---------------------------------------------------------------------------
// Eigenvalue blockIdx.x * 4 + warp (ascending) of the tridiagonal matrix: each
// lane counts the eigenvalues below one of 32 points of the bracket by the signs
// of the leading principal minors (Sturm sequence; T scaled to norm 1, the
// minors rescaled before they leave the range), which narrows it 33-fold a
// round.  No division in the recurrence: two dependent multiply-adds a row.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_bisect(const double *__restrict__ d, const double *__restrict__ e, int k,
                                                double *__restrict__ w) {
  __shared__ double sd[EIG_MAXK], se[EIG_MAXK];
  const int lane = threadIdx.x & 31, idx = blockIdx.x * 4 + (threadIdx.x >> 5);
  double lo, hi;
  gersh(d, e, k, lane, lo, hi);
  double nrm = fmax(fabs(lo), fabs(hi));
  if (!(nrm > 0.0)) nrm = 1.0;
  const double inv = 1.0 / nrm;
  for (int i = threadIdx.x; i < k; i += 128) {
    sd[i] = d[i] * inv;
    const double t = i > 0 ? e[i - 1] * inv : 0.0;
    se[i] = t * t;
  }
  __syncthreads();
  if (idx >= k) return;
  lo = lo * inv - 1e-14;
  hi = hi * inv + 1e-14;
  for (int round = 0; round < 12; ++round) {
    const double x = lo + (hi - lo) * ((double)(lane + 1) / 33.0);
    double p1 = 1.0, p0 = 0.0;
    int cnt = 0;
    for (int i0 = 0; i0 < k; i0 += 4) {
      // signs and magnitudes by integer tests, off the chain of multiply-adds;
      // a row grows the minors at most threefold and shrinks them by at most
      // 1e-18, so four rows stay in range between rescalings
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + u;
        if (i < k) {
          double p = (sd[i] - x) * p1 - se[i] * p0;
          // a zero minor takes the sign opposite to the one before it
          if ((__double_as_longlong(p) << 1) == 0) p = __double2hiint(p1) < 0 ? 1e-100 : -1e-100;
          cnt += ((unsigned)(__double2hiint(p) ^ __double2hiint(p1))) >> 31;
          p0 = p1;
          p1 = p;
        }
      }
      const int e1 = (__double2hiint(p1) >> 20) & 0x7ff, e0 = (__double2hiint(p0) >> 20) & 0x7ff;
      const int m = e1 > e0 ? e1 : e0;
      const double f = m > 1023 + 200 ? 0x1p-400 : m < 1023 - 200 ? 0x1p400 : 1.0;
      p1 *= f;
      p0 *= f;
    }
    // points with cnt <= idx lie at or below the wanted eigenvalue
    const unsigned below = __ballot_sync(0xffffffffu, cnt <= idx);
    const int n = __popc(below);
    const double xl = __shfl_sync(0xffffffffu, x, n > 0 ? n - 1 : 0), xh = __shfl_sync(0xffffffffu, x, n < 32 ? n : 31);
    if (n > 0) lo = xl;
    if (n < 32) hi = xh;
  }
  if (lane == 0) w[idx] = 0.5 * (lo + hi) * nrm;
}

// ---------------------------------------------------------------------------
// Eigenvector of w[k - nv + c] by inverse iteration, thread c: LU of T - w with
// partial pivoting (T scaled to norm 1, tiny pivots raised to eps), three solves
// from a random start.  The factors and the vector of the block's INV_VEC threads
// lie in shared memory ([5][k][INV_VEC]): a chain of k rows with loads from L2
// took twice as long.  Y (k x nv, column-major) gets unit vectors; *check the
// largest residual |T y - w y| (times ||T||^-1, as the bits of a nonnegative
// double).
// ---------------------------------------------------------------------------
#define INV_VEC 8
__global__ void __launch_bounds__(32) k_invit(const double *__restrict__ d, const double *__restrict__ e, int k,
                                              const double *__restrict__ w, int nv, double *__restrict__ Y,
                                              unsigned long long *__restrict__ check) {
  extern __shared__ double fac[];
  __shared__ double sd[EIG_MAXK], se[EIG_MAXK];
  const int lane = threadIdx.x;
  double lo, hi;
  gersh(d, e, k, lane, lo, hi);
  double nrm = fmax(fabs(lo), fabs(hi));
  if (!(nrm > 0.0)) nrm = 1.0;
  const double inv = 1.0 / nrm;
  for (int i = lane; i < k; i += 32) {
    sd[i] = d[i] * inv;
    se[i] = i + 1 < k ? e[i] * inv : 0.0;
  }
  __syncwarp();
  const int c = blockIdx.x * INV_VEC + lane;
  if (lane >= INV_VEC || c >= nv) return;
  const double lam = w[k - nv + c] * inv, eps = 2.2e-16;
  const int ks = k * INV_VEC;
  double *U0 = fac + lane, *U1 = U0 + ks, *U2 = U1 + ks, *Lm = U2 + ks, *X = Lm + ks;
  // LU; U0 holds the reciprocal pivots, Lm the multipliers, a row swap as the
  // multiplier + 4 (multipliers are at most 1 in magnitude)
  {
    double a = sd[0] - lam, b = se[0];
    for (int i = 0; i + 1 < k; ++i) {
      const double lowr = se[i], dn = sd[i + 1] - lam, en = se[i + 1];
      if (fabs(a) >= fabs(lowr)) {
        double p = a;
        if (fabs(p) < eps) p = p < 0.0 ? -eps : eps;
        const double r = 1.0 / p, m = lowr * r;
        U0[i * INV_VEC] = r;
        U1[i * INV_VEC] = b;
        U2[i * INV_VEC] = 0.0;
        Lm[i * INV_VEC] = m;
        a = dn - m * b;
        b = en;
      } else {
        const double r = 1.0 / lowr, m = a * r;
        U0[i * INV_VEC] = r;
        U1[i * INV_VEC] = dn;
        U2[i * INV_VEC] = en;
        Lm[i * INV_VEC] = m + 4.0;
        a = b - m * dn;
        b = -m * en;
      }
    }
    if (fabs(a) < eps) a = a < 0.0 ? -eps : eps;
    U0[(k - 1) * INV_VEC] = 1.0 / a;
  }
  unsigned rng = 0x9E3779B9u * (unsigned)(c + 1) ^ 0x7F4A7C15u;
  for (int i = 0; i < k; ++i) {
    rng ^= rng << 13;
    rng ^= rng >> 17;
    rng ^= rng << 5;
    X[i * INV_VEC] = (double)rng * (2.0 / 4294967296.0) - 1.0;
  }
  double scale = 1.0;
  for (int it = 0; it < 3; ++it) {
    double cur = X[0] * scale;
    for (int i = 0; i + 1 < k; ++i) {
      double m = Lm[i * INV_VEC];
      const double nxt = X[(i + 1) * INV_VEC] * scale;
      if (m > 2.0) {
        m -= 4.0;
        X[i * INV_VEC] = nxt;
        cur = cur - m * nxt;
      } else {
        X[i * INV_VEC] = cur;
        cur = nxt - m * cur;
      }
    }
    double x1 = cur * U0[(k - 1) * INV_VEC], x2 = 0.0, big = fabs(x1);
    X[(k - 1) * INV_VEC] = x1;
    for (int i = k - 2; i >= 0; --i) {
      const double x0 = (X[i * INV_VEC] - U1[i * INV_VEC] * x1 - U2[i * INV_VEC] * x2) * U0[i * INV_VEC];
      X[i * INV_VEC] = x0;
      big = fmax(big, fabs(x0));
      x2 = x1;
      x1 = x0;
    }
    scale = big > 0.0 ? 1.0 / big : 1.0;
  }
  double nn = 0.0;
  for (int i = 0; i < k; ++i) {
    const double x = X[i * INV_VEC] * scale;
    nn += x * x;
  }
  const double f = scale / sqrt(nn);
  double res = 0.0, xm = 0.0, x0 = X[0] * f;
  for (int i = 0; i < k; ++i) {
    const double xp = i + 1 < k ? X[(i + 1) * INV_VEC] * f : 0.0;
    const double r = (sd[i] - lam) * x0 + se[i] * xp + (i > 0 ? se[i - 1] * xm : 0.0);
    const double ar = fabs(r);
    res = ar > res || ar != ar ? (ar != ar ? 1e300 : ar) : res;
    Y[(long long)c * k + i] = x0;
    xm = x0;
    x0 = xp;
  }
  atomicMax(check, (unsigned long long)__double_as_longlong(res));
}

// ---------------------------------------------------------------------------
// Y <- H_0 H_1 ... H_(k-3) Y, a warp per column, the column in its registers, two
// reflectors at a time (their sums v^T z, u^T z and u^T v run together) while the
// next two load; bound by the chain of warp sums.
// ---------------------------------------------------------------------------
template <int NB>
__global__ void __launch_bounds__(32) k_backtr(const double *__restrict__ V, const double *__restrict__ tau, int k,
                                               double *__restrict__ Y) {
  const int lane = threadIdx.x;
  double *y = Y + (long long)blockIdx.x * k;
  double z[NB], nv[NB], nu[NB], tv, tu;
  // reflector j of the pair (j, j - 1); zero (tau 0) below column 0
  auto load = [&](int j, double *r, double &t) {
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int c = 32 * b + lane;
      r[b] = j >= 0 && c < k ? V[(long long)j * k + c] : 0.0;
    }
    t = j >= 0 ? tau[j] : 0.0;
  };
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int c = 32 * b + lane;
    z[b] = c < k ? y[c] : 0.0;
  }
  load(k - 3, nv, tv);
  load(k - 4, nu, tu);
  for (int j = k - 3; j >= 0; j -= 2) {
    double v[NB], u[NB];
    const double t0 = tv, t1 = tu;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      v[b] = nv[b];
      u[b] = nu[b];
    }
    load(j - 2, nv, tv);
    load(j - 3, nu, tu);
    double vz = 0.0, uz = 0.0, uv = 0.0;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      vz += v[b] * z[b];
      uz += u[b] * z[b];
      uv += u[b] * v[b];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      vz += __shfl_xor_sync(0xffffffffu, vz, o);
      uz += __shfl_xor_sync(0xffffffffu, uz, o);
      uv += __shfl_xor_sync(0xffffffffu, uv, o);
    }
    const double s0 = t0 * vz, s1 = t1 * (uz - s0 * uv);
#pragma unroll
    for (int b = 0; b < NB; ++b) z[b] = z[b] - s0 * v[b] - s1 * u[b];
  }
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int c = 32 * b + lane;
    if (c < k) y[c] = z[b];
  }
}

extern "C" size_t bdgd_eig_work(int k) {
  // V, tau, d, e
  return sizeof(double) * ((size_t)k * k + 3 * (size_t)k);
}

template <int NB>
static void launch_eig(bdgd_ctx *c, const double *A, int k, int nv, double *w, double *Y, double *work,
                       unsigned long long *check) {
  double *V = work, *tau = V + (size_t)k * k, *d = tau + k, *e = d + k;
  k_tridiag<NB><<<1, tri_threads<NB>(), 0, c->stream>>>(A, k, V, tau, d, e);
  k_bisect<<<(k + 3) / 4, 128, 0, c->stream>>>(d, e, k, w);
  k_invit<<<(nv + INV_VEC - 1) / INV_VEC, 32, 5 * INV_VEC * sizeof(double) * k, c->stream>>>(d, e, k, w, nv, Y, check);
  k_backtr<NB><<<nv, 32, 0, c->stream>>>(V, tau, k, Y);
}

extern "C" int bdgd_eig_top(bdgd_ctx *c, const double *A, int k, int nv, double *w, double *Y, double *work,
                            double *d_check) {
  if (k < 3 || k > EIG_MAXK || nv < 1 || nv > k) return BDGD_ERR_UNSUPPORTED;
  if (const int rc = bdgd_smem_attr(k_invit, 5 * INV_VEC * sizeof(double) * EIG_MAXK)) return rc;
  BDGD_CK(cudaMemsetAsync(d_check, 0, sizeof(double), c->stream));
  unsigned long long *chk = (unsigned long long *)d_check;
  for (int i = 0; i < 4; ++i) bdgd_count_launch();
  switch ((k + 31) / 32) {
    case 1: launch_eig<1>(c, A, k, nv, w, Y, work, chk); break;
    case 2: launch_eig<2>(c, A, k, nv, w, Y, work, chk); break;
    case 3: launch_eig<3>(c, A, k, nv, w, Y, work, chk); break;
    case 4: launch_eig<4>(c, A, k, nv, w, Y, work, chk); break;
    case 5: launch_eig<5>(c, A, k, nv, w, Y, work, chk); break;
    default: launch_eig<6>(c, A, k, nv, w, Y, work, chk); break;
  }
  BDGD_CK(cudaGetLastError());
  return BDGD_OK;
}
