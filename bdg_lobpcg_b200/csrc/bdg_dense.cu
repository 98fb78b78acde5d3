// bdg_dense.cu -- small dense factorisations of the Rayleigh-Ritz step, one
// thread block each.
//
// The Gram blocks of the iteration (X^H X, [X, P]^H [X, P], W^H W, S^H A S; k up
// to 3 sizeSub) need orthonormalising coefficients Z with Z^T G Z = I.  The
// eigen-decomposition that gives them with dropped directions costs 0.45 ms at
// k = 48 and 1.2 ms at k = 96 (cuSOLVER syevd: a chain of small launches).  Where
// G is well conditioned, as it is nearly always, its Cholesky factor serves as
// well: Z = D L^-T with D G D = L L^T of unit diagonal.  k_chol_inverse factors
// and inverts in one pass over the columns and reports the smallest pivot, by
// which the caller decides whether to take it.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include "bdg_blas.h"
#include "bdg_dev.h"
#include "bdg_dft.cuh"

#define CHOL_THREADS 512

// Column j of the elimination applied to the trailing matrix and to the
// inverse at once.  The lower triangle e holds, at step j, the trailing Schur
// complement in columns c > j and the rows of L^-1 (unit lower L of L D' L^T)
// built so far in columns c < j; row i > j becomes
//   c < j: e -= a_ij e_jc / p    c = j: -a_ij / p    c > j: e -= a_ij a_cj / p
// with a_ij = e(i, j) and p = e(j, j) before the step.  Thread (ty, tx) of 16 x 32
// holds the elements i = ty (mod 16), c = tx (mod 32) in registers; a step
// exchanges one column and one row through shared memory (two buffers, so one
// barrier a step).  Bound by the latency of the k steps, 1/p and the barrier: 27,
// 65 and 223 us at k = 48, 96 and 192 (0.56, 0.68 and 1.16 us a step), the
// multiply-adds of a thread adding to it at 192.
template <int NB>
__global__ void __launch_bounds__(CHOL_THREADS) k_chol_inverse(const double *__restrict__ G, int k, int ldg,
                                                               double *__restrict__ Z, double *__restrict__ minpiv) {
  constexpr int K = 32 * NB, NR = 2 * NB;
  __shared__ double colv[2][K], vec[2][K], rp[2], sd[K], piv[K];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < K; i += CHOL_THREADS) {
    const double g = i < k ? G[(long long)i * ldg + i] : 1.0;
    sd[i] = g > 0.0 ? 1.0 / sqrt(g) : 1.0;
    piv[i] = 1.0;
  }
  __syncthreads();
  double e[NR][NB];
#pragma unroll
  for (int a = 0; a < NR; ++a)
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int i = 16 * a + ty, c = 32 * b + tx;
      e[a][b] = i == c ? 1.0 : 0.0;
      if (16 * a + 15 >= 32 * b && i < k && c < k)
        e[a][b] = sd[i] * (0.5 * (G[(long long)c * ldg + i] + G[(long long)i * ldg + c])) * sd[c];
    }
  double low = 1e300;  // smallest pivot (thread 0)
  for (int j = 0; j < k; ++j) {
    const int s = j & 1, ja = j >> 4, jb = j >> 5;
    // publish column j (zeros for rows i <= j, which the step leaves), row j
    // (columns c < j) and 1/p; column j itself restarts from zero, 1 on the diagonal
    sfor<0, NB>([&](auto B) {
      constexpr int b = CV(B);
      if (b == jb && tx == (j & 31)) {
#pragma unroll
        for (int a = 0; a < NR; ++a) {
          const int i = 16 * a + ty;
          if (16 * a + 15 >= 32 * b) {
            const double x = e[a][b];
            colv[s][i] = i > j ? x : 0.0;
            if (i > j) {
              vec[s][i] = x;
              e[a][b] = 0.0;
            } else if (i == j) {
              const bool bad = !(x > 0.0);  // NaN too
              piv[j] = bad ? -1.0 : x;
              rp[s] = 1.0 / (bad ? 1.0 : x);
              vec[s][j] = 1.0;
              e[a][b] = 1.0;
            }
          } else {
            colv[s][i] = 0.0;
          }
        }
      }
    });
    if (ty == (j & 15)) {
      sfor<0, NR>([&](auto R) {
        constexpr int a = CV(R);
        if (a == ja) {
#pragma unroll
          for (int b = 0; b < NB; ++b)
            if (16 * a + 15 >= 32 * b && 32 * b + tx < j) vec[s][32 * b + tx] = e[a][b];
        }
      });
    }
    __syncthreads();
    const double q = rp[s];
    double v[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) v[b] = vec[s][32 * b + tx];
#pragma unroll
    for (int a = 0; a < NR; ++a) {
      const double l = colv[s][16 * a + ty] * q;
#pragma unroll
      for (int b = 0; b < NB; ++b)
        if (16 * a + 15 >= 32 * b) e[a][b] -= l * v[b];
    }
  }
  __syncthreads();
  // Z(c, i) = d_c L^-1(i, c) / sqrt(p_i), column-major
#pragma unroll
  for (int a = 0; a < NR; ++a) {
    const int i = 16 * a + ty;
    if (i < k) {
      const double p = piv[i];
      const double si = p > 0.0 ? 1.0 / sqrt(p) : 1.0;
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int c = 32 * b + tx;
        if (c < k) Z[(long long)i * k + c] = c <= i ? sd[c] * e[a][b] * si : 0.0;
      }
    }
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < k; ++i) low = fmin(low, piv[i]);
    *minpiv = low;
  }
}

extern "C" int bdgd_chol_inverse(bdgd_ctx *c, const double *G, int k, int ldg, double *Z, double *minpiv) {
  if (k < 1 || k > BDGD_CHOL_MAX) return BDGD_ERR_UNSUPPORTED;
  bdgd_count_launch();
  switch ((k + 31) / 32) {
    case 1: k_chol_inverse<1><<<1, CHOL_THREADS, 0, c->stream>>>(G, k, ldg, Z, minpiv); break;
    case 2: k_chol_inverse<2><<<1, CHOL_THREADS, 0, c->stream>>>(G, k, ldg, Z, minpiv); break;
    case 3: k_chol_inverse<3><<<1, CHOL_THREADS, 0, c->stream>>>(G, k, ldg, Z, minpiv); break;
    case 4: k_chol_inverse<4><<<1, CHOL_THREADS, 0, c->stream>>>(G, k, ldg, Z, minpiv); break;
    case 5: k_chol_inverse<5><<<1, CHOL_THREADS, 0, c->stream>>>(G, k, ldg, Z, minpiv); break;
    default: k_chol_inverse<6><<<1, CHOL_THREADS, 0, c->stream>>>(G, k, ldg, Z, minpiv); break;
  }
  BDGD_CK(cudaGetLastError());
  return BDGD_OK;
}
