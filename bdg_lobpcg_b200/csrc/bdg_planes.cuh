// bdg_planes.cuh -- FFT operator passes that keep an xy plane on chip.
//
// A 3D operator apply is three passes: k_plane_fwd transforms whole xy planes
// (prologue, x lines, y lines), k_zlines the z lines (forward * k-space
// multiplier * inverse), k_plane_inv the planes back (y, x, epilogue).  The
// five line passes they replace moved every spectrum eight times through the
// memory system, these move it four times.  Every axis length n = n1 * n2
// (n1, n2 <= 16) is transformed in two register DFTs with one exchange in
// shared memory, the factors chosen on the host and the DFT sizes by a
// switch, so one kernel serves all lengths:
//
//   first   item t < n2 holds x[n2*i + t], i < n1: DFT of size n1, twiddle
//           w_n^(t*k1), stored at slot n2*k1 + t
//   second  item k1 < n1 holds slots n2*k1 + i, i < n2: DFT of size n2, its
//           output k2 is X[k1 + n1*k2]
//
// and back by the transposed steps.  Both steps work in place: what a plane
// holds between them is permuted, and the permutation is undone by indexing
// (columns by colpos(), rows when a plane leaves the chip), never by a copy.
//
// Real rows y and y + ny/2 are transformed as one complex row z = a + i b, so
// a plane of n real rows takes n/2 complex ones, and split where the y step
// reads them, 2 A_k = Z_k + conj Z_(n-k), 2 B_k = -i (Z_k - conj Z_(n-k)) (the
// factor 2 goes into the k-space multiplier).  The first y step is of even
// size, so the item of column k that reads Z_k and Z_(n-k) of its rows gets
// all the y values that it needs, and what it returns fits the slots that it
// read: y slots of the upper half of a column lie in column n-k (columns 0
// and n/2, which have no partner, use two extra columns).  The inverse mirrors
// this with its second y step.  With ny odd, real rows are transformed as
// complex rows with a zero imaginary part (PL_WHOLE).
//
// Columns lie at x2p*(k % x1) + k / x1 with x2p odd after an in-place x
// transform (PlaneGeo), or in natural order where the items of the second x
// step fit the registers across a barrier (PlaneCT).
//
// What bounds them (ncu, 64^3 FP64, 32 columns of Lrep): the L1 data path,
// 80% busy in k_plane_fwd: an element of 16 bytes crosses shared memory six
// times (4 cycles a warp each) and global memory twice (8 cycles).  Hence the
// twiddles of the y and z steps come from the constant bank and occupancy is
// bought with registers (72 a thread at 64^3: three blocks of 288 threads, one
// item a thread; 128 registers and two blocks took 121 + 227 us for the two
// plane kernels against 119 + 128).  128^3 FP64 planes take 139 KB, one block an
// SM.  Whole applies, line passes before against plane passes: Lrep 64^3 FP64, 32
// columns 459 -> 320 us; T 128^3 FP64, 64 columns 4849 -> 3556 us; Lrep 128^3
// FP32, 64 columns 4448 -> 2800 us; M 48^3, one column 30 -> 25 us; 50x45x36 FP64
// (run-time sized stages before), 16 columns 599 -> 110 us.  Chunks of columns
// whose spectra stay in L2 were slower at every size (64^3: 360 us at 120 MB):
// the last waves of the many small launches cost more than DRAM does.
//
// The spectrum layout (x extent nx/2+1 or nx, x fastest) is that of the other
// pass families and of FFTW's r2c (src/fft_helpers_impl.inc:24-82 of the
// reference).
#pragma once

#include "bdg_dft.cuh"
#include "bdg_planes.h"

enum { PL_REAL = 0, PL_CPLX = 1, PL_WHOLE = 2 };

// i / d for i, d < 2^16: the high word of i * ceil(2^32 / d)
struct FDiv {
  unsigned d, m;
};
__device__ __forceinline__ int fdiv(int i, FDiv f) { return f.d == 1 ? i : (int)__umulhi((unsigned)i, f.m); }

struct PlaneGeo {
  int nx, ny, nz, nxk;
  int rows;            // complex rows of a plane on chip: ny/2 (PL_REAL) or ny
  int x1, x2, x2p;     // nx = x1 * x2, see colpos()
  int ye, yo;          // ny = ye * yo, ye even for PL_REAL
  int z1, z2;          // nz = z1 * z2
  int ld;              // row stride of a plane in shared memory
  int ex;              // first of the two extra columns
  FDiv dx1, dx2, dnxk, dyr;  // dyr: rows per group of the inverse, ye/2 or ye
  int tx;              // z lines per block
  int mode;            // PL_REAL, PL_CPLX or PL_WHOLE
};
// RM: largest DFT size of the switches.  Without the sizes above 8 the kernels
// need 80 registers, not 128, and three blocks fit an SM, not two.
template <int RM>
struct PlanePar : PlaneGeo {
  static constexpr bool CT = false;
  static constexpr int RMAX = RM;
};
__device__ __forceinline__ int colpos(const PlaneGeo &q, int k) {
  const int a = fdiv(k, q.dx1);
  return q.x2p * (k - a * q.x1) + a;
}

// n = s * (n / s) with s <= n / s <= 16 and s largest
__host__ __device__ constexpr int split_small(int n) {
  for (int s = 16; s >= 2; --s)
    if (n % s == 0 && s * s <= n && n / s <= 16) return s;
  return 0;
}

// i / D
template <int D> struct CDiv {};
template <int D>
__device__ __forceinline__ int fdiv(int i, CDiv<D>) { return (int)((unsigned)i / (unsigned)D); }

// The parameters of real N^3 grids as constants (members as in PlanePar).
// ld: with it the lanes of the x steps, which run over the items of a row and
// then over rows, fall into distinct banks.
template <int N>
struct PlaneCT {
  static constexpr bool CT = true;
  static constexpr int nx = N, ny = N, nz = N, nxk = N / 2 + 1, rows = N / 2;
  static constexpr int x1 = split_small(N), x2 = N / x1, x2p = x2 + 1 - (x2 & 1);
  static constexpr int ye = x1, yo = x2, z1 = x2, z2 = x1;
  static constexpr int ld0 = x1 * x2p > N + 2 ? x1 * x2p : N + 2, ldm = x2 % 8 ? x2 % 8 : x1 % 8;
  static constexpr int ld = ld0 + (ldm - ld0 % 8 + 8) % 8;
  static constexpr int ex = N, tx = 16;
  static_assert(ye % 2 == 0, "pairs of rows");
  CDiv<x1> dx1;
  CDiv<x2> dx2;
  CDiv<nxk> dnxk;
  CDiv<ye / 2> dyr;
};
template <int N>
__device__ __forceinline__ int colpos(const PlaneCT<N> &, int k) { return k; }
// the column that holds the upper y slots of column k
template <typename Q>
__device__ __forceinline__ int colb(const Q &q, int k) {
  return k == 0 ? q.ex : 2 * k == q.nx ? q.ex + 1 : colpos(q, q.nx - k);
}

// f(integral_constant<R>) for the DFT size r in 2..RMAX (8 or 16)
template <int RMAX, typename F>
__device__ __forceinline__ void rswitch(int r, F &&f) {
  switch (r) {
#define RCASE(R) case R: if constexpr (R <= RMAX) f(std::integral_constant<int, R>{}); break
    RCASE(2); RCASE(3); RCASE(4); RCASE(5); RCASE(6); RCASE(7); RCASE(8); RCASE(9);
    RCASE(10); RCASE(11); RCASE(12); RCASE(13); RCASE(14); RCASE(15); RCASE(16);
#undef RCASE
    default: break;
  }
}

// f(integral_constant) with the DFT size of one step: a constant of the
// parameters, or by the switch
#define PLANE_STEP(M)                                              \
  template <typename Q, typename F>                                \
  __device__ __forceinline__ void step_##M(const Q &q, F &&f) {    \
    if constexpr (Q::CT) f(std::integral_constant<int, Q::M>{});   \
    else rswitch<Q::RMAX>(q.M, f);                                 \
  }
PLANE_STEP(x1)
PLANE_STEP(x2)
PLANE_STEP(ye)
PLANE_STEP(yo)
PLANE_STEP(z1)
PLANE_STEP(z2)
#undef PLANE_STEP

template <int R, int SGN, typename C>
__device__ __forceinline__ void twiddle(C *v, const C *roots, int step) {
#pragma unroll
  for (int k = 1; k < R; ++k) v[k] = cmul(v[k], rootv(roots, step * k, SGN));
}

// threads of a plane block and resident blocks per SM
template <typename T, typename Q>
constexpr int plane_threads() {
  if constexpr (Q::CT) return Q::nx == 128 ? 512 : Q::nx == 96 ? 384 : Q::nx == 64 ? 288 : Q::nx == 48 ? 224 : Q::nx == 32 ? 160 : 64;
  else return 256;
}
template <typename T, typename Q>
constexpr int plane_blocks() {
  if constexpr (Q::CT) return sizeof(T) == 8 ? (Q::nx == 128 ? 1 : Q::nx == 96 ? 2 : Q::nx == 64 ? 3 : Q::nx == 48 ? 4 : 5)
                                             : (Q::nx == 128 ? 2 : Q::nx == 96 ? 3 : Q::nx == 64 ? 4 : Q::nx == 48 ? 5 : 8);
  else return sizeof(T) == 8 ? (Q::RMAX > 8 ? 2 : 3) : (Q::RMAX > 8 ? 2 : 4);
}
// roots exp(-2 pi i m / n) of one axis as a kernel parameter.  In the y and z
// steps the lanes of a warp hold one or two values of t, so a twiddle comes
// from the constant bank; a 16-byte load of it through L1 would cost as much
// of the L1 data path, the limit of these kernels, as an element does.
template <typename C, typename Q>
constexpr int tw_size() {
  if constexpr (Q::CT) return Q::nx;
  else return 256;
}
template <typename C, typename Q>
struct TwTab {
  C w[tw_size<C, Q>()];
};
template <int R, int SGN, typename C, typename Q>
__device__ __forceinline__ void twiddle_c(C *v, const TwTab<C, Q> &tab, int step) {
#pragma unroll
  for (int k = 1; k < R; ++k) {
    C w = tab.w[step * k];
    if (SGN > 0) w.y = -w.y;
    v[k] = cmul(v[k], w);
  }
}

constexpr int kZThreads = 128;
template <typename T, typename Q>
constexpr int z_blocks() {
  if constexpr (Q::CT) return sizeof(T) == 8 ? (Q::nz == 128 ? 4 : Q::nz == 96 ? 5 : 6) : (Q::nz >= 96 ? 7 : 9);
  else return sizeof(T) == 8 ? (Q::RMAX > 8 ? 4 : 6) : (Q::RMAX > 8 ? 6 : 9);
}

// The kernels are launched programmatically: the blocks of one become resident
// while the last blocks of the kernel before it run, and wait here for its
// results (the launch latency of a small apply overlaps).  So x, y and the
// spectra may be written while a kernel that reads them is already resident (x
// by the inverse of an apply before this one): they are read by ordinary loads,
// through pointers without __restrict__, after this wait.  The read-only path
// (__ldg) wants data that no one writes during the kernel's life: the fields and
// tables, whose uploads end with a wait of the host or a copy, which a launch
// does not overlap.
__device__ __forceinline__ void grid_wait() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Barrier between two steps.  The thread index becomes opaque with it: the
// compiler would otherwise load the twiddles and form the addresses of later
// steps ahead of it, and spill the elements.
__device__ __forceinline__ void step_sync(int &tid) {
  __syncthreads();
  asm volatile("" : "+r"(tid));
}

// the block's threads ask L2 for the `bytes` from p on
template <int THR> __device__ __forceinline__ void prefetch_l2(const void *p, int bytes) {
  for (int i = threadIdx.x * 128; i < bytes; i += THR * 128)
    asm volatile("prefetch.global.L2 [%0];" ::"l"((const char *)p + i));
}

// ---------------------------------------------------------------------------
// prologue, x and y forward of one plane.  grid.x: spectra (column * J +
// job), grid.y: planes, so that blocks of all columns read a plane of the
// coefficients together.
// ---------------------------------------------------------------------------
template <typename T, int MODE, typename Q, bool PF>
__global__ void __launch_bounds__((plane_threads<T, Q>()), (plane_blocks<T, Q>()))
    k_plane_fwd(GeoDev g, Prog p, FieldsDev f, Q q, const __grid_constant__ TwTab<typename Cx<T>::t, Q> tw,
                const void *xin, long long ldx, typename Cx<T>::t *spec,
                void *yout, long long ldy, int ahead) {
  typedef typename Cx<T>::t C;
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int THR = plane_threads<T, Q>();
  C *P = (C *)smraw;
  int tid = threadIdx.x;
  const int z = blockIdx.y, job = blockIdx.x;
  const int col = job / p.J, jj = job - col * p.J;
  const int hf = p.jh[jj], kind = p.pre[hf][p.jf[jj]];
  // K and M: y <- lt x here, where x is at hand; the inverse adds to it
  const bool local = p.jf[jj] == 0 && (p.post[hf] == POST_K || p.post[hf] == POST_M);
  const T *lt = (const T *)post_coef(f, p.post[hf]);
  const long long plane = (long long)z * q.nx * q.ny;
  const C *rx = roots_of<C>(g.ax[0]);
  grid_wait();
  // x, first step: rows from global memory
  step_x1(q, [&](auto RC) {
    constexpr int R = CV(RC);
    const int tot = q.rows * q.x2;
#pragma unroll 1
    for (int i = tid; i < tot; i += THR) {
      const int row = fdiv(i, q.dx2), t = i - row * q.x2;
      const int o = row * q.nx + t;
      C v[R];
      if constexpr (MODE == PL_REAL) {
        const long long oc = col * ldx + hf * g.S + plane + o;
        const int hs = q.rows * q.nx;  // to row y + ny/2
        const T *sa = (const T *)xin + oc;
        const T *cf = (const T *)pre_coef(f, kind);
#pragma unroll
        for (int r = 0; r < R; ++r) v[r].x = sa[r * q.x2];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r].y = sa[hs + r * q.x2];
        if (local) {
          T *y = (T *)yout + col * ldy + hf * g.S + plane + o;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const T *l = lt + plane + o + u * hs;
            T c[R];
#pragma unroll
            for (int r = 0; r < R; ++r) c[r] = __ldg(l + r * q.x2);
#pragma unroll
            for (int r = 0; r < R; ++r) y[u * hs + r * q.x2] = c[r] * (u ? v[r].y : v[r].x);
          }
        }
        if (cf) {
          const T *ca = cf + plane + o;
          T c[R];
#pragma unroll
          for (int r = 0; r < R; ++r) c[r] = __ldg(ca + r * q.x2);
#pragma unroll
          for (int r = 0; r < R; ++r) v[r].x = pre_real<T>(kind, v[r].x, c[r]);
#pragma unroll
          for (int r = 0; r < R; ++r) c[r] = __ldg(ca + hs + r * q.x2);
#pragma unroll
          for (int r = 0; r < R; ++r) v[r].y = pre_real<T>(kind, v[r].y, c[r]);
        } else {
#pragma unroll
          for (int r = 0; r < R; ++r) {
            v[r].x = pre_real<T>(kind, v[r].x, (T)0);
            v[r].y = pre_real<T>(kind, v[r].y, (T)0);
          }
        }
      } else if constexpr (MODE == PL_WHOLE) {
        const T *src = (const T *)xin + col * ldx + hf * g.S + plane + o;
        const T *cf = (const T *)pre_coef(f, kind);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          v[r].x = src[r * q.x2];
          v[r].y = cf ? __ldg(cf + plane + o + r * q.x2) : (T)0;
        }
        if (local) {
          T *y = (T *)yout + col * ldy + hf * g.S + plane + o;
#pragma unroll
          for (int r = 0; r < R; ++r) y[r * q.x2] = __ldg(lt + plane + o + r * q.x2) * v[r].x;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = cmk<C>(pre_real<T>(kind, v[r].x, v[r].y), 0.0);
      } else {
        const C *src = (const C *)xin + col * ldx + hf * g.S + plane + o;
        const T *cr = (kind == PRE_PK || kind == PRE_PM) ? (const T *)pre_coef(f, kind) : nullptr;
        const C *cw = (kind == PRE_CONJWF || kind == PRE_DENS) ? (const C *)f.w : nullptr;
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[r * q.x2];
        if (local) {
          C *y = (C *)yout + col * ldy + hf * g.S + plane + o;
          T c[R];
#pragma unroll
          for (int r = 0; r < R; ++r) c[r] = __ldg(lt + plane + o + r * q.x2);
#pragma unroll
          for (int r = 0; r < R; ++r) y[r * q.x2] = cscale(v[r], c[r]);
        }
        C w[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          w[r] = cw ? __ldg(cw + plane + o + r * q.x2) : czero<C>();
          if (cr) w[r].x = __ldg(cr + plane + o + r * q.x2);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = pre_cplx<T, C>(kind, v[r], w[r].x, w[r]);
      }
      rdft<R, -1>(v);
      twiddle<R, -1>(v, rx, t);
      C *d = P + row * q.ld + t;
#pragma unroll
      for (int k = 0; k < R; ++k) d[k * q.x2p] = v[k];
    }
  });
  if (PF && ahead > 0) {
    const unsigned b = blockIdx.y * gridDim.x + blockIdx.x + ahead, zn = b / gridDim.x;
    if (zn < gridDim.y) {
      constexpr int es = MODE == PL_CPLX ? (int)sizeof(C) : (int)sizeof(T);
      const int jn = b - zn * gridDim.x, cn = jn / p.J, hn = p.jh[jn - cn * p.J];
      prefetch_l2<THR>((const char *)xin + (cn * ldx + hn * g.S + (long long)zn * q.nx * q.ny) * es, es * q.nx * q.ny);
    }
  }
  step_sync(tid);
  // x, second step
  step_x2(q, [&](auto RC) {
    constexpr int R = CV(RC);
    const int tot = q.rows * q.x1;
    if constexpr (Q::CT) {
      // items stay in registers while every one is read, then are stored in
      // natural column order
      constexpr int IT = (Q::rows * Q::x1 + THR - 1) / THR;
      C v[IT][R];
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int i = tid + it * THR;
        if (IT * THR == Q::rows * Q::x1 || i < tot) {
          const int row = fdiv(i, q.dx1), k1 = i - row * q.x1;
          const C *d = P + row * q.ld + q.x2p * k1;
#pragma unroll
          for (int r = 0; r < R; ++r) v[it][r] = d[r];
          rdft<R, -1>(v[it]);
        }
      }
      step_sync(tid);
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int i = tid + it * THR;
        if (IT * THR == Q::rows * Q::x1 || i < tot) {
          const int row = fdiv(i, q.dx1), k1 = i - row * q.x1;
          C *d = P + row * q.ld + k1;
#pragma unroll
          for (int r = 0; r < R; ++r) d[r * q.x1] = v[it][r];
        }
      }
    } else {
#pragma unroll 1
      for (int i = tid; i < tot; i += THR) {
        const int row = fdiv(i, q.dx1), k1 = i - row * q.x1;
        C *d = P + row * q.ld + q.x2p * k1;
        C v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = d[r];
        rdft<R, -1>(v);
#pragma unroll
        for (int r = 0; r < R; ++r) d[r] = v[r];
      }
    }
  });
  step_sync(tid);
  // y, first step
  step_ye(q, [&](auto RC) {
    constexpr int R = CV(RC);
    const int tot = q.nxk * q.yo;
#pragma unroll 1
    for (int i = tid; i < tot; i += THR) {
      const int t = fdiv(i, q.dnxk), k = i - t * q.nxk;
      C *pa = P + t * q.ld + colpos(q, k);
      const int rs = q.yo * q.ld;  // rows yo*r + t
      C a[R];
      if constexpr (MODE == PL_REAL) {
        if constexpr (R % 2 == 0) {
          C *pb = P + t * q.ld + colb(q, k);
          const C *pz = (k == 0 || 2 * k == q.nx) ? pa : pb;  // Z_(n-k)
#pragma unroll
          for (int r = 0; r < R / 2; ++r) {
            const C za = pa[r * rs], zb = pz[r * rs];
            a[r].x = za.x + zb.x;
            a[r].y = za.y - zb.y;
            a[r + R / 2].x = za.y + zb.y;  // -i (za - conj zb)
            a[r + R / 2].y = zb.x - za.x;
          }
          rdft<R, -1>(a);
          twiddle_c<R, -1>(a, tw, t);
#pragma unroll
          for (int r = 0; r < R / 2; ++r) {
            pa[r * rs] = a[r];
            pb[r * rs] = a[r + R / 2];
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = pa[r * rs];
        rdft<R, -1>(a);
        twiddle_c<R, -1>(a, tw, t);
#pragma unroll
        for (int r = 0; r < R; ++r) pa[r * rs] = a[r];
      }
    }
  });
  step_sync(tid);
  // y, second step: out to the spectrum
  C *out = spec + (long long)job * g.H + (long long)z * q.ny * q.nxk;
  step_yo(q, [&](auto RC) {
    constexpr int R = CV(RC);
    const int tot = q.nxk * q.ye;
#pragma unroll 1
    for (int i = tid; i < tot; i += THR) {
      const int k1 = fdiv(i, q.dnxk), k = i - k1 * q.nxk;
      const bool up = MODE == PL_REAL && 2 * k1 >= q.ye;
      const C *s = P + q.yo * (up ? k1 - q.ye / 2 : k1) * q.ld + (up ? colb(q, k) : colpos(q, k));
      C v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = s[r * q.ld];
      rdft<R, -1>(v);
      C *o = out + k1 * q.nxk + k;
#pragma unroll
      for (int r = 0; r < R; ++r) o[r * q.ye * q.nxk] = v[r];
    }
  });
}

// ---------------------------------------------------------------------------
// z lines: forward * k-space multiplier * inverse.  Lines are numbered along
// (kx, ky), consecutive ones are consecutive addresses.  grid.x: spectra,
// grid.y: line blocks.  sc: 1/2 when the plane pass left a factor 2.
// ---------------------------------------------------------------------------
template <typename T, typename Q>
__global__ void __launch_bounds__(kZThreads, (z_blocks<T, Q>()))
    k_zlines(GeoDev g, Prog p, FieldsDev f, Q q, const __grid_constant__ TwTab<typename Cx<T>::t, Q> tw, typename Cx<T>::t *spec, double sc) {
  typedef typename Cx<T>::t C;
  extern __shared__ __align__(16) unsigned char smraw[];
  C *P = (C *)smraw;
  const int tx = q.tx, sh = 31 - __clz(tx);  // tx is a power of two
  const int nlines = q.nxk * q.ny;
  const int l0 = blockIdx.y * tx, job = blockIdx.x;
  const int jj = job % p.J;
  const int kind = p.mul[p.jh[jj]][p.jf[jj]];
  C *base = spec + (long long)job * g.H + l0;
  const int nl = min(tx, nlines - l0);
  grid_wait();
  step_z1(q, [&](auto RC) {
    constexpr int R = CV(RC);
#pragma unroll 1
    for (int i = threadIdx.x; i < q.z2 << sh; i += kZThreads) {
      const int t = i >> sh, l = i & (tx - 1);
      if (l >= nl) continue;
      const C *s = base + (long long)t * nlines + l;
      const long long st = (long long)q.z2 * nlines;
      C v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = s[r * st];
      rdft<R, -1>(v);
      twiddle_c<R, -1>(v, tw, t);
      C *d = P + i;
#pragma unroll
      for (int r = 0; r < R; ++r) d[(r * q.z2) << sh] = v[r];
    }
  });
  __syncthreads();
  step_z2(q, [&](auto RC) {
    constexpr int R = CV(RC);
    const double *tab = kind == MUL_DIP ? f.vdd : kind == MUL_PRE ? f.ptab : nullptr;
    const double tsc = kind == MUL_DIP ? f.inv_size * sc : sc;
#pragma unroll 1
    for (int i = threadIdx.x; i < q.z1 << sh; i += kZThreads) {
      const int k1 = i >> sh, l = i & (tx - 1);
      if (l >= nl) continue;
      C *d = P + ((k1 * q.z2) << sh) + l;
      C v[R];
      double m[R];
      if (tab) {
        const double *tb = tab + (long long)k1 * nlines + l0 + l;
#pragma unroll
        for (int r = 0; r < R; ++r) m[r] = __ldg(tb + (long long)r * q.z1 * nlines) * tsc;
      } else {
        // k^2 = kx2[0][ix] + kx2[1][iy] + kx2[2][iz] summed in that order
        const int iy = fdiv(l0 + l, q.dnxk), ix = l0 + l - iy * q.nxk;
        const double kxy = __ldg(g.kx2[0] + ix) + __ldg(g.kx2[1] + iy);
#pragma unroll
        for (int r = 0; r < R; ++r) m[r] = kmult_k2(f, kind, kxy + __ldg(g.kx2[2] + k1 + r * q.z1)) * sc;
      }
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = d[r << sh];
      rdft<R, -1>(v);
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = cscale(v[r], (T)m[r]);
      rdft<R, +1>(v);
      twiddle_c<R, +1>(v, tw, k1);
#pragma unroll
      for (int r = 0; r < R; ++r) d[r << sh] = v[r];
    }
  });
  __syncthreads();
  step_z1(q, [&](auto RC) {
    constexpr int R = CV(RC);
#pragma unroll 1
    for (int i = threadIdx.x; i < q.z2 << sh; i += kZThreads) {
      const int t = i >> sh, l = i & (tx - 1);
      if (l >= nl) continue;
      C v[R];
      const C *d = P + i;
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = d[(r * q.z2) << sh];
      rdft<R, +1>(v);
      C *s = base + (long long)t * nlines + l;
      const long long st = (long long)q.z2 * nlines;
#pragma unroll
      for (int r = 0; r < R; ++r) s[r * st] = v[r];
    }
  });
}

// ---------------------------------------------------------------------------
// y and x inverse of one plane and the epilogue.  grid.x: column * nhs +
// half - h0 (the nhs halves from h0), grid.y: planes; field fi of each half.
// K and M add to the local term that k_plane_fwd left in y, so the epilogue
// has one operand to wait for, not three.  A half with two fields (M with
// dipolar exchange) takes two launches, the second field's first: y <- ltM x +
// 2 g w o1, then + o0.
// ---------------------------------------------------------------------------
template <typename T, int MODE, typename Q, bool PF>
__global__ void __launch_bounds__((plane_threads<T, Q>()), (plane_blocks<T, Q>()))
    k_plane_inv(GeoDev g, Prog p, FieldsDev f, Q q, const __grid_constant__ TwTab<typename Cx<T>::t, Q> tw,
                const typename Cx<T>::t *spec, void *yout, long long ldy, int h0, int nhs, int fi, int ahead) {
  typedef typename Cx<T>::t C;
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int THR = plane_threads<T, Q>();
  C *P = (C *)smraw;
  int tid = threadIdx.x;
  const int z = blockIdx.y;
  const int col = blockIdx.x / nhs;
  const int hf = h0 + (blockIdx.x - col * nhs);
  const int post = p.post[hf];
  const long long plane = (long long)z * q.nx * q.ny;
  const C *rx = roots_of<C>(g.ax[0]);
  const C *in = spec + ((long long)col * p.J + p.j0[hf] + fi) * g.H + (long long)z * q.ny * q.nxk;
  grid_wait();
  // y, first step: from the spectrum.  Slot ye*k1 + t of a column lies in
  // row ye*k1 + t (PL_REAL: ye/2*k1 + t % (ye/2), of colb(k) for the upper t)
  step_yo(q, [&](auto RC) {
    constexpr int R = CV(RC);
    const int tot = q.nxk * q.ye;
#pragma unroll 1
    for (int i = tid; i < tot; i += THR) {
      const int t = fdiv(i, q.dnxk), k = i - t * q.nxk;
      C v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = in[(q.ye * r + t) * q.nxk + k];
      rdft<R, +1>(v);
      twiddle_c<R, +1>(v, tw, t);
      const bool up = MODE == PL_REAL && 2 * t >= q.ye;
      C *d = P + (up ? t - q.ye / 2 : t) * q.ld + (up ? colb(q, k) : colpos(q, k));
      const int rs = (MODE == PL_REAL ? q.ye / 2 : q.ye) * q.ld;
#pragma unroll
      for (int r = 0; r < R; ++r) d[r * rs] = v[r];
    }
  });
  if (PF && ahead > 0) {
    const unsigned nx = blockIdx.y * gridDim.x + blockIdx.x + ahead, zn = nx / gridDim.x;
    if (zn < gridDim.y) {
      const int bx = nx - zn * gridDim.x, cn = bx / nhs, hn = h0 + (bx - cn * nhs);
      prefetch_l2<THR>(spec + ((long long)cn * p.J + p.j0[hn] + fi) * g.H + (long long)zn * q.ny * q.nxk,
                       (int)sizeof(C) * q.ny * q.nxk);
    }
  }
  if (PF && (post == POST_K || post == POST_M)) {
    constexpr int es = MODE == PL_CPLX ? (int)sizeof(C) : (int)sizeof(T);
    prefetch_l2<THR>((const char *)yout + (col * ldy + hf * g.S + plane) * es, es * q.nx * q.ny);
  }
  step_sync(tid);
  // y, second step: output r of item k1 is y = k1 + yo*r
  step_ye(q, [&](auto RC) {
    constexpr int R = CV(RC);
    const int tot = q.nxk * q.yo;
#pragma unroll 1
    for (int i = tid; i < tot; i += THR) {
      const int k1 = fdiv(i, q.dnxk), k = i - k1 * q.nxk;
      const bool real_col = MODE != PL_CPLX && (k == 0 || 2 * k == q.nx);
      C a[R];
      if constexpr (MODE == PL_REAL) {
        if constexpr (R % 2 == 0) {
          C *pa = P + R / 2 * k1 * q.ld + colpos(q, k), *pb = P + R / 2 * k1 * q.ld + colb(q, k);
#pragma unroll
          for (int r = 0; r < R / 2; ++r) {
            a[r] = pa[r * q.ld];
            a[r + R / 2] = pb[r * q.ld];
          }
          rdft<R, +1>(a);
          if (real_col) {
            // a real row's DC and Nyquist terms are real (as in a c2r transform)
#pragma unroll
            for (int r = 0; r < R; ++r) a[r].y = (T)0;
          }
#pragma unroll
          for (int r = 0; r < R / 2; ++r) {
            const C u = a[r], w = a[r + R / 2];
            C za, zb;  // u + i w and conj(u - i w)
            za.x = u.x - w.y;
            za.y = u.y + w.x;
            zb.x = u.x + w.y;
            zb.y = w.x - u.y;
            pa[r * q.ld] = za;
            if (!real_col) pb[r * q.ld] = zb;
          }
        }
      } else {
        C *pa = P + R * k1 * q.ld + colpos(q, k);
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = pa[r * q.ld];
        rdft<R, +1>(a);
        if (real_col) {
#pragma unroll
          for (int r = 0; r < R; ++r) a[r].y = (T)0;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) pa[r * q.ld] = a[r];
        if (MODE == PL_WHOLE && !real_col) {
          C *pb = P + R * k1 * q.ld + colpos(q, q.nx - k);
#pragma unroll
          for (int r = 0; r < R; ++r) pb[r * q.ld] = cconj(a[r]);
        }
      }
    }
  });
  step_sync(tid);
  // x, first step
  step_x2(q, [&](auto RC) {
    constexpr int R = CV(RC);
    const int tot = q.rows * q.x1;
    if constexpr (Q::CT) {
      // from natural column order, through registers
      constexpr int IT = (Q::rows * Q::x1 + THR - 1) / THR;
      C v[IT][R];
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int i = tid + it * THR;
        if (IT * THR == Q::rows * Q::x1 || i < tot) {
          const int row = fdiv(i, q.dx1), k1 = i - row * q.x1;
          const C *d = P + row * q.ld + k1;
#pragma unroll
          for (int r = 0; r < R; ++r) v[it][r] = d[r * q.x1];
          rdft<R, +1>(v[it]);
          twiddle<R, +1>(v[it], rx, k1);
        }
      }
      step_sync(tid);
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int i = tid + it * THR;
        if (IT * THR == Q::rows * Q::x1 || i < tot) {
          const int row = fdiv(i, q.dx1), k1 = i - row * q.x1;
          C *d = P + row * q.ld + q.x2p * k1;
#pragma unroll
          for (int r = 0; r < R; ++r) d[r] = v[it][r];
        }
      }
    } else {
#pragma unroll 1
      for (int i = tid; i < tot; i += THR) {
        const int row = fdiv(i, q.dx1), k1 = i - row * q.x1;
        C *d = P + row * q.ld + q.x2p * k1;
        C v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = d[r];
        rdft<R, +1>(v);
        twiddle<R, +1>(v, rx, k1);
#pragma unroll
        for (int r = 0; r < R; ++r) d[r] = v[r];
      }
    }
  });
  step_sync(tid);
  // x, second step, and the epilogue
  step_x1(q, [&](auto RC) {
    constexpr int R = CV(RC);
    const int tot = q.rows * q.x2;
    const T gg = (T)f.g_ddi;
    const bool add = post == POST_K || post == POST_M;
    const bool needw = fi > 0 || post == POST_DIPCONV;
#pragma unroll 1
    for (int i = tid; i < tot; i += THR) {
      const int row = fdiv(i, q.dx2), t = i - row * q.x2;
      const C *s = P + row * q.ld + t;
      C v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = s[r * q.x2p];
      rdft<R, +1>(v);
      const int yr = MODE == PL_REAL ? q.ye / 2 : q.ye;
      const int k1 = fdiv(row, q.dyr);
      const int o = (k1 + q.yo * (row - k1 * yr)) * q.nx + t;  // row element of v[0]; v[r] at o + r*x2
      if constexpr (MODE == PL_CPLX) {
        C *ys = (C *)yout + col * ldy + hf * g.S + plane + o;
        const C *cw = (const C *)f.w + plane + o;
        if (add) {
          if (needw) {
            C w[R];
#pragma unroll
            for (int r = 0; r < R; ++r) w[r] = __ldg(cw + r * q.x2);
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = cscale(cmul(cscale(w[r], gg), v[r]), (T)2);
          }
          C yv[R];
#pragma unroll
          for (int r = 0; r < R; ++r) yv[r] = ys[r * q.x2];
#pragma unroll
          for (int r = 0; r < R; ++r) ys[r * q.x2] = cadd(yv[r], v[r]);
        } else {
          const T *cl = (const T *)post_coef(f, post);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const T c = cl ? __ldg(cl + plane + o + r * q.x2) : (T)0;
            const C w = needw ? __ldg(cw + r * q.x2) : czero<C>();
            ys[r * q.x2] = epi_cplx<T, C>(post, 1, v[r], v[r], czero<C>(), c, w, gg);
          }
        }
      } else {
        // PL_REAL: row y in the real parts, row y + ny/2 in the imaginary ones
        const int hs = q.rows * q.nx;
        T *ys = (T *)yout + col * ldy + hf * g.S + plane + o;
        const T *cw = (const T *)f.w + plane + o;
        const T *cl = (const T *)post_coef(f, post) + plane + o;
#pragma unroll
        for (int u = 0; u < (MODE == PL_REAL ? 2 : 1); ++u) {
          T c[R], o1[R];
#pragma unroll
          for (int r = 0; r < R; ++r) o1[r] = u ? v[r].y : v[r].x;
          if (add) {
            if (needw) {
#pragma unroll
              for (int r = 0; r < R; ++r) c[r] = __ldg(cw + u * hs + r * q.x2);
#pragma unroll
              for (int r = 0; r < R; ++r) o1[r] = (T)2 * ((gg * c[r]) * o1[r]);
            }
#pragma unroll
            for (int r = 0; r < R; ++r) c[r] = ys[u * hs + r * q.x2];
#pragma unroll
            for (int r = 0; r < R; ++r) ys[u * hs + r * q.x2] = c[r] + o1[r];
          } else {
            const bool coef = post == POST_TK || post == POST_TM;
#pragma unroll
            for (int r = 0; r < R; ++r)
              c[r] = coef ? __ldg(cl + u * hs + r * q.x2) : needw ? __ldg(cw + u * hs + r * q.x2) : (T)0;
#pragma unroll
            for (int r = 0; r < R; ++r)
              ys[u * hs + r * q.x2] = epi_real<T>(post, 1, o1[r], (T)0, (T)0, c[r], c[r], gg);
          }
        }
      }
    }
  });
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// geometry of context c, false when the kernels cannot run it
bool bdgd_plane_par(const bdgd_ctx *c, PlaneGeo *q);

template <typename C> static const C *host_roots(const bdgd_ctx *c, int d);
template <> const double2 *host_roots<double2>(const bdgd_ctx *c, int d) { return c->h_roots64[d]; }
template <> const float2 *host_roots<float2>(const bdgd_ctx *c, int d) { return c->h_roots32[d]; }

// Launch on the context's stream behind the kernel before it (see grid_wait).
template <typename K, typename... A>
static int launch_after(bdgd_ctx *c, K kern, dim3 grid, int threads, size_t sm, const A &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = c->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  bdgd_count_launch();
  BDGD_CK(cudaLaunchKernelEx(&cfg, kern, args...));
  return BDGD_OK;
}

// Applies whose blocks and spectra together exceed kL2Bytes (what the 126 MB L2
// keeps of data read and written once) prefetch into L2.  The inverse asks for
// the local term in y, its epilogue's operand, before its second step; where
// one plane fills an SM (128^3 FP64: 139 KB) nothing else hides the loads, so
// both plane kernels also ask for the plane of the block kAhead = 148 SMs
// later.  Without -> with: Lrep 48x64x96
// complex 667 -> 651 us; T 128^3 FP64, 64 columns 3659 -> 3552 (the inverse's
// lookahead alone gave nearly all of it); Lrep 64^3 FP64, 32 columns 333.8 ->
// 331.8; Lrep 128^3 FP32, 64 columns 2901 -> 2882.  Elsewhere they cost: y below kL2Bytes 106.6 -> 107.4
// (50x45x36, 16 columns), lookahead of both with two or more blocks an SM
// 106.6 -> 112 there and 325 -> 330 at 64^3.  PF is a template argument: as
// run-time branches they cost the small applies (50x45x36) 1.4%.
static const size_t kL2Bytes = (size_t)80 << 20, kSmemSM = 227 * 1024;
static const int kAhead = 148;

template <typename T, int MODE, bool PF, typename Q, typename Qz>
static int planes_launch_pf(bdgd_ctx *c, const Prog &p, const FieldsDev &fd, const Q &q, const Qz &qz, const void *x,
                         long long ldx, void *y, long long ldy, void *spec, int nc) {
  typedef typename Cx<T>::t C;
  const size_t sm = sizeof(C) * (size_t)q.rows * q.ld;
  const size_t smz = sizeof(C) * (size_t)q.tx * q.nz;
  int rc;
  if (sm > 48 * 1024) {
    if ((rc = bdgd_smem_attr(k_plane_fwd<T, MODE, Q, PF>, sm))) return rc;
    if ((rc = bdgd_smem_attr(k_plane_inv<T, MODE, Q, PF>, sm))) return rc;
  }
  if (smz > 48 * 1024 && (rc = bdgd_smem_attr(k_zlines<T, Qz>, smz))) return rc;
  TwTab<C, Q> ty;
  TwTab<C, Qz> tz;
  const C *hy = host_roots<C>(c, 1), *hz = host_roots<C>(c, 2);
  for (int i = 0; i < q.ny; ++i) ty.w[i] = hy[i];
  for (int i = 0; i < q.nz; ++i) tz.w[i] = hz[i];
  const unsigned nzb = (unsigned)((q.nxk * q.ny + q.tx - 1) / q.tx);
  const int thr = plane_threads<T, Q>();
  C *sp = (C *)spec;
  const int ahead = PF && 2 * (sm + 1024) > kSmemSM ? kAhead : 0;
  if ((rc = launch_after(c, k_plane_fwd<T, MODE, Q, PF>, dim3(nc * p.J, q.nz), thr, sm, c->geo, p, fd, q, ty, x, ldx, sp, y, ldy, ahead)))
    return rc;
  if ((rc = launch_after(c, k_zlines<T, Qz>, dim3(nc * p.J, nzb), kZThreads, smz, c->geo, p, fd, qz, tz, sp,
                         MODE == PL_REAL ? 0.5 : 1.0)))
    return rc;
  const C *csp = sp;
  for (int h = 0; h < p.nh; ++h)
    if (p.nf[h] > 1 && (rc = launch_after(c, k_plane_inv<T, MODE, Q, PF>, dim3(nc, q.nz), thr, sm, c->geo, p, fd, q, ty, csp, y,
                                          ldy, h, 1, 1, ahead)))
      return rc;
  return launch_after(c, k_plane_inv<T, MODE, Q, PF>, dim3(nc * p.nh, q.nz), thr, sm, c->geo, p, fd, q, ty, csp, y, ldy, 0,
                      p.nh, 0, ahead);
}

template <typename T, int MODE, typename Q, typename Qz>
static int planes_launch(bdgd_ctx *c, const Prog &p, const FieldsDev &fd, const Q &q, const Qz &qz, const void *x,
                         long long ldx, void *y, long long ldy, void *spec, int nc) {
  typedef typename Cx<T>::t C;
  const size_t bytes = (size_t)nc * (2 * p.nh * c->geo.S * (MODE == PL_CPLX ? sizeof(C) : sizeof(T)) +
                                     p.J * c->geo.H * sizeof(C));
  if (bytes > kL2Bytes) return planes_launch_pf<T, MODE, true>(c, p, fd, q, qz, x, ldx, y, ldy, spec, nc);
  return planes_launch_pf<T, MODE, false>(c, p, fd, q, qz, x, ldx, y, ldy, spec, nc);
}

template <typename T, int MODE>
static int planes_launch_rt(bdgd_ctx *c, const Prog &p, const FieldsDev &fd, const PlaneGeo &g, const void *x,
                            long long ldx, void *y, long long ldy, void *spec, int nc) {
  const PlanePar<8> q8 = {g};
  const PlanePar<16> q16 = {g};
  const bool xy8 = g.x1 <= 8 && g.x2 <= 8 && g.ye <= 8 && g.yo <= 8, z8 = g.z1 <= 8 && g.z2 <= 8;
  if (xy8) {
    if (z8) return planes_launch<T, MODE>(c, p, fd, q8, q8, x, ldx, y, ldy, spec, nc);
    return planes_launch<T, MODE>(c, p, fd, q8, q16, x, ldx, y, ldy, spec, nc);
  }
  if (z8) return planes_launch<T, MODE>(c, p, fd, q16, q8, x, ldx, y, ldy, spec, nc);
  return planes_launch<T, MODE>(c, p, fd, q16, q16, x, ldx, y, ldy, spec, nc);
}

template <typename T>
static int planes_apply(bdgd_ctx *c, const Prog &p, const FieldsDev &fd, const void *x, long long ldx, void *y,
                        long long ldy, void *spec, int nc) {
  PlaneGeo q;
  if (!bdgd_plane_par(c, &q)) return BDGD_ERR_UNSUPPORTED;
  if (q.mode == PL_CPLX) return planes_launch_rt<T, PL_CPLX>(c, p, fd, q, x, ldx, y, ldy, spec, nc);
  if (q.mode == PL_WHOLE) return planes_launch_rt<T, PL_WHOLE>(c, p, fd, q, x, ldx, y, ldy, spec, nc);
  // Compiled-in against run-time sizes, FP64 (FP32), us: Lrep of 16 columns 16^3
  // 16 : 22 (12 : 19), 32^3 32 : 47 (24 : 35); 24 columns 48^3 115 : 151 (76 : 97);
  // 32 columns 64^3 315 : 385 (207 : 267), 96^3 1215 : 1338 (686 : 953); 64
  // columns 128^3 5562 : 6801 (2785 : 3707).  One column: 1.05 to 1.6 times.
  if (q.nx == q.ny && q.ny == q.nz) {
    switch (q.nx) {
#define PLANE_CUBE(N) \
  case N: return planes_launch<T, PL_REAL>(c, p, fd, PlaneCT<N>(), PlaneCT<N>(), x, ldx, y, ldy, spec, nc)
      PLANE_CUBE(16);
      PLANE_CUBE(32);
      PLANE_CUBE(48);
      PLANE_CUBE(64);
      PLANE_CUBE(96);
      PLANE_CUBE(128);
#undef PLANE_CUBE
      default: break;
    }
  }
  return planes_launch_rt<T, PL_REAL>(c, p, fd, q, x, ldx, y, ldy, spec, nc);
}
