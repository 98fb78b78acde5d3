// bdg_dft.cuh -- small DFTs in registers with compile-time twiddles, and the
// operator prologues and epilogues with hoisted coefficient loads, shared by
// the FFT pass kernels.  Internal to the library.
#pragma once

#include <type_traits>

#include "bdg_kern.cuh"

// ---------------------------------------------------------------------------
// compile-time trigonometry for the in-register DFT twiddles
// ---------------------------------------------------------------------------
// Taylor series on [0, pi/2) after an exact reduction of the angle 2*pi*j/n
// to a quadrant, in pairs of doubles (Dekker's and Knuth's error-free sums and
// products), so that every constant is the double nearest to its value.  In
// plain doubles they were up to 10 units of the last place off (n = 13), an
// error that every element of a transform shares: T on 50x50x36 was 4.57e-16 off
// (now 3.49e-16, the runtime-sized kernels with rounded tables 3.62e-16).
struct cx_dd {
  double h, l;
};
__host__ __device__ constexpr cx_dd cx_two_sum(double a, double b) {
  const double s = a + b, t = s - a;
  return {s, (a - (s - t)) + (b - t)};
}
__host__ __device__ constexpr cx_dd cx_two_prod(double a, double b) {
  const double ca = 134217729.0 * a, ah = ca - (ca - a), al = a - ah;
  const double cb = 134217729.0 * b, bh = cb - (cb - b), bl = b - bh;
  const double p = a * b;
  return {p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
__host__ __device__ constexpr cx_dd cx_add(cx_dd a, cx_dd b) {
  const cx_dd s = cx_two_sum(a.h, b.h);
  return cx_two_sum(s.h, s.l + (a.l + b.l));
}
__host__ __device__ constexpr cx_dd cx_mul(cx_dd a, cx_dd b) {
  const cx_dd p = cx_two_prod(a.h, b.h);
  return cx_two_sum(p.h, p.l + (a.h * b.l + a.l * b.h));
}
__host__ __device__ constexpr cx_dd cx_div(cx_dd a, double b) {
  const double q = a.h / b;
  const cx_dd p = cx_two_prod(q, b);
  return cx_two_sum(q, ((a.h - p.h) - p.l + a.l) / b);
}
// sin (odd = 1) or cos (odd = 0) of x
__host__ __device__ constexpr double cx_series(cx_dd x, int odd) {
  const cx_dd x2 = cx_mul(x, x), m = {-x2.h, -x2.l};
  cx_dd t = odd ? x : cx_dd{1.0, 0.0}, s = t;
  for (int i = 1; i < 22; ++i) {
    t = cx_div(cx_mul(t, m), (2.0 * i) * (2.0 * i + (odd ? 1.0 : -1.0)));
    s = cx_add(s, t);
  }
  return s.h;
}
__host__ __device__ constexpr int cx_quadrant(int j, int n) { return (4 * j) / n; }
__host__ __device__ constexpr cx_dd cx_rem(int j, int n) {
  const cx_dd half_pi = {1.5707963267948966, 6.123233995736766e-17};
  return cx_div(cx_mul(half_pi, {(double)(4 * j - cx_quadrant(j, n) * n), 0.0}), (double)n);
}
// cos(2 pi j / n), sin(2 pi j / n) for 0 <= j < n
__host__ __device__ constexpr double cx_cos(int j, int n) {
  const int q = cx_quadrant(j, n);
  const double v = cx_series(cx_rem(j, n), q & 1);
  return q == 1 || q == 2 ? -v : v;
}
__host__ __device__ constexpr double cx_sin(int j, int n) {
  const int q = cx_quadrant(j, n);
  const double v = cx_series(cx_rem(j, n), !(q & 1));
  return q >= 2 ? -v : v;
}

#define CV(I) decltype(I)::value

template <int B, int E, typename F>
__device__ __forceinline__ void sfor(F &&f) {
  if constexpr (B < E) {
    f(std::integral_constant<int, B>{});
    sfor<B + 1, E>(f);
  }
}

// a * w_R^M with w_R = exp(SGN * 2 pi i / R), M a compile-time constant
template <int M, int R, int SGN, typename C>
__device__ __forceinline__ C ctw(C a) {
  constexpr int m = ((M % R) + R) % R;
  if constexpr (m == 0) {
    return a;
  } else if constexpr (2 * m == R) {
    a.x = -a.x;
    a.y = -a.y;
    return a;
  } else if constexpr (4 * m == R) {
    return cmul_si(a, SGN);
  } else if constexpr (4 * m == 3 * R) {
    return cmul_si(a, -SGN);
  } else {
    typedef decltype(a.x) E;
    constexpr double c = cx_cos(m, R), s = SGN * cx_sin(m, R);
    C r;
    r.x = a.x * (E)c - a.y * (E)s;
    r.y = a.x * (E)s + a.y * (E)c;
    return r;
  }
}

template <int R>
__host__ __device__ constexpr int rdft_split() {
  return (R % 16 == 0) ? 4 : (R % 8 == 0) ? 8 : (R % 4 == 0) ? 4 : (R % 2 == 0) ? 2 : 3;
}

template <typename C>
__device__ __forceinline__ C czero() {
  C z;
  z.x = 0;
  z.y = 0;
  return z;
}

// Odd prime size: with t_j = v_j + v_(R-j) and s_j = v_j - v_(R-j),
// X_k = v_0 + sum_j cos(2 pi jk/R) t_j +- SGN i sum_j sin(2 pi jk/R) s_j gives
// X_k and X_(R-k) from one pair of real-coefficient sums.
template <int R, int SGN, typename C>
__device__ __forceinline__ void prime_dft(C *v) {
  typedef decltype(v[0].x) E;
  constexpr int Hf = (R - 1) / 2;
  C t[Hf], s[Hf];
  C x0 = v[0];
  sfor<0, Hf>([&](auto J) {
    constexpr int j = CV(J);
    t[j] = cadd(v[j + 1], v[R - 1 - j]);
    s[j] = csub(v[j + 1], v[R - 1 - j]);
    x0 = cadd(x0, t[j]);
  });
  sfor<1, Hf + 1>([&](auto K) {
    constexpr int k = CV(K);
    C m = v[0], n = czero<C>();
    sfor<0, Hf>([&](auto J) {
      constexpr int j = CV(J);
      constexpr double c = cx_cos((j + 1) * k % R, R), d = cx_sin((j + 1) * k % R, R);
      m.x += t[j].x * (E)c;
      m.y += t[j].y * (E)c;
      n.x += s[j].x * (E)d;
      n.y += s[j].y * (E)d;
    });
    const C in = cmul_si(n, SGN);
    // v[k] and v[R - k] are read only through t and s from here on
    v[k] = cadd(m, in);
    v[R - k] = csub(m, in);
  });
  v[0] = x0;
}

// In-register DFT of size R (natural order in and out), sign SGN.
template <int R, int SGN, typename C>
__device__ __forceinline__ void rdft(C *v) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    bfly2(v);
  } else if constexpr (R == 3) {
    bfly3(v, SGN);
  } else if constexpr (R == 4) {
    bfly4(v[0], v[1], v[2], v[3], SGN);
  } else if constexpr (R == 8) {
    bfly8(v, SGN);
  } else if constexpr (R == 5 || R == 7 || R == 11 || R == 13) {
    prime_dft<R, SGN>(v);
  } else {
    constexpr int R1 = rdft_split<R>(), R2 = R / R1;
    // n = R2*n1 + n2, k = k1 + R1*k2
    sfor<0, R2>([&](auto I2) {
      constexpr int n2 = CV(I2);
      C u[R1];
      sfor<0, R1>([&](auto I1) { u[CV(I1)] = v[R2 * CV(I1) + n2]; });
      rdft<R1, SGN>(u);
      sfor<0, R1>([&](auto K1) { v[R2 * CV(K1) + n2] = ctw<n2 * CV(K1), R, SGN>(u[CV(K1)]); });
    });
    C w[R];
    sfor<0, R1>([&](auto K1) {
      constexpr int k1 = CV(K1);
      C u[R2];
      sfor<0, R2>([&](auto I2) { u[CV(I2)] = v[R2 * k1 + CV(I2)]; });
      rdft<R2, SGN>(u);
      sfor<0, R2>([&](auto K2) { w[k1 + R1 * CV(K2)] = u[CV(K2)]; });
    });
    sfor<0, R>([&](auto I) { v[CV(I)] = w[CV(I)]; });
  }
}

// ---------------------------------------------------------------------------
// prologue / epilogue with the coefficient loads hoisted: the operator kind
// is uniform over a launch, so the array it reads is chosen once and every
// load of a row chunk is issued before the arithmetic (a per-element switch
// with the load inside would expose one memory latency per element).  The
// arithmetic is that of prologue() and epilogue() in bdg_kern.cuh.
// ---------------------------------------------------------------------------
// real-valued coefficient array of a prologue kind (pK, pM; the wavefunction
// for the real path), or null
__device__ __forceinline__ const void *pre_coef(const FieldsDev &f, int kind) {
  switch (kind) {
    case PRE_PK: return f.pK;
    case PRE_PM: return f.pM;
    case PRE_CONJWF:
    case PRE_DENS: return f.w;
    default: return nullptr;
  }
}
template <typename T>
__device__ __forceinline__ T pre_real(int kind, T x, T c) {
  switch (kind) {
    case PRE_PK:
    case PRE_PM:
    case PRE_CONJWF: return c * x;
    case PRE_DENS: {
      const T a = fabs(c);
      return a * a;
    }
    case PRE_XDENS: return x * x;
    default: return x;
  }
}
// complex path: c is the real coefficient (pK, pM), w the wavefunction value
template <typename T, typename C>
__device__ __forceinline__ C pre_cplx(int kind, C x, T c, C w) {
  switch (kind) {
    case PRE_PK:
    case PRE_PM: return cscale(x, c);
    case PRE_CONJWF: return cmul(cconj(w), x);
    case PRE_DENS: {
      const T a = hypot(w.x, w.y);
      return cmk<C>(a * a, 0.0);
    }
    case PRE_XDENS: return cmk<C>(x.x * x.x + x.y * x.y, 0.0);
    default: return x;
  }
}
// real-valued coefficient array of an epilogue kind (ltK, ltM, pK, pM), or null
__device__ __forceinline__ const void *post_coef(const FieldsDev &f, int post) {
  switch (post) {
    case POST_K: return f.ltK;
    case POST_M: return f.ltM;
    case POST_TK: return f.pK;
    case POST_TM: return f.pM;
    default: return nullptr;
  }
}
template <typename T>
__device__ __forceinline__ T epi_real(int post, int nf, T y0, T y1, T x, T c, T w, T g) {
  switch (post) {
    case POST_K: return y0 + c * x;
    case POST_M:
      if (nf > 1) {
        const T dc = (g * w) * y1;
        return y0 + (c * x + (T)2 * dc);
      }
      return y0 + c * x;
    case POST_TK:
    case POST_TM: return y0 * c;
    case POST_DIPCONV: return (g * w) * y0;
    case POST_PHI: return g * y0;
    default: return y0;
  }
}
template <typename T, typename C>
__device__ __forceinline__ C epi_cplx(int post, int nf, C o0, C o1, C x, T c, C w, T g) {
  switch (post) {
    case POST_K: return cadd(o0, cscale(x, c));
    case POST_M:
      if (nf > 1) {
        const C dc = cmul(cscale(w, g), o1);
        return cadd(o0, cadd(cscale(x, c), cscale(dc, (T)2)));
      }
      return cadd(o0, cscale(x, c));
    case POST_TK:
    case POST_TM: return cscale(o0, c);
    case POST_DIPCONV: return cmul(cscale(w, g), o0);
    case POST_PHI: return cmk<C>(g * o0.x, 0.0);
    default: return o0;
  }
}
