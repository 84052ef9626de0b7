// harmonic.cuh -- the FP64 far field in solid harmonics: what COMP_TCOEFF and
// COMPP_TREE_PB (treecode3d_pb.f:439-486, 684-855) evaluate, term for term the
// same truncated Taylor sum, in another basis.
//
// For a cluster centred at 0, source charges q = A x2 (a monopole at y) and
// d = A x1 n (a dipole there) and a target at x, the reference's sums are
//   P_f = sum_s q  sum_{|k| <= p} y^k/k! D^k f(x - y)|_{y=0},
//   G_f = sum_s d.grad_y of the same sum to |k| <= p + 1,
// for f = 1/r and f = e^{-kappa r}/r (D in y), combined to
//   out1 = (P - G)[1/r] - (P - eps G)[e^{-kappa r}/r],
//   out2 = n0.grad_x { (P - G)[1/r] - (P / eps - G)[e^{-kappa r}/r] }.
// The degree-n part of the sum is (-1)^n/n! (y.D)^n f, and (y.D)^n splits into
// |y|^{2j} |D|^{2j} times harmonic parts of degree l = n - 2j.  Away from the
// origin |D|^2 f = kappa^2 f (0 for 1/r), and a harmonic polynomial H of degree l
// acts on a radial f as H(D) f = f_l(r) H(x), f_l = ((1/r) d/dr)^l f.  So
//   out1 = sum_l c_l(r) U_l(x) + y_l(r) V_l(x),
//   out2 = n0.grad [ sum_l c_l U_l ] + (1/eps) n0.grad [ sum_l y_l V_l ]
// with l <= p + 1, c_l and y_l the radial functions of 1/r and e^{-kappa r}/r,
// and per cluster one harmonic polynomial U_l and V_l of 2l + 1 coefficients:
//   U_l = (-1)^l w_lm/(2l-1)!! sum_s [ q (l <= p) - d.grad_y ] S_lm(y),
//   V_l = (-1)^l w_lm sum_s [ -q b_l^p(|y|^2) + eps d.grad_y b_l^{p+1}(|y|^2) ] S_lm(y),
//   b_l^N(t) = sum_{j <= (N-l)/2} (2l+1)/(2^j j! (2l+2j+1)!!) (kappa^2 t)^j.
// grad(f_l H_l) = f_{l+1} H_l x + f_l grad H_l, and grad H_l, of degree l - 1, is
// kept as three more coefficient sets.
//
// Basis: S_lm = Z_lm(z, r^2) (x + iy)^m, real and imaginary part, with
// Z_mm = 1 and Z_l = z Z_{l-1} - ((l-1)^2 - m^2)/((2l-1)(2l-3)) r^2 Z_{l-2};
// w_lm = (2 - [m=0]) (2l-1)!!^2/((l-m)! (l+m)!).  Element index l^2 for m = 0,
// l^2 + 2m - 1 (real) and l^2 + 2m (imaginary).
//
// Work per (target, cluster): 2 (p+2)^2 + 6 (p+1)^2 multiply-adds of the
// contraction and a short recurrence, about 310 FP64 instructions at p = 3 and
// 870 at p = 6; the Cartesian form took about 1,640 and 5,300 (two passes of a
// 3-index recurrence and 16 moment sets each).  Bound by the FP64 pipe.  Measured
// per operator apply: order 3, 3.29 M interactions, 0.375 -> 0.097 ms; order 6,
// 10.4 M, 4.59 -> 0.79 ms.
#pragma once

#include "fast_math.cuh"

namespace tabi {

// doubles per cluster: per element of degree <= p U, V and the gradients of
// U_{l+1} and V_{l+1}; per element of degree p + 1 U and V
__host__ __device__ constexpr int harm_size(int p) {
  return 8 * (p + 1) * (p + 1) + 2 * (2 * p + 3);
}
// raw sums per source chunk: U and V of every element of degree <= p + 1
__host__ __device__ constexpr int harm_raw(int p) { return 2 * (p + 2) * (p + 2); }

__host__ __device__ constexpr double harm_b(int l, int m) {
  return (double)((l - 1) * (l - 1) - m * m) / (double)((2 * l - 1) * (2 * l - 3));
}
// b_l^p and b_l^{p+1} as polynomials in |y|^2 (kappa^{2j} included), a kernel
// argument: [l][j], 0 past the truncation
template <int P>
struct HarmBeta {
  double p[P + 2][(P + 1) / 2 + 1], q[P + 2][(P + 1) / 2 + 1];
};
template <int P>
HarmBeta<P> harm_beta(double kappa) {
  HarmBeta<P> t{};
  for (int l = 0; l <= P + 1; ++l) {
    double v = 2 * l + 1;  // (2l+1) kappa^{2j} / (2^j j! (2l+2j+1)!!)
    for (int k = 2 * l + 1; k > 1; k -= 2) v /= k;
    for (int j = 0; l + 2 * j <= P + 1; ++j) {
      if (j > 0) v *= kappa * kappa / (2.0 * j * (2 * l + 2 * j + 1));
      t.q[l][j] = v;
      if (l + 2 * j <= P) t.p[l][j] = v;
    }
  }
  return t;
}

// One source's contributions to the raw sums: out[2 e] for U, out[2 e + 1] for
// V of element e (without the constants of l and m).
template <int P>
__device__ __forceinline__ void harm_source(double x, double y, double z, double q, double d0,
                                            double d1, double d2, const HarmBeta<P>& beta,
                                            double eps, double* __restrict__ out) {
  constexpr int L = P + 1;
  const double r2 = fma(x, x, fma(y, y, z * z));
  const double dy = fma(d0, x, fma(d1, y, d2 * z));
  const double dr2 = 2.0 * dy;
  // V = va_l S + vb_l (d.grad S)
  double va[L + 1], vb[L + 1];
#pragma unroll
  for (int l = 0; l <= L; ++l) {
    double bp = 0.0, bq = 0.0, db = 0.0;  // b^p, b^{p+1} and its derivative
#pragma unroll
    for (int j = (L - l) / 2; j >= 0; --j) {
      bp = fma(bp, r2, beta.p[l][j]);
      bq = fma(bq, r2, beta.q[l][j]);
      if (j > 0) db = fma(db, r2, j * beta.q[l][j]);
    }
    va[l] = fma(-q, bp, eps * db * dr2);
    vb[l] = eps * bq;
  }
  double a = 1.0, b = 0.0, da = 0.0, db = 0.0;  // (x + iy)^m and d.grad of it
#pragma unroll
  for (int m = 0; m <= L; ++m) {
    double z0 = 0.0, dz0 = 0.0, z1 = 1.0, dz1 = 0.0;
#pragma unroll
    for (int l = m; l <= L; ++l) {
      if (l > m) {
        const double zn = l == m + 1 ? z : fma(z, z1, -(harm_b(l, m) * r2) * z0);
        const double dzn = l == m + 1 ? d2
                                      : fma(d2, z1, fma(z, dz1, -harm_b(l, m) *
                                                                    fma(dr2, z0, r2 * dz0)));
        z0 = z1;
        dz0 = dz1;
        z1 = zn;
        dz1 = dzn;
      }
      const double ql = l <= P ? q : 0.0;
      double* o = out + 2 * (l * l + (m == 0 ? 0 : 2 * m - 1));
      double s = z1 * a, ds = fma(dz1, a, z1 * da);
      o[0] = fma(ql, s, -ds);
      o[1] = fma(va[l], s, vb[l] * ds);
      if (m > 0) {
        s = z1 * b;
        ds = fma(dz1, b, z1 * db);
        o[2] = fma(ql, s, -ds);
        o[3] = fma(va[l], s, vb[l] * ds);
      }
    }
    const double an = fma(x, a, -y * b), bn = fma(x, b, y * a);
    const double dan = fma(d0, a, fma(x, da, -fma(d1, b, y * db)));
    const double dbn = fma(d0, b, fma(x, db, fma(d1, a, y * da)));
    a = an;
    b = bn;
    da = dan;
    db = dbn;
  }
}

// a_lm = (2l-1)!!/((l-m)! (l+m)!): R_lm = a_lm S_lm is the normalisation in
// which derivatives have unit coefficients
__device__ __forceinline__ double harm_a(int l, int m) {
  double v = 1.0, w = 1.0;
  for (int k = 2 * l - 1; k > 1; k -= 2) v *= k;
  for (int k = 2; k <= l - m; ++k) w *= k;
  for (int k = 2; k <= l + m; ++k) w *= k;
  return v / w;
}

// (-1)^l w_lm/(2l-1)!! / a_lm (set 0, U) and (-1)^l w_lm / a_lm (set 1, V): raw
// sums to coefficients of the R_lm
__device__ __forceinline__ double harm_scale(int l, int m, int set) {
  double v = m == 0 ? 1.0 : 2.0;
  if (set == 1)
    for (int k = 2 * l - 1; k > 1; k -= 2) v *= k;
  return (l & 1) ? -v : v;
}

// Coefficient of Re or Im R_l^k in d/dx_dim of H_{l+1}, whose coefficients are
// c[2 * element]: d/dz R_l^m = R_{l-1}^m, (d/dx + i d/dy) R_l^m = -R_{l-1}^{m+1},
// (d/dx - i d/dy) R_l^m = R_{l-1}^{m-1}.
__device__ __forceinline__ double harm_grad(const double* c, int l, int k, bool im, int dim) {
  const int h = l + 1, base = h * h;
  // coefficient of Re / Im R_h^m, 0 outside 0..h
  auto re = [&](int m) {
    return m < 0 || m > h ? 0.0 : c[2 * (base + (m == 0 ? 0 : 2 * m - 1))];
  };
  auto imc = [&](int m) { return m < 1 || m > h ? 0.0 : c[2 * (base + 2 * m)]; };
  if (dim == 2) return im ? imc(k) : re(k);
  const double low = k == 1 ? 2.0 * re(0) : re(k - 1);  // m = 0 counts for m = +-1
  if (dim == 0) return 0.5 * (im ? imc(k + 1) - imc(k - 1) : re(k + 1) - low);
  return 0.5 * (im ? -(low + re(k + 1)) : imc(k - 1) + imc(k + 1));
}

// out1 and out2 (before 1/(4 pi)) of NT targets at (x, y, z) from the cluster's
// centre, unit normals (n0, n1, n2); M: the cluster's harm_size(P) coefficients,
// 16-byte aligned, read in order, once for the NT targets.
template <int P, int NT>
__device__ __forceinline__ void harm_eval(const double (&x)[NT], const double (&y)[NT],
                                          const double (&z)[NT], const double (&n0)[NT],
                                          const double (&n1)[NT], const double (&n2)[NT],
                                          double kappa, double inv_eps,
                                          const double* __restrict__ M, double (&out1)[NT],
                                          double (&out2)[NT]) {
  constexpr int L = P + 1;
  const double k2 = kappa * kappa;
  double r2[NT], ri2[NT], xn[NT], c[NT], y0[NT], y1[NT], o2y[NT];  // c_l, y_l, y_{l+1}
  double za[NT][L + 1], zb[NT][L + 1], a[NT][L + 1], b[NT][L + 1];  // Z_{l-1}, Z_{l-2}, (x + iy)^m
#pragma unroll
  for (int k = 0; k < NT; ++k) {
    r2[k] = fma(x[k], x[k], fma(y[k], y[k], z[k] * z[k]));
    const double ri = fast_rsqrt(r2[k]);
    ri2[k] = ri * ri;
    const double kr = kappa * (r2[k] * ri);
    const double ex = exp(-kr);
    xn[k] = fma(n0[k], x[k], fma(n1[k], y[k], n2[k] * z[k]));
    c[k] = ri;
    y0[k] = ex * ri;
    y1[k] = -fma(kr, ex, ex) * ri * ri2[k];
    out1[k] = out2[k] = o2y[k] = 0.0;
    a[k][0] = 1.0;
    b[k][0] = 0.0;
  }
#pragma unroll
  for (int l = 0; l <= L; ++l) {
    // sums over the degree's elements: U, V, grad U_{l+1}, grad V_{l+1}
    double s[NT][8] = {};
    const double* Ml = l <= P ? M + 8 * l * l : M + 8 * (P + 1) * (P + 1);
#pragma unroll
    for (int m = 0; m <= l; ++m) {
      double zl[NT];
#pragma unroll
      for (int k = 0; k < NT; ++k) {
        if (m == l && l > 0) {
          a[k][l] = l == 1 ? x[k] : fma(x[k], a[k][l - 1], -y[k] * b[k][l - 1]);
          b[k][l] = l == 1 ? y[k] : fma(x[k], b[k][l - 1], y[k] * a[k][l - 1]);
        }
        zl[k] = m == l       ? 1.0
                : m == l - 1 ? z[k]
                             : fma(z[k], za[k][m], -(harm_b(l, m) * r2[k]) * zb[k][m]);
        if (m < l) zb[k][m] = za[k][m];
        za[k][m] = zl[k];
      }
#pragma unroll
      for (int im = 0; im < (m > 0 ? 2 : 1); ++im) {
        const int e = m == 0 ? 0 : 2 * m - 1 + im;
        const double2* v = reinterpret_cast<const double2*>(Ml + (l <= P ? 8 : 2) * e);
#pragma unroll
        for (int q = 0; q < (l <= P ? 4 : 1); ++q) {
          const double2 w = v[q];
#pragma unroll
          for (int k = 0; k < NT; ++k) {
            const double t = im == 0 ? a[k][m] : b[k][m];
            const double f = m == 0 ? zl[k] : m == l ? t : zl[k] * t;
            s[k][2 * q] = fma(f, w.x, s[k][2 * q]);
            s[k][2 * q + 1] = fma(f, w.y, s[k][2 * q + 1]);
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < NT; ++k) {
      out1[k] = fma(c[k], s[k][0], fma(y0[k], s[k][1], out1[k]));
      c[k] *= -(double)(2 * l + 1) * ri2[k];
      double tu = xn[k] * s[k][0], tv = xn[k] * s[k][1];
      if (l <= P) {
        tu = fma(n0[k], s[k][2], fma(n1[k], s[k][3], fma(n2[k], s[k][4], tu)));
        tv = fma(n0[k], s[k][5], fma(n1[k], s[k][6], fma(n2[k], s[k][7], tv)));
      }
      out2[k] = fma(c[k], tu, out2[k]);
      o2y[k] = fma(y1[k], tv, o2y[k]);
      const double yn = fma(k2, y0[k], -(double)(2 * l + 3) * y1[k]) * ri2[k];
      y0[k] = y1[k];
      y1[k] = yn;
    }
  }
#pragma unroll
  for (int k = 0; k < NT; ++k) out2[k] = fma(inv_eps, o2y[k], out2[k]);
}

}  // namespace tabi
