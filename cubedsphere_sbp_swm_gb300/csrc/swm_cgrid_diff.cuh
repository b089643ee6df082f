// swm_cgrid_diff.cuh -- the passes of the C-grid hyperdiffusion with its 2/1
// operators (hordiff_Cgrid_mod.f90:59-140, hordiff_scalar_mod.f90:33-53):
//   XF    contravariant components from covariant ones, or back
//         (co2contra_Cgrid_mod.f90:135-203): both interpolations in one pass,
//         a face needs only its two centres
//   DIV   divergence with its SAT penalties onto the centres
//   GRAD  gradient with its SAT penalties onto the faces
//   CURL  curl with its SAT penalties onto the corners, before the corner sync
//   GPERP grad_perp of a corner field onto the faces, the field's corner sync
//         taken as it is read
// The three chains of the operator (curl part, divergence part, h) are six
// passes each and independent, so launch k runs pass k of all three: a role
// of grid.z per chain.  Six launches fill the GPU at sizes where a pass of one
// chain does not, and need no side streams.  Columns and rows are mapped as in
// swm_cgrid_rhs.cuh.  FP32 takes the roundings of the table-driven operators, so
// that results do not depend on the path (spelled out where the compiler has a
// choice of contraction).
// Measured, one diffusion step at N=384 against 29 launches in three streams:
// FP32 0.181 -> 0.142 ms, FP64 0.345 -> 0.317 ms.
#pragma once

enum DiffKind { DK_NONE = 0, DK_XF, DK_XF_CO, DK_DIV, DK_GRAD, DK_CURL, DK_GPERP };

template <class T>
struct DiffRole {
  int kind;
  const T *x, *y;   // inputs (x alone for GRAD and GPERP)
  T *o1, *o2;       // outputs (o1 alone for DIV and CURL)
};
template <class T>
struct DiffArgs {
  RhsArgs<T> r;          // geometry, halo table and the 2/1 operators
  DiffRole<T> role[3];
  int zs;                // grid.z slabs of one role
  // metric: J Qi12, Qi11, Qi22 and, for the way back, J Q12, Q11, Q22; 1/J on
  // the faces; 1/(J hx a) on corners, centres and faces
  const T *jq, *q1, *q3, *jqc, *q1c, *q3c, *rju, *rjv, *rjq, *rjp, *rjuh, *rjvh;
};

// 2/1 interpolation of two values in the order of the table-driven operator
template <class T>
__device__ __forceinline__ T half_sum(T f0, T f1) {
  T s = T(0.5) * f0;
  s += T(0.5) * f1;
  return s;
}

// A face's component from its own q x, the cross terms A0, A1 = jq (y + y') of
// its two centres (twice the interpolated ones) and 1/J; at a panel side the
// one centre counts twice.  FP64 halves once, FP32 as the operators do.
template <class T>
__device__ __forceinline__ T xf_out(T q, T x, T A0, T A1, bool side, T rj) {
  if constexpr (sizeof(T) == 4) {
    const T t = side ? A0 : half_sum(A0, A1);
    return q * x + t * rj;
  } else {
    return q * x + (T(0.25) * (A0 + A1)) * rj;
  }
}
template <class T>
__device__ __forceinline__ void diff_xf(const DiffArgs<T>& a, const DiffRole<T>& R, const RhsPoint& r, bool co) {
  const int N = a.r.N, P = a.r.g.P, i = r.i, j = r.j, e = at(a.r.g, r.p, i, j);
  const T *jq = co ? a.jqc : a.jq, *x = R.x, *y = R.y;
  auto cross = [&](const T* f, int c, int st) {   // of centre c
    if constexpr (sizeof(T) == 4) return ro(jq + c) * half_sum(ro(f + c), ro(f + c + st));
    else return ro(jq + c) * (ro(f + c) + ro(f + c + st));
  };
  if (j < N) {
    const int c0 = i == 0 ? e : e - 1, c1 = i == N ? e - 1 : e;
    R.o1[e] = xf_out(ro((co ? a.q1c : a.q1) + e), ro(x + e), cross(y, c0, P), cross(y, c1, P), c0 == c1, ro(a.rju + e));
  }
  if (i < N) {
    const int c0 = j == 0 ? e : e - P, c1 = j == N ? e - P : e;
    R.o2[e] = xf_out(ro((co ? a.q3c : a.q3) + e), ro(y + e), cross(x, c0, 1), cross(x, c1, 1), c0 == c1, ro(a.rjv + e));
  }
}

// Divergence along one line at centre k: div_line21, in FP64 as it is written
// in div_c2_mod.f90:97-177.
template <bool ALONG_X, class T, class Fn, class Jn>
__device__ __forceinline__ T div_line21_any(int N, int k, Fn F, Jn J) {
  if constexpr (sizeof(T) == 4) {
    return div_line21<ALONG_X, T>(N, k, F, J);
  } else {
    if (k == 0) return J(1) * F(1) - J(0) * (T(0.25) * F(0) + T(0.75) * F(-1));
    if (k == N - 1) return J(N) * (T(0.75) * F(N + 1) + T(0.25) * F(N)) - J(N - 1) * F(N - 1);
    T s = J(k + 1) * F(k + 1) - J(k) * F(k);
    if (k == 1) s -= T(0.25) * J(0) * (F(0) - F(-1));
    if (k == N - 2) s += T(0.25) * J(N) * (F(N) - F(N + 1));
    return s;
  }
}

template <class T>
__device__ __forceinline__ void diff_div(const DiffArgs<T>& a, const DiffRole<T>& R, const RhsPoint& r) {
  const RhsArgs<T>& b = a.r;
  const int N = b.N, P = b.g.P, p = r.p, i = r.ip, j = r.j;
  if (i < 0 || j >= N) return;
  const int e = at(b.g, p, i, j);
  const T *x = R.x, *y = R.y;
  T dx, dy;
  if (!r.strip && rhs_yin(N, j)) {
    const T *X = x + e, *Y = y + e, *Ju = b.Ju + e, *Jv = b.Jv + e;
    if constexpr (sizeof(T) == 4) {
      dx = __fmaf_rn(-ro(Ju), ro(X), __fmul_rn(ro(Ju + 1), ro(X + 1)));
      dy = __fmaf_rn(-ro(Jv), ro(Y), __fmul_rn(ro(Jv + P), ro(Y + P)));
    } else {
      dx = ro(Ju + 1) * ro(X + 1) - ro(Ju) * ro(X);
      dy = ro(Jv + P) * ro(Y + P) - ro(Jv) * ro(Y);
    }
  } else {
    const int row = at(b.g, p, 0, j), col = at(b.g, p, i, 0);
    dx = div_line21_any<true, T>(N, i, [&](int m) {
      return m < 0 ? rhs_halo(b, 1, 0, p, 1, j, x, y) : m > N ? rhs_halo(b, 1, 1, p, 1, j, x, y) : x[row + m];
    }, [&](int m) { return b.Ju[row + m]; });
    dy = div_line21_any<false, T>(N, j, [&](int m) {
      return m < 0 ? rhs_halo(b, 2, 2, p, 1, i, y, x) : m > N ? rhs_halo(b, 2, 3, p, 1, i, y, x) : y[col + m * P];
    }, [&](int m) { return b.Jv[col + m * P]; });
  }
  if constexpr (sizeof(T) == 4) R.o1[e] = __fmul_rn(__fadd_rn(dx, dy), ro(a.rjp + e));
  else R.o1[e] = (dx + dy) * ro(a.rjp + e);
}

template <class T>
__device__ __forceinline__ T mul_rn(T x, T y) {
  if constexpr (sizeof(T) == 4) return __fmul_rn(x, y);
  else return x * y;
}

template <class T>
__device__ __forceinline__ void diff_grad(const DiffArgs<T>& a, const DiffRole<T>& R, const RhsPoint& r) {
  const RhsArgs<T>& b = a.r;
  const int N = b.N, P = b.g.P, p = r.p, i = r.i, j = r.j, e = at(b.g, p, i, j);
  const T* f = R.x;
  if (j < N) {
    const int row = at(b.g, p, 0, j);
    R.o1[e] = i > 0 && i < N
                  ? mul_rn(ro(f + e) - ro(f + e - 1), b.dx1)
                  : grad_edge<T>(b, i, [&](int k) {
                      return k < 0 ? rhs_halo(b, 0, 0, p, -k, j, f, f)
                                   : k >= N ? rhs_halo(b, 0, 1, p, k - N + 1, j, f, f) : f[row + k];
                    });
  }
  if (i < N) {
    const int col = at(b.g, p, i, 0);
    R.o2[e] = j > 0 && j < N
                  ? mul_rn(ro(f + e) - ro(f + e - P), b.dx1)
                  : grad_edge<T>(b, j, [&](int k) {
                      return k < 0 ? rhs_halo(b, 0, 2, p, -k, i, f, f)
                                   : k >= N ? rhs_halo(b, 0, 3, p, k - N + 1, i, f, f) : f[col + k * P];
                    });
  }
}

template <class T>
__device__ __forceinline__ void diff_curl(const DiffArgs<T>& a, const DiffRole<T>& R, const RhsPoint& r) {
  const RhsArgs<T>& b = a.r;
  const int N = b.N, P = b.g.P, p = r.p, i = r.i, j = r.j, e = at(b.g, p, i, j);
  const T *u = R.x, *v = R.y;
  const T* vrow = v + at(b.g, p, 0, j);
  const T* ucol = u + at(b.g, p, i, 0);
  const T dv = i > 0 && i < N ? ro(v + e) - ro(v + e - 1)
                              : d_c2i_sat<21, T>(b, i, [&](int m) { return vrow[m]; },
                                                 [&](int s, int d) { return rhs_halo(b, 2, s, p, d, j, v, u); });
  const T du = j > 0 && j < N ? ro(u + e) - ro(u + e - P)
                              : d_c2i_sat<21, T>(b, j, [&](int m) { return ucol[m * P]; },
                                                 [&](int s, int d) { return rhs_halo(b, 1, 2 + s, p, d, i, u, v); });
  R.o1[e] = (dv - du) * ro(a.rjq + e);
}

// The synced value of corner field w at a neighbour's copy of a point (depth 1
// of side `side`, position k).
template <class T>
__device__ __forceinline__ T corner_copy_synced(const RhsArgs<T>& b, const T* w, int side, int p, int k) {
  const int o = __ldg(&b.halo[(((3 * 4 + side) * 6 + p) * kHaloDepth) * b.L + k]) >> 2;
  const int q = o / (int)b.g.ps, rest = o - q * (int)b.g.ps, jq = rest / b.g.P;
  return rhs_corner_synced(b, w, q, rest - jq * b.g.P, jq);
}

template <class T>
__device__ __forceinline__ void diff_gperp(const DiffArgs<T>& a, const DiffRole<T>& R, const RhsPoint& r) {
  const RhsArgs<T>& b = a.r;
  const int N = b.N, P = b.g.P, p = r.p, i = r.i, j = r.j, e = at(b.g, p, i, j);
  const T* w = R.x;
  const bool yin = rhs_yin(N, j);
  if (j < N) {  // x-face: along the column
    const T s = !r.strip && yin ? ro(w + e + P) - ro(w + e)
                                : d_i2c_sat<21, T>(b, j, [&](int m) { return rhs_corner_synced(b, w, p, i, m); },
                                                   [&](int sd) { return corner_copy_synced(b, w, 2 + sd, p, i); });
    R.o1[e] = -s * ro(a.rjuh + e);
  }
  if (i < N) {  // y-face: along the row
    const T s = !r.strip && yin ? ro(w + e + 1) - ro(w + e)
                                : d_i2c_sat<21, T>(b, i, [&](int m) { return rhs_corner_synced(b, w, p, m, j); },
                                                   [&](int sd) { return corner_copy_synced(b, w, sd, p, j); });
    R.o2[e] = s * ro(a.rjvh + e);
  }
}

template <class T>
__global__ void __launch_bounds__(kRhsX * kRhsY, kRhsBlocks<T>) diff_pass_kernel(const __grid_constant__ DiffArgs<T> a) {
  const int k = blockIdx.z / a.zs;
  const DiffRole<T>& R = a.role[k];
  RhsPoint r;
  if (R.kind == DK_NONE || !rhs_map(a.r, (int)blockIdx.z - k * a.zs, r)) return;
  switch (R.kind) {
    case DK_XF: diff_xf(a, R, r, false); break;
    case DK_XF_CO: diff_xf(a, R, r, true); break;
    case DK_DIV: diff_div(a, R, r); break;
    case DK_GRAD: diff_grad(a, R, r); break;
    case DK_CURL: diff_curl(a, R, r); break;
    default: diff_gperp(a, R, r); break;
  }
}
