// swm_cgrid_rhs.cuh -- the fused C-grid right-hand side (operator_swm_mod
// .f90:61-113 with the C-grid operators) and its RK4 stage epilogue, in four
// passes over the panels:
//   rhs1  p, q   J Qi12 times the other covariant component interpolated to
//                the centres; the curl at the corners (before its corner sync)
//   rhs2  u, v   contravariant components, J * mass flux and kinetic-energy
//                densities on the faces; the synced curl at the x-faces
//   rhs3  p      kinetic energy + g (h + hs), divergence (h tendency),
//                Coriolis terms at the centres
//   rhs4  u, v   gradient and the Coriolis terms back on the faces (u, v
//                tendencies)
//
// What bounds the passes: in FP64 the FP64 instructions (GB300 issues one warp
// instruction to an SM quarter in 64 cycles), in FP32 instruction issue and
// the L2 traffic between passes.  So:
//   - The interior stencils are straight-line code on pointers.
//   - FP64 takes their sums and differences before any scaling and leaves the
//     leading coefficient out: the intermediate fields hold values scaled by
//     the inverse leading coefficients (Sc<ORD>), which return in the metric
//     fields and constants that multiply them anyway (M_S* fields).  The
//     closure rows come scaled the same way.  An interpolation or difference
//     takes 3 FP64 instructions instead of 4, and the difference of two 7
//     instead of 9.  FP32, where an instruction more is cheap, keeps the
//     coefficients and the order of the unfused operators' sums, so that its
//     results are bit for bit what table-driven passes gave.
//   - The first and last four columns are run by warps of their own (rhs_map), in
//     FP64 along the column, so that a warp's closure row along x is uniform, and
//     no other warp branches on x.  Along y a warp is one row, and uniform already.
//   - The six passes of the operators one by one pair up where one does not
//     read the other's output: 16 launches an RK4 step.
// Measured at N=384, 4/2 (RK4 step): FP64 1.058 -> 0.705 ms against six
// passes with table-driven stencils in warps along the row; FP32 model step
// (with hyperdiffusion) 0.481 -> 0.365 ms.
#pragma once

// Leading coefficients of the interior stencils: interpolation sW (f0 + f1 +
// rW (f-1 + f2)), difference sD (f1 - f0 + rD (f2 - f-1)).
template <int ORD>
struct Sc {
  static constexpr double sW = ORD == 42 ? 9.0 / 16.0 : 0.5, rW = -1.0 / 9.0;
  static constexpr double sD = ORD == 42 ? 9.0 / 8.0 : 1.0, rD = -1.0 / 27.0;
};
inline double scale_w(int ord) { return ord == 42 ? Sc<42>::sW : Sc<21>::sW; }
inline double scale_d(int ord) { return ord == 42 ? Sc<42>::sD : Sc<21>::sD; }

// The operators with their leading interior coefficient taken out.
template <class T>
struct ScaledOps {
  StagOpT<T> wc2i, wi2c, dc2i, di2c;
  int np;
  T proj[3];
  T pen[3];   // SAT of the divergence: pen_c / 2
  T csat;     // SAT of the curl: 1 / (2 a_i0)
  T gsat;     // SAT of the gradient: 1 / (2 sq1)
};
template <class T>
ScaledOps<T> scaled_ops(const COps& o, int ord) {
  const double w = 1.0 / scale_w(ord), d = 1.0 / scale_d(ord);
  auto scaled = [](StagOp s, double f) {
    for (double& x : s.Ql) x *= f;
    return stag_cast<T>(s);
  };
  ScaledOps<T> r{};
  r.wc2i = scaled(o.wc2i, w); r.wi2c = scaled(o.wi2c, w);
  r.dc2i = scaled(o.dc2i, d); r.di2c = scaled(o.di2c, d);
  r.np = o.np;
  for (int k = 0; k < 3; ++k) { r.proj[k] = T(o.proj[k]); r.pen[k] = T(0.5 * o.pen_c[k] * d); }
  r.csat = T(0.5 * d / o.a_i0);
  r.gsat = T(0.5 * d / o.sq1);
  return r;
}

template <class T>
struct RhsArgs {
  FieldGeom g;
  int N, L, strips;   // strips: grid.z slabs of the side columns
  const int* halo;
  std::conditional_t<sizeof(T) == 8, ScaledOps<T>, COpsT<T>> ops;
  // metric: JQi2p, f, Ju, Jv, Qi1u, Qi3v and 1/J (u, v), 1/(J hx a) (corners),
  // 1/(2J) and 1/(J hx a) (centres) scaled; FP32: unscaled, and 1/J for 1/(2J)
  const T *jq, *fp, *Ju, *Jv, *Qi1u, *Qi3v, *sju, *sjv, *sjq, *sjp, *sdiv;
  const T *h, *u, *v, *hs;
  T *Ap, *Bp, *Gu, *Gv, *KEu, *KEv, *curl, *fu, *KE, *cup, *cvp;
  T *hu, *hv;   // FP32 at 2/1: the raw fluxes, whose divergence multiplies by J
  T grav, cg, cw, cw2;   // g; FP64: scale of the gradient, the Coriolis terms, the curl
  T dx1;                 // FP32: 1 / (a hx)
  T hdt, dt, c3, c6;     // the RK4 stages, as in CArgsT
  T *tend, *y0, *Y, *Kb, *acc, *lo;
};

constexpr int kRhsX = 32, kRhsY = 8, kRhsEdge = 4;
// Resident blocks per SM the passes are compiled for.  FP32 waits on memory
// and wants every warp slot on large panels: 8 blocks (32 registers) 0.365 ms a
// model step at N=384, unconstrained 0.380, 6 blocks 0.394, 4 blocks 0.455; up to
// N=160, where few blocks are resident at all, 3, 4 and 6 blocks measured 0 to 5%
// faster (RK4 step 4/2, side columns still in warps along the column: N=48 119 us
// for 123, N=96 111 for 115), which two compiled variants of every pass are not
// worth.  FP64 waits on
// its pipe and measures the same at 6 and 8 (3% slower unconstrained).
template <class T>
constexpr int kRhsBlocks = sizeof(T) == 4 ? 8 : 6;

// Point of this thread in slab z: i for the interface outputs along x (0..N) and ip for
// the centre outputs (0..N-1, or -1 where a thread has none).  The first grid.z
// slabs hold the warps of the four columns at either side, a block 32 rows of
// them; the others hold the columns between.
struct RhsPoint {
  int p, i, ip, j;
  bool strip;
};
template <class T>
__device__ __forceinline__ bool rhs_map(const RhsArgs<T>& a, int z, RhsPoint& r) {
  const int N = a.N;
  if (z < a.strips) {
    const int nb = (N + kRhsX) / kRhsX;   // blocks of 32 rows along 0..N
    const int b = (z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    r.p = b / nb;
    if (r.p >= 6) return false;
    // FP64: a column a warp.  FP32, which waits on memory, 8 rows of the four
    // columns of a side: 8 cache lines a load and not 32, at the price of closure
    // rows that differ between lanes.  RK4 step 4/2, us, against columns: N=16 117 ->
    // 94, N=48 123 -> 109, N=56 125 -> 107, N=80 127 -> 108, N=384 211 -> 207 (2/1: N=56
    // 102 -> 94, N=192 107 -> 110); FP64 at N=16 195 -> 141 but the FP64 diffusion at
    // N=128 77 -> 84.
    const int w = threadIdx.y, l = threadIdx.x;
    const bool tile = sizeof(T) == 4;
    r.j = (b - r.p * nb) * kRhsX + (tile ? (w >> 1) * 8 + (l >> 2) : l);
    const int c = tile ? (w & 1) * kRhsEdge + (l & 3) : w;
    r.i = c < kRhsEdge ? c : N - 2 * kRhsEdge + 1 + c;
    r.ip = c < kRhsEdge ? c : N - 2 * kRhsEdge + c;
    r.strip = true;
    return r.j <= N;
  }
  r.p = z - a.strips;
  r.i = kRhsEdge + blockIdx.x * kRhsX + threadIdx.x;
  r.j = blockIdx.y * kRhsY + threadIdx.y;
  r.ip = r.i < N - kRhsEdge ? r.i : -1;
  r.strip = false;
  return r.i <= N - kRhsEdge && r.j <= N;
}

// Load of a value no thread of the kernel writes: the compiler may move it
// above the kernel's stores, so that all loads of a point are in flight at once
// (FP32 model step at N=384 0.398 -> 0.380 ms).
template <class T>
__device__ __forceinline__ T ro(const T* p) { return __ldg(p); }

// Interior stencils at f (the input f0 sits at f, stride st).
template <int ORD, class T>
__device__ __forceinline__ T w_in(const T* __restrict__ f, int st) {
  if constexpr (sizeof(T) == 4) {
    T s = T(0.0);
    if constexpr (ORD == 42) {
      s += T(-1.0 / 16.0) * ro(f + (-st));
      s += T(9.0 / 16.0) * ro(f);
      s += T(9.0 / 16.0) * ro(f + (st));
      s += T(-1.0 / 16.0) * ro(f + (2 * st));
    } else {
      s += T(0.5) * ro(f);
      s += T(0.5) * ro(f + (st));
    }
    return s;
  } else if constexpr (ORD == 21) return ro(f) + ro(f + (st));
  else return (ro(f) + ro(f + (st))) + T(Sc<ORD>::rW) * (ro(f + (-st)) + ro(f + (2 * st)));
}
template <int ORD, class T>
__device__ __forceinline__ T d_in(const T* __restrict__ f, int st) {
  if constexpr (sizeof(T) == 4) {
    T s = T(0.0);
    if constexpr (ORD == 42) {
      s += T(1.0 / 24.0) * ro(f + (-st));
      s += T(-9.0 / 8.0) * ro(f);
      s += T(9.0 / 8.0) * ro(f + (st));
      s += T(-1.0 / 24.0) * ro(f + (2 * st));
    } else {
      s = ro(f + (st)) - ro(f);
    }
    return s;
  } else if constexpr (ORD == 21) return ro(f + (st)) - ro(f);
  else return (ro(f + (st)) - ro(f)) + T(Sc<ORD>::rD) * (ro(f + (2 * st)) - ro(f + (-st)));
}
// f along x plus s times g along y, differences (d) or interpolations
template <int ORD, class T>
__device__ __forceinline__ T d_in2(const T* __restrict__ f, int sf, const T* __restrict__ q, int sq, T s) {
  if constexpr (sizeof(T) == 4) return d_in<ORD, T>(f, sf) + s * d_in<ORD, T>(q, sq);
  else if constexpr (ORD == 21) return (ro(f + (sf)) - ro(f)) + s * (ro(q + (sq)) - ro(q));
  else
    return ((ro(f + (sf)) - ro(f)) + s * (ro(q + (sq)) - ro(q))) +
           T(Sc<ORD>::rD) * ((ro(f + (2 * sf)) - ro(f + (-sf))) + s * (ro(q + (2 * sq)) - ro(q + (-sq))));
}
template <int ORD, class T>
__device__ __forceinline__ T w_in2(const T* __restrict__ f, int sf, const T* __restrict__ q, int sq) {
  if constexpr (sizeof(T) == 4) return w_in<ORD, T>(f, sf) + w_in<ORD, T>(q, sq);
  else if constexpr (ORD == 21) return (ro(f) + ro(f + (sf))) + (ro(q) + ro(q + (sq)));
  else
    return ((ro(f) + ro(f + (sf))) + (ro(q) + ro(q + (sq)))) +
           T(Sc<ORD>::rW) * ((ro(f + (-sf)) + ro(f + (2 * sf))) + (ro(q + (-sq)) + ro(q + (2 * sq))));
}

// Any output row k of nout: the interior form or the scaled closure rows.
// off: input index of f0 at output k (k-1 for c2i, k for i2c); F(m) reads
// input m.
template <int ORD, bool DIFF, class T, class Fn>
__device__ __forceinline__ T any_row(const StagOpT<T>& s, int nout, int k, int off, Fn F) {
  if constexpr (sizeof(T) == 4) return stag_at_f<ORD == 42 ? 4 : 2, T>(s, F, nout, k);
  if (k >= s.ne && k < nout - s.ne) {
    if constexpr (ORD == 21) return DIFF ? F(off + 1) - F(off) : F(off) + F(off + 1);
    else if constexpr (DIFF)
      return (F(off + 1) - F(off)) + T(Sc<ORD>::rD) * (F(off + 2) - F(off - 1));
    else
      return (F(off) + F(off + 1)) + T(Sc<ORD>::rW) * (F(off - 1) + F(off + 2));
  }
  return stag_closure<ORD == 42 ? 4 : 2, T>(s, F, nout, k);
}
template <int ORD, class T, class Fn>
__device__ __forceinline__ T w_c2i(const RhsArgs<T>& a, int k, Fn F) {
  return any_row<ORD, false, T>(a.ops.wc2i, a.N + 1, k, k - 1, F);
}
template <int ORD, class T, class Fn>
__device__ __forceinline__ T w_i2c(const RhsArgs<T>& a, int k, Fn F) {
  return any_row<ORD, false, T>(a.ops.wi2c, a.N, k, k, F);
}
template <int ORD, class T, class Fn>
__device__ __forceinline__ T d_c2i(const RhsArgs<T>& a, int k, Fn F) {
  return any_row<ORD, true, T>(a.ops.dc2i, a.N + 1, k, k - 1, F);
}
template <int ORD, class T, class Fn>
__device__ __forceinline__ T d_i2c(const RhsArgs<T>& a, int k, Fn F) {
  return any_row<ORD, true, T>(a.ops.di2c, a.N, k, k, F);
}

// A neighbour's point (see halo_at).
template <class T>
__device__ __forceinline__ T rhs_halo(const RhsArgs<T>& a, int mesh, int side, int p, int d, int k,
                                      const T* __restrict__ f, const T* __restrict__ g) {
  const int c = __ldg(&a.halo[((((mesh * 4 + side) * 6 + p) * kHaloDepth + (d - 1)) * a.L) + k]);
  const T x = ((c & 2) ? g : f)[c >> 2];
  return (c & 1) ? -x : x;
}

// Difference onto interface k of a line of centres F with the SAT penalty of
// its two ends (the curl's, curl_c_sbp_mod.f90:44-127); H(side, d) is the
// neighbour's point d layers out at the low (side 0) or high end.
template <int ORD, class T, class Fn, class Hn>
__device__ __forceinline__ T d_c2i_sat(const RhsArgs<T>& a, int k, Fn F, Hn H) {
  const int N = a.N;
  T s = d_c2i<ORD, T>(a, k, F);
  if (k == 0 || k == N) {
    T dj = T(0.0);
#pragma unroll
    for (int m = 0; m < (ORD == 42 ? 3 : 2); ++m)
      dj = dj + a.ops.proj[m] * (k == 0 ? F(m) - H(0, m + 1) : H(1, m + 1) - F(N - 1 - m));
    if constexpr (sizeof(T) == 8) s += a.ops.csat * dj;
    else s = s + T(0.5) * dj / a.ops.a_i0;
  }
  return s;
}
// Difference onto centre k of a line of interfaces with the SAT penalty on the
// duplicated edge points (div_c_sbp42_mod.f90:67-107, div_c2_mod.f90:97-177).
template <int ORD, class T, class Fn, class Hn>
__device__ __forceinline__ T d_i2c_sat(const RhsArgs<T>& a, int k, Fn F, Hn H) {
  const int N = a.N;
  T s = d_i2c<ORD, T>(a, k, F);
  if constexpr (sizeof(T) == 8) {
    if (k < a.ops.np) s += a.ops.pen[k] * (F(0) - H(0));
    if (k >= N - a.ops.np) s += a.ops.pen[N - 1 - k] * (H(1) - F(N));
  } else {
    if (k < a.ops.np) s = s + T(0.5) * a.ops.pen_c[k] * (F(0) - H(0));
    if (k >= N - a.ops.np) s = s + T(0.5) * a.ops.pen_c[N - 1 - k] * (H(1) - F(N));
  }
  return s;
}
// The gradient (without FP64's scale) at interface k of a line of centres:
// F(m) reads the panel for 0 <= m < N and the o halo outside.
template <int ORD, class T, class Fn>
__device__ __forceinline__ T grad_any(const RhsArgs<T>& a, int k, Fn F) {
  if constexpr (sizeof(T) == 4) {
    return grad_line<ORD, T>(a, a.N, k, F);
  } else {
    const int N = a.N;
    T s = d_c2i<ORD, T>(a, k, F);
    if (k == 0 || k == N) {
      T dj = T(0);
#pragma unroll
      for (int m = 0; m < (ORD == 42 ? 3 : 2); ++m)
        dj += a.ops.proj[m] * (k == 0 ? F(m) - F(-1 - m) : F(N + m) - F(N - 1 - m));
      s += a.ops.gsat * dj;
    }
    return s;
  }
}
// The 2/1 gradient at the two panel-edge interfaces (k = 0, N), scaled.
template <class T, class Fn>
__device__ __forceinline__ T grad_edge(const RhsArgs<T>& a, int k, Fn F) {
  if constexpr (sizeof(T) == 4) return grad_line<21, T>(a, a.N, k, F);
  else return grad_any<21, T>(a, k, F) * a.dx1;   // the 2/1 difference has the scale 1
}
// The 2/1 divergence along one line in FP32 from the raw fluxes F (with the
// neighbour's at -1 and N+1) and J at the interfaces (div_c2_mod.f90:97-177).
// The roundings are those of centre_b_kernel, spelled out; at the high end
// they differ between x and y (ALONG_X).
template <bool ALONG_X, class T, class Fn, class Jn>
__device__ __forceinline__ T div_line21(int N, int k, Fn F, Jn J) {
  // a b - c d with one product rounded: the first or the second
  auto sub1 = [](T a, T b, T c, T d) { return __fmaf_rn(-c, d, __fmul_rn(a, b)); };
  auto sub2 = [](T a, T b, T c, T d) { return __fmaf_rn(a, b, -__fmul_rn(c, d)); };
  if (k == 0) return sub2(J(1), F(1), J(0), __fmaf_rn(T(0.25), F(0), __fmul_rn(T(0.75), F(-1))));
  if (k == N - 1) {
    const T x = ALONG_X ? __fmaf_rn(T(0.25), F(N), __fmul_rn(T(0.75), F(N + 1)))
                        : __fmaf_rn(T(0.75), F(N + 1), __fmul_rn(T(0.25), F(N)));
    return sub2(J(N), x, J(N - 1), F(N - 1));
  }
  if (k == 1)
    return __fmaf_rn(-__fmul_rn(T(0.25), J(0)), __fadd_rn(F(0), -F(-1)), sub2(J(2), F(2), J(1), F(1)));
  if (k == N - 2) {
    const T s = ALONG_X ? sub1(J(N - 1), F(N - 1), J(N - 2), F(N - 2)) : sub2(J(N - 1), F(N - 1), J(N - 2), F(N - 2));
    return __fmaf_rn(__fmul_rn(T(0.25), J(N)), __fadd_rn(F(N), -F(N + 1)), s);
  }
  return sub1(J(k + 1), F(k + 1), J(k), F(k));
}

// RK4 stage epilogue of one value (mode 0 stores the tendency; 1..4 are
// the stages of rk4_mod.f90:20-42: y0, Y, Kb, acc are 3 fields each, fs apart;
// FP32: y0 / lo the state pair, acc the running increment, no Kb), with the
// inputs loaded by rk_in beforehand.
template <class T>
struct RkIn {
  T y0, kb, acc, lo;
};
template <int MODE, class T>
__device__ __forceinline__ RkIn<T> rk_in(const RhsArgs<T>& a, int o) {
  RkIn<T> r{};
  if (MODE >= 1 && (MODE < 4 || sizeof(T) == 4)) r.y0 = a.y0[o];
  if (sizeof(T) == 8 && (MODE == 2 || MODE == 4)) r.kb = a.Kb[o];
  if (MODE == 4 || (sizeof(T) == 4 && (MODE == 2 || MODE == 3))) r.acc = a.acc[o];
  if (sizeof(T) == 4 && MODE == 4) r.lo = a.lo[o];
  return r;
}
template <int MODE, class T>
__device__ __forceinline__ void rk_out(const RhsArgs<T>& a, int o, T k, const RkIn<T>& r) {
  if constexpr (MODE == 0) {
    a.tend[o] = k;
  } else if constexpr (sizeof(T) == 8) {
    if constexpr (MODE == 1) { a.Kb[o] = k; a.Y[o] = r.y0 + a.hdt * k; }
    else if constexpr (MODE == 2) { a.acc[o] = (r.y0 + a.c6 * r.kb) + a.c3 * k; a.Y[o] = r.y0 + a.hdt * k; }
    else if constexpr (MODE == 3) { a.Kb[o] = k; a.Y[o] = r.y0 + a.dt * k; }
    else a.y0[o] = (r.acc + a.c3 * r.kb) + a.c6 * k;
  } else {
    if constexpr (MODE == 1) { a.Y[o] = r.y0 + a.hdt * k; a.acc[o] = a.c6 * k; }
    else if constexpr (MODE == 2) { a.Y[o] = r.y0 + a.hdt * k; a.acc[o] = r.acc + a.c3 * k; }
    else if constexpr (MODE == 3) { a.Y[o] = r.y0 + a.dt * k; a.acc[o] = r.acc + a.c3 * k; }
    else {
      const T d = r.acc + a.c6 * k;
      const T t = r.lo + d;
      const T s = r.y0 + t;
      const T bb = s - r.y0;
      a.y0[o] = s;
      a.lo[o] = (r.y0 - (s - bb)) + (t - bb);
    }
  }
}

// rows whose y stencils (centre and interface outputs) are interior
__device__ __forceinline__ bool rhs_yin(int N, int j) { return j >= kRhsEdge && j < N - kRhsEdge; }

template <int ORD, class T>
__global__ void __launch_bounds__(kRhsX * kRhsY, kRhsBlocks<T>) rhs1_kernel(const __grid_constant__ RhsArgs<T> a) {
  RhsPoint r;
  if (!rhs_map(a, blockIdx.z, r)) return;
  const int N = a.N, P = a.g.P, p = r.p, j = r.j;
  const bool yin = rhs_yin(N, j);
  {  // corner (i, j): the curl, curl_c_sbp_mod.f90:44-127
    const int e = at(a.g, p, r.i, j);
    const T* u = a.u + e;
    const T* v = a.v + e;
    T z;
    if (!r.strip && yin) {
      z = d_in2<ORD, T>(v - 1, 1, u - P, P, T(-1));
    } else {
      const T* vrow = a.v + at(a.g, p, 0, j);
      const T* ucol = a.u + at(a.g, p, r.i, 0);
      const T dv = r.strip ? d_c2i_sat<ORD, T>(a, r.i, [&](int m) { return vrow[m]; },
                                               [&](int s, int d) { return rhs_halo(a, 2, s, p, d, j, a.v, a.u); })
                           : d_in<ORD, T>(v - 1, 1);
      const T du = yin ? d_in<ORD, T>(u - P, P)
                       : d_c2i_sat<ORD, T>(a, j, [&](int m) { return ucol[m * P]; },
                                           [&](int s, int d) { return rhs_halo(a, 1, 2 + s, p, d, r.i, a.u, a.v); });
      z = dv - du;
    }
    a.curl[e] = z * ro(a.sjq + e);
  }
  if (r.ip >= 0 && j < N) {  // centre (ip, j): co2contra_Cgrid_mod.f90:292-437, first half
    const int e = at(a.g, p, r.ip, j);
    const T* u = a.u + e;
    const T* v = a.v + e;
    const T* urow = a.u + at(a.g, p, 0, j);
    const T* vcol = a.v + at(a.g, p, r.ip, 0);
    const T jq = ro(a.jq + e);
    a.Ap[e] = jq * (yin ? w_in<ORD, T>(v, P) : w_i2c<ORD, T>(a, j, [&](int m) { return vcol[m * P]; }));
    a.Bp[e] = jq * (r.strip ? w_i2c<ORD, T>(a, r.ip, [&](int m) { return urow[m]; }) : w_in<ORD, T>(u, 1));
  }
}

// A corner field with its Ah-type sync (halo_Ah_scalar_sync_mod.f90:38-93, in the
// order of the sync kernel) taken as it is read.
template <class T>
__device__ __forceinline__ T rhs_corner_synced(const RhsArgs<T>& a, const T* c, int p, int i, int j) {
  const int N = a.N;
  const T own = c[at(a.g, p, i, j)];
  const bool lr = i == 0 || i == N, bt = j == 0 || j == N;
  if (!lr && !bt) return own;
  const T x = lr ? rhs_halo(a, 3, i == 0 ? 0 : 1, p, 1, j, c, c) : T(0);
  const T y = bt ? rhs_halo(a, 3, j == 0 ? 2 : 3, p, 1, i, c, c) : T(0);
  return lr && bt ? (own + x + y) / T(3.0) : T(0.5) * (own + (lr ? x : y));
}

// A face's J * mass flux and kinetic-energy density (FP64: twice that) from
// its velocity w, the interpolated cross term t and the interpolated depth h;
// FP32 at 2/1 also stores the raw flux.
template <int ORD, class T>
__device__ __forceinline__ void flux_out(T qi, T w, T t, T sj, T J, T h, T* G, T* KE, T* raw) {
  const T wt = qi * w + t * sj;
  if constexpr (sizeof(T) == 8) {
    const T jw = J * wt;
    *G = jw * h;
    *KE = jw * w;
  } else {
    const T f = wt * h;
    if (ORD == 21) *raw = f;
    *G = f * J;
    *KE = J * (w * wt) * T(0.5);
  }
}

template <int ORD, class T>
__global__ void __launch_bounds__(kRhsX * kRhsY, kRhsBlocks<T>) rhs2_kernel(const __grid_constant__ RhsArgs<T> a) {
  RhsPoint r;
  if (!rhs_map(a, blockIdx.z, r)) return;
  const int N = a.N, P = a.g.P, p = r.p, i = r.i, j = r.j;
  const bool yin = rhs_yin(N, j);
  const int e = at(a.g, p, i, j);
  if (j < N) {  // x-face: co2contra, massflux * J, KE density; interpolator_w2h's first half
    const T* Arow = a.Ap + at(a.g, p, 0, j);
    const T* hrow = a.h + at(a.g, p, 0, j);
    const T t = r.strip ? w_c2i<ORD, T>(a, i, [&](int m) { return Arow[m]; }) : w_in<ORD, T>(a.Ap + e - 1, 1);
    const T hu = r.strip ? w_c2i<ORD, T>(a, i, [&](int m) { return hrow[m]; }) : w_in<ORD, T>(a.h + e - 1, 1);
    flux_out<ORD, T>(ro(a.Qi1u + e), ro(a.u + e), t, ro(a.sju + e), ro(a.Ju + e), hu, a.Gu + e, a.KEu + e, a.hu + e);
    a.fu[e] = !r.strip && yin ? w_in<ORD, T>(a.curl + e, P)
                              : w_i2c<ORD, T>(a, j, [&](int m) { return rhs_corner_synced(a, a.curl, p, i, m); });
  }
  if (i < N) {  // y-face
    const T* Bcol = a.Bp + at(a.g, p, i, 0);
    const T* hcol = a.h + at(a.g, p, i, 0);
    const T t = yin ? w_in<ORD, T>(a.Bp + e - P, P) : w_c2i<ORD, T>(a, j, [&](int m) { return Bcol[m * P]; });
    const T hv = yin ? w_in<ORD, T>(a.h + e - P, P) : w_c2i<ORD, T>(a, j, [&](int m) { return hcol[m * P]; });
    flux_out<ORD, T>(ro(a.Qi3v + e), ro(a.v + e), t, ro(a.sjv + e), ro(a.Jv + e), hv, a.Gv + e, a.KEv + e, a.hv + e);
  }
}

template <int ORD, int MODE, class T>
__global__ void __launch_bounds__(kRhsX * kRhsY, kRhsBlocks<T>) rhs3_kernel(const __grid_constant__ RhsArgs<T> a) {
  RhsPoint r;
  if (!rhs_map(a, blockIdx.z, r) || r.ip < 0 || r.j >= a.N) return;
  const int N = a.N, P = a.g.P, p = r.p, i = r.ip, j = r.j;
  const int e = at(a.g, p, i, j);
  const RkIn<T> rk = rk_in<MODE, T>(a, e);
  // read before the epilogue of stages 2 and 3 writes the new h over it
  const T h = a.h[e];
  T ke, dv, gu, gv, cp;
  if (!r.strip && rhs_yin(N, j)) {
    ke = w_in2<ORD, T>(a.KEu + e, 1, a.KEv + e, P);
    if constexpr (ORD == 21 && sizeof(T) == 4) {
      const T *hu = a.hu + e, *hv = a.hv + e, *Ju = a.Ju + e, *Jv = a.Jv + e;
      dv = __fadd_rn(__fmaf_rn(-Ju[0], hu[0], __fmul_rn(Ju[1], hu[1])),
                     __fmaf_rn(-Jv[0], hv[0], __fmul_rn(Jv[P], hv[P])));
    } else {
      dv = d_in2<ORD, T>(a.Gu + e, 1, a.Gv + e, P, T(1));
    }
    gu = w_in<ORD, T>(a.Gu + e, 1);
    gv = w_in<ORD, T>(a.Gv + e, P);
    cp = w_in<ORD, T>(a.fu + e, 1);
  } else {
    const int row = at(a.g, p, 0, j), col = at(a.g, p, i, 0);
    auto X = [&](const T* f) { return [f, row](int m) { return f[row + m]; }; };
    auto Y = [&](const T* f) { return [f, col, P](int m) { return f[col + m * P]; }; };
    ke = w_i2c<ORD, T>(a, i, X(a.KEu)) + w_i2c<ORD, T>(a, j, Y(a.KEv));
    if constexpr (ORD == 21 && sizeof(T) == 4) {
      auto U = [&](int m) {
        return m < 0 ? rhs_halo(a, 1, 0, p, 1, j, a.hu, a.hv) : m > N ? rhs_halo(a, 1, 1, p, 1, j, a.hu, a.hv) : a.hu[row + m];
      };
      auto V = [&](int m) {
        return m < 0 ? rhs_halo(a, 2, 2, p, 1, i, a.hv, a.hu) : m > N ? rhs_halo(a, 2, 3, p, 1, i, a.hv, a.hu) : a.hv[col + m * P];
      };
      dv = __fadd_rn(div_line21<true, T>(N, i, U, X(a.Ju)), div_line21<false, T>(N, j, V, Y(a.Jv)));
    } else {
      dv = d_i2c_sat<ORD, T>(a, i, X(a.Gu), [&](int s) { return rhs_halo(a, 1, s, p, 1, j, a.Gu, a.Gv); }) +
           d_i2c_sat<ORD, T>(a, j, Y(a.Gv), [&](int s) { return rhs_halo(a, 2, 2 + s, p, 1, i, a.Gv, a.Gu); });
    }
    gu = w_i2c<ORD, T>(a, i, X(a.Gu));
    gv = w_i2c<ORD, T>(a, j, Y(a.Gv));
    cp = w_i2c<ORD, T>(a, i, X(a.fu));
  }
  // KE_Cgrid_mod.f90:60-75 plus g (h + hs) (operator_swm_mod.f90:84-85)
  if constexpr (sizeof(T) == 8) {
    T k = ke * ro(a.sjp + e) + a.grav * h;
    if (a.hs) k = k + a.grav * a.hs[e];
    a.KE[e] = k;
  } else {
    ke = __fmaf_rn(a.grav, h, __fmul_rn(ke, ro(a.sjp + e)));
    if (a.hs) ke = __fmaf_rn(a.grav, a.hs[e], ke);
    a.KE[e] = ke;
  }
  // coriolis_Cgrid_mod.f90:98-118; one division per point
  T q;
  if constexpr (sizeof(T) == 8) q = (ro(a.fp + e) + a.cw2 * cp) / h;
  else q = (ro(a.fp + e) + cp) / h;
  a.cup[e] = q * gv;
  a.cvp[e] = -q * gu;
  // div_c_sbp42_mod.f90:67-107, div_c2_mod.f90:97-177
  if constexpr (sizeof(T) == 4) rk_out<MODE, T>(a, e, -__fmul_rn(dv, ro(a.sdiv + e)), rk);
  else rk_out<MODE, T>(a, e, -(dv * ro(a.sdiv + e)), rk);
}

// Interior gradient at a face (FP64 without its scale) and the tendency of a
// velocity component.
template <int ORD, class T>
__device__ __forceinline__ T grad_fast(const RhsArgs<T>& a, const T* __restrict__ f, int st) {
  if constexpr (sizeof(T) == 8) return d_in<ORD, T>(f, st);
  else return __fmul_rn(d_in<ORD, T>(f, st), a.dx1);
}
template <class T>
__device__ __forceinline__ T uv_tend(const RhsArgs<T>& a, T g, T c) {
  if constexpr (sizeof(T) == 8) return a.cw * c - a.cg * g;
  else return __fadd_rn(c, -g);
}

template <int ORD, int MODE, class T>
__global__ void __launch_bounds__(kRhsX * kRhsY, kRhsBlocks<T>) rhs4_kernel(const __grid_constant__ RhsArgs<T> a) {
  RhsPoint r;
  if (!rhs_map(a, blockIdx.z, r)) return;
  const int N = a.N, P = a.g.P, p = r.p, i = r.i, j = r.j, fs = (int)a.g.fs;
  const int e = at(a.g, p, i, j);
  const bool yin = rhs_yin(N, j), onu = j < N, onv = i < N;
  RkIn<T> ru{}, rv{};
  if (onu) ru = rk_in<MODE, T>(a, fs + e);
  if (onv) rv = rk_in<MODE, T>(a, 2 * fs + e);
  const T* f = a.KE;
  if (onu) {  // grad_c_sbp42_mod.f90:44-139, grad_c2_ecs_mod.f90:234-293
    const int row = at(a.g, p, 0, j);
    T gx, cu;
    if (!r.strip) {
      gx = grad_fast<ORD, T>(a, f + e - 1, 1);
      cu = w_in<ORD, T>(a.cup + e - 1, 1);
    } else {
      gx = grad_any<ORD, T>(a, i, [&](int k) {
        return k < 0 ? rhs_halo(a, 0, 0, p, -k, j, f, f) : k >= N ? rhs_halo(a, 0, 1, p, k - N + 1, j, f, f) : f[row + k];
      });
      cu = w_c2i<ORD, T>(a, i, [&](int m) { return a.cup[row + m]; });
    }
    rk_out<MODE, T>(a, fs + e, uv_tend<T>(a, gx, cu), ru);
  }
  if (onv) {
    const int col = at(a.g, p, i, 0);
    T gy, cv;
    if (yin) {
      gy = grad_fast<ORD, T>(a, f + e - P, P);
      cv = w_in<ORD, T>(a.cvp + e - P, P);
    } else {
      gy = grad_any<ORD, T>(a, j, [&](int k) {
        return k < 0 ? rhs_halo(a, 0, 2, p, -k, i, f, f)
                     : k >= N ? rhs_halo(a, 0, 3, p, k - N + 1, i, f, f) : f[col + k * P];
      });
      cv = w_c2i<ORD, T>(a, j, [&](int m) { return a.cvp[col + m * P]; });
    }
    rk_out<MODE, T>(a, 2 * fs + e, uv_tend<T>(a, gy, cv), rv);
  }
}

template <int ORD, class T>
cudaError_t rhs_passes(const RhsArgs<T>& a, int mode, dim3 grid, cudaStream_t st) {
  const dim3 blk(kRhsX, kRhsY);
  rhs1_kernel<ORD, T><<<grid, blk, 0, st>>>(a);
  rhs2_kernel<ORD, T><<<grid, blk, 0, st>>>(a);
  switch (mode) {
#define SWM_RHS_MODE(M)                                \
  case M:                                              \
    rhs3_kernel<ORD, M, T><<<grid, blk, 0, st>>>(a);   \
    rhs4_kernel<ORD, M, T><<<grid, blk, 0, st>>>(a);   \
    break;
    SWM_RHS_MODE(0) SWM_RHS_MODE(1) SWM_RHS_MODE(2) SWM_RHS_MODE(3) SWM_RHS_MODE(4)
#undef SWM_RHS_MODE
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}
