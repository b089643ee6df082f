// swm_stage.cuh -- SBP derivatives, the RHS tendency and RK stage epilogue,
// the FP64 stage kernels, and the cube-edge pass that finishes the
// panel-boundary nodes of an FP32 stage (whose stage kernel is in
// swm_stage_tma.cuh).
//
// One FP64 RK stage:
//   point_derive_kernel  (first stage of a step only) the pointwise stencil
//                        inputs of the state: 2(KE + g(h+hs)), J h ut, J h vt,
//                        J ut, J vt
//   point_stage_kernel   every node: SBP grad(KE), curl and div(h u) with
//                        their one-sided closures from those fields, the
//                        cube-edge syncs at panel-boundary nodes, Coriolis,
//                        the tendency, the RK stage combination and the next
//                        stage's stencil inputs.
// An FP32 stage is its stage kernel and the
//   edge_kernel          every panel-boundary node, from the pre-sync
//                        (gx, gy, zeta, div) of the stage kernel: the
//                        reference's cube-edge syncs (2-way average on edges,
//                        3-way at cube corners, metric-weighted for the
//                        covariant gradient), then the tendency and the RK
//                        epilogue.
// Reference: operator_swm_mod.f90:61-113, rk4_mod.f90:20-42,
// sbp_operator_mod.f90:152-228, div_ah_sbp_mod.f90:46-96,
// grad_ah_sbp_mod.f90:51-88, curl_div_based_mod.f90:26-66,
// coriolis_colocated_mod.f90:79-103, halo_Ah_scalar_sync_mod.f90:38-93,
// ecs_Ah_vec_sync_mod.f90:62-125.
#pragma once

#include "swm_device.cuh"

namespace swm {

template <int ORD> struct Ord;
template <> struct Ord<21> { static constexpr int idx = 0, NE = 1, NW = 2, H = 1, RMAX = 1; };
template <> struct Ord<42> { static constexpr int idx = 1, NE = 4, NW = 6, H = 2, RMAX = 3; };
template <> struct Ord<43> { static constexpr int idx = 2, NE = 4, NW = 6, H = 2, RMAX = 5; };
template <> struct Ord<63> { static constexpr int idx = 3, NE = 6, NW = 9, H = 3, RMAX = 5; };

// Stencil-input fields of the FP64 stage (InstDev::der, der_out).
enum { DR_K2 = 0, DR_GU, DR_GV, DR_JUT, DR_JVT, DR_N };

// Interior central difference with the antisymmetric coefficients of the
// order's interior stencil; fm(o) returns the value at offset o.
template <int ORD, class T, class F>
__device__ __forceinline__ T d_interior(F fm) {
  if constexpr (Ord<ORD>::H == 1) {
    return T(0.5) * (fm(1) - fm(-1));
  } else if constexpr (Ord<ORD>::H == 2) {
    return T(2.0 / 3.0) * (fm(1) - fm(-1)) + T(-1.0 / 12.0) * (fm(2) - fm(-2));
  } else {
    return T(3.0 / 4.0) * (fm(1) - fm(-1)) + T(-3.0 / 20.0) * (fm(2) - fm(-2)) +
           T(1.0 / 60.0) * (fm(3) - fm(-3));
  }
}

// SBP derivative at line index k of a line of n nodes; fa(m) returns the value
// at absolute line index m.
template <int ORD, class T, class FA>
__device__ __forceinline__ T d_line(int k, int n, FA fa) {
  constexpr int NE = Ord<ORD>::NE, NW = Ord<ORD>::NW, ID = Ord<ORD>::idx;
  if (k < NE) {
    T acc = T(0);
    const int last = c_sbp[ID].last[k];
#pragma unroll
    for (int m = 0; m < NW; ++m)
      if (m < last) acc += sbp_ql<T>(ID, k, m) * fa(m);
    return acc;
  } else if (k >= n - NE) {
    const int r = n - 1 - k;
    const int last = c_sbp[ID].last[r];
    T acc = T(0);
#pragma unroll
    for (int m = NW - 1; m >= 0; --m)
      if (m < last) acc += sbp_qr<T>(ID, r, m) * fa(n - 1 - m);
    return acc;
  }
  return d_interior<ORD, T>([&](int o) { return fa(k + o); });
}

// RK stage epilogue of one node from its tendency and its RK inputs: rb =
// base (FP32 RK4: the state's high part), ra = running sum, rl = state's low
// part.  FP64 keeps the reference's order: y = 1*v0 + c*k; w = v0 + dt/6 k1,
// w += dt/3 k2, w += dt/3 k3, v0 = w + dt/6 k4 (rk4_mod.f90:28-40).  FP32
// compensated form: the stage increments accumulate apart from the state, and
// the last stage adds them to the (hi, lo) state pair with an exact two-sum,
// so the FP32 state keeps the low-order bits across steps.  A null acc (FP64)
// skips the running sum: the stage states of the adjoint need none.
template <class T>
__device__ __forceinline__ void stage_epilogue_pre(const InstDev<T>& I, int mode, long long idx,
                                                   T kh, T ku, T kv, const T* rb, const T* ra,
                                                   const T* rl, T* y) {
  const long long fs = I.fs;
  const T kk[3] = {kh, ku, kv};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const long long o = c * fs + idx;
    if (mode == MODE_APPLY) {
      I.out[o] = kk[c];
    } else if (sizeof(T) == 8) {
      if (mode == MODE_RK4) {
        I.base_out[o] = ra[c] + I.c_acc * kk[c];
      } else {
        y[c] = T(1.0) * rb[c] + I.c_in * kk[c];   // the next stage's state
        I.out[o] = y[c];
        if (I.acc) I.acc[o] = (mode == MODE_RK1 ? rb[c] : ra[c]) + I.c_acc * kk[c];
      }
    } else {
      if (mode == MODE_RK1) {
        I.out[o] = rb[c] + I.c_in * kk[c];
        I.acc[o] = I.c_acc * kk[c];
      } else if (mode == MODE_RK4) {
        const T d = ra[c] + I.c_acc * kk[c];
        const T t = rl[c] + d;
        const T s = rb[c] + t;
        const T bb = s - rb[c];
        I.base_out[o] = s;
        I.base_lo[o] = (rb[c] - (s - bb)) + (t - bb);
      } else {
        I.out[o] = rb[c] + I.c_in * kk[c];
        I.acc[o] = ra[c] + I.c_acc * kk[c];
      }
    }
  }
}

// Coriolis + tendency at a node, given the synced gx, gy, zeta, div.
// cor_u = (f+zeta)*hv/h*J with hv/h = vt (coriolis_colocated_mod.f90:93-100).
template <class T>
__device__ __forceinline__ void node_tendency(T gx, T gy, T zeta, T dv, T f, T J, T ut, T vt,
                                              T& kh, T& ku, T& kv) {
  const T fz = f + zeta;
  ku = -gx + fz * (J * vt);
  kv = -gy - fz * (J * ut);
  kh = -dv;
}
// ---------------------------------------------------------------------------
// FP64 stage.  GB300 issues a warp-wide FP64 instruction to an SM quarter
// once in 64 cycles, so the FP64 instructions per node are the cost and
// memory traffic is nearly free beside them.  Hence:
//   - the pointwise stencil inputs are formed once per node, by the kernel
//     that makes the state, and kept in fields (the earlier row-streaming
//     kernel formed them for its halo rows and columns as well: units of 8 rows
//     had 6 halo rows at N=192);
//   - one thread per node and no work units, so that every SM quarter gets
//     the same number of warps at any size;
//   - the nodes of the NE closure columns at either panel side are separate
//     warps that run along the column, so that a warp's closure row is
//     uniform and the other warps never meet one (in warps along the row, 2
//     of 13 at N=384 ran closures and interior one after the other);
//   - panel-boundary nodes form their neighbours' pre-sync terms themselves, a
//     lane for their own panel and one for the neighbour's, in warps that start
//     first, instead of a second launch that exchanges them (one lane for
//     both: 0.126 against 0.073 ms a step at N=48, before the Taps);
//   - differences are taken before they are scaled, and the constants come
//     from the host: 32 FP64 instructions an inner node and 11 for its stencil
//     inputs (4/2), against 58 (constants formed per thread would be 5 more).
// Measured, RK4 steps d42 of one instance back to back, against the row-streaming
// kernel: N=48 0.237 -> 0.049 ms, N=384 0.546 -> 0.345 ms, N=1024 2.93 -> 2.17
// ms.  The FP64 pipe is 82% busy in a launch at N=384.  Blocks of 64 and 256 threads
// measured within 1% of 128; compiled for 4 blocks an SM 4% slower at N=384 and 8%
// faster at N=48 than for 5, for 7 the reverse: 5 gives up 1% at N=384 (0.342 ms
// before the taps and the bound) for the small panels.
// ---------------------------------------------------------------------------
constexpr int PT_TPB = 128;

// Node of thread tid: first the E columns at either panel side (threads along
// the column), then the others (along the row).  False past the last node.
// Panels of fewer than 2 E columns split in the middle: the columns between
// are then not free of closures, so kernels test the node, not the thread.
template <int E>
__device__ __forceinline__ bool point_node(int n, int tid, int& p, int& i, int& j) {
  const int ne = min(E, n / 2), nclosed = 12 * ne * n, ni = n - 2 * ne;
  if (tid < nclosed) {
    const int r = tid / n;
    j = tid - r * n;
    const int s = r / ne, c = r - s * ne;
    i = (s & 1) ? n - 1 - c : c;
    p = s >> 1;
    return true;
  }
  const int t = tid - nclosed, row = ni > 0 ? t / ni : 6 * n;
  p = row / n;
  j = row - p * n;
  i = ne + t - row * ni;
  return p < 6;
}

// boundary node b of a panel (0 <= b < 4n-4) -> (i, j); bottom and top rows
// own the corners.
__device__ __forceinline__ void boundary_node(int b, int n, int& i, int& j) {
  if (b < n) { i = b; j = 0; }
  else if (b < 2 * n) { i = b - n; j = n - 1; }
  else if (b < 3 * n - 2) { i = 0; j = b - 2 * n + 1; }
  else { i = n - 1; j = b - (3 * n - 2) + 1; }
}

// Stencil inputs of a node with state (h, u, v).
template <class T>
__device__ __forceinline__ void derive_store(T* der, long long fs, long long idx, T h, T u, T v, T J,
                                             T q1, T q2, T q3, T grav2, const T* hs) {
  const T ut = q1 * u + q2 * v, vt = q2 * u + q3 * v;
  const T jut = J * ut, jvt = J * vt;
  T k2 = (u * ut + v * vt) + grav2 * h;   // twice the Bernoulli function: ghs takes the half
  if (hs) k2 = k2 + grav2 * hs[idx];
  der[DR_K2 * fs + idx] = k2;
  der[DR_GU * fs + idx] = h * jut;
  der[DR_GV * fs + idx] = h * jvt;
  der[DR_JUT * fs + idx] = jut;
  der[DR_JVT * fs + idx] = jvt;
}

// Instance of this block and its first thread: a batch has a grid row per
// instance, each as long as the largest needs, or, where that leaves most blocks
// without a node, a table of (instance, block).
template <class T>
__device__ __forceinline__ const InstDev<T>& point_inst(const InstDev<T>& one, const InstDev<T>* many,
                                                        const int2* blocks, int& tid) {
  const int2 b = blocks ? blocks[blockIdx.x] : make_int2(blockIdx.y, blockIdx.x);
  tid = b.y * PT_TPB + threadIdx.x;
  return many ? many[b.x] : one;
}

template <class T>
__global__ void __launch_bounds__(PT_TPB)
    point_derive_kernel(const __grid_constant__ InstDev<T> one, const InstDev<T>* many, const int2* blocks) {
  int t;
  const InstDev<T>& I = point_inst<T>(one, many, blocks, t);
  const int row = t / I.n;
  if (row >= 6 * I.n) return;
  const long long fs = I.fs, x = (long long)row * I.P + (t - row * I.n);
  derive_store<T>(const_cast<T*>(I.der), fs, x, I.in[x], I.in[fs + x], I.in[2 * fs + x],
                  I.metric[MJ * fs + x], I.metric[MQI1 * fs + x], I.metric[MQI2 * fs + x],
                  I.metric[MQI3 * fs + x], I.grav2, I.hs);
}

// Interior coefficients of the first derivative (offset o = 1..H) and their
// ratios to the first: sum_o c_o dif(o) = c_1 d_ratio(dif).
template <int ORD>
__host__ __device__ constexpr double d_coef(int o) {
  return Ord<ORD>::H == 1 ? 0.5 : Ord<ORD>::H == 2 ? (o == 1 ? 2.0 / 3.0 : -1.0 / 12.0)
                                : (o == 1 ? 3.0 / 4.0 : o == 2 ? -3.0 / 20.0 : 1.0 / 60.0);
}
template <int ORD, class T, class F>
__device__ __forceinline__ T d_ratio(F dif) {
  T s = dif(1);
#pragma unroll
  for (int o = 2; o <= Ord<ORD>::H; ++o) s += T(d_coef<ORD>(o) / d_coef<ORD>(1)) * dif(o);
  return s;
}
template <int ORD, class T, class F>
__device__ __forceinline__ T d_scaled(const T (&c)[3], F dif) {
  T s = c[0] * dif(1);
#pragma unroll
  for (int o = 2; o <= Ord<ORD>::H; ++o) s += c[o - 1] * dif(o);
  return s;
}

// The SBP derivative at line index k as one row of taps: sum_m c[m] f(s + m) over
// the taps m in the bit set `on`, closure or interior alike.  All taps are loaded
// and a value of one that the row does not have is replaced by zero (a select, not
// a product with a zero coefficient), so that an infinity or NaN outside the
// row's stencil stays out of the sum.  With predicated loads in its place the
// stage kernel spilled 80 to 180 bytes (N=384 d42 0.356 ms a step, 0.345 so),
// with predicated sums it waited longer (N=64 0.059 against 0.055).
// No branch separates the loads of one derivative from the next, so a
// panel-boundary node waits for memory once a direction and not once a
// derivative (with d_line in its place the RK4 step took 0.085 ms at N=48 and
// 0.141 at N=192, against 0.052 and 0.112).
template <int ORD>
struct Taps {
  static constexpr int NT = Ord<ORD>::NW > 2 * Ord<ORD>::H + 1 ? Ord<ORD>::NW : 2 * Ord<ORD>::H + 1;
  int s;
  unsigned on;
  double c[NT];
  __device__ __forceinline__ bool has(int m) const { return on >> m & 1u; }
};
template <int ORD>
__device__ __forceinline__ Taps<ORD> taps_of(int k, int n) {
  constexpr int NE = Ord<ORD>::NE, NT = Taps<ORD>::NT, ID = Ord<ORD>::idx, H = Ord<ORD>::H;
  Taps<ORD> t;
  const bool left = k < NE, right = k >= n - NE;
  const int r = left ? k : right ? n - 1 - k : 0, last = c_sbp[ID].last[r];
  t.s = left ? 0 : right ? n - NT : k - H;
  const unsigned row = (1u << last) - 1u;
  t.on = left ? row : right ? row << (NT - last) : ((1u << (2 * H + 1)) - 1u) & ~(1u << H);
#pragma unroll
  for (int m = 0; m < NT; ++m) {
    const int mm = right ? NT - 1 - m : m;
    const double q = mm < last && mm < MAXNW ? c_sbp[ID].Ql[r * MAXNW + mm] : 0.0;
    t.c[m] = left ? q : right ? -q : m <= 2 * H ? c_sbp[ID].Qin[m <= 2 * H ? m : 0] : 0.0;
  }
  return t;
}
// f at the node, st the stride along the line, k the node's line index
template <int ORD>
__device__ __forceinline__ double taps_sum(const Taps<ORD>& t, const double* __restrict__ f, int k, int st) {
  const double* q = f + (long long)(t.s - k) * st;
  double v[Taps<ORD>::NT], s = 0.0;
#pragma unroll
  for (int m = 0; m < Taps<ORD>::NT; ++m) v[m] = __ldg(q + m * st);
#pragma unroll
  for (int m = 0; m < Taps<ORD>::NT; ++m) s += t.c[m] * (t.has(m) ? v[m] : 0.0);
  return s;
}

// Pre-sync gx, gy, curl and divergence of any node from the stencil inputs.
template <int ORD, class T>
__device__ __forceinline__ void raw_terms(const InstDev<T>& I, int p, int i, int j, T& gx, T& gy, T& zeta,
                                          T& dv) {
  const int n = I.n, P = I.P;
  const long long fs = I.fs, x = (long long)p * I.ps + (long long)j * P + i;
  const T rJ = I.metric[MRJ * fs + x];
  const T *K = I.der + DR_K2 * fs + x, *GU = I.der + DR_GU * fs + x, *GV = I.der + DR_GV * fs + x;
  const T *U = I.in + fs + x, *V = I.in + 2 * fs + x;
  T z, d;
  {
    const Taps<ORD> t = taps_of<ORD>(i, n);
    gx = taps_sum<ORD>(t, K, i, 1) * I.ghs2;
    z = taps_sum<ORD>(t, V, i, 1);
    d = taps_sum<ORD>(t, GU, i, 1);
  }
  {
    const Taps<ORD> t = taps_of<ORD>(j, n);
    gy = taps_sum<ORD>(t, K, j, P) * I.ghs2;
    z -= taps_sum<ORD>(t, U, j, P);
    d += taps_sum<ORD>(t, GV, j, P);
  }
  zeta = z * rJ;
  dv = d * rJ;
}

// Threads of one instance: the panel-boundary nodes (two lanes each), the
// other closure columns, the other nodes, each padded to whole blocks.
struct PointRanges {
  int nb, closed, total;
};
template <int ORD>
__host__ __device__ inline PointRanges point_ranges(int n) {
  auto pad = [](int k) { return (k + PT_TPB - 1) / PT_TPB * PT_TPB; };
  constexpr int NE = Ord<ORD>::NE;
  PointRanges r;
  r.nb = pad(2 * 6 * (4 * n - 4));
  r.closed = r.nb + pad(12 * (NE - 1) * (n - 2));
  r.total = r.closed + pad(6 * (n - 2 * NE) * (n - 2));
  return r;
}

// Node of thread tid of these ranges; false where it has none.  The lanes of
// boundary blocks past the last node stay (live false) for the shuffles of the
// pairs; the even lane of a pair is the node's own.
struct PointAt {
  int p, i, j;
  bool boundary, live;
};
template <int ORD>
__device__ __forceinline__ bool point_at(int n, int tid, PointAt& o) {
  constexpr int NE = Ord<ORD>::NE;
  const PointRanges rg = point_ranges<ORD>(n);
  o.live = true;
  o.boundary = tid < rg.nb;
  if (o.boundary) {
    const int nb = 4 * n - 4, t = min(tid >> 1, 6 * nb - 1);
    o.live = (tid >> 1) < 6 * nb;
    o.p = t / nb;
    boundary_node(t - o.p * nb, n, o.i, o.j);
    return true;
  }
  if (tid < rg.closed) {   // along the column: rows 1..n-2
    const int t = tid - rg.nb, r = t / (n - 2);
    if (r >= 12 * (NE - 1)) return false;
    o.j = 1 + t - r * (n - 2);
    const int s = r / (NE > 1 ? NE - 1 : 1), c = 1 + r - s * (NE - 1);
    o.i = (s & 1) ? n - 1 - c : c;
    o.p = s >> 1;
    return true;
  }
  const int t = tid - rg.closed, ni = n - 2 * NE, row = t / ni;
  o.p = row / (n - 2);
  o.j = 1 + row - o.p * (n - 2);
  o.i = NE + t - row * ni;
  return o.p < 6;
}

template <class T, int ORD, int MODE>
__global__ void __launch_bounds__(PT_TPB, 5)
    point_stage_kernel(const __grid_constant__ InstDev<T> one, const InstDev<T>* many,
                       const __grid_constant__ Topology tp, const int2* blocks) {
  constexpr int NE = Ord<ORD>::NE;
  constexpr bool needB = MODE == MODE_RK1 || MODE == MODE_RK2 || MODE == MODE_RK3;
  constexpr bool needA = MODE == MODE_RK2 || MODE == MODE_RK3 || MODE == MODE_RK4;
  int tid;
  const InstDev<T>& I = point_inst<T>(one, many, blocks, tid);
  const int n = I.n, P = I.P;
  PointAt at;
  if (!point_at<ORD>(n, tid, at)) return;
  const int p = at.p, i = at.i, j = at.j;
  const long long fs = I.fs, x = (long long)p * I.ps + (long long)j * P + i;
  T rb[3] = {}, ra[3] = {}, rl[3] = {};
  auto rk_load = [&]() {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (needB) rb[c] = I.base[c * fs + x];
      if (needA) ra[c] = I.acc ? I.acc[c * fs + x] : T(0);
    }
  };
  // At 6/3 the nine taps and these inputs together spill 68 bytes in stages 2 and
  // 3 (N=256 0.218 ms a step, 0.216 so), so a boundary node reads them last.
  constexpr bool late = Taps<ORD>::NT > 6 && needA && needB;
  if (!(late && at.boundary)) rk_load();
  const T f = I.metric[MF * fs + x];
  const T jut = I.der[DR_JUT * fs + x], jvt = I.der[DR_JVT * fs + x];
  T kh, ku, kv;
  if (at.boundary) {
    // A boundary node: one lane forms the raw terms of its own panel, the other
    // those of the panels that hold copies of it (formed here again rather
    // than exchanged); then their sync (2-way average on edges, 3-way at cube
    // corners; the covariant gradient with the metric weights;
    // halo_Ah_scalar_sync_mod.f90:38-93, ecs_Ah_vec_sync_mod.f90:62-125).
    const int e = n - 1;
    const bool lr = (i == 0) | (i == e), bt = (j == 0) | (j == e);
    T sgx = T(0), sgy = T(0), sz = T(0), sd = T(0);
    const bool own = (tid & 1) == 0;
    const int copies = !own && lr && bt ? 2 : 1;
#pragma unroll 1
    for (int s = 0; s < copies; ++s) {
      const bool side_lr = lr && s == 0;
      int q = p, iq = i, jq = j;
      EdgeLink L{};
      if (!own) {
        L = tp.link[p][side_lr ? (i == 0 ? SIDE_L : SIDE_R) : (j == 0 ? SIDE_B : SIDE_T)];
        const int k = side_lr ? j : i, kk = L.rev ? e - k : k;
        q = L.q;
        iq = L.side_q == SIDE_L ? 0 : L.side_q == SIDE_R ? e : kk;
        jq = L.side_q == SIDE_B ? 0 : L.side_q == SIDE_T ? e : kk;
      }
      T gx, gy, z, d;
      raw_terms<ORD, T>(I, q, iq, jq, gx, gy, z, d);
      if (!own) {   // the neighbour's components in this panel's frame
        const T a = L.dim_i ? T(L.istep) * gx : T(L.jstep) * gy;
        const T b = L.dim_i ? T(L.jstep) * gy : T(L.istep) * gx;
        gx = a;
        gy = b;
        if (side_lr) gx += I.qw[(i == 0 ? 2 : 3) * n + j] * b;
        else gy += I.qw[(j == 0 ? 0 : 1) * n + i] * a;
      }
      sgx += gx; sgy += gy; sz += z; sd += d;
    }
    sgx += __shfl_xor_sync(0xffffffffu, sgx, 1);
    sgy += __shfl_xor_sync(0xffffffffu, sgy, 1);
    sz += __shfl_xor_sync(0xffffffffu, sz, 1);
    sd += __shfl_xor_sync(0xffffffffu, sd, 1);
    if (!own || !at.live) return;
    if (late) rk_load();
    const T w = lr && bt ? T(1.0 / 3.0) : T(0.5);
    const T fz = f + w * sz;
    kh = -(w * sd);
    ku = fz * jvt - w * sgx;
    kv = -(fz * jut) - w * sgy;
  } else {
    T gx, gy, fz;
    if (i >= NE && i < n - NE && j >= NE && j < n - NE) {
      const T* __restrict__ K = I.der + DR_K2 * fs + x;
      const T* __restrict__ GU = I.der + DR_GU * fs + x;
      const T* __restrict__ GV = I.der + DR_GV * fs + x;
      const T* __restrict__ U = I.in + fs + x;
      const T* __restrict__ V = I.in + 2 * fs + x;
      const T rJ = I.metric[MRJ * fs + x] * T(d_coef<ORD>(1));
      gx = d_scaled<ORD, T>(I.gc, [&](int o) { return K[o] - K[-o]; });
      gy = d_scaled<ORD, T>(I.gc, [&](int o) { return K[o * P] - K[-o * P]; });
      const T zw = d_ratio<ORD, T>([&](int o) { return (V[o] - V[-o]) - (U[o * P] - U[-o * P]); });
      const T dw = d_ratio<ORD, T>([&](int o) { return (GU[o] - GU[-o]) + (GV[o * P] - GV[-o * P]); });
      fz = f + zw * rJ;
      kh = -(dw * rJ);
    } else {
      const T* __restrict__ K = I.der + DR_K2 * fs + x;
      const T* __restrict__ GU = I.der + DR_GU * fs + x;
      const T* __restrict__ GV = I.der + DR_GV * fs + x;
      const T* __restrict__ U = I.in + fs + x;
      const T* __restrict__ V = I.in + 2 * fs + x;
      const T rJ = I.metric[MRJ * fs + x];
      auto dx = [&](const T* q) { return d_line<ORD, T>(i, n, [&](int m) { return q[m - i]; }); };
      auto dy = [&](const T* q) { return d_line<ORD, T>(j, n, [&](int m) { return q[(m - j) * P]; }); };
      gx = dx(K) * I.ghs2;
      gy = dy(K) * I.ghs2;
      fz = f + (dx(V) - dy(U)) * rJ;
      kh = -((dx(GU) + dy(GV)) * rJ);
    }
    ku = fz * jvt - gx;
    kv = -(fz * jut) - gy;
  }
  T y[3];
  stage_epilogue_pre<T>(I, MODE, x, kh, ku, kv, rb, ra, rl, y);
  if (needB && I.der_out)
    derive_store<T>(I.der_out, fs, x, y[0], y[1], y[2], I.metric[MJ * fs + x], I.metric[MQI1 * fs + x],
                    I.metric[MQI2 * fs + x], I.metric[MQI3 * fs + x], I.grav2, I.hs);
}

// Stencil inputs of I.in, then (launch_point_stage) one stage from them, over
// the instances of B.
template <class T>
cudaError_t launch_point_derive(const InstDev<T>& one, const PointBatch<T>& B, cudaStream_t st) {
  // with a table: the stage's blocks, which hold at least as many threads
  const dim3 g = B.blocks ? dim3(B.nblocks) : dim3((6 * B.max_n * B.max_n + PT_TPB - 1) / PT_TPB, B.ninst);
  point_derive_kernel<T><<<g, PT_TPB, 0, st>>>(one, B.many, B.blocks);
  return cudaGetLastError();
}
template <class T, int ORD>
cudaError_t launch_point_stage_ord(const InstDev<T>& one, const PointBatch<T>& B, const Topology& tp, int mode,
                                   cudaStream_t st) {
  const dim3 g = B.blocks ? dim3(B.nblocks) : dim3(point_ranges<ORD>(B.max_n).total / PT_TPB, B.ninst);
  switch (mode) {
    case MODE_APPLY: point_stage_kernel<T, ORD, MODE_APPLY><<<g, PT_TPB, 0, st>>>(one, B.many, tp, B.blocks); break;
    case MODE_RK1: point_stage_kernel<T, ORD, MODE_RK1><<<g, PT_TPB, 0, st>>>(one, B.many, tp, B.blocks); break;
    case MODE_RK2: point_stage_kernel<T, ORD, MODE_RK2><<<g, PT_TPB, 0, st>>>(one, B.many, tp, B.blocks); break;
    case MODE_RK3: point_stage_kernel<T, ORD, MODE_RK3><<<g, PT_TPB, 0, st>>>(one, B.many, tp, B.blocks); break;
    case MODE_RK4: point_stage_kernel<T, ORD, MODE_RK4><<<g, PT_TPB, 0, st>>>(one, B.many, tp, B.blocks); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Cube-edge syncs at one panel-boundary node (p, i, j): returns the synced
// gx, gy (covariant gradient), zeta and div.  E points at the edge buffer of
// the instance; ring values come from the neighbour panels' entries.
// ---------------------------------------------------------------------------
template <class T>
struct EdgeView {
  const T* E;
  int n;
  __device__ __forceinline__ T get(int p, int side, int v, int k) const {
    return E[((long long)(p * 4 + side) * 4 + v) * n + k];
  }
};

template <class T>
__device__ __forceinline__ void ring_scalar(const EdgeView<T>& ev, const Topology& tp, int p,
                                            int side, int v, int k, T& out) {
  const EdgeLink L = tp.link[p][side];
  const int kk = L.rev ? ev.n - 1 - k : k;
  out = ev.get(L.q, L.side_q, v, kk);
}

template <class T>
__device__ __forceinline__ void ring_vector(const EdgeView<T>& ev, const Topology& tp, int p,
                                            int side, int k, T& rx, T& ry) {
  const EdgeLink L = tp.link[p][side];
  const int kk = L.rev ? ev.n - 1 - k : k;
  const T gxq = ev.get(L.q, L.side_q, EV_GX, kk), gyq = ev.get(L.q, L.side_q, EV_GY, kk);
  if (L.dim_i) { rx = T(L.istep) * gxq; ry = T(L.jstep) * gyq; }
  else { rx = T(L.jstep) * gyq; ry = T(L.istep) * gxq; }
}

// Scalar sync of value slot v at node (p,i,j) (halo_Ah_scalar_sync_mod.f90:38-93).
template <class T>
__device__ T sync_scalar_node(const EdgeView<T>& ev, const Topology& tp, int p, int i, int j,
                              int v, T own) {
  const int e = ev.n - 1;
  T a, b;
  if (i == 0 && j == 0) { ring_scalar(ev, tp, p, SIDE_L, v, 0, a); ring_scalar(ev, tp, p, SIDE_B, v, 0, b); return (own + a + b) / T(3.0); }
  if (i == e && j == 0) { ring_scalar(ev, tp, p, SIDE_R, v, 0, a); ring_scalar(ev, tp, p, SIDE_B, v, e, b); return (own + a + b) / T(3.0); }
  if (i == 0 && j == e) { ring_scalar(ev, tp, p, SIDE_L, v, e, a); ring_scalar(ev, tp, p, SIDE_T, v, 0, b); return (own + a + b) / T(3.0); }
  if (i == e && j == e) { ring_scalar(ev, tp, p, SIDE_R, v, e, a); ring_scalar(ev, tp, p, SIDE_T, v, e, b); return (own + a + b) / T(3.0); }
  if (i == 0) { ring_scalar(ev, tp, p, SIDE_L, v, j, a); return T(0.5) * (a + own); }
  if (i == e) { ring_scalar(ev, tp, p, SIDE_R, v, j, a); return T(0.5) * (own + a); }
  if (j == 0) { ring_scalar(ev, tp, p, SIDE_B, v, i, a); return T(0.5) * (own + a); }
  ring_scalar(ev, tp, p, SIDE_T, v, i, a);
  return T(0.5) * (own + a);
}

// Covariant vector sync at node (p,i,j): syncronize_grad_on_edges with U = gy,
// V = gx (ecs_Ah_vec_sync_mod.f90:52, 62-125).  qw = qb|qt|ql|qr (n each).
template <class T>
__device__ void sync_vector_node(const EdgeView<T>& ev, const Topology& tp, const double* qw,
                                 int p, int i, int j, T& gx, T& gy) {
  const int n = ev.n, e = n - 1;
  const double* qb = qw;
  const double* qt = qw + n;
  const double* ql = qw + 2 * n;
  const double* qr = qw + 3 * n;
  T V = gx, U = gy;
  T rx, ry, sx, sy;
  if (i == 0 && j == 0) {
    ring_vector(ev, tp, p, SIDE_L, 0, rx, ry); ring_vector(ev, tp, p, SIDE_B, 0, sx, sy);
    gy = (U + ry + sy + T(qb[0]) * sx) / T(3.0);
    gx = (V + rx + sx + T(ql[0]) * ry) / T(3.0);
  } else if (i == e && j == 0) {
    ring_vector(ev, tp, p, SIDE_R, 0, rx, ry); ring_vector(ev, tp, p, SIDE_B, e, sx, sy);
    gy = (U + ry + sy + T(qb[e]) * sx) / T(3.0);
    gx = (V + rx + sx + T(qr[0]) * ry) / T(3.0);
  } else if (i == 0 && j == e) {
    ring_vector(ev, tp, p, SIDE_L, e, rx, ry); ring_vector(ev, tp, p, SIDE_T, 0, sx, sy);
    gy = (U + ry + sy + T(qt[0]) * sx) / T(3.0);
    gx = (V + rx + sx + T(ql[e]) * ry) / T(3.0);
  } else if (i == e && j == e) {
    ring_vector(ev, tp, p, SIDE_R, e, rx, ry); ring_vector(ev, tp, p, SIDE_T, e, sx, sy);
    gy = (U + ry + sy + T(qt[e]) * sx) / T(3.0);
    gx = (V + rx + sx + T(qr[e]) * ry) / T(3.0);
  } else if (i == 0) {
    ring_vector(ev, tp, p, SIDE_L, j, rx, ry);
    gy = T(0.5) * (ry + U);
    gx = T(0.5) * (V + rx + T(ql[j]) * ry);
  } else if (i == e) {
    ring_vector(ev, tp, p, SIDE_R, j, rx, ry);
    gy = T(0.5) * (U + ry);
    gx = T(0.5) * (V + rx + T(qr[j]) * ry);
  } else if (j == 0) {
    ring_vector(ev, tp, p, SIDE_B, i, sx, sy);
    gx = T(0.5) * (sx + V);
    gy = T(0.5) * (sy + U + T(qb[i]) * sx);
  } else {
    ring_vector(ev, tp, p, SIDE_T, i, sx, sy);
    gx = T(0.5) * (V + sx);
    gy = T(0.5) * (U + sy + T(qt[i]) * sx);
  }
}


// ---------------------------------------------------------------------------
// FP32 edge kernel: finishes every panel-boundary node of every instance.
// blockIdx.y = instance, x covers 6*(4n-4) nodes.
// ---------------------------------------------------------------------------
template <class T>
__global__ void edge_kernel(InstDev<T> one, const InstDev<T>* many, Topology tp, int mode) {
  const InstDev<T>& I = many ? many[blockIdx.y] : one;
  const int n = I.n, nb = 4 * n - 4, e = n - 1;
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= 6 * nb) return;
  const int p = g / nb;
  int i, j;
  boundary_node(g - p * nb, n, i, j);
  // The node lies on a left/right side (lr), a bottom/top side (bt), or both
  // (cube corner).  Every address below is known before any load, so all
  // loads of the node issue together.
  const bool lr = (i == 0) | (i == e), bt = (j == 0) | (j == e);
  const int sLR = i == 0 ? SIDE_L : SIDE_R, sBT = j == 0 ? SIDE_B : SIDE_T;
  const EdgeLink LL = tp.link[p][sLR], LB = tp.link[p][sBT];
  const T* E = I.edge;
  auto at = [&](int q, int s, int v, int k) { return E[((q * 4 + s) * 4 + v) * n + k]; };
  const int so = lr ? sLR : sBT, ko = lr ? j : i;          // own values
  const int kl = LL.rev ? e - j : j, kb = LB.rev ? e - i : i;  // neighbour positions
  T own[4], nl[4], nbt[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    own[v] = at(p, so, v, ko);
    nl[v] = lr ? at(LL.q, LL.side_q, v, kl) : T(0);
    nbt[v] = bt ? at(LB.q, LB.side_q, v, kb) : T(0);
  }
  const double* qw = I.qw;
  const T qlr = lr ? T(qw[(i == 0 ? 2 : 3) * n + j]) : T(0);   // ql / qr at j
  const T qbt = bt ? T(qw[(j == 0 ? 0 : 1) * n + i]) : T(0);   // qb / qt at i
  const long long fs = I.fs;
  const long long idx = (long long)p * I.ps + (long long)j * I.P + i;
  const T u = I.in[fs + idx], v = I.in[2 * fs + idx];
  const T q1 = I.metric[MQI1 * fs + idx], q2 = I.metric[MQI2 * fs + idx],
          q3 = I.metric[MQI3 * fs + idx];
  const T J = I.metric[MJ * fs + idx], f = I.metric[MF * fs + idx];
  // RK inputs of the node, loaded with everything else
  static_assert(sizeof(T) == 4, "the FP64 stage kernel finishes its boundary nodes itself");
  const bool needB = mode != MODE_APPLY;
  const bool needA = mode == MODE_RK2 || mode == MODE_RK3 || mode == MODE_RK4;
  const bool needL = mode == MODE_RK4;
  const T* bsrc = mode == MODE_RK4 ? I.base_out : I.base;
  T rb[3], ra[3], rlo[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    rb[c] = needB ? bsrc[c * fs + idx] : T(0);
    ra[c] = needA ? I.acc[c * fs + idx] : T(0);
    rlo[c] = needL ? I.base_lo[c * fs + idx] : T(0);
  }

  // neighbour vectors in this panel's frame (pack_to_buf_vec component map)
  auto rot = [](const EdgeLink& L, T gxq, T gyq, T& rx, T& ry) {
    if (L.dim_i) { rx = T(L.istep) * gxq; ry = T(L.jstep) * gyq; }
    else { rx = T(L.jstep) * gyq; ry = T(L.istep) * gxq; }
  };
  T rx, ry, sx, sy;
  rot(LL, nl[EV_GX], nl[EV_GY], rx, ry);
  rot(LB, nbt[EV_GX], nbt[EV_GY], sx, sy);
  const T U = own[EV_GY], V = own[EV_GX];
  T gx, gy, zeta, dv;
  if (lr && bt) {
    // cube corner: 3-way averages (halo_Ah_scalar_sync_mod.f90:56-85,
    // ecs_Ah_vec_sync_mod.f90:77-100)
    gy = (U + ry + sy + qbt * sx) / T(3.0);
    gx = (V + rx + sx + qlr * ry) / T(3.0);
    zeta = (own[EV_ZETA] + nl[EV_ZETA] + nbt[EV_ZETA]) / T(3.0);
    dv = (own[EV_DIV] + nl[EV_DIV] + nbt[EV_DIV]) / T(3.0);
  } else if (lr) {
    gy = T(0.5) * (U + ry);
    gx = T(0.5) * (V + rx + qlr * ry);
    zeta = T(0.5) * (own[EV_ZETA] + nl[EV_ZETA]);
    dv = T(0.5) * (own[EV_DIV] + nl[EV_DIV]);
  } else {
    gx = T(0.5) * (V + sx);
    gy = T(0.5) * (U + sy + qbt * sx);
    zeta = T(0.5) * (own[EV_ZETA] + nbt[EV_ZETA]);
    dv = T(0.5) * (own[EV_DIV] + nbt[EV_DIV]);
  }
  const T ut = q1 * u + q2 * v, vt = q2 * u + q3 * v;
  T kh, ku, kv;
  node_tendency<T>(gx, gy, zeta, dv, f, J, ut, vt, kh, ku, kv);
  T y[3] = {};
  stage_epilogue_pre<T>(I, mode, idx, kh, ku, kv, rb, ra, rlo, y);
}

}  // namespace swm
